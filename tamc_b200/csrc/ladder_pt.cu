// ladder_pt.cu -- the ladder form of PT-ICM (TAMC_MODE_FAST): one run spread
// over the GPU by replica.
//
// A CTA keeps one replica (chain c, temperature slot t) in shared memory, a
// sign word per colour-ordered site, with the instance's rows beside it when
// they fit.  A sweep involves one replica and runs inside its CTA; a Houdayer
// move involves the two replicas of a slot, whose CTAs exchange their spins as
// n / 8 bytes through L2 (one flag each) and then both grow the same cluster
// and each flip it in their own replica.  All CTAs meet once per round, at the
// exchange: every CTA publishes its replica and energies, passes one barrier
// over the run's CTAs, makes the exchange decisions of its chain (one warp, the
// same decisions in every CTA of the chain) and fetches the replica that moved
// into its slot.
//
// Why: the fused form runs a whole ladder on one SM (195 us a round for a QUBO
// of 2039 sites and 21 temperatures, 16.5 us for a 256-site lattice and 32), the
// plain form five dependent launches a round with its Houdayer move on one CTA
// per slot (43 us at 4096 sites and 64 temperatures, 176 us at 13824 and 24).
// What bounds a round here is latency and issue inside one SM per replica: the
// CTA barriers, one barrier through L2, and the sweep's instructions.
//
// The chain is the one of the other forms bit for bit: the same Philox
// counters, the same float sums in row order, fixed-point energy sums, the
// same seed rule, and clusters that are exact components.
#include "fast_pt.cuh"

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <map>
#include <mutex>
#include <tuple>

namespace tamc {
namespace {

extern __shared__ __align__(16) unsigned char lad_smem[];

__device__ __forceinline__ uint32_t lad_ld_acquire(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void lad_st_release(uint32_t* p, uint32_t v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;\n" ::"l"(p), "r"(v) : "memory");
}

// Waits (the calling thread) until *p has reached `target`: at most `limit`
// polls of about 0.5 us each, after which the run's error flag is set.
__device__ bool lad_wait(const uint32_t* p, uint32_t target, uint32_t limit, uint32_t* err) {
  uint32_t polls = 0;
  while ((int32_t)(lad_ld_acquire(p) - target) < 0)
    if (++polls > limit) {
      *err = 1u;
      return false;
    }
  return true;
}

// Barrier over the run's CTAs: arrivals counted up without reset, `target`
// arrivals in all.  What a CTA wrote before it is visible to every CTA's
// loads through L2 after it.  A CTA that gives up waiting leaves (false in
// every thread), the others then give up too, and the commit kernel stores
// nothing.
__device__ bool lad_barrier(uint32_t* bar, uint32_t target, uint32_t limit, uint32_t* err, uint32_t* s_ok) {
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;\n" ::"l"(bar) : "memory");
    *s_ok = lad_wait(bar, target, limit, err);
  }
  __syncthreads();
  return *s_ok != 0;
}

// How a run's rows are read.  DEG > 0: every row has DEG entries.  MSC: +-J
// instance with multi-spin-coded decisions (PtJob::msc).
enum { LAD_ROWS = 0, LAD_DEG3, LAD_DEG4, LAD_DEG6, LAD_MSC4, LAD_MSC6 };
template <int MODE>
struct LadMode {
  static constexpr bool MSC = MODE == LAD_MSC4 || MODE == LAD_MSC6;
  static constexpr uint32_t DEG =
      MODE == LAD_DEG3 ? 3u : (MODE == LAD_DEG4 || MODE == LAD_MSC4) ? 4u : (MODE == LAD_DEG6 || MODE == LAD_MSC6) ? 6u : 0u;
};

// Shared memory of a CTA.  The sign words come first (offset 0), so that a
// neighbour's word is one load at its byte offset.  Everything a round reads is
// here: each barrier's acquire drops the SM's L1, so a table in HBM would cost
// an L2 round trip at every use.  Rows in shared memory:
//  * rows of one length: byte offsets of the columns, 16 bits each, two per
//    word, [ceil(DEG/2)][n], and the couplings in pairs [DEG/2][n] (DEG 3:
//    single [3][n]): lanes on consecutive sites read without bank conflicts;
//    MSC needs only the couplings' signs, kept in bit 0 of the offsets;
//  * other rows: sliced rows (FastInst::sl_*): 32 sites of a colour class with
//    about the same row length are a slice, entry e of its lane l at
//    (slice start + e) * 32 + l, short rows padded with (own column, 0).
// Byte offsets, so that every access is a shared-memory instruction with the
// base known (pointers kept in a struct turn into generic loads).
struct LadSm {
  uint32_t own;    // [nwb] this replica's spin bits
  uint32_t D;      // [nwb] where the slot's two replicas differ
  uint32_t C;      // [nwb] cluster
  uint32_t list;   // [n] u16 the cluster's sites
  uint32_t Dr;     // lattices: [rows] q<0 bits per lattice row, file order
  uint32_t Cr;     // lattices: [rows] cluster bits
  uint32_t flat;   // lattices: [nwb + 1] a bitmap in file order
  uint32_t perm, iperm;  // lattices: [n] u16 colour -> file order and back
  uint32_t coff;   // [ncolors + 1] first site of each colour class (sliced rows: first slice)
  uint32_t ex;     // [2][64] f32 exchange: beta differences, uniforms
  uint32_t E;      // [64][2] f64 the chain's energies at the exchange (cached, energy_ref)
  uint32_t red;    // [32][2] i64
  uint32_t tags;   // [nt] bytes: bookkeeping of the chain (slot 0's CTA)
  uint32_t acc;    // [nt]
  uint32_t dhist;  // [nt][2]
  uint32_t bias, colp, J;            // rows: see above
  uint32_t site, pos, soff, kd;      // sliced rows: [32 slices] u16 site, [n] u16 position, [slices + 1], [n] f32
  uint32_t bytes;
};
struct LadDims {
  uint32_t n, nt, ncolors, lat_rows;  // lat_rows 0: not a lattice
  uint32_t deg, msc, rows;            // deg 0: sliced rows
  uint32_t nslice, nsl;               // slices; their rows of 32 entries
  uint32_t self;
};
__host__ __device__ inline LadSm lad_carve(const LadDims d) {
  uint32_t o = 0;
  auto take = [&](uint32_t bytes) {
    const uint32_t p = o;
    o = (o + bytes + 15u) & ~15u;
    return p;
  };
  const uint32_t n = d.n, nwb = (n + 31) / 32;
  take(n * 4);  // sign words
  LadSm S{};
  S.own = take(nwb * 4);
  S.D = take(nwb * 4);
  S.C = take(nwb * 4);
  S.list = take(n * 2);
  S.Dr = take(d.lat_rows * 4);
  S.Cr = take(d.lat_rows * 4);
  S.flat = take(d.lat_rows ? (nwb + 1) * 4 : 0);
  S.perm = take(d.lat_rows ? n * 2 : 0);
  S.iperm = take(d.lat_rows ? n * 2 : 0);
  S.coff = take((d.ncolors + 1) * 4);
  S.ex = take(2 * 64 * 4);
  S.E = take(64 * 16);
  S.red = take(32 * 2 * 8);
  S.tags = take(d.nt);
  S.acc = take(d.nt * 4);
  S.dhist = take(d.nt * 8);
  if (!d.deg) {
    S.site = take(d.nslice * 64);
    S.pos = take(n * 2);
    S.soff = take((d.nslice + 1) * 4);
  }
  if (d.rows) {
    S.bias = take(d.msc ? 0 : n * 4);
    S.colp = take(d.deg ? (d.deg + 1) / 2 * n * 4 : d.nsl * 64);
    S.J = take(d.msc ? 0 : d.deg ? d.deg * n * 4 : d.nsl * 128);
    S.kd = take(d.self && !d.deg ? n * 4 : 0);
  }
  S.bytes = o;
  return S;
}
__host__ __device__ inline LadDims lad_dims(const PtJob& j, int rows, uint32_t deg, bool msc) {
  return LadDims{j.n, j.nt, j.F.ncolors, j.F.lat_any ? j.n / j.F.lat_any : 0u, deg, (uint32_t)msc, (uint32_t)rows,
                 j.F.sl_n, j.F.sl_rows, (uint32_t)j.self_loops};
}
template <class T>
__device__ __forceinline__ T* lad_at(uint32_t offset) {
  return reinterpret_cast<T*>(lad_smem + offset);
}

// The sign word (0 or 0x80000000) of the site at byte offset c4.
__device__ __forceinline__ uint32_t lad_sign(uint32_t c4) {
  return *reinterpret_cast<const uint32_t*>(lad_smem + c4);
}
__device__ __forceinline__ uint32_t& lad_word(uint32_t s) { return reinterpret_cast<uint32_t*>(lad_smem)[s]; }
__device__ __forceinline__ uint32_t bm_bit(const uint32_t* m, uint32_t s) { return (m[s >> 5] >> (s & 31u)) & 1u; }

// The rows of the instance, from shared memory (RS) or from L2.
template <int MODE, bool RS>
struct LadRows {
  static constexpr uint32_t DEG = LadMode<MODE>::DEG;
  static constexpr bool MSC = LadMode<MODE>::MSC;
  const uint32_t n;
  const float* const bias_s;
  const uint32_t* const colp;
  const float* const js;
  const uint16_t* const pos;
  const uint32_t* const soff;
  const uint2* __restrict__ const ent_g;  // sliced rows: FastInst::sl_ent
  const float* __restrict__ const bias_g;
  __device__ __forceinline__ LadRows(const PtJob& j, const LadSm& S)
      : n(j.n), bias_s(lad_at<float>(S.bias)), colp(lad_at<uint32_t>(S.colp)), js(lad_at<float>(S.J)),
        pos(lad_at<uint16_t>(S.pos)), soff(lad_at<uint32_t>(S.soff)), ent_g(DEG ? j.F.ent : j.F.sl_ent),
        bias_g(j.F.bias) {}
  __device__ __forceinline__ float bias(uint32_t s) const {
    if (MSC) return 0.0f;
    return RS ? bias_s[s] : __ldg(bias_g + s);
  }
  // entry x of the sliced rows
  __device__ __forceinline__ void sliced(uint32_t x, uint32_t& c4, float& j) const {
    if (RS) {
      c4 = reinterpret_cast<const uint16_t*>(colp)[x];
      j = js[x];
    } else {
      const uint2 v = __ldg(ent_g + x);
      c4 = v.x;
      j = __uint_as_float(v.y);
    }
  }
  // f(byte offset, coupling) for `w` entries (even) of the sliced row at x, in
  // row order (pads add 0): up to eight entries' loads ahead of their sums
  // (without that a long row took 58 cycles an entry)
  template <uint32_t N, typename Fn>
  __device__ __forceinline__ void chunk(uint32_t x, Fn f) const {
    uint32_t c[N];
    float j[N];
#pragma unroll
    for (uint32_t m = 0; m < N; ++m) sliced(x + 32 * m, c[m], j[m]);
#pragma unroll
    for (uint32_t m = 0; m < N; ++m) f(c[m], j[m]);
  }
  template <typename Fn>
  __device__ __forceinline__ void each_sliced(uint32_t x, uint32_t w, Fn f) const {
#pragma unroll 1
    for (; w >= 8; w -= 8, x += 256) chunk<8>(x, f);
    if (w & 4u) {
      chunk<4>(x, f);
      x += 128;
    }
    if (w & 2u) chunk<2>(x, f);
  }
  // f(byte offset, coupling) for every entry of row s, in row order
  template <typename Fn>
  __device__ __forceinline__ void each(uint32_t s, Fn f) const {
    if (DEG) {
      uint32_t c[DEG ? DEG : 1];
      float j[DEG ? DEG : 1];
      if (RS) {
        uint32_t v[DEG ? (DEG + 1) / 2 : 1];
#pragma unroll
        for (uint32_t m = 0; m < (DEG + 1) / 2; ++m) v[m] = colp[m * n + s];
        if (!MSC && DEG % 2 == 0) {
#pragma unroll
          for (uint32_t m = 0; m < DEG / 2; ++m) {
            const float2 w = reinterpret_cast<const float2*>(js)[m * n + s];
            j[2 * m] = w.x;
            j[2 * m + 1] = w.y;
          }
        } else if (!MSC) {
#pragma unroll
          for (uint32_t m = 0; m < DEG; ++m) j[m] = js[m * n + s];
        }
#pragma unroll
        for (uint32_t m = 0; m < DEG; ++m) {
          const uint32_t h = (m & 1u) ? v[m / 2] >> 16 : v[m / 2] & 0xffffu;
          if (MSC) {
            c[m] = h & ~3u;
            j[m] = __uint_as_float(0x3f800000u | (h << 31));
          } else {
            c[m] = h;
          }
        }
      } else if (DEG % 2 == 0) {  // rows of 32 or 48 bytes, 16-byte aligned
        const uint4* r = reinterpret_cast<const uint4*>(ent_g + s * DEG);
#pragma unroll
        for (uint32_t m = 0; m < DEG / 2; ++m) {
          const uint4 v = __ldg(r + m);
          c[2 * m] = 4 * v.x;
          j[2 * m] = __uint_as_float(v.y);
          c[2 * m + 1] = 4 * v.z;
          j[2 * m + 1] = __uint_as_float(v.w);
        }
      } else {
#pragma unroll
        for (uint32_t m = 0; m < DEG; ++m) {
          const uint2 v = __ldg(ent_g + s * DEG + m);
          c[m] = 4 * v.x;
          j[m] = __uint_as_float(v.y);
        }
      }
#pragma unroll
      for (uint32_t m = 0; m < DEG; ++m) f(c[m], j[m]);
    } else {
      const uint32_t q = pos[s], g = q >> 5;
      const uint32_t o = soff[g];
      each_sliced(32 * o + (q & 31u), soff[g + 1] - o, f);
    }
  }
  // the number of entries of row s and its e-th column (the search)
  __device__ __forceinline__ uint32_t count(uint32_t s) const {
    if (DEG) return DEG;
    const uint32_t g = pos[s] >> 5;
    return soff[g + 1] - soff[g];
  }
  __device__ __forceinline__ uint32_t col(uint32_t s, uint32_t e) const {
    if (DEG) {
      if (RS) return reinterpret_cast<const uint16_t*>(colp)[2 * ((e >> 1) * n + s) + (e & 1u)] >> 2;
      return __ldg(&ent_g[s * DEG + e].x);
    }
    const uint32_t q = pos[s], x = 32 * (soff[q >> 5] + e) + (q & 31u);
    return RS ? reinterpret_cast<const uint16_t*>(colp)[x] >> 2 : __ldg(&ent_g[x].x) >> 2;
  }
};

struct LadClock {  // per-phase cycles (thread 0), PtJob::prof
  unsigned long long* out;
  long long t;
  __device__ __forceinline__ void start(unsigned long long* o) {
    out = o;
    if (out && threadIdx.x == 0) t = clock64();
  }
  __device__ __forceinline__ void lap(int phase) {
    if (out && threadIdx.x == 0) {
      const long long now = clock64();
      atomicAdd(&out[phase], (unsigned long long)(now - t));
      t = now;
    }
  }
};

// Sum of a over the block, in thread 0 of every warp's view of red (integers:
// any order); the caller's next barrier must come before red is used again.
__device__ __forceinline__ long long lad_warp_sum(long long a) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
  return a;
}

// Barrier over the first `count` threads on barrier 1, returning whether any
// of them passed a non-zero `pred`.
__device__ __forceinline__ int lad_bar1_or(int pred, uint32_t count) {
  int r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.s32 q, %1, 0;\n\tbar.red.or.pred p, 1, %2, q;\n\tselp.s32 %0, 1, 0, p;\n\t}"
      : "=r"(r)
      : "r"(pred), "r"(count)
      : "memory");
  return r;
}

// Growth on a periodic square or cubic lattice of side L in file order: a
// thread owns the lattice rows r = tid + k T (L bits along the last axis).  A
// step takes in the cluster bits of the neighbouring rows and of the row's own
// ends (the periodic wrap) and fills the row's q<0 runs from them: the carry
// of d + c runs from each seed to the top of its run, bit reversal gives the
// other direction.  Threads run ahead of one another between barriers (words
// only gain bits, and only their owner writes them); a batch of steps in which
// nothing grew anywhere ends the search, so the result is the exact component.
// (4096 sites: a step of this kind takes about a third of one on words of two
// rows closed twice, which is what the plain form's kernel does.)
__device__ __forceinline__ uint32_t lad_fill(uint32_t c, uint32_t d) {
  const uint32_t rd = __brev(d), rc = __brev(c);
  return ((((d + c) ^ d) & d) | c) | __brev((((rd + rc) ^ rd) & rd) | rc);
}
template <uint32_t DIM>
__device__ void lad_grow_lattice(const LadSm S, uint32_t L, uint32_t nrow) {
  const uint32_t tid = threadIdx.x, T = blockDim.x;
  const uint32_t G = min(T, (nrow + 31u) & ~31u);
  if (tid >= G) return;
  volatile uint32_t* const Cr = lad_at<uint32_t>(S.Cr);
  const uint32_t* const Dr = lad_at<uint32_t>(S.Dr);
  const uint32_t up = L - 1;
  // the rows next to row r along the other axes
  auto next = [&](uint32_t r, uint32_t* q) {
    if (DIM == 2) {
      q[0] = r ? r - 1 : up;
      q[1] = r == up ? 0 : r + 1;
    } else {
      const uint32_t x = r / L, y = r - x * L;
      q[0] = y ? r - 1 : r + up;
      q[1] = y == up ? r - up : r + 1;
      q[2] = x ? r - L : r + nrow - L;
      q[3] = x == up ? r + L - nrow : r + L;
    }
  };
  if (nrow <= T) {  // a row per thread, its state in registers
    const bool has = tid < nrow;
    uint32_t q[4] = {0, 0, 0, 0}, d = 0, c = 0;
    if (has) {
      next(tid, q);
      d = Dr[tid];
      c = Cr[tid];
    }
    for (uint32_t batch = 0; batch < 32u * nrow + 2u; ++batch) {
      const uint32_t c_in = c;
#pragma unroll 1
      for (int step = 0; step < 4; ++step) {
        if (c == d) continue;
        uint32_t nb = Cr[q[0]] | Cr[q[1]];
        if (DIM == 3) nb |= Cr[q[2]] | Cr[q[3]];
        nb |= (c << 1) | (c >> up) | (c >> 1) | (c << up);
        const uint32_t c1 = lad_fill(c | (d & nb), d);
        if (c1 != c) Cr[tid] = c = c1;
      }
      if (!lad_bar1_or(c != c_in, G)) break;
    }
  } else {
    for (uint32_t batch = 0; batch < 32u * nrow + 2u; ++batch) {
      int grew = 0;
#pragma unroll 1
      for (int step = 0; step < 2; ++step)
        for (uint32_t r = tid; r < nrow; r += G) {
          const uint32_t d = Dr[r], c = Cr[r];
          if (c == d) continue;
          uint32_t q[4];
          next(r, q);
          uint32_t nb = Cr[q[0]] | Cr[q[1]];
          if (DIM == 3) nb |= Cr[q[2]] | Cr[q[3]];
          nb |= (c << 1) | (c >> up) | (c >> 1) | (c << up);
          const uint32_t c1 = lad_fill(c | (d & nb), d);
          if (c1 != c) {
            Cr[r] = c1;
            grew = 1;
          }
        }
      if (!lad_bar1_or(grew, G)) break;
    }
  }
}

// Growth on any graph: a breadth-first search from the seed, one barrier per
// level.  A frontier site is expanded by a team of lanes, an edge each; a site
// that joins (an atomicOr on the cluster bitmap decides who adds it) is appended
// to the list, whose consecutive segments are the levels, with one atomic per
// warp and step.  The levels' counters rotate over three cells, so that one
// barrier separates reading, filling and clearing them.  Leaves the cluster's
// sites in the list and returns their number.  (What a level costs is its chain
// of dependent shared loads and two atomics, so a team covers most rows in one
// step: rows of up to 32 entries on teams of four took twice as long, and so
// did passes in which every site watches its own bit.)
template <int MODE, bool RS>
__device__ uint32_t lad_bfs(const PtJob& J, const LadSm S, uint32_t seed, uint32_t* cells) {
  constexpr uint32_t DEG = LadMode<MODE>::DEG;
  constexpr uint32_t TEAM = DEG == 0 ? 16u : DEG <= 4 ? 4u : 8u;
  const LadRows<MODE, RS> R(J, S);
  const uint32_t tid = threadIdx.x, T = blockDim.x, lane = tid & 31u, warp = tid >> 5;
  uint32_t *const Db = lad_at<uint32_t>(S.D), *const Cb = lad_at<uint32_t>(S.C);
  uint16_t* const list = lad_at<uint16_t>(S.list);
  if (tid == 0) {
    list[0] = (uint16_t)seed;
    Cb[seed >> 5] = 1u << (seed & 31u);
    cells[0] = 1;
    cells[1] = 0;
    cells[2] = 0;
  }
  __syncthreads();
  const uint32_t lt = (1u << lane) - 1u;
  uint32_t lo = 0;
  for (uint32_t lvl = 0; lvl < J.n + 2u; ++lvl) {
    const uint32_t ncur = cells[lvl % 3u];
    if (ncur == 0) break;
    uint32_t* const qn = &cells[(lvl + 1u) % 3u];
    uint16_t* const nxt = list + lo + ncur;
    const uint32_t items = TEAM * ncur;
    for (uint32_t b0 = warp * 32u; b0 < items; b0 += T) {  // warp-uniform trip count
      const uint32_t x = b0 + lane;
      uint32_t s = 0, w = 0;
      if (x < items) {
        s = list[lo + x / TEAM];
        w = R.count(s);
      }
      const uint32_t wmax = DEG ? DEG : __reduce_max_sync(0xffffffffu, w);
      for (uint32_t e = lane % TEAM; e - lane % TEAM < wmax; e += TEAM) {
        uint32_t c = 0;
        bool join = false;
        if (e < w) {
          c = R.col(s, e);
          const uint32_t bit = 1u << (c & 31u);
          if (Db[c >> 5] & ~Cb[c >> 5] & bit) join = !(atomicOr(&Cb[c >> 5], bit) & bit);
        }
        const uint32_t b = __ballot_sync(0xffffffffu, join);
        if (!b) continue;
        uint32_t o = 0;
        if (lane == 0) o = atomicAdd(qn, (uint32_t)__popc(b));
        o = __shfl_sync(0xffffffffu, o, 0);
        if (join) nxt[o + __popc(b & lt)] = (uint16_t)c;
      }
    }
    lo += ncur;
    if (tid == 0) cells[(lvl + 2u) % 3u] = 0;
    __syncthreads();
  }
  return lo;
}

// Houdayer move of this CTA's slot at sweep i: as icm_group (the k-th q<0 site
// in colour order from the same draw, the exact component of it, the same f32
// boundary terms in fixed point).  `mate`: the other replica's spin bits.  The
// terms are summed for the pair's first replica and the second's change is the
// negative sum, as there: every neighbour outside the cluster has the same spin in
// both replicas and every cluster site opposite ones, so in the second's CTA the
// own spins are turned (misc[7]: 2^31 there; in a register it cost the search on
// lattices 1 to 2 % of a round).  (Its own sum would be the negative one too, but
// not where a term is beyond the fixed point's range: -2^63 to 2^63 - 1.)
// Returns whether the slot had a q<0 site; *dE: the energy change (thread 0).
template <int MODE, bool RS>
__device__ __noinline__ bool lad_icm(const PtJob& J, const LadSm S, const uint32_t* mate, uint32_t t, uint32_t p,
                                     uint32_t i, uint32_t* misc, long long* dE, LadClock& pc) {
  const LadRows<MODE, RS> R(J, S);
  const uint32_t tid = threadIdx.x, T = blockDim.x, lane = tid & 31u, warp = tid >> 5, nwarp = T >> 5;
  const uint32_t n = J.n, nwb = (n + 31) / 32;
  const uint32_t L = J.F.lat_any, nrow = L ? n / L : 0u;
  uint32_t *const own = lad_at<uint32_t>(S.own), *const Db = lad_at<uint32_t>(S.D), *const Cb = lad_at<uint32_t>(S.C),
           *const flat = lad_at<uint32_t>(S.flat), *const Dr = lad_at<uint32_t>(S.Dr),
           *const Cr = lad_at<uint32_t>(S.Cr);
  const uint16_t *const perm = lad_at<uint16_t>(S.perm), *const iperm = lad_at<uint16_t>(S.iperm);
  uint16_t* const list = lad_at<uint16_t>(S.list);
  long long* const red = lad_at<long long>(S.red);
  for (uint32_t w = tid; w < nwb; w += T) {
    Db[w] = own[w] ^ __ldcg(mate + w);
    if (!L) Cb[w] = 0;
  }
  if (tid == 0) misc[3] = 0;
  __syncthreads();
  if (L) {
    for (uint32_t w = warp; w < nwb; w += nwarp) {
      const uint32_t o = 32 * w + lane;
      const uint32_t b = __ballot_sync(0xffffffffu, o < n && bm_bit(Db, o < n ? iperm[o] : 0u));
      if (lane == 0) flat[w] = b;
    }
    if (tid == 0) flat[nwb] = 0;
  }
  if (warp == nwarp - 1) {
    // the seed: count, draw k, the word holding the k-th site, the site
    uint32_t cnt = 0, seed = 0;
    for (uint32_t w = lane; w < nwb; w += 32) cnt += __popc(Db[w]);
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (cnt) {
      const uint32_t u = philox4x32_10w(make_uint4(t, i, p, PTAG_ICM), J.key).x;
      uint32_t kk = (uint32_t)(((uint64_t)u * cnt) >> 32);
      for (uint32_t w0 = 0; w0 < nwb; w0 += 32) {
        const uint32_t m = w0 + lane < nwb ? Db[w0 + lane] : 0u;
        const uint32_t cc = __popc(m);
        uint32_t incl = cc;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= (uint32_t)o) incl += v;
        }
        const uint32_t tot = __shfl_sync(0xffffffffu, incl, 31);
        if (kk < tot) {
          const uint32_t src = __ffs(__ballot_sync(0xffffffffu, kk < incl)) - 1;
          const uint32_t m2 = __shfl_sync(0xffffffffu, m, src);
          const uint32_t k2 = kk - __shfl_sync(0xffffffffu, incl - cc, src);
          // lane b holds bit b: the set bit with k2 set bits below it
          const bool is = ((m2 >> lane) & 1u) && (uint32_t)__popc(m2 & ((1u << lane) - 1u)) == k2;
          seed = (w0 + src) * 32 + __ffs(__ballot_sync(0xffffffffu, is)) - 1;
          break;
        }
        kk -= tot;
      }
    }
    if (lane == 0) {
      misc[0] = cnt;
      misc[1] = cnt ? (L ? perm[seed] : seed) : 0u;
    }
  }
  __syncthreads();
  pc.lap(PHASE_ICM_INIT);
  if (!misc[0]) return false;
  uint32_t nlist;
  if (L) {
    const uint32_t so = misc[1], sr = so / L, mask = L == 32 ? 0xffffffffu : (1u << L) - 1u;
    for (uint32_t r = tid; r < nrow; r += T) {
      const uint32_t b = r * L;
      Dr[r] = __funnelshift_r(flat[b >> 5], flat[(b >> 5) + 1], b & 31u) & mask;
      Cr[r] = r == sr ? 1u << (so - sr * L) : 0u;
    }
    __syncthreads();
    if (nrow == L) lad_grow_lattice<2>(S, L, nrow);
    else lad_grow_lattice<3>(S, L, nrow);
    __syncthreads();
    pc.lap(PHASE_ICM_GROW);
    // back to one bitmap in file order, then to colour order
    for (uint32_t w = tid; w < nwb; w += T) {
      uint32_t v = 0;
      for (uint32_t r = 32 * w / L; r < nrow && r * L < 32 * w + 32; ++r) {
        const int sh = (int)(r * L) - (int)(32 * w);
        v |= sh >= 0 ? Cr[r] << sh : Cr[r] >> -sh;
      }
      flat[w] = v;
    }
    __syncthreads();
    for (uint32_t w = warp; w < nwb; w += nwarp) {
      const uint32_t s = 32 * w + lane;
      const uint32_t b = __ballot_sync(0xffffffffu, s < n && bm_bit(flat, s < n ? perm[s] : 0u));
      if (lane == 0) Cb[w] = b;
    }
    __syncwarp();
    // the cluster's sites as a list (each warp its own words, in one piece)
    uint32_t cnt = 0;
    for (uint32_t w = warp + nwarp * lane; w < nwb; w += 32 * nwarp) cnt += __popc(Cb[w]);
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    uint32_t o = 0;
    if (lane == 0 && cnt) o = atomicAdd(&misc[3], cnt);
    o = __shfl_sync(0xffffffffu, o, 0);
    for (uint32_t w = warp; w < nwb; w += nwarp) {
      const uint32_t b = Cb[w];
      if ((b >> lane) & 1u) list[o + __popc(b & ((1u << lane) - 1u))] = (uint16_t)(32 * w + lane);
      o += __popc(b);
    }
    __syncthreads();
    nlist = misc[3];
  } else {
    nlist = lad_bfs<MODE, RS>(J, S, misc[1], misc + 4);
    pc.lap(PHASE_ICM_GROW);
  }
  // boundary terms -2 s (h + sum over neighbours outside the cluster)
  long long a0 = 0;
  for (uint32_t x = tid; x < nlist; x += T) {
    const uint32_t s = list[x];
    float f = R.bias(s);
    R.each(s, [&](uint32_t c4, float j) {
      if (!bm_bit(Cb, c4 >> 2)) f += __uint_as_float(__float_as_uint(j) ^ lad_sign(c4));
    });
    a0 += to_fx(-2.0f * __uint_as_float(__float_as_uint(f) ^ lad_word(s) ^ misc[7]));
  }
  a0 = lad_warp_sum(a0);
  if (lane == 0) red[2 * warp] = a0;
  __syncthreads();
  for (uint32_t x = tid; x < nlist; x += T) lad_word(list[x]) ^= 0x80000000u;
  for (uint32_t w = tid; w < nwb; w += T) own[w] ^= Cb[w];
  if (warp == 0) {
    const long long a = lad_warp_sum(lane < nwarp ? red[2 * lane] : 0ll);
    if (tid == 0) *dE = misc[7] ? -a : a;
  }
  pc.lap(PHASE_ICM_APPLY);
  return true;
}

// Uniform of the exchange (24 bits, as exchange_decide).
__device__ __forceinline__ float lad_u24(uint32_t r) { return (float)(r >> 8) * (1.0f / 16777216.0f); }

// Exchange decisions of a chain, by one warp: bit j of the result = the
// replicas of slots j and j + 1 swap.  x = LadSm::ex (beta differences and
// uniforms already there), pe = published energies of the chain, kept in E.
__device__ unsigned long long lad_decide(bool threaded, uint32_t nt, const float* x, const double* pe, double2* E,
                                         uint32_t lane) {
  bool d0[2];
  double2 e[2];
  float des0[2] = {0.0f, 0.0f}, db[2] = {0.0f, 0.0f}, u[2] = {1.0f, 1.0f};
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t j = lane + 32u * h;
    e[h] = j < nt ? __ldcg(reinterpret_cast<const double2*>(pe) + j) : make_double2(0.0, 0.0);
    if (j + 1 < nt) {
      db[h] = x[j];
      u[h] = x[64 + j];
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t j = lane + 32u * h;
    const float lo = (float)e[h].x;
    const float up = __shfl_down_sync(0xffffffffu, lo, 1), wrap = __shfl_sync(0xffffffffu, (float)e[1].x, 0);
    const float hi = lane == 31 ? wrap : up;  // (slot 32 follows slot 31; pair 63 does not exist)
    if (j < nt) E[j] = e[h];
    d0[h] = false;
    if (j + 1 < nt) {
      des0[h] = hi - lo;
      const float dlt = db[h] * des0[h];
      d0[h] = dlt >= 0.0f || u[h] < __expf(dlt);
    }
  }
  if (!threaded) return serial_swaps(nt, des0, db, u, d0);
  return (uint64_t)__ballot_sync(0xffffffffu, d0[0]) | ((uint64_t)__ballot_sync(0xffffffffu, d0[1]) << 32);
}

// The slot whose replica moves to slot t under the swaps D.
__device__ __forceinline__ uint32_t lad_src(uint64_t D, uint32_t t) {
  if ((D >> t) & 1ull) return t + 1;
  if (t > 0 && ((D >> (t - 1)) & 1ull)) {
    const uint64_t nd = ~D & ((1ull << t) - 1ull);
    return nd ? (uint32_t)(64 - __clzll((long long)nd)) : 0u;
  }
  return t;
}

// Bookkeeping of a chain's exchange (acceptance, tags, round trips, diffusion
// histogram), by one warp, in shared memory.
__device__ void lad_book(const LadSm S, uint32_t nt, uint64_t D, uint32_t* rtrips, uint32_t lane) {
  uint8_t* const tg = lad_at<uint8_t>(S.tags);
  uint32_t *const acc = lad_at<uint32_t>(S.acc), *const dhist = lad_at<uint32_t>(S.dhist);
  uint8_t t_new[2] = {0, 0};
  for (int q = 0; q < 2; ++q) {
    const uint32_t k = lane + 32u * q;
    if (k >= nt) continue;
    if ((D >> k) & 1ull) acc[k] += 1;
    t_new[q] = tg[lad_src(D, k)];
  }
  __syncwarp();
  for (int q = 0; q < 2; ++q)
    if (lane + 32u * q < nt) tg[lane + 32u * q] = t_new[q];
  __syncwarp();
  if (lane == 0) {  // PTState::update_round_trips (tamc-core/src/pt.rs:54-72)
    uint8_t lo = tg[0];
    if (lo == 0) lo = 1;
    else if (lo == 4) { *rtrips += 1; lo = 1; }
    else if (lo == 2) lo = 3;
    tg[0] = lo;
    uint8_t hi = tg[nt - 1];
    if (hi == 0) hi = 2;
    else if (hi == 3) { *rtrips += 1; hi = 2; }
    else if (hi == 1) hi = 4;
    tg[nt - 1] = hi;
  }
  __syncwarp();
  for (uint32_t k = lane; k < nt; k += 32) {
    const uint8_t v = tg[k];
    if (v == 1 || v == 3) dhist[2 * k] += 1;
    else if (v == 2 || v == 4) dhist[2 * k + 1] += 1;
  }
}

// One Metropolis sweep of the CTA's replica, a thread per site of the colour
// class.  Random numbers, sums and decisions are those of quad_update
// (component t % 4 of the quad's Philox call) or, for MSC, of msc_flip (bit
// t % 32 of its random words against the replica's thresholds thr, four levels
// per call).  Returns the fixed-point energy change (x) and self-coupling
// part (y) summed over the block, in thread 0.
template <int MODE, bool RS>
__device__ __noinline__ longlong2 lad_sweep(const PtJob& J, const LadSm S, uint32_t c, uint32_t t, float b2,
                                            const uint32_t* thr, uint32_t i) {
  constexpr uint32_t DEG = LadMode<MODE>::DEG;
  constexpr bool MSC = LadMode<MODE>::MSC;
  const LadRows<MODE, RS> R(J, S);
  const uint32_t tid = threadIdx.x, T = blockDim.x, lane = tid & 31u, warp = tid >> 5;
  const uint2 key = J.key;
  const uint32_t ncolors = J.F.ncolors, n = J.n;
  const uint32_t* const coff = lad_at<uint32_t>(S.coff);
  const uint32_t* const soff = lad_at<uint32_t>(S.soff);
  const uint16_t* const site = lad_at<uint16_t>(S.site);
  const bool self = MODE == LAD_ROWS && J.self_loops;
  const float* const kd = RS ? lad_at<float>(S.kd) : J.F.kd;
  long long* const red = lad_at<long long>(S.red);
  long long a = 0, q = 0;
  int units = 0;
  const uint32_t tq = t & 3u, qid = c * 16u + (t >> 2), tb = t & 31u, wo = (c * J.wpc + (t >> 5)) << 8;
  const uint32_t th0 = thr[0], th1 = thr[1], th2 = thr[2], thf = thr[3];
  auto decide = [&](uint32_t s, uint32_t own, float g) {
    g = __uint_as_float(__float_as_uint(g) ^ own);
    const uint4 r = philox4x32_10w(make_uint4(s, i, qid, PTAG_SWEEP), key);
    if (accept_g(g, b2, tq == 0 ? r.x : tq == 1 ? r.y : tq == 2 ? r.z : r.w)) {
      lad_word(s) = own ^ 0x80000000u;
      a += to_fx(-2.0f * g);
      if (self) q += to_fx(2.0f * kd[s]);
    }
  };
  uint32_t s1 = coff[0];
  for (uint32_t cl = 0; cl < ncolors; ++cl) {
    const uint32_t s0 = s1;
    s1 = coff[cl + 1];
    if (DEG == 0) {  // a slice per warp
      for (uint32_t sl = s0 + warp; sl < s1; sl += T >> 5) {
        const uint32_t s = site[32 * sl + lane], o = soff[sl], w = soff[sl + 1] - o;
        if (s == 0xffffu) continue;  // beyond the class's last site
        float g = R.bias(s);
        R.each_sliced(32 * o + lane, w,
                      [&](uint32_t c4, float j) { g += __uint_as_float(__float_as_uint(j) ^ lad_sign(c4)); });
        decide(s, lad_word(s), g);
      }
    } else {
      for (uint32_t s = s0 + tid; s < s1; s += T) {
        const uint32_t own = lad_word(s);
        if (MSC) {
          constexpr uint32_t LV = DEG ? DEG / 2 : 1;
          uint32_t sat = 0;
          R.each(s, [&](uint32_t c4, float j) { sat += (lad_sign(c4) ^ own ^ __float_as_uint(j)) >> 31; });
          const uint32_t x = DEG - sat;  // unsatisfied bonds
          bool f = x >= LV;
          if (!f) {
            f = (thf >> x) & 1u;
            if (!f && !((thf >> (8 + x)) & 1u)) {
              const uint32_t Tv = x == 0 ? th0 : x == 1 ? th1 : th2;
              for (uint32_t kk = 0; kk < 8; ++kk) {
                const uint4 r = philox4x32_10w(make_uint4(s, i, wo | kk, PTAG_MSC), key);
                const uint32_t v = ((r.x >> tb) & 1u) << 3 | ((r.y >> tb) & 1u) << 2 | ((r.z >> tb) & 1u) << 1 |
                                   ((r.w >> tb) & 1u);
                const uint32_t w = (Tv >> (28 - 4 * kk)) & 15u;
                if (v != w) {
                  f = v < w;
                  break;
                }
              }
            }
          }
          if (f) {
            lad_word(s) = own ^ 0x80000000u;
            units += 2 * ((int)DEG - 2 * (int)x);
          }
        } else {
          float g = R.bias(s);
          R.each(s, [&](uint32_t c4, float j) { g += __uint_as_float(__float_as_uint(j) ^ lad_sign(c4)); });
          decide(s, own, g);
        }
      }
    }
    __syncthreads();
  }
  if (MSC) a = (long long)units * 4294967296ll;  // to_fx of the integer energy change
  a = lad_warp_sum(a);
  if (MODE == LAD_ROWS) q = lad_warp_sum(q);
  if (lane == 0) {
    red[2 * warp] = a;
    red[2 * warp + 1] = q;
  }
  // the spin bits (a colour class's last flips are behind the barrier above)
  const uint32_t nwb = (n + 31) / 32;
  for (uint32_t w = warp; w < nwb; w += T >> 5) {
    const uint32_t s = 32 * w + lane;
    const uint32_t b = __ballot_sync(0xffffffffu, s < n && lad_word(s < n ? s : 0u));
    if (lane == 0) lad_at<uint32_t>(S.own)[w] = b;
  }
  __syncthreads();
  longlong2 sum = make_longlong2(0, 0);
  if (warp == 0) {
    sum.x = lad_warp_sum(lane < (T >> 5) ? red[2 * lane] : 0ll);
    if (MODE == LAD_ROWS) sum.y = lad_warp_sum(lane < (T >> 5) ? red[2 * lane + 1] : 0ll);
  }
  return sum;
}

// The replica's energy from scratch (energy_terms4: f32 row terms, in fixed
// point), in thread 0.
template <int MODE, bool RS>
__device__ __noinline__ double lad_energy(const PtJob& J, const LadSm S) {
  const LadRows<MODE, RS> R(J, S);
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, nwarp = blockDim.x >> 5;
  const uint32_t n = J.n;
  long long* const red = lad_at<long long>(S.red);
  long long a = 0;
  for (uint32_t s = tid; s < n; s += blockDim.x) {
    float g = R.bias(s);
    R.each(s, [&](uint32_t c4, float j) { g += __uint_as_float(__float_as_uint(0.5f * j) ^ lad_sign(c4)); });
    a += to_fx(__uint_as_float(__float_as_uint(g) ^ lad_word(s)));
  }
  a = lad_warp_sum(a);
  if (lane == 0) red[2 * warp] = a;
  __syncthreads();
  a = 0;
  if (tid == 0)
    for (uint32_t w = 0; w < nwarp; ++w) a += red[2 * w];
  __syncthreads();
  return (double)J.F.offset + (double)a * TAMC_FX_INV;
}

__device__ __forceinline__ bool lad_sched(int64_t period, uint32_t i, uint32_t meas_init, uint32_t num_sweeps) {
  return period >= 0 && i >= meas_init && ((i - meas_init) % (uint32_t)period == 0 || i == num_sweeps - 1);
}

// Overlaps of the slot's two replicas after round i (the even chain's CTA), as
// measure_rest: q and the weights, one warp each, in its summation order.
__device__ __noinline__ void lad_overlaps(const PtJob& J, const LadSm S, const uint32_t* mate, uint32_t p, uint32_t t,
                                          uint32_t m) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const uint32_t n = J.n, P = J.C / 2, nwb = (n + 31) / 32;
  uint32_t *const Db = lad_at<uint32_t>(S.D), *const own = lad_at<uint32_t>(S.own);
  for (uint32_t w = threadIdx.x; w < nwb; w += blockDim.x) Db[w] = own[w] ^ __ldcg(mate + w);
  __syncthreads();
  for (uint32_t k = warp; k <= J.out.nchi; k += nwarp) {
    if (k == 0) {
      uint32_t neg = 0;
      for (uint32_t w = lane; w < nwb; w += 32) neg += __popc(Db[w]);
      neg = __reduce_add_sync(0xffffffffu, neg);
      if (lane == 0) J.out.q[(size_t)t * J.out.M * P + (size_t)m * P + p] = (int32_t)n - 2 * (int32_t)neg;
    } else {
      const double* sus = J.F.sus + (size_t)(k - 1) * n;
      double v = 0.0;
      for (uint32_t s = lane; s < n; s += 32) {
        const double wv = sus[s];
        v += ((Db[s >> 5] >> lane) & 1u) ? -wv : wv;
      }
      for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
      if (lane == 0)
        J.out.sus[((size_t)t * J.out.nchi + (k - 1)) * J.out.M * P + (size_t)m * P + p] = (float)v;
    }
  }
  __syncthreads();
}

// The CTA's part of a run's rounds [sweep_begin, sweep_end).
template <int MODE, bool RS>
__device__ void lad_run(const LadJob& A) {
  const PtJob& J = A.J;
  constexpr uint32_t DEG = LadMode<MODE>::DEG;
  constexpr bool MSC = LadMode<MODE>::MSC;
  __shared__ uint32_t misc[8];      // q<0 count, seed, waits' result, list length, [3] search counters, second replica
  __shared__ unsigned long long s_D; // exchange: swapped slot pairs of the chain
  __shared__ double s_E[2];         // this replica's Ec, Er
  __shared__ float s_be;            // the round's lowest energy, and its slot
  __shared__ uint32_t s_bx, s_rtrips, s_thr[4];
  const uint32_t tid = threadIdx.x, T = blockDim.x, lane = tid & 31u, warp = tid >> 5, nwarp = T >> 5;
  const uint32_t n = J.n, nt = J.nt, C = J.C, nwb = (n + 31) / 32;
  const LadSm S = lad_carve(lad_dims(J, RS, DEG, MSC));
  uint32_t* const own = lad_at<uint32_t>(S.own);
  float* const ex = lad_at<float>(S.ex);
  const uint32_t g = blockIdx.x - A.cta0, c = g / nt, t = g % nt;
  const uint32_t p = c / 2, cm = c ^ 1u;  // pair, the other chain
  const bool two = cm < C;
  const uint32_t nr = J.sweep_end - J.sweep_begin;
  const bool lead = t == 0;  // keeps the bookkeeping of the chain
  const bool moves = J.icm && two && t >= J.lo;
  const size_t bstride = (size_t)C * nt * nwb, estride = (size_t)C * nt * 2, gstride = (size_t)C * nt;
  const uint32_t nh = 2 * ((n + 63) / 64);  // 32-bit halves of a logged state
  const size_t cstride = (size_t)C * nt * nh;
  const uint32_t me = c * nt + t, mate = cm * nt + t;
  if (RS) {
    if (!MSC)
      for (uint32_t x = tid; x < n; x += T) lad_at<float>(S.bias)[x] = J.F.bias[x];
    if (DEG) {
      for (uint32_t x = tid; x < n; x += T) {
        uint32_t h[DEG ? DEG + 1 : 2];
#pragma unroll
        for (uint32_t m = 0; m < DEG; ++m) {
          const uint2 v = J.F.ent[x * DEG + m];
          h[m] = 4 * v.x;
          if (MSC) h[m] |= v.y >> 31;
          else if (DEG % 2 == 0) lad_at<float>(S.J)[2 * ((m / 2) * n + x) + (m & 1u)] = __uint_as_float(v.y);
          else lad_at<float>(S.J)[m * n + x] = __uint_as_float(v.y);
        }
        h[DEG] = 0;
#pragma unroll
        for (uint32_t m = 0; m < (DEG + 1) / 2; ++m) lad_at<uint32_t>(S.colp)[m * n + x] = h[2 * m] | (h[2 * m + 1] << 16);
      }
    } else {
      for (uint32_t x = tid; x < 32 * J.F.sl_rows; x += T) {
        const uint2 v = J.F.sl_ent[x];
        lad_at<uint16_t>(S.colp)[x] = (uint16_t)v.x;
        lad_at<float>(S.J)[x] = __uint_as_float(v.y);
      }
    }
  }
  if (DEG) {
    for (uint32_t x = tid; x <= J.F.ncolors; x += T) lad_at<uint32_t>(S.coff)[x] = J.F.color_off[x];
  } else {
    for (uint32_t x = tid; x <= J.F.ncolors; x += T) lad_at<uint32_t>(S.coff)[x] = J.F.sl_cls[x];
    for (uint32_t x = tid; x < 32 * J.F.sl_n; x += T) lad_at<uint16_t>(S.site)[x] = J.F.sl_site[x];
    for (uint32_t x = tid; x <= J.F.sl_n; x += T) lad_at<uint32_t>(S.soff)[x] = J.F.sl_off[x];
    for (uint32_t x = tid; x < n; x += T) {
      lad_at<uint16_t>(S.pos)[x] = J.F.sl_pos[x];
      if (RS && J.self_loops) lad_at<float>(S.kd)[x] = J.F.kd[x];
    }
  }
  if (J.F.lat_any)
    for (uint32_t x = tid; x < n; x += T) {
      lad_at<uint16_t>(S.perm)[x] = (uint16_t)J.F.perm[x];
      lad_at<uint16_t>(S.iperm)[x] = (uint16_t)J.F.iperm[x];
    }
  const float b2 = J.betas[t] * TAMC_2LOG2E;
  // the replica as the opening kernel left it (second half of the buffer)
  for (uint32_t s = tid; s < n; s += T) {
    const uint32_t v = A.bits[bstride + (size_t)me * nwb + (s >> 5)];
    lad_word(s) = (v >> (s & 31u)) << 31;
    if ((s & 31u) == 0) own[s >> 5] = v;
  }
  for (uint32_t j = tid; j + 1 < nt; j += T) ex[j] = J.betas[j + 1] - J.betas[j];
  if (tid == 0) {
    misc[7] = c << 31;
    s_E[0] = J.Ec[c * J.ntp + t];
    s_E[1] = J.Er[c * J.ntp + t];
    if (MSC) {
      uint32_t f = 0;
      for (uint32_t l = 0; l < DEG / 2; ++l) {  // as msc_planes
        const double pr = exp(-(double)J.betas[t] * (double)(2 * ((int)DEG - 2 * (int)l)));
        const bool al = !(pr < 1.0);
        const uint32_t Tv = al ? 0xffffffffu : (uint32_t)(pr * 4294967296.0);
        s_thr[l] = Tv;
        if (al) f |= 1u << l;
        if (!al && Tv == 0) f |= 1u << (8 + l);
      }
      s_thr[3] = f;
    }
    if (lead) s_rtrips = J.rtrips[c];
  }
  if (lead)
    for (uint32_t x = tid; x < nt; x += T) {
      const size_t o = (size_t)c * nt + x;
      lad_at<uint8_t>(S.tags)[x] = J.tags[o];
      lad_at<uint32_t>(S.acc)[x] = J.acc[o];
      lad_at<uint32_t>(S.dhist)[2 * x] = J.dhist[2 * o];
      lad_at<uint32_t>(S.dhist)[2 * x + 1] = J.dhist[2 * o + 1];
    }
  // running minimum of the ground-state log (every CTA keeps it)
  int gs_have = *J.log.have;
  float gs_min = *J.log.minE;
  uint32_t gs_count = *J.log.count;
  __syncthreads();
  if (J.init) {
    const double e = lad_energy<MODE, RS>(J, S);
    if (tid == 0) s_E[0] = s_E[1] = e;
  }
  LadClock pc;
  pc.start(J.prof);
  uint32_t m_cur = J.m_base, s_cur = J.s_base;
  for (uint32_t r = 0; r <= nr; ++r) {  // r == nr: publish the final replicas and close the last round
    const uint32_t i = J.sweep_begin + r, par = r & 1u;
    if (r < nr && moves) {
      // the other replica's bits as its last sweep left them
      if (r) {
        if (tid == 0) misc[2] = lad_wait(A.flag + mate, r, A.polls, A.err);
        __syncthreads();
        if (!misc[2]) return;
      }
      pc.lap(PHASE_ICM_SCAN);
      long long dE = 0;
      const uint32_t* mb = r ? A.post + (size_t)mate * nwb : A.bits + bstride + (size_t)mate * nwb;
      if (lad_icm<MODE, RS>(J, S, mb, t, p, i, misc, &dE, pc) && tid == 0) {
        // the reference invalidates both caches; the next energy() is energy_ref
        s_E[1] += (double)dE * TAMC_FX_INV;
        s_E[0] = s_E[1];
      }
      __syncthreads();
    }
    // publish the replica and its energies
    uint32_t* const bits = A.bits + par * bstride;
    double* const pe = A.pe + par * estride;
    for (uint32_t w = tid; w < nwb; w += T) __stcg(&bits[(size_t)me * nwb + w], own[w]);
    if (tid == 0) {
      __stcg(pe + 2 * me, s_E[0]);
      __stcg(pe + 2 * me + 1, s_E[1]);
    }
    // the exchange's uniforms while the stores drain
    if (r < nr && warp == nwarp - 1)
      for (uint32_t j = lane; j + 1 < nt; j += 32)
        ex[64 + j] = lad_u24(philox4x32_10w(make_uint4(j, i, c, PTAG_EXCH), J.key).x);
    pc.lap(PHASE_ICM_SCAN);
    if (!lad_barrier(A.bar, (r + 1) * A.ncta, A.polls, A.err, &misc[2])) return;
    pc.lap(PHASE_OTHER);
    // the two replicas most likely to move into this slot, read while the
    // decisions are made (threads below nwb: slot t + 1's, the next nwb: t - 1's)
    uint32_t fetched = 0;
    if (r < nr && tid < 2 * nwb) {
      const uint32_t ts = tid < nwb ? t + 1 : t - 1;
      if (ts < nt) fetched = __ldcg(&bits[((size_t)c * nt + ts) * nwb + (tid < nwb ? tid : tid - nwb)]);
    }
    // ground-state tracking of the round before (apply_measurements,
    // src/pt.rs:542-583): first minimum over slots, then over chains
    const bool track = r > 0 && i - 1 >= J.meas_init;
    if (track && warp == nwarp - 2) {
      const float* pg = A.pg + (par ^ 1u) * gstride;
      float be = INFINITY;
      uint32_t bx = 0xffffffffu;
      for (uint32_t x = lane; x < C * nt; x += 32) {
        const float e = __ldcg(pg + x);
        if (e < be || (e == be && x < bx)) {
          be = e;
          bx = x;
        }
      }
      for (int off = 16; off > 0; off >>= 1) {
        const float oe = __shfl_xor_sync(0xffffffffu, be, off);
        const uint32_t ox = __shfl_xor_sync(0xffffffffu, bx, off);
        if (oe < be || (oe == be && ox < bx)) {
          be = oe;
          bx = ox;
        }
      }
      if (lane == 0) {
        s_bx = bx == 0xffffffffu ? 0u : bx;
        s_be = be;
      }
    }
    if (r < nr && warp == nwarp - 1) {
      const unsigned long long D = lad_decide(J.threaded, nt, ex, pe + (size_t)c * nt * 2, lad_at<double2>(S.E), lane);
      if (lane == 0) s_D = D;
    }
    __syncthreads();
    if (track) {
      const float be = s_be;
      if (!gs_have || be < gs_min) {
        gs_have = 1;
        gs_min = be;
        if (gs_count < J.log.cap && g == 0) {
          if (tid == 0) {
            J.log.steps[gs_count] = i - 1;
            J.log.E[gs_count] = be;
          }
          const uint32_t* src = A.cand + (par ^ 1u) * cstride + (size_t)s_bx * nh;
          uint32_t* dst = reinterpret_cast<uint32_t*>(J.log.words + (size_t)gs_count * (nh / 2));
          for (uint32_t h = tid; h < nh; h += T) dst[h] = __ldcg(src + h);
        }
        ++gs_count;
      }
    }
    if (r == nr) break;
    // the replica that moved into this CTA's slot
    const uint64_t D = s_D;
    const uint32_t src = lad_src(D, t);
    if (src != t) {
      if (tid == 0) {
        const double2 e = lad_at<double2>(S.E)[src];
        s_E[0] = e.x;
        s_E[1] = e.y;
      }
      if (2 * nwb <= T && (src == t + 1 || src + 1 == t)) {
        const uint32_t x0 = src == t + 1 ? 0u : nwb;
        if (tid >= x0 && tid < x0 + nwb) own[tid - x0] = fetched;
      } else {
        const uint32_t* b = bits + ((size_t)c * nt + src) * nwb;
        for (uint32_t w = tid; w < nwb; w += T) own[w] = __ldcg(b + w);
      }
      __syncthreads();
      for (uint32_t s = tid; s < n; s += T) lad_word(s) = (own[s >> 5] >> (s & 31u)) << 31;
    }
    if (lead && warp == nwarp - 1) lad_book(S, nt, D, &s_rtrips, lane);
    __syncthreads();
    pc.lap(PHASE_EXCH);
    const longlong2 dE = lad_sweep<MODE, RS>(J, S, c, t, b2, s_thr, i);
    pc.lap(PHASE_SWEEP);
    // IsingSampler::sweep: energy += sum of accepted dE (src/ising.rs:226-232)
    if (tid == 0) {
      s_E[0] += (double)dE.x * TAMC_FX_INV;
      s_E[1] += (double)(dE.x + dE.y) * TAMC_FX_INV;
    }
    const bool meas = lad_sched(J.sample, i, J.meas_init, J.num_sweeps);
    const bool snap = lad_sched(J.sample_states, i, J.meas_init, J.num_sweeps);
    if (moves || (meas && two)) {  // this replica's bits for its mate
      for (uint32_t w = tid; w < nwb; w += T) __stcg(A.post + (size_t)me * nwb + w, own[w]);
      __syncthreads();
      if (tid == 0) lad_st_release(A.flag + me, r + 1);
    }
    if (i >= J.meas_init) {
      // for the tracking after the next barrier: the energy, and the state of a
      // replica below the running minimum (it may become it)
      __syncthreads();
      const float ef = (float)s_E[0];
      if (tid == 0) __stcg(A.pg + par * gstride + me, ef);
      const bool low = !gs_have || !(ef >= gs_min);
      if (low || snap) {
        uint32_t* dst = A.cand + par * cstride + (size_t)me * nh;
        uint32_t z = 0xffffffffu;  // sample slot of temperature t, if sampled
        if (snap) {
          const uint32_t Z = J.level == 0 ? nt : (J.level == 1 ? nt / 2 : 1);
          if (J.level == 0) z = t;
          else if (J.level == 1) z = nt - 1 - t < Z ? nt - 1 - t : 0xffffffffu;
          else z = t == nt - 1 ? 0u : 0xffffffffu;
        }
        const uint32_t nb = (n + 7) / 8;
        if (low || z != 0xffffffffu)
          for (uint32_t h = warp; h < nh; h += nwarp) {
            const uint32_t s = 32 * h + lane;
            const uint32_t v = __ballot_sync(0xffffffffu, s < n && bm_bit(own, s < n ? J.F.iperm[s] : 0u));
            if (low && lane == 0) __stcg(dst + h, v);
            if (z != 0xffffffffu && lane < 4 && 4 * h + lane < nb)
              J.out.samp[(((size_t)z * J.out.S + s_cur) * C + c) * nb + 4 * h + lane] = (uint8_t)(v >> (8 * lane));
          }
      }
      if (snap) ++s_cur;
      if (meas) {
        if (tid == 0) J.out.e[(size_t)t * J.out.M * C + (size_t)m_cur * C + c] = ef;
        if (two && !(c & 1u)) {
          if (tid == 0) misc[2] = lad_wait(A.flag + mate, r + 1, A.polls, A.err);
          __syncthreads();
          if (!misc[2]) return;
          lad_overlaps(J, S, A.post + (size_t)mate * nwb, p, t, m_cur);
        }
        ++m_cur;
      }
      pc.lap(PHASE_MEASURE);
    }
  }
  // the bookkeeping for the commit kernel
  if (lead) {
    const LadBook B = lad_book_view(A.book, C, nt);
    for (uint32_t x = tid; x < nt; x += T) {
      const size_t o = (size_t)c * nt + x;
      B.tags[o] = lad_at<uint8_t>(S.tags)[x];
      B.acc[o] = lad_at<uint32_t>(S.acc)[x];
      B.dhist[2 * o] = lad_at<uint32_t>(S.dhist)[2 * x];
      B.dhist[2 * o + 1] = lad_at<uint32_t>(S.dhist)[2 * x + 1];
    }
    if (tid == 0) {
      B.rtrips[c] = s_rtrips;
      if (g == 0) *B.gs = LadGs{gs_have, gs_min, gs_count};
    }
  }
}

template <int MODE>
__device__ __forceinline__ void lad_rows_dispatch(const LadJob& A) {
  if (A.rows_smem) lad_run<MODE, true>(A);
  else lad_run<MODE, false>(A);
}

// One replica of one run; `cta_job` maps CTAs to runs (null: one run).
__global__ void __launch_bounds__(1024, 1) k_pt_ladder(const LadJob* __restrict__ jobs,
                                                       const uint32_t* __restrict__ cta_job) {
  __shared__ LadJob s_A;
  const LadJob* src = jobs + (cta_job ? cta_job[blockIdx.x] : 0u);
  static_assert(sizeof(LadJob) % 8 == 0, "copied as 8-byte words");
  for (uint32_t x = threadIdx.x; x < sizeof(LadJob) / 8; x += blockDim.x)
    reinterpret_cast<uint2*>(&s_A)[x] = reinterpret_cast<const uint2*>(src)[x];
  __syncthreads();
  switch (s_A.mode) {
    case LAD_DEG3: lad_rows_dispatch<LAD_DEG3>(s_A); break;
    case LAD_DEG4: lad_rows_dispatch<LAD_DEG4>(s_A); break;
    case LAD_DEG6: lad_rows_dispatch<LAD_DEG6>(s_A); break;
    case LAD_MSC4: lad_rows_dispatch<LAD_MSC4>(s_A); break;
    case LAD_MSC6: lad_rows_dispatch<LAD_MSC6>(s_A); break;
    default: lad_rows_dispatch<LAD_ROWS>(s_A); break;
  }
}

// The replicas of the runs (blockIdx.y) from their words W[n][nw] (or fresh
// random ones) into bitmaps per slot, a 32 x 32 block of bits per warp.
__global__ void k_ladder_open(const LadJob* __restrict__ jobs) {
  const LadJob& A = jobs[blockIdx.y];
  const PtJob& J = A.J;
  const uint32_t lane = threadIdx.x & 31u, nwb = (J.n + 31) / 32;
  const uint64_t total = (uint64_t)nwb * J.nw;
  uint32_t* const bits = A.bits + (size_t)J.C * J.nt * nwb;
  for (uint64_t x = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; x < total;
       x += ((uint64_t)gridDim.x * blockDim.x) >> 5) {
    const uint32_t blk = (uint32_t)(x % nwb), o = (uint32_t)(x / nwb), c = o / J.wpc, w = o % J.wpc;
    const uint32_t s = 32 * blk + lane;
    uint32_t v = 0;
    if (s < J.n) {
      if (J.init == 1) {
        for (uint32_t qq = 0; qq < 8; ++qq) {
          const uint32_t q = 8 * w + qq;
          if (q >= J.qpc) break;
          v |= init_nibble(philox4x32_10(make_uint4(s, 0xffffffffu, c * 16u + q, PTAG_INIT), J.key)) << (4 * qq);
        }
      } else {
        v = J.W[(size_t)s * J.nw + o];
      }
    }
    v = transpose32(v, lane);
    const uint32_t t = 32 * w + lane;
    if (t < J.nt) bits[((size_t)c * J.nt + t) * nwb + blk] = v;
  }
}

// The results of the runs' rounds into their words, energies and bookkeeping;
// nothing (and LAD_GAVE_UP as the log count) where a CTA gave up.
__global__ void k_ladder_commit(const LadJob* __restrict__ jobs) {
  const LadJob& A = jobs[blockIdx.y];
  const PtJob& J = A.J;
  if (*A.err) {
    if (blockIdx.x == 0 && threadIdx.x == 0 && J.count_out) *J.count_out = LAD_GAVE_UP;
    return;
  }
  const uint32_t lane = threadIdx.x & 31u, nwb = (J.n + 31) / 32;
  const uint64_t total = (uint64_t)nwb * J.nw;
  const uint32_t par = (J.sweep_end - J.sweep_begin) & 1u;
  const uint32_t* bits = A.bits + (size_t)par * J.C * J.nt * nwb;
  const uint64_t gt = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, GT = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t x = gt >> 5; x < total; x += GT >> 5) {
    const uint32_t blk = (uint32_t)(x % nwb), o = (uint32_t)(x / nwb), c = o / J.wpc, w = o % J.wpc;
    const uint32_t t = 32 * w + lane;
    const uint32_t v = transpose32(t < J.nt ? bits[((size_t)c * J.nt + t) * nwb + blk] : 0u, lane);
    const uint32_t s = 32 * blk + lane;
    if (s < J.n) J.W[(size_t)s * J.nw + o] = v;
  }
  const double* pe = A.pe + (size_t)par * J.C * J.nt * 2;
  const LadBook B = lad_book_view(A.book, J.C, J.nt);
  for (uint64_t x = gt; x < (uint64_t)J.C * J.nt; x += GT) {
    const uint32_t c = (uint32_t)(x / J.nt), t = (uint32_t)(x % J.nt);
    J.Ec[c * J.ntp + t] = pe[2 * x];
    J.Er[c * J.ntp + t] = pe[2 * x + 1];
    J.tags[x] = B.tags[x];
    J.acc[x] = B.acc[x];
    J.dhist[2 * x] = B.dhist[2 * x];
    J.dhist[2 * x + 1] = B.dhist[2 * x + 1];
  }
  for (uint64_t x = gt; x < J.C; x += GT) J.rtrips[x] = B.rtrips[x];
  if (gt == 0) {
    *J.log.have = B.gs->have;
    *J.log.minE = B.gs->minE;
    *J.log.count = B.gs->count;
    if (J.count_out) *J.count_out = B.gs->count;
  }
}

int lad_mode(const PtJob& j) {
  if (j.msc) return j.F.udeg == 4 ? LAD_MSC4 : LAD_MSC6;
  if (j.self_loops) return LAD_ROWS;
  return j.F.udeg == 3 ? LAD_DEG3 : j.F.udeg == 4 ? LAD_DEG4 : j.F.udeg == 6 ? LAD_DEG6 : LAD_ROWS;
}

}  // namespace

size_t ladder_scratch_bytes(const PtJob& j) {
  LadJob a{};
  a.J = j;
  return ladder_bind(a, nullptr);
}

size_t ladder_bind(LadJob& a, char* base) {
  const PtJob& j = a.J;
  size_t o = 0;
  auto take = [&](size_t bytes) {
    char* p = base ? base + o : nullptr;
    o = (o + bytes + 255) & ~(size_t)255;
    return p;
  };
  const size_t R = (size_t)j.C * j.nt, nwb = (j.n + 31) / 32, nh = 2 * ((size_t)(j.n + 63) / 64);
  a.bar = (uint32_t*)take(4 + R * 4);  // the barrier's arrivals, then the replicas' flags: cleared together
  a.flag = a.bar ? a.bar + 1 : nullptr;
  a.bits = (uint32_t*)take(2 * R * nwb * 4);
  a.post = (uint32_t*)take(R * nwb * 4);
  a.pe = (double*)take(2 * R * 2 * 8);
  a.pg = (float*)take(2 * R * 4);
  a.cand = (uint32_t*)take(2 * R * nh * 4);
  a.book = take(lad_book_bytes(j.C, j.nt));
  return o;
}

static uint32_t lad_deg(int mode) {
  return mode == LAD_DEG3 ? 3u : mode == LAD_DEG4 || mode == LAD_MSC4 ? 4u : mode == LAD_DEG6 || mode == LAD_MSC6 ? 6u : 0u;
}

size_t ladder_smem(const PtJob& j, int rows) {
  const int m = lad_mode(j);
  const uint32_t deg = lad_deg(m);
  if (rows && j.n > 16383) return SIZE_MAX;  // 16-bit byte offsets
  // (the layout below counts in 32 bits; rows of more than a megabyte, which could be
  // read from L2, were not measured in this form)
  if (j.n > 65535 || (uint64_t)j.F.sl_rows * 192 > (1u << 20)) return SIZE_MAX;
  if (!deg && !j.F.sl_ent) return SIZE_MAX;
  return lad_carve(lad_dims(j, rows, deg, m == LAD_MSC4 || m == LAD_MSC6)).bytes;
}

size_t ladder_sync_bytes(const PtJob& j) { return 4 + (size_t)j.C * j.nt * 4; }

void ladder_shape(LadJob& a, int rows, uint32_t cta0) {
  const PtJob& j = a.J;
  a.ncta = j.C * j.nt;
  a.cta0 = cta0;
  a.mode = lad_mode(j);
  a.rows_smem = rows;
  a.polls = 8u << 20;  // some seconds
  if (const char* e = getenv("TAMC_LADDER_POLLS")) a.polls = (uint32_t)strtoul(e, nullptr, 10);
}

static void ladder_attr(size_t smem) { kernel_smem(reinterpret_cast<const void*>(k_pt_ladder), smem); }

size_t ladder_smem_limit(const tamc_gpu* g) {
  static std::atomic<size_t> own{0};  // the kernel's static shared memory
  size_t b = own.load(std::memory_order_relaxed);
  if (!b) {
    cudaFuncAttributes a{};
    TAMC_CUDA(cudaFuncGetAttributes(&a, k_pt_ladder));
    own.store(b = a.sharedSizeBytes, std::memory_order_relaxed);
  }
  return g->smem_block - b;
}

// Resident CTAs per SM for each CTA size and shared-memory size asked about (at
// most one entry per 16 bytes of shared memory and CTA size): a server plans every
// step anew, and asking the runtime for every candidate of a plan cost 0.9 ms a step
// with 512 requests.
static std::atomic<uint64_t> g_ladder_queries{0};
uint64_t ladder_queries() { return g_ladder_queries.load(std::memory_order_relaxed); }

uint32_t ladder_capacity(const tamc_gpu* g, uint32_t T, size_t smem) {
  static std::mutex mu;
  static std::map<std::tuple<int, uint32_t, size_t>, int> known;
  std::lock_guard<std::mutex> lk(mu);
  auto it = known.find(std::make_tuple(g->device, T, smem));
  if (it == known.end()) {
    ladder_attr(smem);
    int nb = 0;
    TAMC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_pt_ladder, (int)T, smem));
    g_ladder_queries.fetch_add(1, std::memory_order_relaxed);
    it = known.emplace(std::make_tuple(g->device, T, smem), nb).first;
  }
  return (uint32_t)it->second * (uint32_t)g->num_sms;
}

void ladder_launch(cudaStream_t st, const LadJob* d_jobs, const uint32_t* d_cta_job, uint32_t njobs, uint32_t grid,
                   uint32_t T, size_t smem, uint32_t open_grid) {
  ladder_attr(smem);
  k_ladder_open<<<dim3(open_grid, njobs), 256, 0, st>>>(d_jobs);
  TAMC_CUDA(cudaGetLastError());
  // cooperative: every CTA of the launch is resident, as the barrier needs
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(T);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  TAMC_CUDA(cudaLaunchKernelEx(&cfg, k_pt_ladder, d_jobs, d_cta_job));
  k_ladder_commit<<<dim3(open_grid, njobs), 256, 0, st>>>(d_jobs);
  TAMC_CUDA(cudaGetLastError());
}

}  // namespace tamc
