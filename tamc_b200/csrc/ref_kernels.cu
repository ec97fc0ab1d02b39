// ref_kernels.cu -- reference-order replay kernels (TAMC_MODE_REF).
//
// These kernels reproduce the reference's Markov chain bit for bit: every
// replica is swept in site order 0..n-1 with the replica's Xoshiro256++
// stream, ΔE is summed in CSR row order in f32, acceptance uses the
// glibc-identical expf, the ICM seed is drawn with rand's gen_range and the
// cluster is the connected q<0 component of the petgraph node range.
//
// What is sequential in the reference is its random stream: which draw a site
// uses depends on how many sites before it needed one.  Three things take the
// rest of the work off that chain:
//  * the stream itself does not depend on the replicas, so a warp generates it
//    ahead into a small ring while another consumes it;
//  * a warp decides 32 consecutive sites at once (a lane each): given which
//    sites of the block flip, every lane's ΔE, the draws before it (a popcount)
//    and its decision follow, so the decisions are iterated to a fixed point.
//    A lane depends only on the lanes before it: there is one fixed point, the
//    sequential one, reached in a few steps;
//  * the exact expf is only asked when the draw lies within 3e-5 of the fast
//    one, far outside its error (about one draw in 10^5).
// The replicas of one stream still follow one another; independent streams and
// the Houdayer moves of different slots run side by side.  What bounds a sweep
// is the latency of a block's few decision steps and, in cold replicas, the
// generator (about 18 cycles an output).  Measured, whole rounds: 64 replicas
// of 256 sites (2-D +-J, 32 temperatures) 1.0 ms -> 55 us, the serial loop over
// 24 replicas of 100 sites (random 3-regular) 2.15 ms -> 103 us, against one
// thread per stream with every load from HBM or L2 and the exact expf per site.
#include "ref_kernels.cuh"

#include <algorithm>
#include <cstdlib>

namespace tamc {
namespace refk {

// ΔE of flipping site i (src/ising.rs:468-480), f32 in row order.
__device__ __forceinline__ float delta_e(const RefInst& I, const int8_t* s, uint32_t i) {
  float d = 0.0f;
  d = __fadd_rn(d, I.bias[i]);
  const uint32_t e1 = I.rp[i + 1];
  for (uint32_t e = I.rp[i]; e < e1; ++e) d = __fadd_rn(d, __fmul_rn(I.J[e], (float)s[I.col[e]]));
  const float si = (float)s[i];
  return __fmul_rn(d, __fmul_rn(-2.0f, si));
}

// MetropolisSampler::advance_impl (tamc-core/src/metropolis.rs:43-57).
__device__ __forceinline__ bool advance(const RefInst& I, const ExpTable& X, float beta, int8_t* s, uint32_t i,
                                        Xo& rng, float& de) {
  const float d = delta_e(I, s, i);
  if (d < 0.0f) {
    s[i] = (int8_t)-s[i];
    de = d;
    return true;
  }
  const float p = tamc_expf_exact(__fmul_rn(-beta, d), X.off, X.keys, X.vals);
  const float x = rng.std_f32();
  if (x < p) {
    s[i] = (int8_t)-s[i];
    de = d;
    return true;
  }
  return false;
}

// IsingSampler::sweep (src/ising.rs:225-233): returns Σ accepted ΔE in f32 site order.
__device__ float sweep_tracked(const RefInst& I, const ExpTable& X, float beta, int8_t* s, Xo& rng) {
  float de = 0.0f;
  for (uint32_t i = 0; i < I.n; ++i) {
    float d = 0.0f;
    de = __fadd_rn(de, advance(I, X, beta, s, i, rng, d) ? d : 0.0f);
  }
  return de;
}

// Row term h_i * s_i of energy_ref (src/ising.rs:438-454).
__device__ __forceinline__ float energy_row(const RefInst& I, const int8_t* s, uint32_t i) {
  float h = __fadd_rn(0.0f, I.bias[i]);
  const uint32_t e1 = I.rp[i + 1];
  for (uint32_t e = I.rp[i]; e < e1; ++e) h = __fadd_rn(h, __fmul_rn(I.J[e], (float)s[I.col[e]]) / 2.0f);
  return __fmul_rn(h, (float)s[i]);
}
// All row terms, one row per thread; the caller sums them in order.
__device__ void energy_rows(const RefInst& I, const int8_t* s, float* rows) {
  for (uint32_t i = threadIdx.x; i < I.n; i += blockDim.x) rows[i] = energy_row(I, s, i);
}

__device__ __forceinline__ uint32_t block_sum_u32(uint32_t v, uint32_t* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[w] = v;
  __syncthreads();
  uint32_t t = 0;
  for (int k = 0; k < nw; ++k) t += sh[k];
  __syncthreads();
  return t;
}

// ------------------------------------------------------------ init ----
// energy_ref of every replica (rand_ising_state caches it, src/ising.rs:175), a
// CTA each: row terms in parallel, their sum in row order by one thread (64
// replicas of 256 sites: all of it by one thread took 125 us).
__global__ void __launch_bounds__(128) k_energy_all(RefInst I, const int8_t* spins, float* energy) {
  __shared__ float rows[1024];
  const int8_t* s = spins + (size_t)blockIdx.x * I.n;
  float total = I.offset;
  for (uint32_t i0 = 0; i0 < I.n; i0 += 1024) {
    const uint32_t m = min(1024u, I.n - i0);
    for (uint32_t x = threadIdx.x; x < m; x += blockDim.x) rows[x] = energy_row(I, s, i0 + x);
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t x = 0;
      for (; x + 8 <= m; x += 8) {
        float w[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) w[k] = rows[x + k];
#pragma unroll
        for (int k = 0; k < 8; ++k) total = __fadd_rn(total, w[k]);
      }
      for (; x < m; ++x) total = __fadd_rn(total, rows[x]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) energy[blockIdx.x] = total;
}

// ------------------------------------------------------------- ICM ----
// apply_icm (src/pt.rs:521-540) + houdayer_cluster_move (src/pt.rs:31-77), one
// CTA, pairs in the reference's order.  scratch: visited[max(n,1)] u32,
// queue[n] u32, rows[n] f32.
__global__ void __launch_bounds__(512) k_icm(RefInst I, RefPt P, ExpTable X, Xo* rng, int* err) {
  __shared__ uint32_t sh[32];
  __shared__ uint32_t s_k, s_tail, s_found;
  const uint32_t n = I.n;
  for (uint32_t c = 0; c + 1 < P.C; c += 2) {
    for (uint32_t t = P.lo; t < P.nt; ++t) {
      const uint32_t r1 = P.perm[c * P.nt + t], r2 = P.perm[(c + 1) * P.nt + t];
      int8_t* s1 = P.spins + (size_t)r1 * n;
      int8_t* s2 = P.spins + (size_t)r2 * n;
      uint32_t cnt = 0;
      for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) cnt += (s1[i] != s2[i]);
      cnt = block_sum_u32(cnt, sh);
      if (cnt == 0) continue;  // `idxs.choose` returns None: no draw, no invalidation
      if (threadIdx.x == 0) {
        Xo x = *rng;
        s_k = x.gen_range(cnt);
        *rng = x;
        s_found = 0xffffffffu;
      }
      __syncthreads();
      // the k-th site with q<0 (idxs is in increasing site order)
      uint32_t base = 0;
      for (uint32_t i0 = 0; i0 < n; i0 += blockDim.x) {
        const uint32_t i = i0 + threadIdx.x;
        const bool f = i < n && s1[i] != s2[i];
        const uint32_t bal = __ballot_sync(0xffffffffu, f);
        const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
        if (lane == 0) sh[w] = __popc(bal);
        __syncthreads();
        uint32_t before = base;
        for (int k = 0; k < w; ++k) before += sh[k];
        before += __popc(bal & ((1u << lane) - 1u));
        if (f && before == s_k) s_found = i;
        uint32_t tot = 0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) tot += sh[k];
        base += tot;
        __syncthreads();
        if (s_found != 0xffffffffu) break;
      }
      const uint32_t seed = s_found;
      if (seed >= I.g_nodes) {  // petgraph's FixedBitSet would panic here
        if (threadIdx.x == 0) *err = TAMC_E_REFPANIC;
        return;
      }
      // BFS over the q<0 subgraph (order-free: only the discovered set matters)
      for (uint32_t i = threadIdx.x; i < I.g_nodes; i += blockDim.x) P.visited[i] = 0;
      __syncthreads();
      if (threadIdx.x == 0) {
        P.visited[seed] = 1;
        P.queue[0] = seed;
        s_tail = 1;
      }
      __syncthreads();
      uint32_t lvl_begin = 0;
      for (;;) {
        const uint32_t lvl_end = s_tail;
        __syncthreads();  // everyone has read the level bound before anyone appends
        if (lvl_begin == lvl_end) break;
        for (uint32_t q = lvl_begin + threadIdx.x; q < lvl_end; q += blockDim.x) {
          const uint32_t u = P.queue[q];
          const uint32_t e1 = I.grp[u + 1];
          for (uint32_t e = I.grp[u]; e < e1; ++e) {
            const uint32_t v = I.gcol[e];
            if (s1[v] != s2[v] && atomicExch(&P.visited[v], 1u) == 0u) P.queue[atomicAdd(&s_tail, 1u)] = v;
          }
        }
        __syncthreads();
        lvl_begin = lvl_end;
      }
      const uint32_t csz = s_tail;
      for (uint32_t q = threadIdx.x; q < csz; q += blockDim.x) {
        const uint32_t v = P.queue[q];
        const int8_t a = s1[v];
        s1[v] = s2[v];
        s2[v] = a;
      }
      __syncthreads();
      // invalidated energies are recomputed by energy_ref exactly as the next
      // Macrostate::energy call would (tamc-core/src/pt.rs:126-129)
      for (int rep = 0; rep < 2; ++rep) {
        const int8_t* s = rep ? s2 : s1;
        energy_rows(I, s, P.rows);
        __syncthreads();
        if (threadIdx.x == 0) {
          float total = I.offset;
          for (uint32_t i = 0; i < n; ++i) total = __fadd_rn(total, P.rows[i]);
          P.energy[rep ? r2 : r1] = total;
        }
        __syncthreads();
      }
    }
  }
}

// ------------------------------------------- block-wise site sweep ----
constexpr uint32_t REF_RING = 256;   // outputs the ring holds
constexpr uint32_t REF_SEG = 64;     // most draws between two meetings of its two warps
constexpr uint32_t REF_CK = 16;      // outputs between kept generator states, and the unit of filling

// A stream generated ahead of its use.  Output k (counted from the kernel's
// start) is u[k % REF_RING]; the generator's state before every REF_CK-th output
// is kept, from which the state after the last output used is rebuilt.
struct RefRing {
  ulonglong2 raw[REF_RING];  // (s0, s3) of the outputs being converted
  float u[REF_RING];         // std_f32
  Xo ck[REF_RING / REF_CK + 2];
  uint32_t used;             // outputs used up to the last meeting
};

// Outputs [from, to) (multiples of REF_CK) into the ring, by one warp: lane 0
// steps the generator and leaves what each output is made of, all lanes turn
// that into floats.
__device__ void ring_fill(RefRing& R, Xo& x, uint32_t from, uint32_t to) {
  const uint32_t lane = threadIdx.x & 31u;
  if (lane == 0)
    for (uint32_t k = from; k < to; k += REF_CK) {
      R.ck[(k / REF_CK) % (REF_RING / REF_CK + 2)] = x;
      ulonglong2* const raw = R.raw + k % REF_RING;
#pragma unroll
      for (uint32_t j = 0; j < REF_CK; ++j) {
        raw[j] = make_ulonglong2(x.s0, x.s3);
        const uint64_t t = x.s1 << 17;
        const uint64_t a = x.s2 ^ x.s0, b = x.s3 ^ x.s1;
        x.s1 ^= a;
        x.s0 ^= b;
        x.s2 = a ^ t;
        x.s3 = (b << 45) | (b >> 19);
      }
    }
  __syncwarp();
  for (uint32_t k = from + lane; k < to; k += 32) {
    const ulonglong2 v = R.raw[k % REF_RING];
    const uint64_t sum = v.x + v.y, r = ((sum << 23) | (sum >> 41)) + v.x;
    R.u[k % REF_RING] = (float)(uint32_t)(r >> 40) * (1.0f / 16777216.0f);
  }
  __syncwarp();
}
// The generator's state after `used` outputs (fewer than were generated).
__device__ Xo ring_state(const RefRing& R, uint32_t used) {
  Xo x = R.ck[(used / REF_CK) % (REF_RING / REF_CK + 2)];
  for (uint32_t k = 0; k < used % REF_CK; ++k) x.next();
  return x;
}
__device__ __forceinline__ void ref_bar(uint32_t threads) {
  asm volatile("bar.sync 1, %0;\n" ::"r"(threads) : "memory");
}
// The warp that generates: `made` outputs are in the ring, at least REF_SEG more
// than are used; `segs` meetings follow, between two of which at most REF_SEG
// are used and at least as many generated (until the ring is full).
__device__ void ring_produce(RefRing& R, Xo& x, uint32_t& made, uint32_t segs, uint32_t threads) {
  for (uint32_t k = 0; k < segs; ++k) {
    ref_bar(threads);
    const uint32_t room = (*(volatile uint32_t*)&R.used + REF_RING) / REF_CK * REF_CK;
    const uint32_t to = min(room, made + REF_SEG + REF_CK);
    ring_fill(R, x, made, to);
    made = to;
  }
}

// x < expf(a) with glibc's expf, for the lanes of `mask` that want it.
__device__ __forceinline__ bool below_exp(uint32_t mask, bool want, float x, float a, const ExpTable& X) {
  const float p = __expf(a);  // relative error at most 3.6e-6 on [-110, 0] (every float there looked at)
  bool r = x < p * (1.0f - 3e-5f);
  const bool close = want && !r && !(x > p * (1.0f + 3e-5f) + 1e-37f);
  if (__any_sync(mask, close))  // (rare)
    if (close) r = x < tamc_expf_exact(a, X.off, X.keys, X.vals);
  return want && r;
}

// The instance as a CTA reads it: entries (column, J bits) in shared memory
// (CS), or the CSR in HBM.
template <bool CS>
struct RefRows {
  uint32_t n;
  const uint32_t* rp;
  const uint2* ent;
  const uint32_t* col;
  const float* J;
  const float* bias;
  __device__ __forceinline__ void at(uint32_t e, uint32_t& c, uint32_t& j) const {
    if (CS) {
      const uint2 v = ent[e];
      c = v.x;
      j = v.y;
    } else {
      c = __ldg(col + e);
      j = __float_as_uint(__ldg(J + e));
    }
  }
};
__host__ __device__ inline size_t ref_rows_bytes(uint32_t n, uint64_t nnz) {
  return ((size_t)(2 * n + 1) * 4 + 15) / 16 * 16 + nnz * 8;
}
template <bool CS>
__device__ RefRows<CS> ref_rows(const RefInst& I, unsigned char* sm) {
  RefRows<CS> R{I.n, I.rp, nullptr, I.col, I.J, I.bias};
  if (CS) {
    uint32_t* rp = (uint32_t*)sm;
    float* bias = (float*)(rp + I.n + 1);
    uint2* ent = (uint2*)(sm + ((size_t)(2 * I.n + 1) * 4 + 15) / 16 * 16);
    for (uint32_t x = threadIdx.x; x <= I.n; x += blockDim.x) rp[x] = I.rp[x];
    for (uint32_t x = threadIdx.x; x < I.n; x += blockDim.x) bias[x] = I.bias[x];
    const uint32_t nnz = I.rp[I.n];
    for (uint32_t x = threadIdx.x; x < nnz; x += blockDim.x) ent[x] = make_uint2(I.col[x], __float_as_uint(I.J[x]));
    R.rp = rp;
    R.bias = bias;
    R.ent = ent;
  }
  return R;
}

// The decisions of a block of 32 sites from site i0 on: field(w) gives this
// lane's h_i + sum_j J_ij s_j in row order (src/ising.rs:471-475; J * +-1 is
// exact) when the block's spins are w.  Returns the accepted lanes; d, need:
// this lane's ΔE, and the lanes that used a draw.
template <class Field>
__device__ __forceinline__ uint32_t ref_block(Field field, uint32_t w0, bool act, float beta, const ExpTable& X,
                                              const RefRing& ring, uint32_t base, float& d, uint32_t& need) {
  const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
  const float side = (w0 >> lane) & 1u ? 2.0f : -2.0f;
  uint32_t a = 0;
  for (int k = 0; k < 34; ++k) {  // (lane l is final after l + 1 steps)
    d = __fmul_rn(field(w0 ^ (a & lt)), side);
    const bool want = act && !(d < 0.0f);
    need = __ballot_sync(0xffffffffu, want);
    const float x = ring.u[(base + __popc(need & lt)) % REF_RING];
    const bool acc = below_exp(0xffffffffu, want, x, __fmul_rn(-beta, d), X) || (act && d < 0.0f);
    const uint32_t b = __ballot_sync(0xffffffffu, acc);
    if (b == a) break;
    a = b;
  }
  return a;
}
// The same with rows of at most K entries, kept in registers: entries outside
// the block with their spins (they do not change meanwhile), short rows padded
// with -0 (x + -0 = x).
template <bool CS, int K>
__device__ __forceinline__ uint32_t ref_block_regs(const RefRows<CS>& R, const uint32_t* S, uint32_t i, uint32_t e0,
                                                   uint32_t len, float bias, uint32_t w0, bool act, float beta,
                                                   const ExpTable& X, const RefRing& ring, uint32_t base, float& d,
                                                   uint32_t& need) {
  uint32_t j[K], sh[K], in[K];
#pragma unroll
  for (int m = 0; m < K; ++m) {
    uint32_t c = 0;
    j[m] = 0x80000000u;
    if ((uint32_t)m < len) R.at(e0 + m, c, j[m]);
    const bool here = (uint32_t)m < len && (c >> 5) == (i >> 5);
    sh[m] = ~c & 31u;
    in[m] = here ? 0x80000000u : 0u;
    if (!here && (uint32_t)m < len) j[m] ^= (S[c >> 5] << sh[m]) & 0x80000000u;
  }
  auto field = [&](uint32_t w) {
    float f = bias;
#pragma unroll
    for (int m = 0; m < K; ++m) f = __fadd_rn(f, __uint_as_float(j[m] ^ ((w << sh[m]) & in[m])));
    return f;
  };
  return ref_block(field, w0, act, beta, X, ring, base, d, need);
}

// One sweep (IsingSampler::sweep, src/ising.rs:225-233) of a replica by the
// consuming warp: spins S as bits (1 = -1), outputs from `base` on.  The accepted
// ΔE of segment g go to dl[g & 1][0 .. cnt[g & 1]) in site order.
template <bool CS>
__device__ void ref_sweep_warp(const RefRows<CS>& R, const ExpTable& X, float beta, uint32_t* S, RefRing& ring,
                               uint32_t& base, float (*dl)[REF_SEG], volatile uint32_t* cnt, uint32_t threads) {
  const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u, n = R.n;
  for (uint32_t g = 0; g * REF_SEG < n; ++g) {
    if (lane == 0) ring.used = base;
    __syncwarp();
    ref_bar(threads);
    uint32_t nd = 0;
    for (uint32_t i0 = g * REF_SEG; i0 < min(n, (g + 1) * REF_SEG); i0 += 32) {
      const uint32_t i = min(i0 + lane, n - 1);
      const bool act = i0 + lane < n;
      const uint32_t w0 = S[i0 >> 5], e0 = R.rp[i], len = R.rp[i + 1] - e0;
      const float bias = __fadd_rn(0.0f, R.bias[i]);
      const uint32_t most = __reduce_max_sync(0xffffffffu, len);
      float d = 0.0f;
      uint32_t need = 0, a;
      if (most <= 4) a = ref_block_regs<CS, 4>(R, S, i, e0, len, bias, w0, act, beta, X, ring, base, d, need);
      else if (most <= 8) a = ref_block_regs<CS, 8>(R, S, i, e0, len, bias, w0, act, beta, X, ring, base, d, need);
      else {
        auto field = [&](uint32_t w) {
          float f = bias;
          for (uint32_t e = e0; e < e0 + len; ++e) {
            uint32_t c, j;
            R.at(e, c, j);
            const uint32_t v = (c >> 5) == (i >> 5) ? w : S[c >> 5];
            f = __fadd_rn(f, __uint_as_float(j ^ ((v << (~c & 31u)) & 0x80000000u)));
          }
          return f;
        };
        a = ref_block(field, w0, act, beta, X, ring, base, d, need);
      }
      if ((a >> lane) & 1u) dl[g & 1][nd + __popc(a & lt)] = d;
      nd += __popc(a);
      base += __popc(need);
      if (lane == 0) S[i0 >> 5] = w0 ^ a;
      __syncwarp();
    }
    if (lane == 0) cnt[g & 1] = nd;
  }
  if (lane == 0) ring.used = base;
  __syncwarp();
  ref_bar(threads);  // the last segment's ΔE are there
}
// The accumulating warp's side: Σ accepted ΔE in f32, in site order (lane 0).
__device__ float ref_sweep_sum(uint32_t n, const float (*dl)[REF_SEG], volatile uint32_t* cnt, uint32_t threads) {
  float de = 0.0f;
  const uint32_t segs = (n + REF_SEG - 1) / REF_SEG;
  for (uint32_t g = 0; g <= segs; ++g) {
    ref_bar(threads);
    if (g > 0 && (threadIdx.x & 31u) == 0) {
      const uint32_t m = cnt[(g - 1) & 1];
      const float* v = dl[(g - 1) & 1];
      uint32_t k = 0;
      for (; k + 4 <= m; k += 4) {
        const float v0 = v[k], v1 = v[k + 1], v2 = v[k + 2], v3 = v[k + 3];
        de = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(de, v0), v1), v2), v3);
      }
      for (; k < m; ++k) de = __fadd_rn(de, v[k]);
    }
    __syncwarp();
  }
  return de;
}

// Spins of a replica as bits (1 = -1) and back, by the warps [w0, w0 + nw) of the CTA.
__device__ void ref_pack(const int8_t* s, uint32_t* S, uint32_t n, uint32_t w0, uint32_t nw) {
  const uint32_t lane = threadIdx.x & 31u;
  for (uint32_t w = (threadIdx.x >> 5) - w0; w < (n + 31) / 32; w += nw) {
    const uint32_t i = 32 * w + lane;
    const uint32_t b = __ballot_sync(0xffffffffu, i < n && s[i < n ? i : 0u] < 0);
    if (lane == 0) S[w] = b;
  }
}
__device__ void ref_unpack(int8_t* s, const uint32_t* S, uint32_t n, uint32_t w0, uint32_t nw) {
  const uint32_t lane = threadIdx.x & 31u;
  for (uint32_t w = (threadIdx.x >> 5) - w0; w < (n + 31) / 32; w += nw) {
    const uint32_t i = 32 * w + lane;
    if (i < n) s[i] = (S[w] >> lane) & 1u ? -1 : 1;
  }
}

extern __shared__ __align__(16) unsigned char ref_smem[];

// ThreadedPTSampler sweeps (parallel/pt.rs:63-68): a CTA per slot (c, t) with
// rng_vec[c][t].  Warp 0 sweeps, warp 1 generates the stream, warp 2 sums ΔE.
template <bool CS>
__global__ void __launch_bounds__(96) k_sweep_threaded_b(RefInst I, RefPt P, ExpTable X, Xo* rngs) {
  __shared__ RefRing ring;
  __shared__ float dl[2][REF_SEG];
  __shared__ uint32_t cnt[2];
  const uint32_t k = blockIdx.x, t = k % P.nt, r = P.perm[k], warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  uint32_t* S = (uint32_t*)ref_smem;
  const uint32_t nwb = (I.n + 31) / 32;
  const RefRows<CS> R = ref_rows<CS>(I, ref_smem + (nwb * 4 + 15) / 16 * 16);
  int8_t* s = P.spins + (size_t)r * I.n;
  Xo x = rngs[k];
  uint32_t made = 0;
  if (warp == 1) {
    made = REF_SEG;
    ring_fill(ring, x, 0, made);
  } else {
    const uint32_t w0 = warp == 0 ? 0u : 1u;  // warps 0 and 2 load the spins
    for (uint32_t w = w0; w < nwb; w += 2) {
      const uint32_t i = 32 * w + lane;
      const uint32_t b = __ballot_sync(0xffffffffu, i < I.n && s[i < I.n ? i : 0u] < 0);
      if (lane == 0) S[w] = b;
    }
  }
  __syncthreads();
  const uint32_t segs = (I.n + REF_SEG - 1) / REF_SEG;
  if (warp == 0) {
    uint32_t base = 0;
    ref_sweep_warp<CS>(R, X, P.betas[t], S, ring, base, dl, cnt, 96);
  } else if (warp == 1) {
    ring_produce(ring, x, made, segs, 96);
    ref_bar(96);
    if (lane == 0) rngs[k] = ring_state(ring, ring.used);
  } else {
    const float de = ref_sweep_sum(I.n, dl, cnt, 96);
    if (lane == 0) P.energy[r] = __fadd_rn(P.energy[r], de);
  }
  __syncthreads();
  ref_unpack(s, S, I.n, 0, 3);
}

__device__ void update_round_trips(uint8_t* tg, uint32_t nt, uint32_t* rtrips, uint32_t* dhist) {
  // tamc-core/src/pt.rs:54-84, by one warp
  const uint32_t lane = threadIdx.x & 31u;
  if (lane == 0) {
    uint8_t& lo = tg[0];
    if (lo == 0) lo = 1;
    else if (lo == 4) { *rtrips += 1; lo = 1; }
    else if (lo == 2) lo = 3;
    uint8_t& hi = tg[nt - 1];
    if (hi == 0) hi = 2;
    else if (hi == 3) { *rtrips += 1; hi = 2; }
    else if (hi == 1) hi = 4;
  }
  __syncwarp();
  for (uint32_t k = lane; k < nt; k += 32) {
    const uint8_t v = tg[k];
    if (v == 1 || v == 3) dhist[2 * k] += 1;
    else if (v == 2 || v == 4) dhist[2 * k + 1] += 1;
  }
}

// A chain's exchange state in shared memory.
struct RefChain {
  float* des;      // [nt] energy differences
  float* db;       // [nt] beta differences
  uint32_t* pm;    // [nt]
  uint32_t* acc;   // [nt]
  uint8_t* tags;   // [nt]
};
__host__ __device__ inline size_t ref_chain_bytes(uint32_t nt) { return ((size_t)nt * 17 + 15) / 16 * 16; }
__device__ RefChain ref_chain(unsigned char* sm, uint32_t nt) {
  RefChain c;
  c.des = (float*)sm;
  c.db = c.des + nt;
  c.pm = (uint32_t*)(c.db + nt);
  c.acc = c.pm + nt;
  c.tags = (uint8_t*)(c.acc + nt);
  return c;
}
__device__ void ref_chain_load(const RefPt& P, uint32_t c, RefChain& Q, uint32_t tid, uint32_t T) {
  for (uint32_t k = tid; k < P.nt; k += T) {
    const size_t o = (size_t)c * P.nt + k;
    const uint32_t r = P.perm[o];
    Q.pm[k] = r;
    Q.tags[k] = P.tags[o];
    Q.acc[k] = P.acc[o];
    if (k + 1 < P.nt) {
      Q.db[k] = P.dbeta[k];
      Q.des[k] = __fsub_rn(P.energy[P.perm[o + 1]], P.energy[r]);
    }
  }
}
__device__ void ref_chain_store(const RefPt& P, uint32_t c, const RefChain& Q, uint32_t tid, uint32_t T) {
  for (uint32_t k = tid; k < P.nt; k += T) {
    const size_t o = (size_t)c * P.nt + k;
    P.perm[o] = Q.pm[k];
    P.tags[o] = Q.tags[k];
    P.acc[o] = Q.acc[k];
  }
}
__device__ __forceinline__ void ref_chain_swap(RefChain& Q, uint32_t j) {  // PTState::swap_states
  const uint32_t a = Q.pm[j];
  Q.pm[j] = Q.pm[j + 1];
  Q.pm[j + 1] = a;
  const uint8_t b = Q.tags[j];
  Q.tags[j] = Q.tags[j + 1];
  Q.tags[j + 1] = b;
  Q.acc[j] += 1;
}

// ThreadedPTSampler exchange (tamc-core/src/parallel/pt.rs:41-59), one warp per
// chain, uniforms from rng_vec[c][0].  The energy differences are those before
// any swap of the pass, so 32 pairs are decided at once (a lane each; the draws
// before a pair counted as in the sweep); the swaps follow in order.
__global__ void __launch_bounds__(32) k_exchange_threaded_b(RefPt P, ExpTable X, Xo* rngs) {
  __shared__ RefRing ring;
  const uint32_t c = blockIdx.x, lane = threadIdx.x, lt = (1u << lane) - 1u;
  RefChain Q = ref_chain(ref_smem, P.nt);
  ref_chain_load(P, c, Q, lane, 32);
  Xo x = rngs[(size_t)c * P.nt];
  uint32_t base = 0, made = 0;
  __syncwarp();
  for (uint32_t j0 = 0; j0 + 1 < P.nt; j0 += 32) {
    const uint32_t to = (base + 48) / REF_CK * REF_CK;  // above base + 32
    ring_fill(ring, x, made, to);
    made = to;
    const uint32_t j = j0 + lane;
    const bool act = j + 1 < P.nt;
    const float dlt = act ? __fmul_rn(Q.db[j], Q.des[j]) : 0.0f;
    const bool need = act && !(dlt >= 0.0f);
    const uint32_t nm = __ballot_sync(0xffffffffu, need);
    const bool sw = below_exp(0xffffffffu, need, ring.u[(base + __popc(nm & lt)) % REF_RING], dlt, X) || (act && !need);
    uint32_t m = __ballot_sync(0xffffffffu, sw);
    base += __popc(nm);
    if (lane == 0)
      for (; m; m &= m - 1) ref_chain_swap(Q, j0 + __ffs(m) - 1);
    __syncwarp();
  }
  update_round_trips(Q.tags, P.nt, P.rtrips + c, P.dhist + (size_t)c * P.nt * 2);
  __syncwarp();
  ref_chain_store(P, c, Q, lane, 32);
  if (lane == 0 && made) rngs[(size_t)c * P.nt] = ring_state(ring, base);
}

// Serial mode (src/pt.rs:493-497, EnsembleSampler over ParallelTemperingSampler):
// one stream; per chain the exchange with ΔE propagation, then sweeps
// t = 0..nt-1.  Warp 0 sweeps, warp 1 generates the stream, warp 2 sums ΔE, warp
// 3 stores the replica swept last and loads the one swept next.
template <bool CS>
__global__ void __launch_bounds__(128) k_serial_round_b(RefInst I, RefPt P, ExpTable X, Xo* rng) {
  __shared__ RefRing ring;
  __shared__ float dl[2][REF_SEG];
  __shared__ uint32_t cnt[2];
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, nt = P.nt;
  const uint32_t nwb = (I.n + 31) / 32, n = I.n;
  const size_t bb = (size_t)nwb * 4;
  uint32_t* const S = (uint32_t*)ref_smem;  // three replicas' bits
  RefChain Q = ref_chain(ref_smem + (3 * bb + 15) / 16 * 16, nt);
  const RefRows<CS> R = ref_rows<CS>(I, ref_smem + (3 * bb + 15) / 16 * 16 + ref_chain_bytes(nt));
  Xo x = *rng;
  uint32_t made = 0, base = 0;
  if (warp == 1) {
    made = REF_SEG;
    ring_fill(ring, x, 0, made);
  }
  if (tid == 0) ring.used = 0;
  const uint32_t segs = (n + REF_SEG - 1) / REF_SEG;
  for (uint32_t c = 0; c < P.C; ++c) {
    __syncthreads();  // the last chain's energies are there
    ref_chain_load(P, c, Q, tid, 128);
    __syncthreads();
    // exchange (tamc-core/src/pt.rs:120-150), REF_SEG pairs per meeting
    for (uint32_t j0 = 0; j0 + 1 < nt; j0 += REF_SEG) {
      if (warp == 1) {
        ring_produce(ring, x, made, 1, 96);
      } else if (warp == 2) {
        ref_bar(96);
      } else if (warp == 0) {
        if (lane == 0) ring.used = base;
        __syncwarp();
        ref_bar(96);
        for (uint32_t j = j0; j < min(j0 + REF_SEG, nt - 1); ++j) {  // every lane walks alike
          const float des = Q.des[j], dlt = __fmul_rn(Q.db[j], des);
          const bool need = !(dlt >= 0.0f);
          const bool sw = below_exp(0xffffffffu, need, ring.u[base % REF_RING], dlt, X) || !need;
          base += need;
          if (sw && lane == 0) {
            ref_chain_swap(Q, j);
            if (j + 2 < nt) Q.des[j + 1] = __fadd_rn(Q.des[j + 1], des);
          }
          __syncwarp();
        }
      }
    }
    __syncthreads();
    if (warp == 2) update_round_trips(Q.tags, nt, P.rtrips + c, P.dhist + (size_t)c * nt * 2);
    ref_pack(P.spins + (size_t)Q.pm[0] * n, S, n, 0, 4);
    __syncthreads();
    ref_chain_store(P, c, Q, tid, 128);
    for (uint32_t t = 0; t < nt; ++t) {
      const uint32_t r = Q.pm[t];
      uint32_t* const cur = S + (size_t)(t % 3) * nwb;
      if (warp == 0) {
        ref_sweep_warp<CS>(R, X, P.betas[t], cur, ring, base, dl, cnt, 96);
      } else if (warp == 1) {
        ring_produce(ring, x, made, segs, 96);
        ref_bar(96);
      } else if (warp == 2) {
        const float de = ref_sweep_sum(n, dl, cnt, 96);
        if (lane == 0) P.energy[r] = __fadd_rn(P.energy[r], de);
      } else {
        if (t > 0) ref_unpack(P.spins + (size_t)Q.pm[t - 1] * n, S + (size_t)((t - 1) % 3) * nwb, n, 3, 1);
        if (t + 1 < nt) ref_pack(P.spins + (size_t)Q.pm[t + 1] * n, S + (size_t)((t + 1) % 3) * nwb, n, 3, 1);
      }
      __syncthreads();
    }
    ref_unpack(P.spins + (size_t)Q.pm[nt - 1] * n, S + (size_t)((nt - 1) % 3) * nwb, n, 0, 4);
  }
  if (warp == 1) {
    __syncwarp();
    if (lane == 0) *rng = ring_state(ring, ring.used);
  }
}

// ------------------------------------------------- ICM, slot by slot ----
// The move of one slot touches only its two replicas; what orders the slots is
// the stream the seed indices are drawn from.  So one CTA counts every slot's
// q<0 sites (a warp each) and draws the indices in the reference's order, and
// the moves then run side by side, a CTA per slot.
// pick[slot] = k + 1 for slots with q<0 sites (0: no move); slots pair-major.
__global__ void __launch_bounds__(1024) k_icm_seeds(RefInst I, RefPt P, Xo* rng, uint32_t* pick) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nact = P.nt - P.lo;
  const uint32_t slots = P.C / 2 * nact;
  for (uint32_t x = warp; x < slots; x += blockDim.x >> 5) {
    const uint32_t c = 2 * (x / nact), t = P.lo + x % nact;
    const int8_t* s1 = P.spins + (size_t)P.perm[(size_t)c * P.nt + t] * I.n;
    const int8_t* s2 = P.spins + (size_t)P.perm[(size_t)(c + 1) * P.nt + t] * I.n;
    uint32_t cnt = 0;
    for (uint32_t i = lane; i < I.n; i += 32) cnt += s1[i] != s2[i];
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (lane == 0) pick[x] = cnt;
  }
  __syncthreads();
  if (warp == 0) {  // 32 counts at a time, drawn for in order
    Xo x = *rng;
    for (uint32_t x0 = 0; x0 < slots; x0 += 32) {
      const uint32_t mine = x0 + lane < slots ? pick[x0 + lane] : 0u;
      uint32_t k = 0;
      for (uint32_t j = 0; j < min(32u, slots - x0); ++j) {
        const uint32_t cnt = __shfl_sync(0xffffffffu, mine, j);
        if (!cnt) continue;  // `idxs.choose` returns None: no draw, no invalidation
        const uint32_t v = x.gen_range(cnt) + 1;  // every lane steps alike
        if (lane == j) k = v;
      }
      if (x0 + lane < slots) pick[x0 + lane] = k;
    }
    if (lane == 0) *rng = x;
  }
}

// apply_icm (src/pt.rs:521-540) + houdayer_cluster_move (src/pt.rs:31-77) of one
// slot.  Shared memory: where the replicas differ, replica 1's spins and the
// cluster as bitmaps, the search's queue [n], and the row terms of both energies
// [2][n] in the same place afterwards; then the rows (CS).  The search runs over
// the rows' off-diagonal entries, the ICM graph's edges (sites past its node
// range have none).
__host__ __device__ inline size_t ref_icm_bytes(uint32_t n) {
  return 3 * (((size_t)n + 31) / 32 * 4 + 16) / 16 * 16 + ((size_t)n * 8 + 15) / 16 * 16;
}
template <bool CS>
__global__ void __launch_bounds__(256) k_icm_move(RefInst I, RefPt P, const uint32_t* pick, int* err) {
  __shared__ uint32_t s_seed, s_n[3], s_pre[9];
  const uint32_t tid = threadIdx.x, T = blockDim.x, lane = tid & 31u, warp = tid >> 5, nwarp = T >> 5;
  const uint32_t x = blockIdx.x, nact = P.nt - P.lo, c = 2 * (x / nact), t = P.lo + x % nact;
  if (!pick[x]) return;
  const uint32_t n = I.n, nwb = (n + 31) / 32, nwp = (nwb + 3) / 4 * 4;
  const RefRows<CS> R = ref_rows<CS>(I, ref_smem + ref_icm_bytes(n));
  const uint32_t r1 = P.perm[(size_t)c * P.nt + t], r2 = P.perm[(size_t)(c + 1) * P.nt + t];
  int8_t* s1 = P.spins + (size_t)r1 * n;
  int8_t* s2 = P.spins + (size_t)r2 * n;
  uint32_t* D = (uint32_t*)ref_smem;
  uint32_t* V = D + nwp;
  uint32_t* A = V + nwp;
  uint32_t* queue = A + nwp;
  // bitmap of the differing sites; each warp a contiguous range of words, so
  // that their counts order the sites
  const uint32_t per = (nwb + nwarp - 1) / nwarp, w0 = min(nwb, warp * per), w1 = min(nwb, w0 + per);
  uint32_t cnt = 0;
  for (uint32_t w = w0; w < w1; ++w) {
    const uint32_t i = 32 * w + lane;
    const int8_t a = i < n ? s1[i] : 0, b2 = i < n ? s2[i] : 0;
    const uint32_t b = __ballot_sync(0xffffffffu, a != b2), m = __ballot_sync(0xffffffffu, a < 0);
    if (lane == 0) {
      D[w] = b;
      V[w] = 0;
      A[w] = m;
    }
    cnt += __popc(b);
  }
  if (lane == 0) s_pre[warp] = cnt;
  __syncthreads();
  uint32_t k = pick[x] - 1;
  for (uint32_t v = 0; v < warp; ++v) k -= s_pre[v];  // (wraps in warps past the one that holds it)
  if (k < cnt)
    for (uint32_t w = w0; w < w1; ++w) {
      const uint32_t b = D[w], m = __popc(b);
      if (k < m) {
        if (((b >> lane) & 1u) && (uint32_t)__popc(b & ((1u << lane) - 1u)) == k) s_seed = 32 * w + lane;
        break;
      }
      k -= m;
    }
  __syncthreads();
  const uint32_t seed = s_seed;
  if (seed >= I.g_nodes) {  // petgraph's FixedBitSet would panic here
    if (tid == 0) *err = TAMC_E_REFPANIC;
    return;
  }
  // BFS over the q<0 subgraph (order-free: only the discovered set matters), a
  // team of four lanes per frontier site; the levels are consecutive segments of
  // the queue, their sizes rotate over three cells (one barrier per level)
  if (tid == 0) {
    V[seed >> 5] = 1u << (seed & 31u);
    queue[0] = seed;
    s_n[0] = 1;
    s_n[1] = 0;
    s_n[2] = 0;
  }
  __syncthreads();
  uint32_t lo = 0;
  for (uint32_t lvl = 0; lvl < n + 2u; ++lvl) {
    const uint32_t ncur = s_n[lvl % 3u];
    if (ncur == 0) break;
    uint32_t* const nxt = queue + lo + ncur;
    for (uint32_t q = tid; q < 4 * ncur; q += T) {
      const uint32_t u = queue[lo + q / 4], e1 = R.rp[u + 1];
      for (uint32_t e = R.rp[u] + q % 4; e < e1; e += 4) {
        uint32_t v, j;
        R.at(e, v, j);
        const uint32_t bit = 1u << (v & 31u);
        if ((D[v >> 5] & ~V[v >> 5] & bit) && !(atomicOr(&V[v >> 5], bit) & bit))
          nxt[atomicAdd(&s_n[(lvl + 1u) % 3u], 1u)] = v;
      }
    }
    lo += ncur;
    if (tid == 0) s_n[(lvl + 2u) % 3u] = 0;
    __syncthreads();
  }
  // the replicas trade the cluster's spins: each flips it
  for (uint32_t q = tid; q < lo; q += T) {
    const uint32_t v = queue[q];
    const int8_t a = (A[v >> 5] >> (v & 31u)) & 1u ? 1 : -1;
    s1[v] = a;
    s2[v] = (int8_t)-a;
  }
  __syncthreads();
  for (uint32_t w = tid; w < nwb; w += T) {
    const uint32_t a = A[w] ^ V[w];
    A[w] = a;
    D[w] ^= a;  // replica 2's spins
  }
  __syncthreads();
  // invalidated energies are recomputed by energy_ref exactly as the next
  // Macrostate::energy call would (tamc-core/src/pt.rs:126-129): the row terms in
  // parallel, their sums in order by a thread per replica
  float* rows = (float*)queue;
  for (uint32_t y = tid; y < 2 * n; y += T) {
    const uint32_t i = y < n ? y : y - n;
    const uint32_t* B = y < n ? A : D;
    float h = __fadd_rn(0.0f, R.bias[i]);
    const uint32_t e1 = R.rp[i + 1];
    for (uint32_t e = R.rp[i]; e < e1; ++e) {
      uint32_t v, j;
      R.at(e, v, j);
      h = __fadd_rn(h, __uint_as_float(j ^ ((B[v >> 5] >> (v & 31u)) << 31)) / 2.0f);
    }
    rows[y] = __uint_as_float(__float_as_uint(h) ^ ((B[i >> 5] >> (i & 31u)) << 31));
  }
  __syncthreads();
  if (tid == 0 || tid == 32) {
    const float* v = rows + (tid ? n : 0u);
    float total = I.offset;
    uint32_t i = 0;
    for (; i + 8 <= n; i += 8) {
      float w[8];
#pragma unroll
      for (int m = 0; m < 8; ++m) w[m] = v[i + m];
#pragma unroll
      for (int m = 0; m < 8; ++m) total = __fadd_rn(total, w[m]);
    }
    for (; i < n; ++i) total = __fadd_rn(total, v[i]);
    P.energy[tid ? r2 : r1] = total;
  }
}

// ------------------------------------------------------- exchange ----
__device__ void update_round_trips(const RefPt& P, uint32_t c) {  // tamc-core/src/pt.rs:54-84
  uint8_t* tg = P.tags + (size_t)c * P.nt;
  uint8_t& lo = tg[0];
  if (lo == 0) lo = 1;
  else if (lo == 4) { P.rtrips[c] += 1; lo = 1; }
  else if (lo == 2) lo = 3;
  uint8_t& hi = tg[P.nt - 1];
  if (hi == 0) hi = 2;
  else if (hi == 3) { P.rtrips[c] += 1; hi = 2; }
  else if (hi == 1) hi = 4;
  for (uint32_t k = 0; k < P.nt; ++k) {
    const uint8_t v = tg[k];
    if (v == 1 || v == 3) P.dhist[((size_t)c * P.nt + k) * 2] += 1;
    else if (v == 2 || v == 4) P.dhist[((size_t)c * P.nt + k) * 2 + 1] += 1;
  }
}

__device__ __forceinline__ void swap_slots(const RefPt& P, uint32_t c, uint32_t j) {  // PTState::swap_states
  uint32_t* pm = P.perm + (size_t)c * P.nt;
  const uint32_t a = pm[j];
  pm[j] = pm[j + 1];
  pm[j + 1] = a;
  uint8_t* tg = P.tags + (size_t)c * P.nt;
  const uint8_t b = tg[j];
  tg[j] = tg[j + 1];
  tg[j + 1] = b;
  P.acc[(size_t)c * P.nt + j] += 1;
}

// ThreadedPTSampler exchange (tamc-core/src/parallel/pt.rs:41-59), one thread per chain,
// uniforms from rng_vec[c][0].
__global__ void k_exchange_threaded(RefPt P, ExpTable X, Xo* rngs) {
  const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= P.C) return;
  Xo x = rngs[(size_t)c * P.nt];
  const uint32_t* pm = P.perm + (size_t)c * P.nt;
  for (uint32_t j = 0; j + 1 < P.nt; ++j) {
    // stale differences: E taken before any swap of this pass
    const float dlt = __fmul_rn(P.dbeta[j], __fsub_rn(P.e_stale[(size_t)c * P.nt + j + 1], P.e_stale[(size_t)c * P.nt + j]));
    if (dlt >= 0.0f || x.std_f32() < tamc_expf_exact(dlt, X.off, X.keys, X.vals)) swap_slots(P, c, j);
  }
  (void)pm;
  update_round_trips(P, c);
  rngs[(size_t)c * P.nt] = x;
}
// snapshot of the slot energies for the stale-difference exchange
__global__ void k_snapshot_energies(RefPt P) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < P.C * P.nt) P.e_stale[k] = P.energy[P.perm[k]];
}

// --------------------------------------------------------- sweeps ----
// ThreadedPTSampler sweeps (parallel/pt.rs:63-68): slot (c,t) with rng_vec[c][t].
__global__ void k_sweep_threaded(RefInst I, RefPt P, ExpTable X, Xo* rngs) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= P.C * P.nt) return;
  const uint32_t t = k % P.nt;
  const uint32_t r = P.perm[k];
  Xo x = rngs[k];
  const float de = sweep_tracked(I, X, P.betas[t], P.spins + (size_t)r * I.n, x);
  P.energy[r] = __fadd_rn(P.energy[r], de);
  rngs[k] = x;
}

// Serial mode (src/pt.rs:493-497, EnsembleSampler over ParallelTemperingSampler):
// one stream, per chain: exchange with ΔE propagation, then sweeps t = 0..nt-1.
__global__ void k_serial_round(RefInst I, RefPt P, ExpTable X, Xo* rng) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  Xo x = *rng;
  for (uint32_t c = 0; c < P.C; ++c) {
    uint32_t* pm = P.perm + (size_t)c * P.nt;
    float* des = P.e_stale;  // scratch [nt]
    for (uint32_t k = 0; k + 1 < P.nt; ++k) des[k] = __fsub_rn(P.energy[pm[k + 1]], P.energy[pm[k]]);
    for (uint32_t j = 0; j + 1 < P.nt; ++j) {
      const float dlt = __fmul_rn(P.dbeta[j], des[j]);
      if (dlt >= 0.0f || x.std_f32() < tamc_expf_exact(dlt, X.off, X.keys, X.vals)) {
        swap_slots(P, c, j);
        if (j + 2 < P.nt) des[j + 1] = __fadd_rn(des[j + 1], des[j]);
        des[j] = -des[j];
      }
    }
    update_round_trips(P, c);
    for (uint32_t t = 0; t < P.nt; ++t) {
      const uint32_t r = pm[t];
      const float de = sweep_tracked(I, X, P.betas[t], P.spins + (size_t)r * I.n, x);
      P.energy[r] = __fadd_rn(P.energy[r], de);
    }
  }
  *rng = x;
}

// ---------------------------------------------------- measurements ----
// PtIcmThermalSamples::measure / sample_states (src/pt.rs:167-226) for one
// measurement index; grid (nt, C).
__global__ void k_measure(RefInst I, RefPt P, MeasOut O, uint32_t m, int do_measure, uint32_t smp, int do_sample) {
  __shared__ uint32_t sh[32];
  const uint32_t t = blockIdx.x, c = blockIdx.y;
  const uint32_t n = I.n;
  const uint32_t r = P.perm[(size_t)c * P.nt + t];
  const int8_t* s1 = P.spins + (size_t)r * n;
  const uint32_t npair = P.C / 2;
  if (do_measure) {
    if (threadIdx.x == 0) O.e[(size_t)t * O.M * P.C + (size_t)m * P.C + c] = P.energy[r];
    if ((c & 1u) == 0 && c / 2 < npair) {
      const uint32_t p = c / 2;
      const int8_t* s2 = P.spins + (size_t)P.perm[(size_t)(c + 1) * P.nt + t] * n;
      uint32_t neg = 0;
      for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) neg += (s1[i] != s2[i]);
      neg = block_sum_u32(neg, sh);
      if (threadIdx.x == 0) O.q[(size_t)t * O.M * npair + (size_t)m * npair + p] = (int32_t)n - 2 * (int32_t)neg;
      for (uint32_t k = threadIdx.x; k < O.nchi; k += blockDim.x) {
        const double* w = I.sus + (size_t)k * n;
        double chi = 0.0;
        for (uint32_t i = 0; i < n; ++i) chi = __dadd_rn(chi, __dmul_rn(w[i], (double)(s1[i] * s2[i])));
        O.sus[((size_t)t * O.nchi + k) * O.M * npair + (size_t)m * npair + p] = (float)chi;
      }
    }
  }
  if (do_sample) {
    int z = -1;
    if (O.level == 0) z = (int)t;
    else if (O.level == 1) { if (t >= P.nt - P.nt / 2) z = (int)(P.nt - 1 - t); }
    else if (t == P.nt - 1) z = 0;
    if (z >= 0) {
      const uint32_t nb = (n + 7) / 8;
      uint8_t* dst = O.samp + (((size_t)z * O.S + smp) * P.C + c) * nb;
      for (uint32_t b = threadIdx.x; b < nb; b += blockDim.x) {
        uint32_t v = 0;
        for (uint32_t k = 0; k < 8 && b * 8 + k < n; ++k) v |= (uint32_t)(s1[b * 8 + k] <= 0) << k;
        dst[b] = (uint8_t)v;
      }
    }
  }
}

// Ground-state tracking of apply_measurements (src/pt.rs:559-581): first
// minimum over slots, then over chains, strictly below the running minimum.  A
// warp reduces by (energy, chain, slot); energies that are not numbers, whose
// comparisons depend on their order, are walked through by one thread.
__global__ void k_gs_track(RefInst I, RefPt P, GsLog L, uint32_t step) {
  __shared__ int s_new;
  __shared__ uint32_t s_rep, s_slot;
  if (threadIdx.x < 32) {
    const uint32_t lane = threadIdx.x, N = P.C * P.nt;
    float best = INFINITY;
    uint32_t bx = 0xffffffffu;
    bool nan = false;
    for (uint32_t x = lane; x < N; x += 32) {
      const float e = P.energy[P.perm[x]];
      nan |= e != e;
      if (e < best || (e == best && x < bx)) {
        best = e;
        bx = x;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float oe = __shfl_xor_sync(0xffffffffu, best, o);
      const uint32_t ox = __shfl_xor_sync(0xffffffffu, bx, o);
      if (oe < best || (oe == best && ox < bx)) {
        best = oe;
        bx = ox;
      }
    }
    nan = __any_sync(0xffffffffu, nan);
    if (lane == 0) {
      uint32_t br = nan ? 0u : P.perm[bx];
      if (nan)
        for (uint32_t c = 0; c < P.C; ++c) {
          uint32_t i1 = 0;
          float e1 = P.energy[P.perm[(size_t)c * P.nt]];
          for (uint32_t t = 1; t < P.nt; ++t) {
            const float e = P.energy[P.perm[(size_t)c * P.nt + t]];
            if (e < e1) { e1 = e; i1 = t; }
          }
          if (c == 0 || e1 < best) { best = e1; br = P.perm[(size_t)c * P.nt + i1]; }
        }
      s_new = 0;
      if (!*L.have || best < *L.minE) {
        *L.have = 1;
        *L.minE = best;
        const uint32_t k = *L.count;
        if (k < L.cap) {
          L.steps[k] = step;
          L.E[k] = best;
          s_new = 1;
          s_slot = k;
          s_rep = br;
        }
        *L.count = k + 1;
      }
    }
  }
  __syncthreads();
  if (!s_new) return;
  const int8_t* s = P.spins + (size_t)s_rep * I.n;
  const uint32_t nw = (I.n + 63) / 64;
  for (uint32_t w = threadIdx.x; w < nw; w += blockDim.x) {
    uint64_t v = 0;
    for (uint32_t k = 0; k < 64 && w * 64 + k < I.n; ++k) v |= (uint64_t)(s[w * 64 + k] <= 0) << k;
    L.words[(size_t)s_slot * nw + w] = v;
  }
}

// ------------------------------------------------------------- SA ----
// sa_loop over one partition (src/sa.rs:167-199, tamc-core/src/sa.rs:27-48):
// for each beta, each replica of the partition is swept in turn with the
// partition's stream.  One thread per partition.
__global__ void k_sa(RefInst I, ExpTable X, int8_t* spins, Xo* rngs, uint32_t parts, uint32_t per,
                     const float* betas, uint32_t nbeta) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= parts) return;
  Xo x = rngs[p];
  for (uint32_t b = 0; b < nbeta; ++b) {
    const float beta = betas[b];
    for (uint32_t r = 0; r < per; ++r) {
      int8_t* s = spins + ((size_t)p * per + r) * I.n;
      for (uint32_t i = 0; i < I.n; ++i) {
        float d;
        advance(I, X, beta, s, i, x, d);
      }
    }
  }
  rngs[p] = x;
}

}  // namespace refk

// ----------------------------------------------------------- launchers ----
void ref_energy_all(cudaStream_t st, const RefInst& I, const int8_t* spins, float* energy, uint32_t R) {
  if (!R) return;
  refk::k_energy_all<<<R, 128, 0, st>>>(I, spins, energy);
}
// Largest dynamic shared memory of the kernels below (they leave room for 8 KB
// of their own).  TAMC_REF_SMEM lowers it, so that a small instance takes the
// kernels for sizes that do not fit.
static size_t ref_smem_limit() {
  int dev = 0, v = 0;
  TAMC_CUDA(cudaGetDevice(&dev));
  TAMC_CUDA(cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  const size_t most = (size_t)v - 8192;
  const char* e = getenv("TAMC_REF_SMEM");
  return e ? std::min<size_t>(most, strtoull(e, nullptr, 10)) : most;
}
template <typename K>
static void ref_smem_attr(K k, size_t bytes) {
  if (bytes > 40960) kernel_smem(reinterpret_cast<const void*>(k), bytes);
}
uint32_t ref_icm(cudaStream_t st, const RefInst& I, uint64_t nnz, const RefPt& P, const ExpTable& X, Xo* rng,
                 int* err) {
  const size_t smem = refk::ref_icm_bytes(I.n), rows = refk::ref_rows_bytes(I.n, nnz);
  const uint32_t slots = P.C / 2 * (P.nt - P.lo);
  if (!slots) return 0;
  if (smem > ref_smem_limit()) {  // (above 27000 sites)
    refk::k_icm<<<1, 512, 0, st>>>(I, P, X, rng, err);
    return 1;
  }
  refk::k_icm_seeds<<<1, 1024, 0, st>>>(I, P, rng, P.pick);
  if (smem + rows <= ref_smem_limit()) {
    ref_smem_attr(refk::k_icm_move<true>, smem + rows);
    refk::k_icm_move<true><<<slots, 256, smem + rows, st>>>(I, P, P.pick, err);
  } else {
    ref_smem_attr(refk::k_icm_move<false>, smem);
    refk::k_icm_move<false><<<slots, 256, smem, st>>>(I, P, P.pick, err);
  }
  return 2;
}
void ref_exchange_threaded(cudaStream_t st, const RefPt& P, const ExpTable& X, Xo* rngs) {
  const size_t smem = refk::ref_chain_bytes(P.nt);
  if (smem > ref_smem_limit()) {  // (above 13000 temperatures)
    const uint32_t k = P.C * P.nt;
    refk::k_snapshot_energies<<<(k + 127) / 128, 128, 0, st>>>(P);
    refk::k_exchange_threaded<<<(P.C + 31) / 32, 32, 0, st>>>(P, X, rngs);
    return;
  }
  ref_smem_attr(refk::k_exchange_threaded_b, smem);
  refk::k_exchange_threaded_b<<<P.C, 32, smem, st>>>(P, X, rngs);
}
void ref_sweep_threaded(cudaStream_t st, const RefInst& I, uint64_t nnz, const RefPt& P, const ExpTable& X, Xo* rngs) {
  const uint32_t k = P.C * P.nt;
  const size_t bits = ((size_t)(I.n + 31) / 32 * 4 + 15) / 16 * 16, rows = refk::ref_rows_bytes(I.n, nnz);
  if (bits > ref_smem_limit()) {  // (above 1.7 million sites)
    refk::k_sweep_threaded<<<(k + 31) / 32, 32, 0, st>>>(I, P, X, rngs);
  } else if (bits + rows <= ref_smem_limit()) {
    ref_smem_attr(refk::k_sweep_threaded_b<true>, bits + rows);
    refk::k_sweep_threaded_b<true><<<k, 96, bits + rows, st>>>(I, P, X, rngs);
  } else {
    ref_smem_attr(refk::k_sweep_threaded_b<false>, bits);
    refk::k_sweep_threaded_b<false><<<k, 96, bits, st>>>(I, P, X, rngs);
  }
}
void ref_serial_round(cudaStream_t st, const RefInst& I, uint64_t nnz, const RefPt& P, const ExpTable& X, Xo* rng) {
  const size_t base = (3 * ((size_t)(I.n + 31) / 32 * 4) + 15) / 16 * 16 + refk::ref_chain_bytes(P.nt);
  const size_t rows = refk::ref_rows_bytes(I.n, nnz);
  if (base > ref_smem_limit()) {  // (hundreds of thousands of sites, or thousands of temperatures)
    refk::k_serial_round<<<1, 1, 0, st>>>(I, P, X, rng);
  } else if (base + rows <= ref_smem_limit()) {
    ref_smem_attr(refk::k_serial_round_b<true>, base + rows);
    refk::k_serial_round_b<true><<<1, 128, base + rows, st>>>(I, P, X, rng);
  } else {
    ref_smem_attr(refk::k_serial_round_b<false>, base);
    refk::k_serial_round_b<false><<<1, 128, base, st>>>(I, P, X, rng);
  }
}
void ref_measure(cudaStream_t st, const RefInst& I, const RefPt& P, const MeasOut& O, uint32_t m, bool meas,
                 uint32_t smp, bool samp) {
  refk::k_measure<<<dim3(P.nt, P.C), 128, 0, st>>>(I, P, O, m, meas ? 1 : 0, smp, samp ? 1 : 0);
}
void ref_gs_track(cudaStream_t st, const RefInst& I, const RefPt& P, const GsLog& L, uint32_t step) {
  refk::k_gs_track<<<1, 128, 0, st>>>(I, P, L, step);
}
void ref_sa(cudaStream_t st, const RefInst& I, const ExpTable& X, int8_t* spins, Xo* rngs, uint32_t parts,
            uint32_t per, const float* betas, uint32_t nbeta) {
  refk::k_sa<<<(parts + 31) / 32, 32, 0, st>>>(I, X, spins, rngs, parts, per, betas, nbeta);
}

}  // namespace tamc
