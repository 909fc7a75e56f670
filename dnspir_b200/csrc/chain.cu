// chain.cu -- the key-switching chain of preprocess / partial_gal
// (crates/pir/src/base_pir.rs:496-594, 782-863) and its fusion with the
// secondary scan (double_pir.rs:195-218).
//
// A chain step on the a-part of a ciphertext is
//     t      = sigma_5(a)                        (the galois lookup of :509-515)
//     v      = centred CRT lift of iNTT(t)        (:544-555)
//     d1     = (v + 2^25) >> 26, d0 = v - 2^26 d1 (:557-570; the second digit's
//              own carry is always 0 since |v| < q/2 < 2^50)
//     a      = NTT(d0) gk_a0 + NTT(d1) gk_a1 + qry_a E_i
// and, for the secondary database evaluated on a query ciphertext (b-part),
//     b      = sigma_5(b) + NTT(d0) gk_b0 + NTT(d1) gk_b1 + qry_b E_i,
// which is the homomorphic evaluation whose b-part main_pir_loop computes
// from the stored digits (its sum/sum_new recurrence equals b up to the
// sigma_5 applied before the final permute, :1072-1073).
//
// Because d0 + 2^26 d1 = v exactly and v = t in each factor, NTT(d0) =
// t - 2^26 NTT(d1): one forward transform per factor and step instead of two.
//
// Forms.  N = 2048, on the register transforms of ntt2048.cuh, by the number of
// chains: two SMs each (a cluster of two blocks, one RNS factor each, which
// exchange their inverse transforms through mbarrier-counted inboxes), one SM each
// (both factors in one block, inboxes in its shared memory), or several chains a
// block or SM (each thread carries both factors).  Other lengths, and preprocessing
// with three stored arrays: a cluster of two blocks with a cluster barrier per step,
// or one block with both factors.  NTT-domain vectors hold slots in bit-reversed
// position order (position q <-> slot brv(q)); the constants are stored the same way.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstring>
#include <type_traits>

#include "kernels.cuh"
#include "ntt2048.cuh"

namespace cg = cooperative_groups;

namespace dnspir {
namespace {

constexpr int CT = 512;  // threads per block of a chain cluster

// ---- Montgomery arithmetic, R = 2^32 (p < 2^26)
__host__ __device__ constexpr uint32_t neg_inv32(uint32_t p) {
  uint32_t x = p;  // Newton iteration for p^-1 mod 2^32
  for (int i = 0; i < 5; i++) x *= 2u - p * x;
  return 0u - x;
}
// x * y R^-1 mod p for products and sums below 2^64 whose result is < 3p; returns [0, p)
__device__ __forceinline__ uint32_t mont_reduce(uint64_t T, uint32_t p, uint32_t pinv) {
  const uint32_t m = (uint32_t)T * pinv;
  uint64_t u = (T + (uint64_t)m * p) >> 32;
  u = u >= p ? u - p : u;
  u = u >= p ? u - p : u;
  return (uint32_t)u;
}

struct ChainPrime {
  uint32_t p, pinv;      // factor and -p^-1 mod 2^32
  uint32_t r2;           // R^2 mod p (to enter Montgomery form)
  uint32_t c26;          // 2^26 R mod p
  uint32_t k1, k1q;      // q2^-1 N^-1 mod q1 with its Shoup companion (CRT, factor 1)
  uint32_t k2, k2q;      // q1^-1 N^-1 mod q2 (CRT, factor 2)
  uint32_t k, kinv;      // this factor's CRT constant (k1 or k2) and its inverse (N times the other factor)
};

// radix-4 / radix-2 transforms of one length-2^logn vector by CT threads, with
// Harvey's lazy butterflies: values stay in [0, 4p) inside a transform (4p <
// 2^28) and are brought back to [0, p) when it ends.
// Forward: natural -> bit-reversed (CT butterflies), input in [0, p).
// Inverse: bit-reversed -> natural, NOT scaled by N^-1 (the caller folds N^-1
// into its next constant), input in [0, p), outputs in [0, 2p).
__device__ __forceinline__ uint32_t shoup_lazy(uint32_t x, uint32_t w, uint32_t wq, uint32_t p) {
  return x * w - __umulhi(x, wq) * p;  // in [0, 2p) for any x < 2^32
}
__device__ __forceinline__ uint32_t red2p(uint32_t x, uint32_t p2) { return x >= p2 ? x - p2 : x; }
// CT butterfly on [0, 4p) inputs: (x, y) -> (x + w y, x - w y), outputs in [0, 4p)
__device__ __forceinline__ void ct_bf(uint32_t& x, uint32_t& y, uint32_t w, uint32_t wq, uint32_t p) {
  const uint32_t a = red2p(x, 2 * p);
  const uint32_t t = shoup_lazy(y, w, wq, p);
  x = a + t;
  y = a - t + 2 * p;
}
// GS butterfly on [0, 2p) inputs: (x, y) -> (x + y, w (x - y)), outputs in [0, 2p)
__device__ __forceinline__ void gs_bf(uint32_t& x, uint32_t& y, uint32_t w, uint32_t wq, uint32_t p) {
  const uint32_t a = x + y;
  const uint32_t d = x - y + 2 * p;
  x = red2p(a, 2 * p);
  y = shoup_lazy(d, w, wq, p);
}

// LOGN > 0 fixes the length at compile time (the stage loop unrolls and every
// index shift is a constant); LOGN = 0 takes logn_rt.
template <int LOGN>
__device__ __forceinline__ void fwd_one(uint32_t* x, int logn_rt, const uint32_t* __restrict__ tw,
                                        const uint32_t* __restrict__ twq, uint32_t p) {
  const int logn = LOGN ? LOGN : logn_rt;
  const int N = 1 << logn;
  int s = 0;
#pragma unroll
  for (; s + 1 < logn; s += 2) {
    const int logt2 = logn - s - 2;
    const int t2 = 1 << logt2, t = 2 * t2, m = 1 << s;
    for (int g = threadIdx.x; g < N / 4; g += CT) {
      const int blk = g >> logt2, r = g & (t2 - 1);
      const int j = (blk << (logt2 + 2)) + r;
      const uint32_t w = tw[m + blk], wq = twq[m + blk];
      const uint32_t w1 = tw[2 * m + 2 * blk], w1q = twq[2 * m + 2 * blk];
      const uint32_t w2 = tw[2 * m + 2 * blk + 1], w2q = twq[2 * m + 2 * blk + 1];
      uint32_t v[4] = {x[j], x[j + t2], x[j + t], x[j + t + t2]};
      ct_bf(v[0], v[2], w, wq, p);
      ct_bf(v[1], v[3], w, wq, p);
      ct_bf(v[0], v[1], w1, w1q, p);
      ct_bf(v[2], v[3], w2, w2q, p);
      x[j] = v[0], x[j + t2] = v[1], x[j + t] = v[2], x[j + t + t2] = v[3];
    }
    __syncthreads();
  }
  if (s < logn) {  // last stage, t = 1
    for (int b = threadIdx.x; b < N / 2; b += CT) {
      uint32_t u = x[2 * b], v = x[2 * b + 1];
      ct_bf(u, v, tw[N / 2 + b], twq[N / 2 + b], p);
      x[2 * b] = red2p(red2p(u, 2 * p), p);
      x[2 * b + 1] = red2p(red2p(v, 2 * p), p);
    }
  } else {
    for (int b = threadIdx.x; b < N; b += CT) x[b] = red2p(red2p(x[b], 2 * p), p);
  }
  __syncthreads();
}

template <int LOGN>
__device__ __forceinline__ void inv_one(uint32_t* x, int logn_rt, const uint32_t* __restrict__ tw,
                                        const uint32_t* __restrict__ twq, uint32_t p) {
  const int logn = LOGN ? LOGN : logn_rt;
  const int N = 1 << logn;
  int s = 0;
#pragma unroll
  for (; s + 1 < logn; s += 2) {
    const int t = 1 << s;
    const int h0 = N >> (s + 1), h1 = N >> (s + 2);
    for (int g = threadIdx.x; g < N / 4; g += CT) {
      const int blk = g >> s, r = g & (t - 1);
      const int j = (blk << (s + 2)) + r;
      const uint32_t w0 = tw[h0 + 2 * blk], w0q = twq[h0 + 2 * blk];
      const uint32_t w1 = tw[h0 + 2 * blk + 1], w1q = twq[h0 + 2 * blk + 1];
      const uint32_t w = tw[h1 + blk], wq = twq[h1 + blk];
      uint32_t v[4] = {x[j], x[j + t], x[j + 2 * t], x[j + 3 * t]};
      gs_bf(v[0], v[1], w0, w0q, p);
      gs_bf(v[2], v[3], w1, w1q, p);
      gs_bf(v[0], v[2], w, wq, p);
      gs_bf(v[1], v[3], w, wq, p);
      x[j] = v[0], x[j + t] = v[1], x[j + 2 * t] = v[2], x[j + 3 * t] = v[3];
    }
    __syncthreads();
  }
  if (s < logn) {  // last stage, t = N/2
    const uint32_t w = tw[1], wq = twq[1];
    for (int j = threadIdx.x; j < N / 2; j += CT) {
      uint32_t u = x[j], v = x[j + N / 2];
      gs_bf(u, v, w, wq, p);
      x[j] = u;
      x[j + N / 2] = v;
    }
    __syncthreads();
  }
}

// High digit of the centred CRT lift from the two factors' unscaled iNTT
// outputs: x = v - k q (v = x1 q2 + x2 q1 < 2q, k = round(v / q)), digit
// floor((x + 2^25) / 2^26).  Computed in double precision, exactly: x1 q2 and
// x2 q1 are below 2^51, v below 2^52 and q = q1 q2 below 2^51, so every sum,
// difference and comparison is exact in the 53-bit significand, and
// x 2^-26 + 1/2 (a power-of-two scaling of an integer below 2^51 in
// magnitude, plus one half) is exact too, leaving floor() the only rounding
// -- the same integer as the 64-bit formula, on the FP64 pipe instead of the
// integer pipes the transforms saturate.
__device__ __forceinline__ int32_t high_digit(uint32_t c1, uint32_t c2, const ChainPrime& P1c, const ChainPrime& P2c) {
  const uint32_t x1 = shoup_mul(c1, P1c.k1, P1c.k1q, P1);
  const uint32_t x2 = shoup_mul(c2, P2c.k2, P2c.k2q, P2);
  constexpr double Q = (double)QQ, HALF_Q = (double)(QQ / 2);  // QQ / 2 = (q - 1) / 2, exact
  double v = fma((double)x1, (double)P2, (double)x2 * (double)P1);
  v = v >= Q ? v - Q : v;
  v = v > HALF_Q ? v - Q : v;
  return __double2int_rd(fma(v, 1.0 / (double)(1u << LOG2_B), 0.5));
}

struct ChainArgs {
  Group g;
  // constants: gk_a digits [d][p][pos], qry_a halves [h][p][pos], sigma_5 map, canonical
  const uint32_t* gka;
  const uint32_t* qa;
  const uint32_t* galb;
  SlotMaps maps;
  NttTables T;
  ChainPrime cp[2];
  // secondary: entries in chain layout, query vectors [q][slot][p][pos], output
  const uint32_t* E;
  const uint32_t* qv;
  size_t qv_stride;
  int nl;
  uint32_t* out;
  // primary: slabs and a-part output
  uint32_t* const* slabs;
  uint32_t* a_out;
  // paired chains: error word, set to 1 when a wait for the peer block gives up;
  // limit of that wait; step that the first chain's second block leaves before (~0u: none)
  uint32_t* err;
  uint64_t wait_ns;
  uint32_t withhold;
  uint32_t c_first, cinv_first, inv5;
};

// Primary chain (preprocessing), one lane per block.  Shared-memory plan (u32
// words, N = 2^logn):
//   A, TC, D           N each    state a, saved sigma_5(a), work vector
//   X[2]               2N        iNTT outputs published to the peer block
//   CG0, CG1, CQA      3N        gk_a0 R, gk_a1 R, qry_a R of this factor and half
//   FW, FWQ, IW, IWQ   4N        twiddles of this factor
template <int LOGN>
__device__ __forceinline__ void primary_body(const ChainArgs& a, int h, int lane, int s, uint32_t* sm) {
  cg::cluster_group cluster = cg::this_cluster();
  const int p = (int)cluster.block_rank();
  const int logn = LOGN ? LOGN : a.g.log2n;
  const int N = 1 << logn;
  const uint32_t mask = 2 * N - 1;
  const ChainPrime cp = a.cp[p];
  const uint32_t pr = cp.p;
  uint32_t* A = sm;
  uint32_t* TC = A + N;
  uint32_t* D = TC + N;
  uint32_t* X = D + N;
  uint32_t* CG0 = X + 2 * N;
  uint32_t* CG1 = CG0 + N;
  uint32_t* CQA = CG1 + N;
  uint32_t* FW = CQA + N;
  uint32_t* FWQ = FW + N;
  uint32_t* IW = FWQ + N;
  uint32_t* IWQ = IW + N;
  for (int b = threadIdx.x; b < N; b += CT) {
    A[b] = 0;
    const size_t o = (size_t)p * N + b;
    CG0[b] = mont_reduce((uint64_t)a.gka[o] * cp.r2, pr, cp.pinv);
    CG1[b] = mont_reduce((uint64_t)a.gka[2 * (size_t)N + o] * cp.r2, pr, cp.pinv);
    CQA[b] = mont_reduce((uint64_t)a.qa[(size_t)h * 2 * N + o] * cp.r2, pr, cp.pinv);
    FW[b] = a.T.fw[p][b];
    FWQ[b] = a.T.fwq[p][b];
    IW[b] = a.T.iw[p][b];
    IWQ[b] = a.T.iwq[p][b];
  }
  cluster.sync();
  uint32_t* peerX = cluster.map_shared_rank(X, p ^ 1);
  uint32_t* slab = a.slabs[s];
  uint32_t ci = a.c_first, cinv = a.cinv_first;
  constexpr int PER = N_MAX / CT;  // positions per thread (N <= N_MAX)
  for (uint32_t i = 0; i < a.g.L; i++) {
    // entries of row i for this thread's positions, consumed at the end of the step
    uint32_t e[PER];
#pragma unroll
    for (int c = 0; c < PER; c++) {
      const int pos = threadIdx.x + c * CT;
      e[c] = 0;
      if (pos < N) {
        const uint32_t j = brv(pos, logn);
        const uint32_t ks = gidx(cinv * (2 * j + 1), mask);
        e[c] = slab[slab_off(a.g, p, h, i, 0, __ldg(a.maps.uof + ks)) + lane];
      }
    }
    // sigma_5 on a
    uint32_t ra[PER];
#pragma unroll
    for (int c = 0; c < PER; c++) {
      const int pos = threadIdx.x + c * CT;
      if (pos < N) ra[c] = A[pos];
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < PER; c++) {
      const int pos = threadIdx.x + c * CT;
      if (pos < N) {
        const uint32_t dst = __ldg(a.galb + pos);
        TC[dst] = ra[c];
        D[dst] = ra[c];
      }
    }
    __syncthreads();
    inv_one<LOGN>(D, logn, IW, IWQ, pr);
    uint32_t* Xc = X + (i & 1) * N;
    for (int b = threadIdx.x; b < N; b += CT) Xc[b] = D[b];
    cluster.sync();
    const uint32_t* Pc = peerX + (i & 1) * N;
    for (int b = threadIdx.x; b < N; b += CT) {
      const uint32_t own = D[b], other = Pc[b];
      const int32_t hd = p == 0 ? high_digit(own, other, a.cp[0], a.cp[1]) : high_digit(other, own, a.cp[0], a.cp[1]);
      D[b] = hd < 0 ? (uint32_t)(hd + (int32_t)pr) : (uint32_t)hd;
    }
    __syncthreads();
    fwd_one<LOGN>(D, logn, FW, FWQ, pr);
#pragma unroll
    for (int c = 0; c < PER; c++) {
      const int pos = threadIdx.x + c * CT;
      if (pos < N) {
        const uint32_t n1 = D[pos];
        const uint32_t n0 = sub_mod(TC[pos], mont_reduce((uint64_t)n1 * cp.c26, pr, cp.pinv), pr);
        A[pos] = mont_reduce((uint64_t)n0 * CG0[pos] + (uint64_t)n1 * CG1[pos] + (uint64_t)e[c] * CQA[pos], pr,
                             cp.pinv);
        TC[pos] = n0;
      }
    }
    __syncthreads();
    // row i in the scan layout: position u (natural slot k with 2k+1 = g[u])
    // holds the values at slot idx(5^(L-1-i) g[u]) -- the new state over the
    // entries and the high digit, or both digits beside the entries (slab_off)
    const bool two = a.g.na == 2;
    for (int u = threadIdx.x; u < N; u += CT) {
      const uint32_t jb = brv(gidx(ci * __ldg(a.maps.g + u), mask), logn);
      slab[slab_off(a.g, p, h, i, two ? 0 : 1, u) + lane] = two ? A[jb] : TC[jb];
      slab[slab_off(a.g, p, h, i, two ? 1 : 2, u) + lane] = D[jb];
    }
    // TC and D are rewritten only after the next step's first barrier
    ci = (ci * a.inv5) & mask;
    cinv = (cinv * 5) & mask;
  }
  uint32_t* o = a.a_out + (((size_t)s * a.g.H + h) * SIMD + lane) * 2 * N;
  for (int b = threadIdx.x; b < N; b += CT) o[(size_t)p * N + b] = A[b];
  cluster.sync();  // keep this block's shared memory alive until the peer's last read
}

// Secondary chain at N < 2048: one of the three parts of one query's secondary
// ciphertext at half h in one block (factor p = rank in the cluster).  The key
// constants gk_a0, gk_a1, qry_a, gk_b0, gk_b1, qry_b (Montgomery form) and the
// sigma_5 destinations of a thread's positions live in its registers.  Each step's
// pointwise stage writes the next step's sigma_5-permuted a and b straight
// into the other buffer of a pair, and the inverse transform is published to
// the peer from its own buffer D[i mod 2] (the peer reads it between the
// cluster barriers of steps i and i + 1; this block rewrites it only at the end
// of step i + 1).  Shared memory (u32 words):
//   FW FWQ IW IWQ             4N   twiddles of this factor
//   TC[2] D[2] B[2] H         7N   sigma_5(a) kept, sigma_5(a) transformed
//                                  (published), sigma_5(b), high digit
constexpr int SEC_PART_WORDS = 7;  // x N
constexpr int SEC_WORDS = 4 + SEC_PART_WORDS;

__device__ __forceinline__ void secondary_body(const ChainArgs& a, int h, int q, int part, uint32_t* sm) {
  cg::cluster_group cluster = cg::this_cluster();
  const int p = (int)cluster.block_rank();
  const int logn = a.g.log2n;
  const int N = 1 << logn;
  const ChainPrime cp = a.cp[p];
  const uint32_t pr = cp.p;
  uint32_t* FW = sm;
  uint32_t* FWQ = FW + N;
  uint32_t* IW = FWQ + N;
  uint32_t* IWQ = IW + N;
  uint32_t* TC = IWQ + N;
  uint32_t* D = TC + 2 * N;
  uint32_t* B = D + 2 * N;
  uint32_t* H = B + 2 * N;
  const uint32_t* qq = a.qv + (size_t)q * a.qv_stride;
  constexpr int PER = N_MAX / CT;  // positions per thread (N <= N_MAX)
  uint32_t kc[6][PER], dst[PER];
#pragma unroll
  for (int c = 0; c < PER; c++) {
    const int pos = threadIdx.x + c * CT;
    if (pos < N) {
      const size_t o = (size_t)p * N + pos;
      kc[0][c] = mont_reduce((uint64_t)a.gka[o] * cp.r2, pr, cp.pinv);
      kc[1][c] = mont_reduce((uint64_t)a.gka[2 * (size_t)N + o] * cp.r2, pr, cp.pinv);
      kc[2][c] = mont_reduce((uint64_t)a.qa[(size_t)h * 2 * N + o] * cp.r2, pr, cp.pinv);
      kc[3][c] = mont_reduce((uint64_t)qq[o] * cp.r2, pr, cp.pinv);
      kc[4][c] = mont_reduce((uint64_t)qq[2 * (size_t)N + o] * cp.r2, pr, cp.pinv);
      kc[5][c] = mont_reduce((uint64_t)qq[(size_t)(4 + h) * 2 * N + o] * cp.r2, pr, cp.pinv);
      dst[c] = __ldg(a.galb + pos);
    }
  }
  for (int b = threadIdx.x; b < N; b += CT) {
    FW[b] = a.T.fw[p][b];
    FWQ[b] = a.T.fwq[p][b];
    IW[b] = a.T.iw[p][b];
    IWQ[b] = a.T.iwq[p][b];
    TC[b] = D[b] = B[b] = 0;  // a = b = 0, so sigma_5(a) = sigma_5(b) = 0
  }
  cluster.sync();
  const uint32_t* peerD = cluster.map_shared_rank(D, p ^ 1);
  for (uint32_t i = 0; i < a.g.L; i++) {
    const int cur = (int)(i & 1) * N, nxt = N - cur;
    // entries of row i, consumed at the end of the step
    const uint32_t* Ei =
        a.E + ((((size_t)p * a.g.H + h) * a.g.L + a.g.L - 1 - i) * a.nl + (size_t)q * CTXT_PARTS + part) * N;
    uint32_t e[PER];
#pragma unroll
    for (int c = 0; c < PER; c++) {
      const int pos = threadIdx.x + c * CT;
      e[c] = pos < N ? __ldg(Ei + pos) : 0;
    }
    inv_one<0>(D + cur, logn, IW, IWQ, pr);
    cluster.sync();
    for (int b = threadIdx.x; b < N; b += CT) {
      const uint32_t own = D[cur + b], other = peerD[cur + b];
      const int32_t hd = p == 0 ? high_digit(own, other, a.cp[0], a.cp[1]) : high_digit(other, own, a.cp[0], a.cp[1]);
      H[b] = hd < 0 ? (uint32_t)(hd + (int32_t)pr) : (uint32_t)hd;
    }
    __syncthreads();
    fwd_one<0>(H, logn, FW, FWQ, pr);
#pragma unroll
    for (int c = 0; c < PER; c++) {
      const int pos = threadIdx.x + c * CT;
      if (pos < N) {
        const uint32_t n1 = H[pos];
        const uint32_t n0 = sub_mod(TC[cur + pos], mont_reduce((uint64_t)n1 * cp.c26, pr, cp.pinv), pr);
        const uint32_t an = mont_reduce(
            (uint64_t)n0 * kc[0][c] + (uint64_t)n1 * kc[1][c] + (uint64_t)e[c] * kc[2][c], pr, cp.pinv);
        const uint32_t bn = mont_reduce(((uint64_t)B[cur + pos] << 32) + (uint64_t)n0 * kc[3][c] +
                                            (uint64_t)n1 * kc[4][c] + (uint64_t)e[c] * kc[5][c],
                                        pr, cp.pinv);
        // sigma_5 for the next step
        TC[nxt + dst[c]] = an;
        D[nxt + dst[c]] = an;
        B[nxt + dst[c]] = bn;
      }
    }
    __syncthreads();
  }
  // the state after the last step sits sigma_5-permuted in buffer L mod 2
  const int fin = (int)(a.g.L & 1) * N;
  uint32_t* o = a.out + ((((size_t)q * a.g.H + h) * CTXT_PARTS + part) * 2) * 2 * N;
#pragma unroll
  for (int c = 0; c < PER; c++) {
    const int pos = threadIdx.x + c * CT;
    if (pos < N) {
      o[(size_t)p * N + pos] = TC[fin + dst[c]];
      o[2 * (size_t)N + (size_t)p * N + pos] = B[fin + dst[c]];
    }
  }
  cluster.sync();  // keep this block's shared memory alive until the peer's last read
}

// ---- secondary chain without a cluster: one block carries one part at half h
// in BOTH factors.  Every transform pass handles the two factors' vectors
// (each with its own twiddles and prime), the high digit reads both inverse
// transforms from this block's shared memory (no cluster barrier, no remote
// reads), and each barrier covers twice the work of the clustered form.
// Shared memory (u32 words): twiddles FW FWQ IW IWQ of each factor (8N), per
// factor TC[2] D[2] B[2] H (7N): 22N.
constexpr int SEC_DUAL_WORDS = 8 + 2 * SEC_PART_WORDS;  // x N

__device__ __forceinline__ void fwd_dual(uint32_t* x0, uint32_t* x1, int logn, const uint32_t* const* tw,
                                         const uint32_t* const* twq, uint32_t p0, uint32_t p1) {
  const int N = 1 << logn;
  uint32_t* xs[2] = {x0, x1};
  const uint32_t ps[2] = {p0, p1};
  int s = 0;
#pragma unroll
  for (; s + 1 < logn; s += 2) {
    const int logt2 = logn - s - 2;
    const int t2 = 1 << logt2, t = 2 * t2, m = 1 << s;
    for (int g = threadIdx.x; g < N / 4; g += CT) {
      const int blk = g >> logt2, r = g & (t2 - 1);
      const int j = (blk << (logt2 + 2)) + r;
      uint32_t v[2][4];
#pragma unroll
      for (int l = 0; l < 2; l++) {
        const uint32_t* x = xs[l];
        v[l][0] = x[j], v[l][1] = x[j + t2], v[l][2] = x[j + t], v[l][3] = x[j + t + t2];
      }
#pragma unroll
      for (int l = 0; l < 2; l++) {
        const uint32_t w = tw[l][m + blk], wq = twq[l][m + blk];
        ct_bf(v[l][0], v[l][2], w, wq, ps[l]);
        ct_bf(v[l][1], v[l][3], w, wq, ps[l]);
        ct_bf(v[l][0], v[l][1], tw[l][2 * m + 2 * blk], twq[l][2 * m + 2 * blk], ps[l]);
        ct_bf(v[l][2], v[l][3], tw[l][2 * m + 2 * blk + 1], twq[l][2 * m + 2 * blk + 1], ps[l]);
      }
#pragma unroll
      for (int l = 0; l < 2; l++) {
        uint32_t* x = xs[l];
        x[j] = v[l][0], x[j + t2] = v[l][1], x[j + t] = v[l][2], x[j + t + t2] = v[l][3];
      }
    }
    __syncthreads();
  }
  if (s < logn) {  // last stage, t = 1
    for (int b = threadIdx.x; b < N / 2; b += CT) {
#pragma unroll
      for (int l = 0; l < 2; l++) {
        uint32_t* x = xs[l];
        uint32_t u = x[2 * b], v = x[2 * b + 1];
        ct_bf(u, v, tw[l][N / 2 + b], twq[l][N / 2 + b], ps[l]);
        x[2 * b] = red2p(red2p(u, 2 * ps[l]), ps[l]);
        x[2 * b + 1] = red2p(red2p(v, 2 * ps[l]), ps[l]);
      }
    }
  } else {
    for (int b = threadIdx.x; b < N; b += CT)
#pragma unroll
      for (int l = 0; l < 2; l++) xs[l][b] = red2p(red2p(xs[l][b], 2 * ps[l]), ps[l]);
  }
  __syncthreads();
}

__device__ __forceinline__ void inv_dual(uint32_t* x0, uint32_t* x1, int logn, const uint32_t* const* tw,
                                         const uint32_t* const* twq, uint32_t p0, uint32_t p1) {
  const int N = 1 << logn;
  uint32_t* xs[2] = {x0, x1};
  const uint32_t ps[2] = {p0, p1};
  int s = 0;
#pragma unroll
  for (; s + 1 < logn; s += 2) {
    const int t = 1 << s;
    const int h0 = N >> (s + 1), h1 = N >> (s + 2);
    for (int g = threadIdx.x; g < N / 4; g += CT) {
      const int blk = g >> s, r = g & (t - 1);
      const int j = (blk << (s + 2)) + r;
      uint32_t v[2][4];
#pragma unroll
      for (int l = 0; l < 2; l++) {
        const uint32_t* x = xs[l];
        v[l][0] = x[j], v[l][1] = x[j + t], v[l][2] = x[j + 2 * t], v[l][3] = x[j + 3 * t];
      }
#pragma unroll
      for (int l = 0; l < 2; l++) {
        gs_bf(v[l][0], v[l][1], tw[l][h0 + 2 * blk], twq[l][h0 + 2 * blk], ps[l]);
        gs_bf(v[l][2], v[l][3], tw[l][h0 + 2 * blk + 1], twq[l][h0 + 2 * blk + 1], ps[l]);
        const uint32_t w = tw[l][h1 + blk], wq = twq[l][h1 + blk];
        gs_bf(v[l][0], v[l][2], w, wq, ps[l]);
        gs_bf(v[l][1], v[l][3], w, wq, ps[l]);
      }
#pragma unroll
      for (int l = 0; l < 2; l++) {
        uint32_t* x = xs[l];
        x[j] = v[l][0], x[j + t] = v[l][1], x[j + 2 * t] = v[l][2], x[j + 3 * t] = v[l][3];
      }
    }
    __syncthreads();
  }
  if (s < logn) {  // last stage, t = N/2
    for (int j = threadIdx.x; j < N / 2; j += CT) {
#pragma unroll
      for (int l = 0; l < 2; l++) {
        uint32_t* x = xs[l];
        uint32_t u = x[j], v = x[j + N / 2];
        gs_bf(u, v, tw[l][1], twq[l][1], ps[l]);
        x[j] = u;
        x[j + N / 2] = v;
      }
    }
    __syncthreads();
  }
}

__device__ __forceinline__ void secondary_dual_body(const ChainArgs& a, int h, int q, int part, uint32_t* sm) {
  const int logn = a.g.log2n;
  const int N = 1 << logn;
  const uint32_t pr0 = a.cp[0].p, pr1 = a.cp[1].p;
  const uint32_t* tws[2] = {sm, sm + 4 * N};
  const uint32_t* twqs[2] = {sm + N, sm + 5 * N};
  const uint32_t* itws[2] = {sm + 2 * N, sm + 6 * N};
  const uint32_t* itwqs[2] = {sm + 3 * N, sm + 7 * N};
  uint32_t* F0 = sm + 8 * N;  // factor blocks: TC[2] at 0, N; D[2] at 2N, 3N; B[2] at 4N, 5N; H at 6N
  const int FS = SEC_PART_WORDS * N;
  const int oTC = 0, oD = 2 * N, oB = 4 * N, oH = 6 * N;
  const uint32_t* qq = a.qv + (size_t)q * a.qv_stride;
  constexpr int PER = N_MAX / CT;
  uint32_t kc[2][6][PER], dst[PER];
#pragma unroll
  for (int c = 0; c < PER; c++) {
    const int pos = threadIdx.x + c * CT;
    if (pos < N) {
#pragma unroll
      for (int p = 0; p < 2; p++) {
        const ChainPrime& cp = a.cp[p];
        const size_t o = (size_t)p * N + pos;
        kc[p][0][c] = mont_reduce((uint64_t)a.gka[o] * cp.r2, cp.p, cp.pinv);
        kc[p][1][c] = mont_reduce((uint64_t)a.gka[2 * (size_t)N + o] * cp.r2, cp.p, cp.pinv);
        kc[p][2][c] = mont_reduce((uint64_t)a.qa[(size_t)h * 2 * N + o] * cp.r2, cp.p, cp.pinv);
        kc[p][3][c] = mont_reduce((uint64_t)qq[o] * cp.r2, cp.p, cp.pinv);
        kc[p][4][c] = mont_reduce((uint64_t)qq[2 * (size_t)N + o] * cp.r2, cp.p, cp.pinv);
        kc[p][5][c] = mont_reduce((uint64_t)qq[(size_t)(4 + h) * 2 * N + o] * cp.r2, cp.p, cp.pinv);
      }
      dst[c] = __ldg(a.galb + pos);
    }
  }
  for (int b = threadIdx.x; b < N; b += CT) {
#pragma unroll
    for (int p = 0; p < 2; p++) {
      sm[4 * p * N + b] = a.T.fw[p][b];
      sm[(4 * p + 1) * N + b] = a.T.fwq[p][b];
      sm[(4 * p + 2) * N + b] = a.T.iw[p][b];
      sm[(4 * p + 3) * N + b] = a.T.iwq[p][b];
      F0[p * FS + oTC + b] = 0;
      F0[p * FS + oD + b] = 0;
      F0[p * FS + oB + b] = 0;
    }
  }
  __syncthreads();
  for (uint32_t i = 0; i < a.g.L; i++) {
    const int cur = (int)(i & 1) * N, nxt = N - cur;
    uint32_t e[2][PER];
#pragma unroll
    for (int p = 0; p < 2; p++) {
      const uint32_t* Ei =
          a.E + ((((size_t)p * a.g.H + h) * a.g.L + a.g.L - 1 - i) * a.nl + (size_t)q * CTXT_PARTS + part) * N;
#pragma unroll
      for (int c = 0; c < PER; c++) {
        const int pos = threadIdx.x + c * CT;
        e[p][c] = pos < N ? __ldg(Ei + pos) : 0;
      }
    }
    inv_dual(F0 + oD + cur, F0 + FS + oD + cur, logn, itws, itwqs, pr0, pr1);
    for (int b = threadIdx.x; b < N; b += CT) {
      const int32_t hd = high_digit(F0[oD + cur + b], F0[FS + oD + cur + b], a.cp[0], a.cp[1]);
      F0[oH + b] = hd < 0 ? (uint32_t)(hd + (int32_t)pr0) : (uint32_t)hd;
      F0[FS + oH + b] = hd < 0 ? (uint32_t)(hd + (int32_t)pr1) : (uint32_t)hd;
    }
    __syncthreads();
    fwd_dual(F0 + oH, F0 + FS + oH, logn, tws, twqs, pr0, pr1);
#pragma unroll
    for (int c = 0; c < PER; c++) {
      const int pos = threadIdx.x + c * CT;
      if (pos < N) {
#pragma unroll
        for (int p = 0; p < 2; p++) {
          const ChainPrime& cp = a.cp[p];
          uint32_t* P = F0 + p * FS;
          const uint32_t n1 = P[oH + pos];
          const uint32_t n0 = sub_mod(P[oTC + cur + pos], mont_reduce((uint64_t)n1 * cp.c26, cp.p, cp.pinv), cp.p);
          const uint32_t an = mont_reduce(
              (uint64_t)n0 * kc[p][0][c] + (uint64_t)n1 * kc[p][1][c] + (uint64_t)e[p][c] * kc[p][2][c], cp.p,
              cp.pinv);
          const uint32_t bn = mont_reduce(((uint64_t)P[oB + cur + pos] << 32) + (uint64_t)n0 * kc[p][3][c] +
                                              (uint64_t)n1 * kc[p][4][c] + (uint64_t)e[p][c] * kc[p][5][c],
                                          cp.p, cp.pinv);
          P[oTC + nxt + dst[c]] = an;
          P[oD + nxt + dst[c]] = an;
          P[oB + nxt + dst[c]] = bn;
        }
      }
    }
    __syncthreads();
  }
  const int fin = (int)(a.g.L & 1) * N;
  uint32_t* o = a.out + ((((size_t)q * a.g.H + h) * CTXT_PARTS + part) * 2) * 2 * N;
#pragma unroll
  for (int c = 0; c < PER; c++) {
    const int pos = threadIdx.x + c * CT;
    if (pos < N) {
#pragma unroll
      for (int p = 0; p < 2; p++) {
        o[(size_t)p * N + pos] = F0[p * FS + oTC + fin + dst[c]];
        o[2 * (size_t)N + (size_t)p * N + pos] = F0[p * FS + oB + fin + dst[c]];
      }
    }
  }
}

// ---- N = 2048, register transforms (ntt2048.cuh): one block carries PARTS of
// the three parts of one query's secondary ciphertext at half h.  A group of
// 256 threads works one part in BOTH factors: thread t owns positions 8t .. 8t
// + 7 of each factor in the first inverse pass, the last forward pass and the
// pointwise stage, and words t + 256 k between the last inverse and the first
// forward pass, where the CRT high digit needs both factors -- so those run
// from registers, the digit needs no exchange, and the groups meet no barrier
// but their own.  The key constants are the same for the three parts and are
// kept once per block.
//
// With r = qry_b / qry_a per slot (both of the secondary query's half) the b
// part is carried as b^ = b - r a, which drops the entries from its recurrence:
//     a' = t ka0 + n1 ka1 + E qa
//     b^' = sigma_5(b^) + t (C + sigma_5(r)) + n1 V
// (t = sigma_5(a), n1 = NTT(d1), ka1 = gk_a1 - 2^26 gk_a0, C = gk_b0 - gk_a0 r,
// V = gk_b1 - 2^26 gk_b0 - ka1 r): five products and five constants a position
// instead of six; b = b^ + r a once at the end.  Where qry_a is zero, r is taken as
// 0 and the slot's b^' keeps its entry, E qry_b: a-parts with such slots (ZEROS) have
// a sixth constant, qry_b there and zero elsewhere.
//
// The state is carried as k a, k the factor's CRT constant: a global scale that
// the constants absorb (ka1 and qa times k, C + sigma_5(r) over k), so that the
// inverse transform's outputs are the CRT terms and the digit needs no products.
//
// Measured (1024 steps, 64 queries): 10.2 ms for the chunk against 16.6 for one
// part per block of 512 threads with one factor per half and a wave of blocks
// per 24 queries.  Three parts keep the heavy FMA pipe 73 % and the L1 /
// shared-memory pipe 83 % busy; the loaded twiddles are a quarter of the latter.
//
// Bounds: a is canonical, b^ below 2p.  The forward transform ends below 2^31
// (ntt.cuh) and n1 is used as it is: t ka0 + n1 ka1 + E qa < 34 p^2, so its
// Montgomery reduction is below 34 p^2 / 2^32 + p < 2p, and b^' stays below 2p
// + 33 p^2 / 2^32 + p < 4p before one subtraction of 2p (p < 2^26).
//
// Shared memory: per part A[2], B[2] (padded polynomials; A is also the
// transforms' work space), then the five constants (Montgomery form) as
// [j][factor][quad half][thread] 16-byte vectors.
constexpr int sec_consts(bool zeros) { return zeros ? 6 : 5; }
constexpr int sec2k_words(bool zeros) { return CTXT_PARTS * 4 * n2k::PS + sec_consts(zeros) * 2 * 2 * 256 * 4; }

// T R^-1 mod p, below T / 2^32 + p (T < 2^62)
__device__ __forceinline__ uint32_t mont_lazy(uint64_t T, uint32_t p, uint32_t pinv) {
  return (uint32_t)((T + (uint64_t)((uint32_t)T * pinv) * p) >> 32);
}

__device__ __forceinline__ double u32_to_double_biased(uint32_t x) {  // 2^52 + x, exactly
  return __hiloint2double(0x43300000, (int)x);
}

// high_digit() from inverse outputs that carry the CRT constants (below 2p):
// the conversions to and from double are additions of 2^52 folded into exact
// fused multiply-adds (x1 P2 and x2 P1 are below 2^51), and floor is the
// rounding mode of the last addition.
__device__ __forceinline__ int32_t high_digit_scaled(uint32_t c1, uint32_t c2) {
  const uint32_t x1 = ntt_detail::red(c1, P1), x2 = ntt_detail::red(c2, P2);
  constexpr double Q = (double)QQ, HALF_Q = (double)(QQ / 2), BIAS = 4503599627370496.0;  // 2^52
  double v = fma(u32_to_double_biased(x1), (double)P2, -BIAS * (double)P2) +
             fma(u32_to_double_biased(x2), (double)P1, -BIAS * (double)P1);
  v = v >= Q ? v - Q : v;
  v = v > HALF_Q ? v - Q : v;
  // 1.5 2^52 + floor(v / 2^26 + 1/2): its low word is the digit
  return __double2loint(__dadd_rd(fma(v, 1.0 / (double)(1u << LOG2_B), 0.5), 1.5 * BIAS));
}

// One radix-8 pass over both factors' polynomials x, x + PS of a 256-thread group.
template <int M, bool INV>
__device__ __forceinline__ void pass8_both(uint32_t* x, int t, const NttTables& T) {
  using Gm = n2k::Geo8<M>;
#pragma unroll
  for (int f = 0; f < 2; f++) {
    const uint32_t p = prime_of(f);
    const n2k::Tw8 tw = n2k::load_tw8(INV ? T.iw2[f] : T.fw2[f], M, Gm::blk(t));
    uint32_t* y = x + f * n2k::PS + Gm::base(t);
    uint32_t v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = y[k * Gm::STR];
    if (INV)
      n2k::inv8_bf(v, tw, p);
    else
      n2k::fwd8_bf(v, tw, p);
#pragma unroll
    for (int k = 0; k < 8; k++) y[k * Gm::STR] = v[k];
  }
}

// Padded words that sigma_5 brings to positions 8t .. 8t + 7, two per register (PS < 2^16).
struct Sources {
  uint32_t w[4];
  __device__ __forceinline__ uint32_t at(int m) const { return m & 1 ? w[m >> 1] >> 16 : w[m >> 1] & 0xFFFFu; }
};

// Transforms of one step on a group's work space x (x, x + PS: the factors):
// from ta = sigma_5(a) at positions 8t .. 8t + 7 to the high digit's forward
// transform after stage 8.  `between` runs before the last pass (loads whose
// latency it covers).  Starts and ends with a barrier of the group.
template <class Sync, class Between>
__device__ __forceinline__ void step_transforms(uint32_t* x, const uint32_t (&ta)[2][8], int t, int qb,
                                                const ChainArgs& a, const Sync& group_sync, const Between& between) {
  using namespace n2k;
  group_sync();
  // inverse stages 0-1 from registers, two quads a factor
#pragma unroll
  for (int f = 0; f < 2; f++) {
    const uint32_t p = prime_of(f);
#pragma unroll
    for (int h4 = 0; h4 < 2; h4++) {
      const Tw4 w = load_tw4(a.T.iw2[f], 2 * t + h4);
      uint4 v = make_uint4(ta[f][4 * h4], ta[f][4 * h4 + 1], ta[f][4 * h4 + 2], ta[f][4 * h4 + 3]);
      gs(v.x, v.y, w.b0, w.b0q, p);
      gs(v.z, v.w, w.b1, w.b1q, p);
      gs(v.x, v.z, w.a, w.aq, p);
      gs(v.y, v.w, w.a, w.aq, p);
      *reinterpret_cast<uint4*>(x + f * PS + qb + 4 * h4) = v;
    }
  }
  group_sync();
  pass8_both<64, true>(x, t, a.T);
  group_sync();
  pass8_both<8, true>(x, t, a.T);
  group_sync();
  {
    // last inverse pass, high digit, first forward pass; words t + 256 k
    uint32_t* const y = x + phys(t);
    constexpr int STR = Geo8<1>::STR;
    uint32_t v[2][8];
#pragma unroll
    for (int f = 0; f < 2; f++) {
#pragma unroll
      for (int k = 0; k < 8; k++) v[f][k] = y[f * PS + k * STR];
      inv8_bf(v[f], param_tw8(a.T.iw7[f]), prime_of(f));
    }
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const int32_t hd = high_digit_scaled(v[0][k], v[1][k]);
      v[0][k] = (uint32_t)(hd + (int32_t)P1), v[1][k] = (uint32_t)(hd + (int32_t)P2);
    }
#pragma unroll
    for (int f = 0; f < 2; f++) {
      fwd8_bf(v[f], param_tw8(a.T.fw7[f]), prime_of(f));
#pragma unroll
      for (int k = 0; k < 8; k++) y[f * PS + k * STR] = v[f][k];
    }
  }
  group_sync();
  pass8_both<8, false>(x, t, a.T);
  group_sync();
  between();
  pass8_both<64, false>(x, t, a.T);
  group_sync();
}

// Forward stages 9-10 at quad h4 of positions 8t .. 8t + 7: values below 2^31.
__device__ __forceinline__ uint4 last_stages(const uint32_t* x, int f, int h4, int t, int qb, const NttTables& T) {
  const uint32_t p = prime_of(f);
  const n2k::Tw4 w = n2k::load_tw4(T.fw2[f], 2 * t + h4);
  uint4 v = *reinterpret_cast<const uint4*>(x + f * n2k::PS + qb + 4 * h4);
  n2k::ct(v.x, v.z, w.a, w.aq, p);
  n2k::ct(v.y, v.w, w.a, w.aq, p);
  n2k::ct(v.x, v.y, w.b0, w.b0q, p);
  n2k::ct(v.z, v.w, w.b1, w.b1q, p);
  return v;
}

// r = qry_b / qry_a of half h of query q at a position of factor f
__device__ __forceinline__ uint32_t query_ratio(const ChainArgs& a, const ScanConsts& sc, int h, int q, int f,
                                                uint32_t pos) {
  const uint32_t p = prime_of(f);
  return mul_mod(__ldg(a.qv + (size_t)q * a.qv_stride + ((size_t)(4 + h) * 2 + f) * N_MAX + pos),
                 __ldg(sc.qinv + (size_t)(h * 2 + f) * N_MAX + __ldg(a.maps.uof + n2k::brv11(pos))), p, barrett_mu(p));
}

// ka0, k ka1, k qa (Montgomery form) at a position of factor f
__device__ __forceinline__ void state_constants(const ChainArgs& a, int h, int f, uint32_t pos, uint32_t* k) {
  const ChainPrime cp = f ? a.cp[1] : a.cp[0];
  const uint64_t mu = barrett_mu(cp.p);
  const size_t o = (size_t)f * N_MAX + pos;
  const uint32_t ga0 = __ldg(a.gka + o);
  const uint32_t ka1 =
      sub_mod(__ldg(a.gka + 2 * (size_t)N_MAX + o), mul_mod(ga0, (1u << LOG2_B) % cp.p, cp.p, mu), cp.p);
  const uint32_t c[3] = {ga0, mul_mod(ka1, cp.k, cp.p, mu),
                         mul_mod(__ldg(a.qa + (size_t)h * 2 * N_MAX + o), cp.k, cp.p, mu)};
#pragma unroll
  for (int j = 0; j < 3; j++) k[j] = mont_reduce((uint64_t)c[j] * cp.r2, cp.p, cp.pinv);
}

// the same, then (C + sigma_5(r)) / k and V (and qry_b where qry_a is zero, for
// ZEROS); from: the position sigma_5 brings here
template <bool ZEROS>
__device__ __forceinline__ void secondary_constants(const ChainArgs& a, const ScanConsts& sc, int h, int q, int f,
                                                    uint32_t pos, uint32_t from, uint32_t* k) {
  state_constants(a, h, f, pos, k);
  const ChainPrime cp = f ? a.cp[1] : a.cp[0];
  const uint64_t mu = barrett_mu(cp.p);
  const size_t o = (size_t)f * N_MAX + pos;
  const uint32_t* qq = a.qv + (size_t)q * a.qv_stride;
  const uint32_t c26 = (1u << LOG2_B) % cp.p, ga0 = __ldg(a.gka + o);
  const uint32_t ka1 = sub_mod(__ldg(a.gka + 2 * (size_t)N_MAX + o), mul_mod(ga0, c26, cp.p, mu), cp.p);
  const uint32_t gb0 = __ldg(qq + o), gb1 = __ldg(qq + 2 * (size_t)N_MAX + o);
  const uint32_t r = query_ratio(a, sc, h, q, f, pos), r5 = query_ratio(a, sc, h, q, f, from);
  const uint32_t C = sub_mod(gb0, mul_mod(ga0, r, cp.p, mu), cp.p);
  const uint32_t V = sub_mod(sub_mod(gb1, mul_mod(gb0, c26, cp.p, mu), cp.p), mul_mod(ka1, r, cp.p, mu), cp.p);
  k[3] = mont_reduce((uint64_t)mul_mod(add_mod(C, r5, cp.p), cp.kinv, cp.p, mu) * cp.r2, cp.p, cp.pinv);
  k[4] = mont_reduce((uint64_t)V * cp.r2, cp.p, cp.pinv);
  if constexpr (ZEROS) {
    const uint32_t qb = __ldg(qq + ((size_t)(4 + h) * 2 + f) * N_MAX + pos);
    k[5] = __ldg(a.qa + (size_t)h * 2 * N_MAX + o) ? 0 : mont_reduce((uint64_t)qb * cp.r2, cp.p, cp.pinv);
  }
}

template <bool ZEROS>
__global__ void __launch_bounds__(256 * CTXT_PARTS, 1) secondary_chain2k_kernel(ChainArgs a, ScanConsts sc) {
  extern __shared__ __align__(16) uint32_t sm[];
  using namespace n2k;
  constexpr int NKC = sec_consts(ZEROS);
  constexpr int PARTS = CTXT_PARTS, NT = 256 * PARTS;
  const int h = blockIdx.x, q = blockIdx.y;
  const int part = threadIdx.x >> 8, t = threadIdx.x & 255;
  uint32_t* const A = sm + part * 4 * PS;
  uint32_t* const B = A + 2 * PS;
  uint4* const KC = reinterpret_cast<uint4*>(sm + PARTS * 4 * PS);
  const int qb = (int)phys(8 * t);  // positions 8t .. 8t + 7 sit in one padded row: qb .. qb + 7
  auto group_sync = [&] { asm volatile("bar.sync %0, 256;" ::"r"(1 + part) : "memory"); };
  // sigma_5 sources of the positions (galb inverted through the constants' space)
  uint32_t* const inv = sm + PARTS * 4 * PS;
  for (int b = threadIdx.x; b < N; b += NT) inv[__ldg(a.galb + b)] = b;
  for (int b = threadIdx.x; b < PARTS * 4 * PS; b += NT) sm[b] = 0;  // a = b^ = 0
  __syncthreads();
  Sources src;
#pragma unroll
  for (int m = 0; m < 4; m++) src.w[m] = phys(inv[8 * t + 2 * m]) | (phys(inv[8 * t + 2 * m + 1]) << 16);
  // the constants of position quads, dealt over the whole block: item = (factor, quad)
  {
    constexpr int PER = (2 * N + NT - 1) / NT;
    uint32_t from[PER];
#pragma unroll
    for (int c = 0; c < PER; c++) from[c] = inv[(threadIdx.x + c * NT) & (N - 1)];
    __syncthreads();  // the table is overwritten by the constants
    // (not unrolled, as in few_chain)
#pragma unroll 1
    for (int c = 0; c < PER; c++) {
      const int it = threadIdx.x + c * NT;
      if (it < 2 * N) {
        const int f = it / N, pos = it & (N - 1);
        uint32_t k[NKC];
        uint32_t src_pos = from[0];
#pragma unroll
        for (int x = 1; x < PER; x++) src_pos = c == x ? from[x] : src_pos;
        secondary_constants<ZEROS>(a, sc, h, q, f, pos, src_pos, k);
#pragma unroll
        for (int j = 0; j < NKC; j++)
          reinterpret_cast<uint32_t*>(KC)[(((j * 2 + f) * 2 + (pos >> 2 & 1)) * 256 + (pos >> 3)) * 4 + (pos & 3)] = k[j];
      }
    }
  }
  __syncthreads();
  const size_t lane = (size_t)q * CTXT_PARTS + part;
  const uint4* Erow = reinterpret_cast<const uint4*>(a.E + ((size_t)h * a.g.L * a.nl + lane) * N) + 2 * t;
  const size_t erow_stride = (size_t)a.nl * N / 4;             // uint4 per row
  const size_t efac = (size_t)a.g.H * a.g.L * a.nl * (N / 4);  // uint4 per factor
  for (uint32_t i = 0; i < a.g.L; i++) {
    // t = sigma_5(a), kept for the pointwise stage
    uint32_t ta[2][8];
#pragma unroll
    for (int f = 0; f < 2; f++)
#pragma unroll
      for (int m = 0; m < 8; m++) ta[f][m] = A[f * PS + src.at(m)];
    uint4 e[2][2];  // entries of the step
    step_transforms(A, ta, t, qb, a, group_sync, [&] {
#pragma unroll
      for (int f = 0; f < 2; f++)
#pragma unroll
        for (int h4 = 0; h4 < 2; h4++) e[f][h4] = __ldg(Erow + f * efac + (a.g.L - 1 - i) * erow_stride + h4);
    });
    // forward stages 9-10 and the pointwise stage at the two quads
    uint4 bn[2][2];
#pragma unroll
    for (int f = 0; f < 2; f++) {
      const uint32_t p = prime_of(f), pinv = f ? a.cp[1].pinv : a.cp[0].pinv;
#pragma unroll
      for (int h4 = 0; h4 < 2; h4++) {
        const uint4 v = last_stages(A, f, h4, t, qb, a.T);
        const uint32_t n1[4] = {v.x, v.y, v.z, v.w};
        const uint32_t es[4] = {e[f][h4].x, e[f][h4].y, e[f][h4].z, e[f][h4].w};
        uint32_t kc[NKC][4], an[4], b4[4];
#pragma unroll
        for (int j = 0; j < NKC; j++) {
          const uint4 c = KC[((j * 2 + f) * 2 + h4) * 256 + t];
          kc[j][0] = c.x, kc[j][1] = c.y, kc[j][2] = c.z, kc[j][3] = c.w;
        }
#pragma unroll
        for (int m = 0; m < 4; m++) {
          const int j = 4 * h4 + m;
          const uint32_t tt = ta[f][j], tb = B[f * PS + src.at(j)];
          an[m] = red(mont_lazy((uint64_t)tt * kc[0][m] + (uint64_t)n1[m] * kc[1][m] + (uint64_t)es[m] * kc[2][m], p,
                                pinv),
                      p);
          uint64_t bt = ((uint64_t)tb << 32) + (uint64_t)tt * kc[3][m] + (uint64_t)n1[m] * kc[4][m];
          if constexpr (ZEROS) bt += (uint64_t)es[m] * kc[5][m];
          b4[m] = red(mont_lazy(bt, p, pinv), 2 * p);
        }
        *reinterpret_cast<uint4*>(A + f * PS + qb + 4 * h4) = make_uint4(an[0], an[1], an[2], an[3]);
        bn[f][h4] = make_uint4(b4[0], b4[1], b4[2], b4[3]);
      }
    }
    group_sync();  // every gather of b^ is done
#pragma unroll
    for (int f = 0; f < 2; f++)
#pragma unroll
      for (int h4 = 0; h4 < 2; h4++) *reinterpret_cast<uint4*>(B + f * PS + qb + 4 * h4) = bn[f][h4];
  }
  uint32_t* o = a.out + ((((size_t)q * a.g.H + h) * CTXT_PARTS + part) * 2) * 2 * N;
#pragma unroll 1
  for (int f = 0; f < 2; f++) {
    const uint32_t p = prime_of(f);
#pragma unroll 1
    for (int m = 0; m < 8; m++) {
      const uint32_t av = mul_mod(A[f * PS + qb + m], f ? a.cp[1].kinv : a.cp[0].kinv, p, barrett_mu(p));
      const uint32_t br = red(B[f * PS + qb + m], p);
      o[(size_t)f * N + 8 * t + m] = av;
      o[2 * (size_t)N + (size_t)f * N + 8 * t + m] =
          add_mod(br, mul_mod(av, query_ratio(a, sc, h, q, f, 8 * t + m), p, barrett_mu(p)), p);
    }
  }
}

// Preprocessing chain at N = 2048 with two stored arrays: one chain (shard,
// half, lane) per block of 256 threads on the same step, without a b part.
// Rows of the chain layout, E on input, take the state k a' in their place; the
// canonical high digits' transforms go to `digits`, the same layout.  Three
// blocks fit an SM (67 KiB, 80 registers).  Taken by calls of more chains than SMs,
// which are of order 512 or less: shards of larger orders fill a call's scratch with
// 104 chains (preprocess_batch).  160 chains of 512 steps 4.2 ms; 144 on one SM
// each (below) 2.05.
constexpr int PRIM2K_KC = 3;
constexpr int PRIM2K_WORDS = 2 * n2k::PS + PRIM2K_KC * 2 * 2 * 256 * 4;

__global__ void __launch_bounds__(256, 3) primary_chain2k_kernel(ChainArgs a, uint32_t* rows, uint32_t* digits,
                                                                 size_t shard_words) {
  extern __shared__ __align__(16) uint32_t sm[];
  using namespace n2k;
  const int t = threadIdx.x, h = blockIdx.x % a.g.H, lane = blockIdx.x / a.g.H, s = blockIdx.y;
  uint32_t* const A = sm;
  uint4* const KC = reinterpret_cast<uint4*>(sm + 2 * PS);
  uint32_t* const inv = sm + 2 * PS;
  const int qb = (int)phys(8 * t);
  for (int b = t; b < N; b += 256) inv[__ldg(a.galb + b)] = b;
  for (int b = t; b < 2 * PS; b += 256) A[b] = 0;
  __syncthreads();
  Sources src;
#pragma unroll
  for (int m = 0; m < 4; m++) src.w[m] = phys(inv[8 * t + 2 * m]) | (phys(inv[8 * t + 2 * m + 1]) << 16);
  __syncthreads();  // the table is overwritten by the constants, each thread reading only its own
#pragma unroll 1
  for (int fm = 0; fm < 16; fm++) {  // (not unrolled, as in few_chain)
    const int f = fm >> 3, m = fm & 7;
    uint32_t k[PRIM2K_KC];
    state_constants(a, h, f, 8 * t + m, k);
#pragma unroll
    for (int j = 0; j < PRIM2K_KC; j++)
      reinterpret_cast<uint32_t*>(KC)[(((j * 2 + f) * 2 + (m >> 2)) * 256 + t) * 4 + (m & 3)] = k[j];
  }
  const size_t first = (size_t)s * shard_words + ((size_t)h * a.g.L * SIMD + lane) * N + 8 * t;
  const size_t row_stride = (size_t)SIMD * N, efac = (size_t)a.g.H * a.g.L * row_stride;
  for (uint32_t i = 0; i < a.g.L; i++) {
    const size_t row = first + (a.g.L - 1 - i) * row_stride;
    uint32_t ta[2][8];
#pragma unroll
    for (int f = 0; f < 2; f++)
#pragma unroll
      for (int m = 0; m < 8; m++) ta[f][m] = A[f * PS + src.at(m)];
    uint4 e[2][2];  // entries of the step (plain loads: the row is rewritten below)
    step_transforms(A, ta, t, qb, a, [] { __syncthreads(); }, [&] {
#pragma unroll
      for (int f = 0; f < 2; f++)
#pragma unroll
        for (int h4 = 0; h4 < 2; h4++) e[f][h4] = *reinterpret_cast<const uint4*>(rows + row + f * efac + 4 * h4);
    });
#pragma unroll
    for (int f = 0; f < 2; f++) {
      const uint32_t p = prime_of(f), pinv = f ? a.cp[1].pinv : a.cp[0].pinv;
#pragma unroll
      for (int h4 = 0; h4 < 2; h4++) {
        const uint4 v = last_stages(A, f, h4, t, qb, a.T);
        const uint32_t n1[4] = {v.x, v.y, v.z, v.w};
        const uint32_t es[4] = {e[f][h4].x, e[f][h4].y, e[f][h4].z, e[f][h4].w};
        const uint4 k0 = KC[(f * 2 + h4) * 256 + t], k1 = KC[((2 + f) * 2 + h4) * 256 + t],
                    k2 = KC[((4 + f) * 2 + h4) * 256 + t];
        const uint32_t kc[PRIM2K_KC][4] = {
            {k0.x, k0.y, k0.z, k0.w}, {k1.x, k1.y, k1.z, k1.w}, {k2.x, k2.y, k2.z, k2.w}};
        uint32_t an[4];
#pragma unroll
        for (int m = 0; m < 4; m++)
          an[m] = red(mont_lazy((uint64_t)ta[f][4 * h4 + m] * kc[0][m] + (uint64_t)n1[m] * kc[1][m] +
                                    (uint64_t)es[m] * kc[2][m],
                                p, pinv),
                      p);
        const uint4 x = make_uint4(an[0], an[1], an[2], an[3]);
        *reinterpret_cast<uint4*>(A + f * PS + qb + 4 * h4) = x;
        *reinterpret_cast<uint4*>(rows + row + f * efac + 4 * h4) = x;
        *reinterpret_cast<uint4*>(digits + row + f * efac + 4 * h4) =
            make_uint4(canon(n1[0], p), canon(n1[1], p), canon(n1[2], p), canon(n1[3], p));
      }
    }
    __syncthreads();
  }
  uint32_t* o = a.a_out + (((size_t)s * a.g.H + h) * SIMD + lane) * 2 * N;
#pragma unroll
  for (int f = 0; f < 2; f++)
#pragma unroll
    for (int m = 0; m < 8; m++)
      o[(size_t)f * N + 8 * t + m] = mul_mod(A[f * PS + qb + m], f ? a.cp[1].kinv : a.cp[0].kinv, prime_of(f),
                                             barrett_mu(prime_of(f)));
}

// ---- The same two chains when they are few: 256 threads per factor, so that a
// step is half as long for a thread.  PAIR: the factors' threads are the two
// blocks of a cluster, on two SMs while there are two for every chain -- a
// chain alone on one SM keeps its heavy FMA pipe 60 % busy, so the second SM
// is what shortens the step (2.06 us against 3.66).  Otherwise they are the two
// halves of one 512-thread block (up to one chain per SM).  The factors send each
// other their inverse outputs:
// every thread writes its eight values into the other's inbox (double-buffered
// by step parity, so that one may run ahead of the other's reads) before the
// one barrier of a step that both meet.  F: the factor, so that primes and
// shared twiddles are constants of its code.
// As pairs the inbox fills by st.async, which counts its bytes on the
// receiver's mbarrier: no barrier of the cluster and no fence in a step.  A wait
// is bounded.  When it gives up, which the threads of a block do together or not at
// all, the block raises the error word and ends there: it arms and sends no more,
// so the peer's next wait runs out too.  That path never comes back, which keeps
// it out of the steps' code: one query's 1024 steps as long as without it (2.64 ms the
// call), a shard's 0.7 % longer; with a way out of the loop, a guard around the
// sends or a flag asked in each step they took 1 to 5 % longer.
// The states a and b^ are kept apart from the transforms' work space and
// transposed, position 8 t + m at word 256 m + t: sigma_5 maps a warp's
// positions of one m to 32 positions whose t differ mod 32, so its gathers have
// no bank conflict (three-way in the padded order), and the first pass may
// write its work space without waiting for them.
constexpr int few_words(int kc) {  // of one factor: work space, a, b^ (secondary), inbox[2], constants, two
                                   // mbarriers, the peer's steps (12 bytes spare)
  return n2k::PS + (kc > 3 ? 4 : 3) * N_MAX + kc * 2 * 256 * 4 + 8;
}
__device__ __forceinline__ uint32_t state_word(uint32_t pos) { return ((pos & 7) << 8) | (pos >> 3); }

__device__ __forceinline__ bool peer_done(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, "
      "p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// The same until limit_ns have passed (and one look after them: the thread may
// have been held up between the last one and the clock).
__device__ __forceinline__ bool peer_done_within(uint32_t bar, uint32_t parity, uint64_t limit_ns) {
  uint64_t t0, t1;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  do {
    if (peer_done(bar, parity)) return true;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
  } while (t1 - t0 <= limit_ns);
  return peer_done(bar, parity);
}
// Waits, in all 256 threads of a block, for the phase of `parity` of a barrier
// that the peer block's copies complete; false in all of them or in none.  A thread
// whose time is up makes the phase wait for one byte more: if the phase was still
// open then, it now stays open for the others too; if it had just completed, the
// byte went to the next phase, which cannot have begun to complete while this
// thread is here, and is taken back.
__device__ __forceinline__ bool wait_peer(uint32_t bar, uint32_t parity, uint64_t limit_ns) {
  if (peer_done_within(bar, parity, limit_ns)) return true;
  asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
  if (!peer_done(bar, parity)) return false;
  asm volatile("mbarrier.complete_tx.relaxed.cta.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
  return true;
}
// Expects the peer's values of one step (256 threads, 32 bytes each).
__device__ __forceinline__ void arm_inbox(uint32_t bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(256 * 32) : "memory");
}
constexpr uint32_t PEER_SENT = 16;  // byte offset of the peer's number of steps sent from the barriers
// End of a paired chain, for all threads of the block: neither block leaves while
// the peer may still write into it.  `waited` steps' values have come, `sent` are
// armed and sent (one more when a wait has given up).  Stores of st.async are not
// ordered by the cluster barrier, so a block that leaves early waits, bounded again,
// for those that its peer had sent besides (at most two steps': a block sends step
// i + 2 only after the peer's step i + 1 has come).
__device__ __noinline__ void leave_pair(uint32_t bars, uint32_t peer_bars, uint32_t waited, uint32_t sent, uint32_t L,
                                        int t, uint64_t limit_ns) {
  if (t == 0 && sent < L)
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(peer_bars + PEER_SENT), "r"(sent) : "memory");
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
  if (t != 0) return;
  if (sent > waited)  // the bytes of the threads' waits that gave up
    asm volatile("mbarrier.complete_tx.relaxed.cta.shared::cta.b64 [%0], 256;" ::"r"(bars + (waited & 1) * 8) : "memory");
  uint32_t peer_sent;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(peer_sent) : "r"(bars + PEER_SENT) : "memory");
  for (uint32_t j = waited; j < peer_sent; j++) {
    const uint32_t bar = bars + (j & 1) * 8;
    if (j >= sent) arm_inbox(bar);
    peer_done_within(bar, (j >> 1) & 1, limit_ns);
  }
}

template <int F, bool SEC, bool PAIR, bool ZEROS>
__device__ __forceinline__ void few_chain(const ChainArgs& a, const ScanConsts& sc, uint32_t* sm, int h, int q,
                                           int unit, uint32_t* rows, uint32_t* digits) {
  using namespace n2k;
  constexpr int NKC = SEC ? sec_consts(ZEROS) : PRIM2K_KC;
  constexpr uint32_t p = F ? P2 : P1;
  constexpr int WORDS = few_words(NKC), XO = PS + (SEC ? 2 : 1) * N;
  const int t = threadIdx.x & 255;
  uint32_t* const A = sm + (PAIR ? 0 : F * WORDS);  // work space
  uint32_t* const S = A + PS;                       // a
  uint32_t* const B = S + N;                        // b^
  uint32_t* const X = A + XO;  // inbox: [parity][half of 8][t] 16-byte vectors
  uint4* const KC = reinterpret_cast<uint4*>(X + 2 * N);  // [j][quad half][t]
  // barrier of this factor's threads, and of both factors'
  auto sync = [] {
    if constexpr (PAIR)
      __syncthreads();
    else
      asm volatile("bar.sync %0, 256;" ::"n"(1 + F) : "memory");
  };
  auto sync_both = [] {
    if constexpr (PAIR)
      asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    else
      asm volatile("bar.sync 3, 512;" ::: "memory");
  };
  const int qb = (int)phys(8 * t);
  // sigma_5 sources (galb inverted through X), a = b^ = 0, constants
  for (int b = t; b < N; b += 256) {
    X[__ldg(a.galb + b)] = b;
    S[b] = 0;
    if (SEC) B[b] = 0;
  }
  sync();
  Sources src;
#pragma unroll
  for (int m = 0; m < 4; m++) src.w[m] = state_word(X[8 * t + 2 * m]) | (state_word(X[8 * t + 2 * m + 1]) << 16);
  // (not unrolled: eight copies of this code, run once, cost more to fetch than to
  // run -- 47 us of set-up instead of 21)
#pragma unroll 1
  for (int m = 0; m < 8; m++) {
    uint32_t k[NKC];
    if constexpr (SEC)
      secondary_constants<ZEROS>(a, sc, h, q, F, 8 * t + m, X[8 * t + m], k);
    else
      state_constants(a, h, F, 8 * t + m, k);
#pragma unroll
    for (int j = 0; j < NKC; j++)
      reinterpret_cast<uint32_t*>(KC)[((j * 2 + (m >> 2)) * 256 + t) * 4 + (m & 3)] = k[j];
  }
  // shared::cluster address of the other factor's inbox
  uint32_t peer = (uint32_t)__cvta_generic_to_shared(PAIR ? X : sm + (1 - F) * WORDS + XO);
  if constexpr (PAIR) asm("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(peer) : "r"(1 - F));
  // PAIR: one mbarrier per parity, behind the constants; its phase i / 2 ends with
  // the peer's 8 KiB of step i.  The steps that the peer has sent lie behind them.
  const uint32_t bars = (uint32_t)__cvta_generic_to_shared(KC + NKC * 2 * 256);
  const uint32_t peer_bars = peer + (bars - (uint32_t)__cvta_generic_to_shared(X));
  const uint32_t steps = PAIR && F == 1 && blockIdx.x < 2 && blockIdx.y == 0 ? min(a.g.L, a.withhold) : a.g.L;
  if (PAIR && t == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n\tmbarrier.init.shared::cta.b64 [%0 + 8], 1;\n\t"
                 "fence.mbarrier_init.release.cluster;" ::"r"(bars)
                 : "memory");
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(bars + PEER_SENT), "r"(a.g.L) : "memory");
  }
  sync_both();  // both run, both inboxes are free and the barriers exist
  const size_t lanes = SEC ? (size_t)a.nl : SIMD;
  const size_t first = (((size_t)F * a.g.H + h) * a.g.L * lanes + unit) * N + 8 * t;
  const Tw4 iw0 = load_tw4(a.T.iw2[F], 2 * t), iw1 = load_tw4(a.T.iw2[F], 2 * t + 1);
  const Tw4 fw0 = load_tw4(a.T.fw2[F], 2 * t), fw1 = load_tw4(a.T.fw2[F], 2 * t + 1);
  constexpr uint32_t pinv = neg_inv32(p);
  // a thread's groups are the same in every step: its twiddles stay in registers
  // (loading them in every pass put their latency behind each barrier: 3.5 ms per
  // 1024 steps instead of 2.7 as pairs, 4.4 instead of 3.8 as wide blocks, although
  // those have 128 registers a thread and spill some)
  const Tw8 i64 = load_tw8(a.T.iw2[F], 64, Geo8<64>::blk(t)), i8 = load_tw8(a.T.iw2[F], 8, Geo8<8>::blk(t));
  const Tw8 f64 = load_tw8(a.T.fw2[F], 64, Geo8<64>::blk(t)), f8 = load_tw8(a.T.fw2[F], 8, Geo8<8>::blk(t));
  auto radix8 = [&](auto m, bool inverse, const Tw8& tw) {
    constexpr int M = decltype(m)::value;
    using Gm = Geo8<M>;
    uint32_t* y = A + Gm::base(t);
    uint32_t v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = y[k * Gm::STR];
    if (inverse)
      inv8_bf(v, tw, p);
    else
      fwd8_bf(v, tw, p);
#pragma unroll
    for (int k = 0; k < 8; k++) y[k * Gm::STR] = v[k];
  };
  for (uint32_t i = 0; i < steps; i++) {
    const size_t row = first + (size_t)(a.g.L - 1 - i) * lanes * N;
    uint32_t ta[8], tb[8];
#pragma unroll
    for (int m = 0; m < 8; m++) ta[m] = S[src.at(m)];
    if (SEC) {
#pragma unroll
      for (int m = 0; m < 8; m++) tb[m] = B[src.at(m)];
    }
    uint4 e[2];  // entries of the step
#pragma unroll
    for (int h4 = 0; h4 < 2; h4++)
      e[h4] = SEC ? __ldg(reinterpret_cast<const uint4*>(a.E + row) + h4)
                  : *(reinterpret_cast<const uint4*>(rows + row) + h4);
#pragma unroll
    for (int h4 = 0; h4 < 2; h4++) {
      const Tw4& w = h4 ? iw1 : iw0;
      uint4 v = make_uint4(ta[4 * h4], ta[4 * h4 + 1], ta[4 * h4 + 2], ta[4 * h4 + 3]);
      gs(v.x, v.y, w.b0, w.b0q, p);
      gs(v.z, v.w, w.b1, w.b1q, p);
      gs(v.x, v.z, w.a, w.aq, p);
      gs(v.y, v.w, w.a, w.aq, p);
      *reinterpret_cast<uint4*>(A + qb + 4 * h4) = v;
    }
    sync();
    radix8(std::integral_constant<int, 64>(), true, i64);
    sync();
    radix8(std::integral_constant<int, 8>(), true, i8);
    sync();
    {
      uint32_t* const y = A + phys(t);
      constexpr int STR = Geo8<1>::STR;
      const uint32_t xo = ((i & 1) * 512 + t) * 16;  // bytes into X
      uint32_t v[8];
#pragma unroll
      for (int k = 0; k < 8; k++) v[k] = y[k * STR];
      inv8_bf(v, param_tw8(a.T.iw7[F]), p);
      if constexpr (PAIR) {
        const uint32_t bo = (i & 1) * 8;
#pragma unroll
        for (int h4 = 0; h4 < 2; h4++)
          asm volatile(
              "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                  peer + xo + h4 * 4096),
              "r"(v[4 * h4]), "r"(v[4 * h4 + 1]), "r"(v[4 * h4 + 2]), "r"(v[4 * h4 + 3]), "r"(peer_bars + bo)
              : "memory");
        // (copies may land before this: the count may run below zero meanwhile)
        if (t == 0) arm_inbox(bars + bo);
        if (!wait_peer(bars + bo, (i >> 1) & 1, a.wait_ns)) {
          if (t == 0) atomicOr(a.err, 1u);
          leave_pair(bars, peer_bars, i, i + 1, a.g.L, t, a.wait_ns);
          asm volatile("exit;");
          __builtin_unreachable();
        }
      } else {
#pragma unroll
        for (int h4 = 0; h4 < 2; h4++)
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(peer + xo + h4 * 4096), "r"(v[4 * h4]),
                       "r"(v[4 * h4 + 1]), "r"(v[4 * h4 + 2]), "r"(v[4 * h4 + 3])
                       : "memory");
        sync_both();
      }
#pragma unroll
      for (int h4 = 0; h4 < 2; h4++) {
        const uint4 x = *reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(X) + xo + h4 * 4096);
        const uint32_t o[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int m = 0; m < 4; m++) {
          uint32_t& w = v[4 * h4 + m];
          w = (uint32_t)((F ? high_digit_scaled(o[m], w) : high_digit_scaled(w, o[m])) + (int32_t)p);
        }
      }
      fwd8_bf(v, param_tw8(a.T.fw7[F]), p);
#pragma unroll
      for (int k = 0; k < 8; k++) y[k * STR] = v[k];
    }
    sync();
    radix8(std::integral_constant<int, 8>(), false, f8);
    sync();
    radix8(std::integral_constant<int, 64>(), false, f64);
    sync();
#pragma unroll
    for (int h4 = 0; h4 < 2; h4++) {
      const Tw4& w = h4 ? fw1 : fw0;
      uint4 v = *reinterpret_cast<const uint4*>(A + qb + 4 * h4);
      ct(v.x, v.z, w.a, w.aq, p);
      ct(v.y, v.w, w.a, w.aq, p);
      ct(v.x, v.y, w.b0, w.b0q, p);
      ct(v.z, v.w, w.b1, w.b1q, p);
      const uint32_t n1[4] = {v.x, v.y, v.z, v.w};
      const uint32_t es[4] = {e[h4].x, e[h4].y, e[h4].z, e[h4].w};
      uint32_t kc[NKC][4], an[4], bn[4];
#pragma unroll
      for (int j = 0; j < NKC; j++) {
        const uint4 c = KC[(j * 2 + h4) * 256 + t];
        kc[j][0] = c.x, kc[j][1] = c.y, kc[j][2] = c.z, kc[j][3] = c.w;
      }
#pragma unroll
      for (int m = 0; m < 4; m++) {
        const uint32_t tt = ta[4 * h4 + m];
        an[m] = red(mont_lazy((uint64_t)tt * kc[0][m] + (uint64_t)n1[m] * kc[1][m] + (uint64_t)es[m] * kc[2][m], p, pinv),
                    p);
        if constexpr (SEC) {
          uint64_t bt = ((uint64_t)tb[4 * h4 + m] << 32) + (uint64_t)tt * kc[3][m] + (uint64_t)n1[m] * kc[4][m];
          if constexpr (ZEROS) bt += (uint64_t)es[m] * kc[5][m];
          bn[m] = red(mont_lazy(bt, p, pinv), 2 * p);
        }
      }
#pragma unroll
      for (int m = 0; m < 4; m++) {
        S[256 * (4 * h4 + m) + t] = an[m];
        if constexpr (SEC) B[256 * (4 * h4 + m) + t] = bn[m];
      }
      if constexpr (!SEC) {
        *(reinterpret_cast<uint4*>(rows + row) + h4) = make_uint4(an[0], an[1], an[2], an[3]);
        *(reinterpret_cast<uint4*>(digits + row) + h4) =
            make_uint4(canon(n1[0], p), canon(n1[1], p), canon(n1[2], p), canon(n1[3], p));
      }
    }
    sync();
  }
  if constexpr (PAIR) leave_pair(bars, peer_bars, steps, steps, a.g.L, t, a.wait_ns);
  constexpr uint64_t mu = barrett_mu(p);
  const uint32_t kinv = a.cp[F].kinv;
#pragma unroll 1
  for (int m = 0; m < 8; m++) {
    const uint32_t av = mul_mod(S[256 * m + t], kinv, p, mu), pos = 8 * t + m;
    if constexpr (SEC) {
      uint32_t* o = a.out + (((size_t)q * a.g.H + h) * CTXT_PARTS + (unit - q * CTXT_PARTS)) * 4 * N + F * N + pos;
      o[0] = av;
      o[2 * N] = add_mod(red(B[256 * m + t], p), mul_mod(av, query_ratio(a, sc, h, q, F, pos), p, mu), p);
    } else {
      a.a_out[((size_t)h * SIMD + unit) * 2 * N + F * N + pos] = av;
    }
  }
}

// grid: x = part * H + half (times 2, + factor, as pairs), y = query
template <bool PAIR, bool ZEROS>
__device__ __forceinline__ void few_secondary(const ChainArgs& a, const ScanConsts& sc, uint32_t* sm) {
  const int c = PAIR ? blockIdx.x >> 1 : blockIdx.x, f = PAIR ? blockIdx.x & 1 : threadIdx.x >> 8;
  const int h = c % a.g.H, q = blockIdx.y, unit = q * CTXT_PARTS + c / a.g.H;
  if (f == 0)
    few_chain<0, true, PAIR, ZEROS>(a, sc, sm, h, q, unit, nullptr, nullptr);
  else
    few_chain<1, true, PAIR, ZEROS>(a, sc, sm, h, q, unit, nullptr, nullptr);
}
template <bool ZEROS>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(256, 1) secondary_chain_pair_kernel(ChainArgs a,
                                                                                               ScanConsts sc) {
  extern __shared__ __align__(16) uint32_t sm[];
  few_secondary<true, ZEROS>(a, sc, sm);
}
template <bool ZEROS>
__global__ void __launch_bounds__(512, 1) secondary_chain_wide_kernel(ChainArgs a, ScanConsts sc) {
  extern __shared__ __align__(16) uint32_t sm[];
  few_secondary<false, ZEROS>(a, sc, sm);
}

// grid: x = lane * H + half (times 2, + factor, as pairs), y = shard
template <bool PAIR>
__device__ __forceinline__ void few_primary(ChainArgs& a, uint32_t* rows, uint32_t* digits, size_t shard_words,
                                            uint32_t* sm) {
  const int c = PAIR ? blockIdx.x >> 1 : blockIdx.x, f = PAIR ? blockIdx.x & 1 : threadIdx.x >> 8;
  const int h = c % a.g.H, s = blockIdx.y, lane = c / a.g.H;
  rows += s * shard_words, digits += s * shard_words;
  a.a_out += (size_t)s * a.g.H * SIMD * 2 * N_MAX;
  if (f == 0)
    few_chain<0, false, PAIR, false>(a, ScanConsts(), sm, h, 0, lane, rows, digits);
  else
    few_chain<1, false, PAIR, false>(a, ScanConsts(), sm, h, 0, lane, rows, digits);
}
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(256, 1)
    primary_chain_pair_kernel(ChainArgs a, uint32_t* rows, uint32_t* digits, size_t shard_words) {
  extern __shared__ __align__(16) uint32_t sm[];
  few_primary<true>(a, rows, digits, shard_words, sm);
}
__global__ void __launch_bounds__(512, 1)
    primary_chain_wide_kernel(ChainArgs a, uint32_t* rows, uint32_t* digits, size_t shard_words) {
  extern __shared__ __align__(16) uint32_t sm[];
  few_primary<false>(a, rows, digits, shard_words, sm);
}

// Rows of the chain layout (bit-reversed positions) to (sign, e) order, in
// place; one block per row.
__global__ void __launch_bounds__(256) order_rows_kernel(uint32_t* rows, const uint32_t* __restrict__ gtab) {
  __shared__ uint4 sm[N_MAX / 4];
  uint4* const row = reinterpret_cast<uint4*>(rows + (size_t)blockIdx.x * N_MAX);
  const uint32_t* w = reinterpret_cast<const uint32_t*>(sm);
#pragma unroll
  for (int c = 0; c < 2; c++) sm[threadIdx.x + 256 * c] = row[threadIdx.x + 256 * c];
  __syncthreads();
#pragma unroll
  for (int c = 0; c < 2; c++) {
    const int q = threadIdx.x + 256 * c;
    const uint4 g = __ldg(reinterpret_cast<const uint4*>(gtab) + q);
    row[q] = make_uint4(w[n2k::brv11((g.x - 1) >> 1)], w[n2k::brv11((g.y - 1) >> 1)], w[n2k::brv11((g.z - 1) >> 1)],
                        w[n2k::brv11((g.w - 1) >> 1)]);
  }
}

// Chain-layout rows of the 8 lanes (states and digits) to a shard's lane
// layout; one block per (factor, half, row) and array.  Position u = (sign, e)
// of row r holds slot (sign, e + r) (slab_off: row i = L - 1 - r).
constexpr int LANE_PAD = N_MAX + 4;
__global__ void __launch_bounds__(512) lane_rows_kernel(const uint32_t* __restrict__ rows,
                                                        const uint32_t* __restrict__ digits,
                                                        uint32_t* __restrict__ slab, Group g,
                                                        const uint32_t* __restrict__ gtab) {
  extern __shared__ __align__(16) uint32_t sm[];  // [8][LANE_PAD]
  const uint32_t r = blockIdx.x % g.L, ph = blockIdx.x / g.L, h = ph % g.H, p = ph / g.H;
  const int arr = blockIdx.y;
  const uint4* src = reinterpret_cast<const uint4*>((arr ? digits : rows) + (size_t)blockIdx.x * SIMD * N_MAX);
  for (int q = threadIdx.x; q < SIMD * N_MAX / 4; q += 512)
    *reinterpret_cast<uint4*>(sm + (q >> 9) * LANE_PAD + 4 * (q & 511)) = __ldg(src + q);
  __syncthreads();
  uint32_t* const dst = slab + slab_off(g, (int)p, (int)h, g.L - 1 - r, arr, 0);
  for (int x = threadIdx.x; x < 2 * N_MAX; x += 512) {
    const uint32_t u = x >> 1, l0 = (x & 1) * 4;
    const uint32_t us = (u & (N_MAX / 2)) | ((u + r) & (N_MAX / 2 - 1));
    const uint32_t* w = sm + l0 * LANE_PAD + n2k::brv11((__ldg(gtab + us) - 1) >> 1);
    reinterpret_cast<uint4*>(dst)[x] = make_uint4(w[0], w[LANE_PAD], w[2 * LANE_PAD], w[3 * LANE_PAD]);
  }
}

// grid: x = part * H + half, y = query (no cluster)
__global__ void __launch_bounds__(CT, 1) secondary_dual_kernel(ChainArgs a) {
  extern __shared__ uint32_t sm[];
  secondary_dual_body(a, blockIdx.x % a.g.H, blockIdx.y, blockIdx.x / a.g.H, sm);
}

// grid: x = factor (cluster of 2), y = part * H + half, z = query
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(CT) secondary_chain_kernel(ChainArgs a) {
  extern __shared__ uint32_t sm[];
  secondary_body(a, blockIdx.y % a.g.H, blockIdx.z, blockIdx.y / a.g.H, sm);
}

// grid: x = factor (cluster of 2), y = lane * H + half, z = shard
template <int LOGN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(CT) primary_chain_kernel(ChainArgs a) {
  extern __shared__ uint32_t sm[];
  const int h = blockIdx.y % a.g.H, lane = blockIdx.y / a.g.H;
  primary_body<LOGN>(a, h, lane, blockIdx.z, sm);
}

// reply_a = a_main + a_conj -> iNTT -> CRT; also the 17-bit mod switch
// (get_a, base_pir.rs:897-903, and double_pir.rs:164).
__global__ void primary_finalize_kernel(const uint32_t* __restrict__ a_out, uint64_t* __restrict__ a_zq,
                                        uint32_t* __restrict__ a_ms, Group g, NttTables T, CrtConst crtc) {
  extern __shared__ uint32_t sm[];  // [2][N]
  const int lane = blockIdx.x, s = blockIdx.y;
  const uint32_t N = g.n;
  for (uint32_t b = threadIdx.x; b < 2 * N; b += blockDim.x) {
    const uint32_t p = b / N;
    uint32_t v = a_out[(((size_t)s * g.H + 0) * SIMD + lane) * 2 * N + b];
    if (g.H == 2) v = add_mod(v, a_out[(((size_t)s * g.H + 1) * SIMD + lane) * 2 * N + b], prime_of(p));
    sm[b] = v;
  }
  __syncthreads();
  ntt_inv_smem2(sm, g.log2n, 1, 1, T);
  for (uint32_t n = threadIdx.x; n < N; n += blockDim.x) {
    const uint64_t v = crt(sm[n], sm[N + n], crtc);
    a_zq[((size_t)s * SIMD + lane) * N + n] = v;
    a_ms[((size_t)s * SIMD + lane) * N + n] = ms_encode(v, PRIM_A_BITS);
  }
}

}  // namespace

CrtConst host_crt_const();

static uint64_t pw(uint64_t b, uint64_t e, uint64_t m) {
  uint64_t r = 1 % m;
  b %= m;
  while (e) {
    if (e & 1) r = (uint64_t)((unsigned __int128)r * b % m);
    b = (uint64_t)((unsigned __int128)b * b % m);
    e >>= 1;
  }
  return r;
}
static uint32_t pow_mod2n(uint32_t b, uint32_t e, uint32_t mask) {
  uint32_t r = 1;
  for (uint32_t k = 0; k < e; k++) r = (r * b) & mask;
  return r;
}
static uint32_t inv5_mod2n(uint32_t two_n) {
  for (uint32_t x = 1; x < two_n; x += 2)
    if ((5 * x) % two_n == 1) return x;
  return 1;
}

constexpr size_t PAIR_SMEM = 116 * 1024;  // more than half an SM's shared memory

static ChainArgs chain_args(const Group& g, const ChainConsts& cc, const NttTables& T) {
  ChainArgs a;
  memset(&a, 0, sizeof(a));
  a.g = g;
  a.gka = cc.gka;
  a.qa = cc.qa;
  a.galb = cc.galb;
  a.maps = cc.maps;
  a.T = T;
  const uint64_t n = g.n;
  const CrtConst crtc = host_crt_const();
  for (int p = 0; p < 2; p++) {
    ChainPrime& c = a.cp[p];
    c.p = p ? P2 : P1;
    c.pinv = neg_inv32(c.p);
    c.r2 = (uint32_t)pw(pw(2, 64, c.p), 1, c.p);
    c.c26 = (uint32_t)((((unsigned __int128)1 << 26) << 32) % c.p);
    const uint64_t ninv1 = pw(n, P1 - 2, P1), ninv2 = pw(n, P2 - 2, P2);
    c.k1 = (uint32_t)((uint64_t)crtc.q2inv1 * ninv1 % P1);
    c.k1q = (uint32_t)(((uint64_t)c.k1 << 32) / P1);
    c.k2 = (uint32_t)((uint64_t)crtc.q1inv2 * ninv2 % P2);
    c.k2q = (uint32_t)(((uint64_t)c.k2 << 32) / P2);
    c.k = p ? c.k2 : c.k1;
    c.kinv = (uint32_t)(n * (p ? P1 : P2) % c.p);
  }
  return a;
}

static void set_limits(ChainArgs& a, uint32_t* err, const WaitLimits& lim) {
  a.err = err;
  a.wait_ns = lim.ns();
  a.withhold = lim.withhold_step < 0 ? ~0u : (uint32_t)lim.withhold_step;
}


void launch_primary_chain(uint32_t* const* slabs_dev, int nshards, uint32_t* a_out, const Group& g,
                          const ChainConsts& cc, const NttTables& T, cudaStream_t st) {
  ChainArgs a = chain_args(g, cc, T);
  a.slabs = slabs_dev;
  a.a_out = a_out;
  const uint32_t mask = 2 * g.n - 1;
  a.inv5 = inv5_mod2n(2 * g.n);
  a.c_first = pow_mod2n(5, g.L - 1, mask);
  a.cinv_first = pow_mod2n(a.inv5, g.L - 1, mask);
  const size_t smem = (size_t)12 * g.n * 4;
  dim3 grid(2, SIMD * g.H, nshards);
  if (g.log2n == LOG2_N_MAX) {  // three arrays a row
    set_smem(primary_chain_kernel<LOG2_N_MAX>, smem);
    primary_chain_kernel<LOG2_N_MAX><<<grid, CT, smem, st>>>(a);
  } else {
    set_smem(primary_chain_kernel<0>, smem);
    primary_chain_kernel<0><<<grid, CT, smem, st>>>(a);
  }
}

int chain_rows_supported(const Group& g) { return g.log2n == LOG2_N_MAX && g.na == 2; }

size_t chain_rows_words(const Group& g) { return (size_t)2 * g.H * g.L * SIMD * g.n; }

void launch_primary_chain_rows(uint32_t* rows, uint32_t* digits, size_t shard_words, int nshards, uint32_t* a_out,
                               uint32_t* err, const WaitLimits& lim, const Group& g, const ChainConsts& cc,
                               const NttTables& T, cudaStream_t st) {
  ChainArgs a = chain_args(g, cc, T);
  a.a_out = a_out;
  set_limits(a, err, lim);
  const int sms = sm_count();
  const long chains = SIMD * (long)g.H * nshards;
  if (2 * chains <= sms) {
    set_smem(primary_chain_pair_kernel, PAIR_SMEM);
    primary_chain_pair_kernel<<<dim3(2 * SIMD * g.H, nshards), 256, PAIR_SMEM, st>>>(a, rows, digits, shard_words);
    return;
  }
  if (chains <= sms) {
    const size_t smem = (size_t)2 * few_words(PRIM2K_KC) * 4;
    set_smem(primary_chain_wide_kernel, smem);
    primary_chain_wide_kernel<<<dim3(SIMD * g.H, nshards), 512, smem, st>>>(a, rows, digits, shard_words);
    return;
  }
  const size_t smem = (size_t)PRIM2K_WORDS * 4;
  set_smem(primary_chain2k_kernel, smem);
  primary_chain2k_kernel<<<dim3(SIMD * g.H, nshards), 256, smem, st>>>(a, rows, digits, shard_words);
}

void launch_order_rows(uint32_t* rows, size_t words, const SlotMaps& maps, cudaStream_t st) {
  order_rows_kernel<<<(unsigned)(words / N_MAX), 256, 0, st>>>(rows, maps.g);
}

void launch_lane_rows(const uint32_t* rows, const uint32_t* digits, uint32_t* slab, const Group& g,
                      const SlotMaps& maps, cudaStream_t st) {
  const size_t smem = (size_t)SIMD * LANE_PAD * 4;
  set_smem(lane_rows_kernel, smem);
  lane_rows_kernel<<<dim3(2 * g.H * g.L, 2), 512, smem, st>>>(rows, digits, slab, g, maps.g);
}

void chain_state_scale(const Group& g, int p, uint32_t* scale, uint32_t* inverse) {
  const uint32_t pr = p ? P2 : P1;
  *inverse = chain_rows_supported(g) ? (uint32_t)((uint64_t)g.n * (p ? P1 : P2) % pr) : 1;
  *scale = (uint32_t)pw(*inverse, pr - 2, pr);
}

void launch_primary_finalize(const uint32_t* a_out, int nshards, uint64_t* a_zq, uint32_t* a_ms, const Group& g,
                             const NttTables& T, cudaStream_t st) {
  const size_t smem = (size_t)2 * g.n * 4;
  dim3 grid(SIMD, nshards);
  primary_finalize_kernel<<<grid, 256, smem, st>>>(a_out, a_zq, a_ms, g, T, host_crt_const());
}

int secondary_chain_wave(const Group& g, int sms) {
  return std::max(1, g.log2n == LOG2_N_MAX ? sms / (int)g.H : 2 * sms / (2 * CTXT_PARTS * (int)g.H));
}

template <bool ZEROS>
static void launch_secondary_2048(const ChainArgs& a, const ScanConsts& sc, int nq, int sms, bool clustered,
                                  cudaStream_t st) {
  const unsigned H = a.g.H;
  const long chains = (long)nq * CTXT_PARTS * H;
  if (clustered || 2 * chains <= sms) {
    // PAIR_SMEM keeps the two blocks off one SM (and fits beside a scan block)
    const size_t smem = clustered && 2 * chains > sms ? (size_t)few_words(sec_consts(ZEROS)) * 4 : PAIR_SMEM;
    set_smem(secondary_chain_pair_kernel<ZEROS>, smem);
    secondary_chain_pair_kernel<ZEROS><<<dim3(2 * CTXT_PARTS * H, nq), 256, smem, st>>>(a, sc);
  } else if (chains <= sms) {
    const size_t smem = (size_t)2 * few_words(sec_consts(ZEROS)) * 4;
    set_smem(secondary_chain_wide_kernel<ZEROS>, smem);
    secondary_chain_wide_kernel<ZEROS><<<dim3(CTXT_PARTS * H, nq), 512, smem, st>>>(a, sc);
  } else {
    const size_t smem = (size_t)sec2k_words(ZEROS) * 4;
    set_smem(secondary_chain2k_kernel<ZEROS>, smem);
    secondary_chain2k_kernel<ZEROS><<<dim3(H, nq), 256 * CTXT_PARTS, smem, st>>>(a, sc);
  }
}

void launch_secondary_chain(const uint32_t* E, const uint32_t* qv, size_t qv_stride, int nq, uint32_t* out,
                            uint32_t* err, const WaitLimits& lim, const Group& g, const ChainConsts& cc,
                            const ScanConsts& sc, bool zeros, const NttTables& T, cudaStream_t st, bool clustered) {
  ChainArgs a = chain_args(g, cc, T);
  set_limits(a, err, lim);
  a.E = E;
  a.qv = qv;
  a.qv_stride = qv_stride;
  a.nl = nq * CTXT_PARTS;
  a.out = out;
  // N = 2048 (1024 steps of order 2048): a part's chain on two SMs while there
  // are two for each (2.1 ms), on one while there is one (3.75), beyond that the
  // three parts of a query and half per block (10.2, the constants kept once).
  // Other lengths: one part and factor per block in two-block clusters while the
  // chunk needs at most one block per SM, then one block per part carrying both
  // factors.  `clustered` asks for the cluster form at any chunk size (its blocks
  // share SMs with a running scan; the pipeline tuner picks it per group size when
  // faster).
  const int sms = sm_count();
  if (g.log2n == LOG2_N_MAX) {
    if (zeros)
      launch_secondary_2048<true>(a, sc, nq, sms, clustered, st);
    else
      launch_secondary_2048<false>(a, sc, nq, sms, clustered, st);
  } else if (clustered || 2 * (long)nq * CTXT_PARTS * g.H <= sms) {
    const size_t smem = (size_t)SEC_WORDS * g.n * 4;
    set_smem(secondary_chain_kernel, smem);
    secondary_chain_kernel<<<dim3(2, CTXT_PARTS * g.H, nq), CT, smem, st>>>(a);
  } else {
    const size_t smem = (size_t)SEC_DUAL_WORDS * g.n * 4;
    set_smem(secondary_dual_kernel, smem);
    secondary_dual_kernel<<<dim3(CTXT_PARTS * g.H, nq), CT, smem, st>>>(a);
  }
}

}  // namespace dnspir
