// scan.cu -- the primary-phase scan (main_pir_loop, crates/pir/src/base_pir.rs:
// 1085-1247) for B queries at once, and its epilogue (perform_pir_split
// :1066-1077, from_simd_element :905-935, double_pir.rs:161-175).
//
// main_pir_loop is the recurrence  sum'[gal(j)] = sum[j] + G0[i,j] gk0[j] +
// G1[i,j] gk1[j] + E[i,j] q[j]  followed by the inverse permutation.  Unrolled,
// output slot k receives from row i the terms at slot j = idx(5^(L-1-i) (2k+1)).
// The slab orders slots by (sign, e) with 2k+1 = +-5^e mod 2N (SlotMaps), so
// sigma_5 is e -> e+1 and output u = (sign, e) reads, at row i, the query
// entry (sign, e + L-1-i mod N/2): for a tile of consecutive e and a chunk of
// rows the query entries needed form one contiguous (cyclic) window, which is
// staged in shared memory for all B queries.  Every row is stored permuted so
// that the data for output u sits at position u (slab_off), so a block streams
// its rows contiguously.  Products of canonical residues are below 2^52, so one
// 64-bit accumulator per (lane, query) absorbs a half (at most 3 L <= 3072
// products) without reduction; it is reduced once between halves and once at
// the end.  Two arrays a row instead of the reference's three (slab_off): at
// 2^22 entries a pass reads 137 GB instead of 206 (a query of a stream of
// one-query passes on the tensor engine 29.0 -> 20.1 ms; 16 queries at 2^20 on
// this engine 43.1 -> 25.8 ms).
// One block per (shard, factor, sign, tile) item, consecutive blocks sharing a
// shard; blocks retire after their item so that the higher-priority secondary
// stream can take SMs while a scan is running.
#include <algorithm>

#include "kernels.cuh"
#include "ntt2048.cuh"

namespace dnspir {
namespace {

constexpr int SCAN_NT = 256;

// Query vectors (launch_scan_vectors).  With C = gk0 - gk_a0 r and r = q / qry_a
// per half, the recurrence's contribution of row i at slot j,
//     t_i gk0 + G1_i (gk1 - 2^26 gk0) + E_i q,
// becomes, with E_i = (a_(i+1) - t_i gk_a0 - G1_i kappa) / qry_a,
//     t_i C + G1_i (gk1 - 2^26 gk0 - kappa r) + a_(i+1) r,
// and t_i[j] C[j] = a_i[5 j] C[j] joins row i - 1, whose slot for the same
// output is 5 j: array 0 of every row but the last meets r[j] + C[5^-1 j].
// The last row's state has no following t, so its C term is taken back (v = 2).
// In (sign, e) order 5^-1 is e - 1.  States stored with a scale (ScanConsts xinv)
// meet vectors divided by it.  One slot u and factor p of one query; at(slot, x):
// the decoded vector of that slot at position x.
template <class At>
__device__ __forceinline__ void scan_vectors(const At& at, uint32_t u, int p, int s_q, int s_gk, uint32_t* o,
                                             const Group& g, const ScanConsts& sc) {
  const uint32_t N = g.n, half = N / 2;
  const uint32_t pr = prime_of(p);
  const uint64_t mu = barrett_mu(pr);
  const uint32_t gk0 = at(s_gk, u), gk1 = at(s_gk + 1, u);
  if (g.na == 3) {
    for (int h = 0; h < (int)g.H; h++) {
      o[scan_vec_off(N, h, 0, p) + u] = at(s_q + h, u);
      o[scan_vec_off(N, h, 1, p) + u] = gk0;
      o[scan_vec_off(N, h, 2, p) + u] = gk1;
    }
    return;
  }
  const uint32_t um = (u & (half - 1)) ? u - 1 : u + half - 1;  // 5^-1 of this slot
  const uint32_t gk0m = at(s_gk, um);
  const uint32_t ga = __ldg(sc.gka0 + (size_t)p * N + um), ka = __ldg(sc.kappa + (size_t)p * N + u);
  const uint32_t g1 = sub_mod(gk1, mul_mod(gk0, 1u << LOG2_B, pr, mu), pr);
  for (int h = 0; h < (int)g.H; h++) {
    const uint32_t* inv = sc.qinv + (size_t)(h * 2 + p) * N;
    const uint32_t r = mul_mod(at(s_q + h, u), __ldg(inv + u), pr, mu);
    const uint32_t rm = mul_mod(at(s_q + h, um), __ldg(inv + um), pr, mu);
    const uint32_t cm = sub_mod(gk0m, mul_mod(ga, rm, pr, mu), pr);
    o[scan_vec_off(N, h, 0, p) + u] = mul_mod(add_mod(r, cm, pr), sc.xinv[p], pr, mu);
    o[scan_vec_off(N, h, 1, p) + u] = sub_mod(g1, mul_mod(ka, r, pr, mu), pr);
    o[scan_vec_off(N, h, 2, p) + u] = cm ? pr - mul_mod(cm, sc.xinv[p], pr, mu) : 0;
  }
}

// One thread per slot, factor and query.  sum: cleared for scan_lanes_kernel (or null).
__global__ void scan_vectors_kernel(const uint32_t* __restrict__ src, size_t q_stride, int s_q, int s_gk, int nb,
                                    uint32_t* __restrict__ qv, uint32_t* __restrict__ sum, Group g, ScanConsts sc,
                                    const uint32_t* __restrict__ gtab) {
  const uint32_t N = g.n;
  const uint32_t u = blockIdx.x * blockDim.x + threadIdx.x;
  if (u >= N) return;
  const int p = blockIdx.y, q = blockIdx.z;
  uint32_t* o = qv + (size_t)q * 2 * SCAN_VECS * 2 * N;
  if (sum) sum[((size_t)p * N + u) * SIMD + q] = 0;
  if (q >= nb) {
    for (int h = 0; h < (int)g.H; h++)
      for (int v = 0; v < SCAN_VECS; v++) o[scan_vec_off(N, h, v, p) + u] = 0;
    return;
  }
  src += (size_t)q * q_stride;
  auto at = [&](int slot, uint32_t x) {
    return __ldg(src + ((size_t)slot * 2 + p) * N + ((__ldg(gtab + x) - 1) >> 1));
  };
  scan_vectors(at, u, p, s_q, s_gk, o, g, sc);
}

// The same from the ring elements of a per-lane query, for N <= 512: one block per
// lane and factor transforms the lane's elements (query, conjugate if the group
// has one, both keys) in shared memory and takes the vectors from there.  A small
// shard's call is a row of short kernels, and this is one instead of two: 45 us the
// call instead of 50 at N = 64, 62 / 64 at 256; at N = 1024 (90 / 88) the 64 blocks of
// separate transforms are worth their launch.
constexpr int LANE_VECS_NT = 512;
__global__ void __launch_bounds__(LANE_VECS_NT) lane_vectors_kernel(const uint64_t* __restrict__ zq,
                                                                    uint32_t* __restrict__ qv,
                                                                    uint32_t* __restrict__ sum, Group g,
                                                                    ScanConsts sc, const uint32_t* __restrict__ gtab,
                                                                    NttTables T) {
  extern __shared__ __align__(16) uint32_t sm[];
  const int lane = blockIdx.x, p = blockIdx.y;
  const uint32_t N = g.n, pr = prime_of(p);
  const uint64_t* src = zq + (size_t)lane * 4 * N;
  const uint32_t gap = g.H == 2 ? 0 : N;  // no conjugate: its element is left out
  for (uint32_t b = threadIdx.x; b < 4 * N - gap; b += LANE_VECS_NT)
    sm[b] = reduce64(__ldg(src + b + (b < N ? 0 : gap)), pr, barrett_mu(pr));
  __syncthreads();
  ntt_fwd_smem(sm, g.log2n, g.H == 2 ? 4 : 3, T, p);
  auto at = [&](int slot, uint32_t x) {
    return sm[slot * N - (slot < 2 ? 0 : gap) + brv((__ldg(gtab + x) - 1) >> 1, g.log2n)];
  };
  for (uint32_t u = threadIdx.x; u < N; u += LANE_VECS_NT) {
    sum[((size_t)p * N + u) * SIMD + lane] = 0;
    scan_vectors(at, u, p, 0, 2, qv + (size_t)lane * 2 * SCAN_VECS * 2 * N, g, sc);
  }
}

struct ScanArgs {
  Group g;
  uint32_t* const* slabs;
  int nshards;
  const uint32_t* qv;  // query vectors, 12 N words a query
  uint32_t* out;       // [b][s][p][u][lane], reduced mod p
  int rows;            // rows per window chunk
  uint32_t groups;     // groups of B queries
};

__device__ __forceinline__ void ld_lanes(const uint32_t* p, uint32_t* v, int lpt) {
  if (lpt == 8) {
    const uint4 a = __ldcs(reinterpret_cast<const uint4*>(p));
    const uint4 b = __ldcs(reinterpret_cast<const uint4*>(p + 4));
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
  } else if (lpt == 4) {
    const uint4 a = __ldcs(reinterpret_cast<const uint4*>(p));
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
  } else {
    const uint2 a = __ldcs(reinterpret_cast<const uint2*>(p));
    v[0] = a.x, v[1] = a.y;
  }
}

// B queries per block, LPT lanes per thread, MINB blocks per SM (0: as many as
// the registers give), UN rows unrolled.  One and two queries are bound by HBM
// and take light threads with many rows in flight (64 full shards: one query 4.65
// ms, 7.4 TB/s; two 4.8, 5.2 as eight lanes a thread).  From four on the wide
// multiply-adds bound it (four cycles a warp on the heavy FMA pipe: 7.5 ms for 8
// queries of 64 full shards), and four lanes a thread halve the shared-memory
// reads per product against two: 8 queries 9.7 ms as two blocks per SM, 16 19.0 as
// two such groups against 21.2 as 16 with two lanes; four queries 5.7 at three
// blocks per SM and four lanes, 8.1 at eight lanes (130 registers; 0.38 / 0.56 at
// 4 half-size shards).  Tried: a third of the queries on the FP64 pipe, exactly,
// with 13-bit halves (8 queries 16 ms).
template <int B, int LPT, int NA, int MINB, int UN>
__global__ void __launch_bounds__(SCAN_NT, MINB) scan_batch_kernel(ScanArgs a) {
  constexpr int LG = SIMD / LPT;     // lane groups per slot
  constexpr int TS = SCAN_NT / LG;   // slots per tile
  extern __shared__ uint32_t win[];  // [NA][B][W]: x fastest, so a warp's slots hit distinct banks
  const Group& g = a.g;
  const uint32_t N = g.n, half = N / 2, L = g.L;
  const uint32_t R = (uint32_t)a.rows;
  const uint32_t W = TS + R - 1;
  const uint32_t tiles = (half + TS - 1) / TS;
  const int slot = threadIdx.x / LG, lg = threadIdx.x % LG;
  const size_t arr = (size_t)N * SIMD, row_stride = NA * arr;
  // item = ((s * 2 + p) * 2 + sgn) * tiles + tile; the groups of B queries of one
  // item are consecutive blocks, so that its rows come from HBM once and from
  // L2 for the others
  const uint32_t item = blockIdx.x / a.groups;
  const size_t qbase = (size_t)(blockIdx.x % a.groups) * B;
  const uint32_t tile = item % tiles;
  const uint32_t sgn = (item / tiles) & 1;
  const int p = (item / (2 * tiles)) & 1;
  const int s = item / (4 * tiles);
  const uint32_t e0 = tile * TS;
  const uint32_t e = e0 + slot;
  const bool active = e < half;
  const uint32_t u = sgn * half + e;
  const uint32_t pr = prime_of(p);
  const uint64_t mu = barrett_mu(pr);
  const uint32_t* slab = a.slabs[s];
  const size_t qs = (size_t)2 * SCAN_VECS * 2 * N;
  uint64_t acc[LPT][B];
#pragma unroll
  for (int l = 0; l < LPT; l++)
#pragma unroll
    for (int b = 0; b < B; b++) acc[l][b] = 0;
  for (uint32_t h = 0; h < g.H; h++) {
    for (uint32_t i0 = 0; i0 < L; i0 += R) {
      const uint32_t i1 = min(L, i0 + R);
      const uint32_t Wr = TS + (i1 - i0) - 1;
      const uint32_t w0 = (e0 + L - i1) % half;
      for (uint32_t idx = threadIdx.x; idx < NA * Wr * B; idx += SCAN_NT) {
        const uint32_t x = idx % Wr, b = (idx / Wr) % B, v = idx / (B * Wr);
        win[(v * B + b) * W + x] =
            __ldg(a.qv + (qbase + b) * qs + scan_vec_off(N, h, v, p) + sgn * half + (w0 + x) % half);
      }
      __syncthreads();
      if (active) {
        const uint32_t* row = slab + slab_off(g, p, h, i0, 0, u) + lg * LPT;
        uint32_t x = slot + (i1 - 1 - i0);
#pragma unroll UN
        for (uint32_t i = i0; i < i1; i++) {
          uint32_t ev[NA][LPT];
#pragma unroll
          for (int v = 0; v < NA; v++) ld_lanes(row + v * arr, ev[v], LPT);
#pragma unroll
          for (int b = 0; b < B; b++) {
            uint32_t q[NA];
#pragma unroll
            for (int v = 0; v < NA; v++) q[v] = win[(v * B + b) * W + x];
#pragma unroll
            for (int l = 0; l < LPT; l++)
#pragma unroll
              for (int v = 0; v < NA; v++) acc[l][b] += (uint64_t)ev[v][l] * q[v];
          }
          row += row_stride;
          x--;
        }
      }
      __syncthreads();
    }
    uint32_t xv[LPT] = {};  // the last row's state once more
    if (NA == 2 && active) ld_lanes(slab + slab_off(g, p, h, L - 1, 0, u) + lg * LPT, xv, LPT);
#pragma unroll
    for (int b = 0; b < B; b++) {
      uint32_t c = 0;
      if (NA == 2 && active) c = __ldg(a.qv + (qbase + b) * qs + scan_vec_off(N, h, 2, p) + u);
#pragma unroll
      for (int l = 0; l < LPT; l++) acc[l][b] = reduce64(acc[l][b] + (uint64_t)xv[l] * c, pr, mu);
    }
  }
  if (active) {
#pragma unroll
    for (int b = 0; b < B; b++) {
      uint32_t* o = a.out + ((((qbase + b) * a.nshards + s) * 2 + p) * N + u) * SIMD + lg * LPT;
#pragma unroll
      for (int l = 0; l < LPT; l++) o[l] = (uint32_t)acc[l][b];
    }
  }
}

// Per-lane queries (perform_pir_split): qv holds lane l's vectors as query l.
// One block: blockDim.x consecutive slots of one sign, factor and half over
// one chunk of rows; the lanes' query entries its rows need are one window in
// shared memory, [vector][lane quad][x][4 lanes], so a thread reads its 8 lanes'
// entries as 16-byte vectors without bank conflicts.  Bound by the slab's bytes;
// with the sums kept per slot instead of per chunk the epilogue reads one word
// where it added up 256 (3.0 ms of a 3.5 ms call at N = 2048; the whole
// set_db + get_a + split call 14.9 -> 11.6 ms);
// the chunks' residues (at most 2 SCAN_MAX_CHUNKS = 32 of them, below 2^31 in
// all) add up in `sum` [p][u][lane], zeroed by the kernel that makes the vectors.
constexpr int LANES_NT = 256;
__global__ void __launch_bounds__(LANES_NT) scan_lanes_kernel(const uint32_t* __restrict__ slab,
                                                              const uint32_t* __restrict__ qv,
                                                              uint32_t* __restrict__ sum, Group g, int R) {
  extern __shared__ __align__(16) uint32_t win[];
  const uint32_t N = g.n, half = N / 2, L = g.L;
  const int na = (int)g.na;
  const int TS = blockDim.x;
  const uint32_t tiles = half / TS;
  const uint32_t e0 = (blockIdx.x % tiles) * TS, sgn = blockIdx.x / tiles;
  const int h = blockIdx.y / R, rc = blockIdx.y % R, p = blockIdx.z;
  const uint32_t rows = (L + R - 1) / R;
  const uint32_t i0 = rc * rows, i1 = min(L, i0 + rows);
  if (i0 >= i1) return;
  const uint32_t W = TS + rows - 1, Wr = TS + (i1 - i0) - 1;
  const uint32_t w0 = (e0 + L - i1) % half;
  const size_t qs = (size_t)2 * SCAN_VECS * 2 * N;
  for (uint32_t idx = threadIdx.x; idx < (uint32_t)na * SIMD * Wr; idx += TS) {
    const uint32_t x = idx % Wr, vl = idx / Wr, l = vl % SIMD, v = vl / SIMD;
    win[((v * 2 + l / 4) * W + x) * 4 + l % 4] =
        __ldg(qv + l * qs + scan_vec_off(N, h, v, p) + sgn * half + (w0 + x) % half);
  }
  __syncthreads();
  const uint32_t u = sgn * half + e0 + threadIdx.x;
  const uint32_t pr = prime_of(p);
  uint64_t acc[SIMD] = {};
  const size_t arr = (size_t)N * SIMD;
  const uint32_t* row = slab + slab_off(g, p, h, i0, 0, u);
  uint32_t x = threadIdx.x + (i1 - 1 - i0);
  if (na == 2) {
#pragma unroll 4
    for (uint32_t i = i0; i < i1; i++, x--, row += 2 * arr) {
      uint32_t xv[SIMD], gv[SIMD];
      ld_lanes(row, xv, SIMD);
      ld_lanes(row + arr, gv, SIMD);
#pragma unroll
      for (int d = 0; d < 2; d++) {
        const uint4 a = *reinterpret_cast<const uint4*>(win + (d * W + x) * 4);
        const uint4 b = *reinterpret_cast<const uint4*>(win + ((2 + d) * W + x) * 4);
        acc[4 * d] += (uint64_t)xv[4 * d] * a.x + (uint64_t)gv[4 * d] * b.x;
        acc[4 * d + 1] += (uint64_t)xv[4 * d + 1] * a.y + (uint64_t)gv[4 * d + 1] * b.y;
        acc[4 * d + 2] += (uint64_t)xv[4 * d + 2] * a.z + (uint64_t)gv[4 * d + 2] * b.z;
        acc[4 * d + 3] += (uint64_t)xv[4 * d + 3] * a.w + (uint64_t)gv[4 * d + 3] * b.w;
      }
    }
    if (i1 == L) {  // the last row's state once more
      uint32_t xv[SIMD];
      ld_lanes(slab + slab_off(g, p, h, L - 1, 0, u), xv, SIMD);
#pragma unroll
      for (int l = 0; l < SIMD; l++)
        acc[l] += (uint64_t)xv[l] * __ldg(qv + l * qs + scan_vec_off(N, h, 2, p) + u);
    }
  } else {
    for (uint32_t i = i0; i < i1; i++, x--, row += 3 * arr)
      for (int v = 0; v < 3; v++) {
        uint32_t xv[SIMD];
        ld_lanes(row + v * arr, xv, SIMD);
#pragma unroll
        for (int l = 0; l < SIMD; l++) acc[l] += (uint64_t)xv[l] * win[((v * 2 + l / 4) * W + x) * 4 + l % 4];
      }
  }
#pragma unroll
  for (int l = 0; l < SIMD; l++)
    atomicAdd(sum + ((size_t)p * N + u) * SIMD + l, reduce64(acc[l], pr, barrett_mu(pr)));
}

// grid: x = shard, y = lane pair, z = query.  b = the query's scan output ->
// iNTT -> CRT -> mod switch to 12 bits; with the shard's 17-bit a-part,
// three base-1025 digits (encode_ciphertext_plaintext, double_pir.rs:70-81).
__global__ void primary_epilogue_kernel(const uint32_t* __restrict__ fin, int nshards,
                                        const uint32_t* __restrict__ a_ms, const int* __restrict__ distinct_of,
                                        uint16_t* __restrict__ sec_in, int nq, int chunk, Group g,
                                        const uint32_t* __restrict__ uof, NttTables T, CrtConst crtc) {
  extern __shared__ uint32_t sm[];  // [l0 q1, l1 q1, l0 q2, l1 q2]
  const int s = blockIdx.x, l0 = blockIdx.y * 2, b = blockIdx.z;
  const int logn = g.log2n;
  const uint32_t N = g.n;
  // position x of factor p holds natural slot brv(x) of both lanes (one 8-byte
  // load per pair; iterating over positions keeps the stores conflict-free)
  for (uint32_t x = threadIdx.x; x < 2 * N; x += blockDim.x) {
    const uint32_t p = x >> logn, xx = x & (N - 1);
    const uint2 v = __ldg(reinterpret_cast<const uint2*>(
        fin + ((((size_t)b * nshards + s) * 2 + p) * N + __ldg(uof + brv(xx, logn))) * SIMD + l0));
    sm[((2 * p) << logn) + xx] = v.x;
    sm[((2 * p + 1) << logn) + xx] = v.y;
  }
  __syncthreads();
  ntt_inv_smem2(sm, logn, 2, 2, T);
  const int ds = distinct_of[s];
  for (uint32_t x = threadIdx.x; x < 2 * N; x += blockDim.x) {
    const uint32_t ll = x >> logn, n = x & (N - 1);
    const uint64_t v = crt(sm[(ll << logn) + n], sm[((2 + ll) << logn) + n], crtc);
    const uint32_t bq = ms_encode(v, PRIM_B_BITS);
    const uint32_t aq = a_ms[((size_t)ds * SIMD + l0 + ll) * N + n];
    uint32_t w = (aq << PRIM_B_BITS) + bq;
    const uint32_t d0 = w % TPLAIN;
    w /= TPLAIN;
    const uint32_t d1 = w % TPLAIN;
    const uint32_t d2 = w / TPLAIN;
    // the secondary input of queries [c * chunk, ...) is one [t][lanes_c][N] block
    const int c = b / chunk, bl = b % chunk;
    const size_t lanes_c = (size_t)CTXT_PARTS * min(chunk, nq - c * chunk);
    const size_t t = (size_t)s * SIMD + l0 + ll;
    uint16_t* o = sec_in + (size_t)c * chunk * CTXT_PARTS * nshards * SIMD * N + (t * lanes_c + (size_t)bl * CTXT_PARTS) * N + n;
    o[0] = (uint16_t)d0;
    o[N] = (uint16_t)d1;
    o[2 * N] = (uint16_t)d2;
  }
}

// ---- N = 2048: the same epilogue on the register transforms of ntt2048.cuh,
// with the encoder's column transforms (encode.cu) in the same block: the three
// digits of a coefficient stay in shared memory as one word, and each digit's
// polynomial is transformed from there into A [t][lane][x].  Grid: x = shard, y =
// LN lanes, z = query of the chunk.  One 16-byte gather per position and factor
// brings four lanes (half a 32-byte sector; the other half is the neighbouring
// block's), the eight inverse transforms run together, the CRT uses Shoup
// companions of its two constants and the 12-bit switch an exact 64-bit rounding
// (v 2^13 + q < 2^64 for v < q).  LN = 1: one lane per block, for few shards and
// queries (launch_epilogue_cols).  Bound by shared memory and
// barriers (three blocks an SM).  Against digits through global memory and a kernel
// for their columns (256 queries of 64 shards): 2.95 + 2.03 -> 4.25 ms, and the
// digits' buffer is not needed.
constexpr int EPI_NT = 512;

__device__ __forceinline__ uint32_t ms_encode12(uint64_t v) {
  // round(v 2^12 / q) = floor((v 2^13 + q) / 2q): a double estimate (v times
  // the rounded constant 2^12 / q, within one of the result), then one exact
  // correction (r <= 2^12, so r 2q < 2^64)
  constexpr double SCALE = (double)(1u << PRIM_B_BITS) / (double)QQ;
  const uint64_t num = (v << (PRIM_B_BITS + 1)) + QQ;
  int64_t r = (int64_t)floor((double)v * SCALE + 0.5);
  r = r < 0 ? 0 : r;
  const uint64_t lo = (uint64_t)r * (2 * QQ);
  if (num < lo) r--;
  else if (num - lo >= 2 * QQ) r++;
  return (uint32_t)r & ((1u << PRIM_B_BITS) - 1);
}

template <int LN>
__global__ void __launch_bounds__(EPI_NT, LN == 4 ? 3 : 0) primary_epilogue2k_kernel(
    const uint32_t* __restrict__ fin, int nshards, const uint32_t* __restrict__ a_ms,
    const int* __restrict__ distinct_of, uint32_t* __restrict__ A, const uint32_t* __restrict__ uof, NttTables T,
    uint32_t k1, uint32_t k1q, uint32_t k2, uint32_t k2q) {
  extern __shared__ __align__(16) uint32_t sm[];  // [q1 lanes l0 .. l0 + LN - 1][q2 lanes], padded
  using namespace n2k;
  const int s = blockIdx.x, l0 = blockIdx.y * LN, b = blockIdx.z;
  // position x of factor p holds natural slot brv(x)
  for (int x = threadIdx.x; x < 2 * N; x += EPI_NT) {
    const int p = x >> 11, xx = x & (N - 1);
    const uint32_t* src = fin + ((((size_t)b * nshards + s) * 2 + p) * N + __ldg(uof + brv11(xx))) * SIMD + l0;
    uint32_t* o = sm + LN * p * PS + phys(xx);
    if constexpr (LN == 4) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(src));
      o[0] = v.x, o[PS] = v.y, o[2 * PS] = v.z, o[3 * PS] = v.w;
    } else {
      o[0] = __ldg(src);
    }
  }
  __syncthreads();
  inv<EPI_NT>(sm, LN, LN, T);
  const int ds = distinct_of[s];
  for (int x = threadIdx.x; x < LN * N; x += EPI_NT) {
    const int ll = x >> 11, n = x & (N - 1);
    const uint32_t o = phys(n);
    const uint32_t x1 = shoup_mul(sm[ll * PS + o], k1, k1q, P1);
    const uint32_t x2 = shoup_mul(sm[(LN + ll) * PS + o], k2, k2q, P2);
    uint64_t v = (uint64_t)x1 * P2 + (uint64_t)x2 * P1;
    v = v >= QQ ? v - QQ : v;
    const uint32_t aq = __ldg(a_ms + ((size_t)ds * SIMD + l0 + ll) * N + n);
    uint32_t w = (aq << PRIM_B_BITS) + ms_encode12(v);
    const uint32_t d0 = w % TPLAIN;
    w /= TPLAIN;
    const uint32_t d1 = w % TPLAIN;
    const uint32_t d2 = w / TPLAIN;  // below 2^29 / 1025^2 < 2^10
    sm[ll * PS + o] = d0 | (d1 << 11) | (d2 << 22);
  }
  __syncthreads();
  uint32_t* const work = sm + LN * PS;
  const size_t nl = (size_t)CTXT_PARTS * gridDim.z;
#pragma unroll 1
  for (int digit = 0; digit < CTXT_PARTS; digit++) {
    {
      const int po = threadIdx.x >> 8, base = (int)phys(threadIdx.x & 255);
      for (int ll = po; ll < LN; ll += EPI_NT / 256) {
        uint32_t v[8];
#pragma unroll
        for (int k = 0; k < 8; k++) v[k] = (sm[ll * PS + base + k * Geo8<1>::STR] >> (11 * digit)) & 0x7FFu;
        fwd8_bf(v, param_tw8(T.fw7[0]), P1);
#pragma unroll
        for (int k = 0; k < 8; k++) work[ll * PS + base + k * Geo8<1>::STR] = v[k];
      }
    }
    __syncthreads();
    pass8<EPI_NT, 8, false>(work, LN, 0, T, (void*)nullptr);
    pass8<EPI_NT, 64, false>(work, LN, 0, T, (void*)nullptr);
    const int g = threadIdx.x;  // quad of transform positions
    const Tw4 tw = load_tw4(T.fw2[0], g);
#pragma unroll
    for (int ll = 0; ll < LN; ll++) {
      uint4 v = *reinterpret_cast<const uint4*>(work + ll * PS + phys(4 * g));
      ct(v.x, v.z, tw.a, tw.aq, P1);
      ct(v.y, v.w, tw.a, tw.aq, P1);
      ct(v.x, v.y, tw.b0, tw.b0q, P1);
      ct(v.z, v.w, tw.b1, tw.b1q, P1);
      reinterpret_cast<uint4*>(A + (((size_t)s * SIMD + l0 + ll) * nl + (size_t)b * CTXT_PARTS + digit) * N)[g] =
          make_uint4(canon(v.x, P1), canon(v.y, P1), canon(v.z, P1), canon(v.w, P1));
    }
    __syncthreads();
  }
}

// One lane per block: sums of scan_lanes_kernel (below 2^31) -> iNTT -> CRT.
constexpr int ZQ_NT = 512;
__global__ void __launch_bounds__(ZQ_NT) epilogue_zq_kernel(const uint32_t* __restrict__ sum,
                                                            uint64_t* __restrict__ out, Group g,
                                                            const uint32_t* __restrict__ uof, NttTables T,
                                                            CrtConst crtc) {
  extern __shared__ __align__(16) uint32_t sm[];
  const int l = blockIdx.x, logn = g.log2n;
  const uint32_t N = g.n;
  const bool full = logn == LOG2_N_MAX;
  const uint32_t PW = full ? n2k::PS : N;  // words between the two factors' polynomials
  for (uint32_t x = threadIdx.x; x < 2 * N; x += ZQ_NT) {
    const uint32_t p = x >> logn, xx = x & (N - 1);  // position xx holds natural slot brv(xx)
    const uint32_t v = __ldg(sum + ((size_t)p * N + __ldg(uof + brv(xx, logn))) * SIMD + l);
    sm[p * PW + (full ? n2k::phys(xx) : xx)] = ntt_detail::canon(v, prime_of(p));
  }
  __syncthreads();
  if (full)
    n2k::inv<ZQ_NT>(sm, 1, 1, T);
  else
    ntt_inv_smem2(sm, logn, 1, 1, T);
  for (uint32_t n = threadIdx.x; n < N; n += ZQ_NT) {
    const uint32_t o = full ? n2k::phys(n) : n;
    out[(size_t)l * N + n] = crt(sm[o], sm[PW + o], crtc);
  }
}

template <int B, int LPT, int NA, int MINB, int UN>
void launch_batch_na(const ScanArgs& a, cudaStream_t st) {
  constexpr int TS = SCAN_NT / (SIMD / LPT);
  const size_t smem = (size_t)NA * (TS + a.rows - 1) * B * 4;
  set_smem(scan_batch_kernel<B, LPT, NA, MINB, UN>, smem);
  const uint32_t tiles = (a.g.n / 2 + TS - 1) / TS;
  const uint32_t items = (uint32_t)a.nshards * 4 * tiles;
  scan_batch_kernel<B, LPT, NA, MINB, UN><<<items * a.groups, SCAN_NT, smem, st>>>(a);
}
template <int B, int LPT, int MINB, int UN>
void launch_batch(const ScanArgs& a, cudaStream_t st) {
  if (a.g.na == 2)
    launch_batch_na<B, LPT, 2, MINB, UN>(a, st);
  else
    launch_batch_na<B, LPT, 3, MINB, 1>(a, st);
}

}  // namespace

CrtConst host_crt_const();

void launch_scan_vectors(const uint32_t* src, size_t q_stride, int s_q, int s_gk, int nb, int nb_pad, uint32_t* qv,
                         const Group& g, const ScanConsts& sc, const SlotMaps& maps, cudaStream_t st) {
  const unsigned nt = g.n < 256 ? g.n : 256;
  scan_vectors_kernel<<<dim3(g.n / nt, 2, nb_pad), nt, 0, st>>>(src, q_stride, s_q, s_gk, nb, qv, nullptr, g, sc,
                                                                maps.g);
}

void launch_lane_vectors(const uint64_t* zq, uint32_t* ntt, uint32_t* qv, uint32_t* sum, const Group& g,
                         const ScanConsts& sc, const SlotMaps& maps, const NttTables& T, cudaStream_t st) {
  if (g.n <= 512) {
    const size_t smem = (size_t)4 * g.n * 4;
    lane_vectors_kernel<<<dim3(SIMD, 2), LANE_VECS_NT, smem, st>>>(zq, qv, sum, g, sc, maps.g, T);
    return;
  }
  launch_ring_to_ntt(zq, SIMD * 4, ntt, nullptr, g.log2n, T, st);
  scan_vectors_kernel<<<dim3(g.n / 256, 2, SIMD), 256, 0, st>>>(ntt, 8 * (size_t)g.n, 0, 2, SIMD, qv, sum, g, sc, maps.g);
}

int scan_batch_supported(int B) { return B >= 1 && B <= 256 && (B & (B - 1)) == 0; }

int launch_scan_batch(uint32_t* const* slabs_dev, int nshards, const uint32_t* qv, int B, int per_block, uint32_t* out,
                      const Group& g, cudaStream_t st) {
  if (!scan_batch_supported(B)) return -1;
  if (per_block <= 0) per_block = B < 8 ? B : 8;
  if (per_block > B || B % per_block) return -1;
  const int groups = B / per_block;
  ScanArgs a;
  a.g = g;
  a.slabs = slabs_dev;
  a.nshards = nshards;
  a.qv = qv;
  a.out = out;
  a.rows = (int)(g.L < 256 ? g.L : 256);
  a.groups = (uint32_t)groups;
  switch (per_block) {
    case 1: {
      // rows in flight per thread against threads: few blocks need the depth,
      // many give it themselves (4 / 11 / 25 half-size and 64 full shards: 4 rows
      // 0.51 / 0.52 / 0.55 / 4.65 ms, 8 rows 0.37 / 0.39 / 0.48 / 4.85, 12 rows at
      // three blocks per SM 0.25 / 0.30 / 0.76 / 4.69)
      const int sms = sm_count();
      const size_t blocks = (size_t)nshards * 4 * ((g.n / 2 + 127) / 128) * groups;
      if (blocks <= (size_t)3 * sms) launch_batch<1, 4, 3, 12>(a, st);
      else if (blocks <= (size_t)7 * sms) launch_batch<1, 4, 0, 8>(a, st);
      else launch_batch<1, 4, 0, 4>(a, st);
      break;
    }
    case 2: launch_batch<2, 4, 3, 6>(a, st); break;
    case 4: launch_batch<4, 4, 3, 6>(a, st); break;
    case 8: launch_batch<8, 4, 2, 4>(a, st); break;
    case 16: launch_batch<16, 2, 2, 6>(a, st); break;
    default: return -1;
  }
  return 0;
}

size_t scan_lanes_sum_words(const Group& g) { return (size_t)2 * g.n * SIMD; }

void launch_scan_lanes(const uint32_t* slab, const uint32_t* qv, uint32_t* sum, const Group& g, cudaStream_t st) {
  const int nt = g.n / 2 < (uint32_t)LANES_NT ? (int)(g.n / 2) : LANES_NT;
  const int R = (int)std::max<uint32_t>(1, std::min<uint32_t>(SCAN_MAX_CHUNKS, g.L / 8));
  const uint32_t rows = (g.L + R - 1) / R;
  const size_t smem = (size_t)g.na * SIMD * (nt + rows - 1) * 4;
  scan_lanes_kernel<<<dim3(2 * (g.n / 2 / nt), g.H * R, 2), nt, smem, st>>>(slab, qv, sum, g, R);
}

void launch_primary_epilogue(const uint32_t* fin, int nq, int nshards, const uint32_t* a_ms, const int* distinct_of,
                             uint16_t* sec_in, int chunk, const Group& g, const SlotMaps& maps, const NttTables& T,
                             cudaStream_t st) {
  const size_t smem = (size_t)4 * g.n * 4;
  dim3 grid(nshards, SIMD / 2, nq);
  set_smem(primary_epilogue_kernel, smem);
  primary_epilogue_kernel<<<grid, 256, smem, st>>>(fin, nshards, a_ms, distinct_of, sec_in, nq, chunk, g,
                                                   maps.uof, T, host_crt_const());
}

int epilogue_cols_supported(const Group& g) { return g.log2n == LOG2_N_MAX; }

void launch_epilogue_cols(const uint32_t* fin, int nq, int nshards, const uint32_t* a_ms, const int* distinct_of,
                          uint32_t* A, const SlotMaps& maps, const NttTables& T, cudaStream_t st) {
  const CrtConst cc = host_crt_const();
  const uint32_t k1q = (uint32_t)(((uint64_t)cc.q2inv1 << 32) / P1);
  const uint32_t k2q = (uint32_t)(((uint64_t)cc.q1inv2 << 32) / P2);
  // one lane per block while three blocks an SM hold them all (one query's first
  // kernel of the secondary phase and what follows, order 512, in us, one lane /
  // four: 8 shards 1162 / 1182, 32 1167 / 1180, 48 1175 / 1179, 64 1185 / 1181)
  if ((size_t)nshards * SIMD * nq <= 3 * (size_t)sm_count()) {
    primary_epilogue2k_kernel<1><<<dim3(nshards, SIMD, nq), EPI_NT, (size_t)2 * n2k::PS * 4, st>>>(
        fin, nshards, a_ms, distinct_of, A, maps.uof, T, cc.q2inv1, k1q, cc.q1inv2, k2q);
    return;
  }
  const size_t smem = (size_t)8 * n2k::PS * 4;
  set_smem(primary_epilogue2k_kernel<4>, smem);
  primary_epilogue2k_kernel<4><<<dim3(nshards, SIMD / 4, nq), EPI_NT, smem, st>>>(
      fin, nshards, a_ms, distinct_of, A, maps.uof, T, cc.q2inv1, k1q, cc.q1inv2, k2q);
}

int preload_pir_split_kernels() {
  // the runtime loads kernels lazily, at their first launch; this loads the
  // single-shard scan kernels now (cudaFuncGetAttributes forces the load)
  cudaFuncAttributes a;
  if (cudaFuncGetAttributes(&a, (const void*)scan_vectors_kernel) != cudaSuccess ||
      cudaFuncGetAttributes(&a, (const void*)lane_vectors_kernel) != cudaSuccess ||
      cudaFuncGetAttributes(&a, (const void*)scan_lanes_kernel) != cudaSuccess ||
      cudaFuncGetAttributes(&a, (const void*)epilogue_zq_kernel) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  return 0;
}

void launch_epilogue_zq(const uint32_t* sum, uint64_t* out, const Group& g, const SlotMaps& maps, const NttTables& T,
                        cudaStream_t st) {
  const size_t smem = (size_t)2 * (g.log2n == LOG2_N_MAX ? n2k::PS : (int)g.n) * 4;
  epilogue_zq_kernel<<<SIMD, ZQ_NT, smem, st>>>(sum, out, g, maps.uof, T, host_crt_const());
}

}  // namespace dnspir
