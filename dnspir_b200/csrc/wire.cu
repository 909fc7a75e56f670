// wire.cu -- query unpacking and reply packing on the device
// (process_queries, crates/pir/src/pir_wrapper.rs:370-408; uncondense :120-158,
// condense :84-113; mod_switch_decode / mod_switch_encode, bfv.rs:52-69).
#include "kernels.cuh"
#include "ntt2048.cuh"

namespace dnspir {
namespace {

// One coefficient of a condense<bits> stream of N values (pir_wrapper.rs:84-113):
// whole bytes first (one plane of N bytes per byte), then a nibble plane,
// a 2-bit plane and a 1-bit plane, each only when the width needs it.
__device__ __forceinline__ uint64_t unpack_one(const uint8_t* __restrict__ b, int bits, uint32_t N, uint32_t n) {
  uint64_t x = 0;
  size_t pos = 0;
  for (int i = 0; i < bits / 8; i++) {
    x |= (uint64_t)b[pos + n] << (8 * i);
    pos += N;
  }
  if (bits % 8 >= 4) {
    const uint8_t s = b[pos + n / 2];
    x |= (uint64_t)((n & 1) ? (s & 0xF) : (s >> 4)) << ((bits / 8) * 8);
    pos += N / 2;
  }
  if (bits % 4 >= 2) {
    const uint8_t s = b[pos + n / 4];
    x |= (uint64_t)((s >> (6 - 2 * (n % 4))) & 3) << ((bits / 4) * 4);
    pos += N / 4;
  }
  if (bits % 2 >= 1) {
    const uint8_t s = b[pos + n / 8];
    x |= (uint64_t)((s >> (7 - n % 8)) & 1) << ((bits / 2) * 2);
  }
  return x;
}

// grid: x = polynomial of the query, y = factor, z = query of the group.
// Outputs natural-order qnat[slot][p][u] and bit-reversed qbrv[slot][p][pos]
// at q * q_stride.  A query with a session takes its Galois-key slots 0 and 1
// from the session cache ([session][slot][p][N], natural and bit-reversed)
// and its bytes start with the first polynomial after the keys.
__global__ void decode_query_kernel(const uint8_t* __restrict__ bytes, const QDesc* __restrict__ desc, PolySpec spec,
                                    uint32_t gk_bytes, uint32_t* __restrict__ qnat, uint32_t* __restrict__ qbrv,
                                    size_t q_stride, const uint32_t* __restrict__ sess_nat,
                                    const uint32_t* __restrict__ sess_brv, int log2n, NttTables T) {
  extern __shared__ uint32_t sm[];
  const int poly = blockIdx.x, p = blockIdx.y, q = blockIdx.z;
  const uint32_t N = 1u << log2n;
  const uint32_t pr = prime_of(p);
  const int bits = spec.bits[poly];
  const QDesc d = desc[q];
  const int slot = spec.slot[poly];
  qnat += (size_t)q * q_stride;
  qbrv += (size_t)q * q_stride;
  if (d.session >= 0 && slot < 2) {
    const size_t o = (((size_t)d.session * 2 + slot) * 2 + p) * N;
    for (uint32_t u = threadIdx.x; u < N; u += blockDim.x) {
      qnat[((size_t)slot * 2 + p) * N + u] = sess_nat[o + u];
      qbrv[((size_t)slot * 2 + p) * N + u] = sess_brv[o + u];
    }
    return;
  }
  const uint8_t* src = bytes + d.byte_off + spec.off[poly] - (d.session >= 0 ? gk_bytes : 0);
  for (uint32_t n = threadIdx.x; n < N; n += blockDim.x) {
    const uint64_t v = ms_decode(unpack_one(src, bits, N, n), bits);
    sm[n] = reduce64(v, pr, barrett_mu(pr));
  }
  __syncthreads();
  ntt_fwd_smem(sm, log2n, 1, T, p);
  uint32_t* on = qnat + ((size_t)slot * 2 + p) * N;
  uint32_t* ob = qbrv + ((size_t)slot * 2 + p) * N;
  for (uint32_t u = threadIdx.x; u < N; u += blockDim.x) {
    on[u] = sm[brv(u, log2n)];
    ob[u] = sm[u];
  }
}

// ---- N = 2048: the codec on the register transforms of ntt2048.cuh, one
// polynomial (both factors of one ciphertext polynomial for replies) per block.
// A single query's codec is latency: decode 20 -> 8.5 us, reply 40 -> 6.6 us.
constexpr int WIRE_NT = 256;

// transformed polynomial in sm (padded positions) -> natural and bit-reversed order
__device__ __forceinline__ void store_both_orders(const uint32_t* sm, uint32_t* on, uint32_t* ob) {
  using namespace n2k;
#pragma unroll
  for (int c = 0; c < 2; c++) {
    const int q = threadIdx.x + WIRE_NT * c;
    if (ob) reinterpret_cast<uint4*>(ob)[q] = *reinterpret_cast<const uint4*>(sm + phys(4 * q));
    if (on)
      reinterpret_cast<uint4*>(on)[q] = make_uint4(sm[phys(brv11(4 * q))], sm[phys(brv11(4 * q + 1))],
                                                   sm[phys(brv11(4 * q + 2))], sm[phys(brv11(4 * q + 3))]);
  }
}

__global__ void __launch_bounds__(WIRE_NT) decode_query2k_kernel(
    const uint8_t* __restrict__ bytes, const QDesc* __restrict__ desc, PolySpec spec, uint32_t gk_bytes,
    uint32_t* __restrict__ qnat, uint32_t* __restrict__ qbrv, size_t q_stride, const uint32_t* __restrict__ sess_nat,
    const uint32_t* __restrict__ sess_brv, NttTables T) {
  using namespace n2k;
  __shared__ __align__(16) uint32_t sm[PS];
  const int poly = blockIdx.x, p = blockIdx.y, q = blockIdx.z;
  const uint32_t pr = prime_of(p);
  const int bits = spec.bits[poly], slot = spec.slot[poly];
  const QDesc d = desc[q];
  qnat += (size_t)q * q_stride + ((size_t)slot * 2 + p) * N;
  qbrv += (size_t)q * q_stride + ((size_t)slot * 2 + p) * N;
  if (d.session >= 0 && slot < 2) {
    const size_t o = (((size_t)d.session * 2 + slot) * 2 + p) * N;
#pragma unroll
    for (int c = 0; c < 2; c++) {
      const int x = threadIdx.x + WIRE_NT * c;
      reinterpret_cast<uint4*>(qnat)[x] = __ldg(reinterpret_cast<const uint4*>(sess_nat + o) + x);
      reinterpret_cast<uint4*>(qbrv)[x] = __ldg(reinterpret_cast<const uint4*>(sess_brv + o) + x);
    }
    return;
  }
  const uint8_t* src = bytes + d.byte_off + spec.off[poly] - (d.session >= 0 ? gk_bytes : 0);
  // coefficients 8t .. 8t + 7: one 8-byte load per whole-byte plane, and their
  // 4, 2 and 1 bytes of the nibble, 2-bit and 1-bit planes (every polynomial
  // starts on a multiple of 8 bytes: plane lengths are multiples of N / 8)
  {
    const int t = threadIdx.x, whole = bits / 8;
    uint64_t plane[7];
#pragma unroll
    for (int i = 0; i < 7; i++) plane[i] = i < whole ? __ldg(reinterpret_cast<const uint64_t*>(src + (size_t)i * N) + t) : 0;
    const uint8_t* rest = src + (size_t)whole * N;
    uint32_t nib = 0, two = 0, one = 0;
    if (bits % 8 >= 4) {
      nib = __ldg(reinterpret_cast<const uint32_t*>(rest) + t);
      rest += N / 2;
    }
    if (bits % 4 >= 2) {
      two = __ldg(reinterpret_cast<const uint16_t*>(rest) + t);
      rest += N / 4;
    }
    if (bits % 2) one = __ldg(rest + t);
    const int o = (int)phys(8 * t);
#pragma unroll
    for (int j = 0; j < 8; j++) {
      uint64_t x = 0;
#pragma unroll
      for (int i = 0; i < 7; i++) x |= ((plane[i] >> (8 * j)) & 0xFF) << (8 * i);
      // each byte of a partial plane holds its first coefficient in its top bits
      x |= (uint64_t)((nib >> (8 * (j / 2) + (j % 2 ? 0 : 4))) & 0xF) << (8 * whole);
      x |= (uint64_t)((two >> (8 * (j / 4) + 6 - 2 * (j % 4))) & 3) << (4 * (bits / 4));
      x |= (uint64_t)((one >> (7 - j)) & 1) << (2 * (bits / 2));
      sm[o + j] = reduce64(ms_decode(x, bits), pr, barrett_mu(pr));
    }
  }
  __syncthreads();
  fwd<WIRE_NT>(sm, p == 0, p == 1, T);
  store_both_orders(sm, qnat, qbrv);
}

__global__ void __launch_bounds__(WIRE_NT) ring_to_ntt2k_kernel(const uint64_t* __restrict__ zq,
                                                                uint32_t* __restrict__ qnat,
                                                                uint32_t* __restrict__ qbrv, NttTables T) {
  using namespace n2k;
  __shared__ __align__(16) uint32_t sm[PS];
  const int i = blockIdx.x, p = blockIdx.y;
  const uint32_t pr = prime_of(p);
#pragma unroll
  for (int c = 0; c < N / WIRE_NT; c++) {
    const uint32_t n = threadIdx.x + WIRE_NT * c;
    sm[phys(n)] = reduce64(__ldg(zq + (size_t)i * N + n), pr, barrett_mu(pr));
  }
  __syncthreads();
  fwd<WIRE_NT>(sm, p == 0, p == 1, T);
  const size_t o = ((size_t)i * 2 + p) * N;
  store_both_orders(sm, qnat ? qnat + o : nullptr, qbrv ? qbrv + o : nullptr);
}

// mod_switch_encode of v in [0, q) to BITS bits, round(v 2^BITS / q) = floor((v
// 2^(BITS+1) + q) / 2q): a double estimate within one of it, corrected by the
// remainder, which is below 4q in magnitude and so exact modulo 2^64 although
// its terms may not be.
template <int BITS>
__device__ __forceinline__ uint32_t ms_encode_small(uint64_t v) {
  constexpr double SCALE = (double)(1u << BITS) / (double)QQ;
  const int64_t r = (int64_t)floor((double)v * SCALE + 0.5);
  const int64_t rem = (int64_t)((v << (BITS + 1)) + QQ - (uint64_t)r * (2 * QQ));
  return (uint32_t)(r + (rem >= (int64_t)(2 * QQ)) - (rem < 0)) & ((1u << BITS) - 1);
}

// Ends the inverse transforms unscaled: N^-1 sits in the CRT constants.
struct PlainStore {
  __device__ __forceinline__ void operator()(uint32_t* y, int, int, uint32_t (&v)[8], uint32_t, uint32_t,
                                             uint32_t) const {
#pragma unroll
    for (int k = 0; k < 8; k++) y[k * n2k::Geo8<1>::STR] = v[k];
  }
};

// grid: x = ciphertext part * 2 + (0: a, 1: b), y = query.
constexpr int REPLY_NT = 512;
__global__ void __launch_bounds__(REPLY_NT) reply2k_kernel(const uint32_t* __restrict__ chain_out, int H,
                                                           uint8_t* __restrict__ reply_bytes, size_t reply_stride,
                                                           uint64_t* __restrict__ reply_zq, NttTables T, uint32_t k1,
                                                           uint32_t k1q, uint32_t k2, uint32_t k2q) {
  using namespace n2k;
  __shared__ __align__(16) uint32_t sm[2 * PS];
  const int part = blockIdx.x >> 1, ab = blockIdx.x & 1, q = blockIdx.y;
#pragma unroll
  for (int p = 0; p < 2; p++) {
    const int x = threadIdx.x;  // quad of positions
    const uint4* src = reinterpret_cast<const uint4*>(
                           chain_out + ((((size_t)q * H * CTXT_PARTS + part) * 2 + ab) * 2 + p) * N) + x;
    uint4 v = __ldg(src);
    if (H == 2) {
      const uint4 w = __ldg(src + (size_t)CTXT_PARTS * 4 * (N / 4));
      const uint32_t pr = prime_of(p);
      v = make_uint4(add_mod(v.x, w.x, pr), add_mod(v.y, w.y, pr), add_mod(v.z, w.z, pr), add_mod(v.w, w.w, pr));
    }
    *reinterpret_cast<uint4*>(sm + p * PS + phys(4 * x)) = v;
  }
  __syncthreads();
  inv<REPLY_NT>(sm, 1, 1, T, PlainStore());
  uint32_t e[4];
#pragma unroll
  for (int c = 0; c < 4; c++) {
    const int n = threadIdx.x + REPLY_NT * c;
    const uint32_t x1 = shoup_mul(sm[phys(n)], k1, k1q, P1), x2 = shoup_mul(sm[PS + phys(n)], k2, k2q, P2);
    uint64_t v = (uint64_t)x1 * P2 + (uint64_t)x2 * P1;
    v = v >= QQ ? v - QQ : v;
    if (reply_zq)
      reply_zq[(((size_t)q * CTXT_PARTS + part) * 2 + ab) * N + n] = v;
    else
      e[c] = ab ? ms_encode_small<SEC_B_BITS>(v) : ms_encode_small<SEC_A_BITS>(v);
  }
  if (reply_zq) return;
  // condense (pir_wrapper.rs:84-113): byte planes, then the a-part's bit plane
  // (first coefficient in the top bit) or the b-part's nibble plane
  constexpr uint32_t abytes = N * SEC_A_BITS / 8, bbytes = N * SEC_B_BITS / 8;
  uint8_t* out = reply_bytes + (size_t)q * reply_stride + (size_t)part * (abytes + bbytes) + (ab ? abytes : 0);
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int c = 0; c < 4; c++) {
    const int n = threadIdx.x + REPLY_NT * c;
    out[n] = (uint8_t)e[c];
    if (!ab) {
      out[N + n] = (uint8_t)(e[c] >> 8);
      const uint32_t m = __ballot_sync(0xffffffffu, (e[c] >> 16) & 1);  // bit i: coefficient of lane i
      if ((lane & 7) == 0) out[2 * N + n / 8] = (uint8_t)(__brev((m >> lane) & 0xffu) >> 24);
    } else {
      const uint32_t next = __shfl_down_sync(0xffffffffu, e[c], 1);
      if ((lane & 1) == 0) out[N + n / 2] = (uint8_t)((((e[c] >> 8) & 0xF) << 4) | ((next >> 8) & 0xF));
    }
  }
}

__global__ void ring_to_ntt_kernel(const uint64_t* __restrict__ zq, uint32_t* __restrict__ qnat,
                                   uint32_t* __restrict__ qbrv, int log2n, NttTables T) {
  extern __shared__ uint32_t sm[];
  const int i = blockIdx.x, p = blockIdx.y;
  const uint32_t N = 1u << log2n;
  const uint32_t pr = prime_of(p);
  for (uint32_t n = threadIdx.x; n < N; n += blockDim.x) sm[n] = reduce64(zq[(size_t)i * N + n], pr, barrett_mu(pr));
  __syncthreads();
  ntt_fwd_smem(sm, log2n, 1, T, p);
  for (uint32_t u = threadIdx.x; u < N; u += blockDim.x) {
    if (qnat) qnat[((size_t)i * 2 + p) * N + u] = sm[brv(u, log2n)];
    if (qbrv) qbrv[((size_t)i * 2 + p) * N + u] = sm[u];
  }
}

// grid: x = ciphertext part, y = query.  Sums the two halves of the secondary
// chain, returns to coefficients, CRT, and either stores Z_q values or the
// mod-switched, condensed reply (pir_wrapper.rs:401-408).
__global__ void reply_kernel(const uint32_t* __restrict__ chain_out, int H, uint8_t* __restrict__ reply_bytes,
                             size_t reply_stride, uint64_t* __restrict__ reply_zq, int log2n, NttTables T,
                             CrtConst crtc) {
  extern __shared__ uint32_t sm[];  // [a q1 | b q1 | a q2 | b q2]
  const int part = blockIdx.x, q = blockIdx.y;
  const uint32_t N = 1u << log2n;
  for (uint32_t b = threadIdx.x; b < 4 * N; b += blockDim.x) {
    const uint32_t poly = b >> log2n, pos = b & (N - 1);
    const uint32_t p = poly >> 1, ab = poly & 1;
    const uint32_t pr = prime_of(p);
    uint32_t v = 0;
    for (int h = 0; h < H; h++)
      v = add_mod(v, chain_out[((((size_t)q * H + h) * CTXT_PARTS + part) * 2 + ab) * 2 * N + p * N + pos], pr);
    sm[b] = v;
  }
  __syncthreads();
  ntt_inv_smem2(sm, log2n, 2, 2, T);
  for (uint32_t n = threadIdx.x; n < N; n += blockDim.x) {
    const uint64_t va = crt(sm[n], sm[2 * N + n], crtc);
    const uint64_t vb = crt(sm[N + n], sm[3 * N + n], crtc);
    if (reply_zq) {
      reply_zq[(((size_t)q * CTXT_PARTS + part) * 2 + 0) * N + n] = va;
      reply_zq[(((size_t)q * CTXT_PARTS + part) * 2 + 1) * N + n] = vb;
    } else {
      sm[n] = ms_encode(va, SEC_A_BITS);
      sm[N + n] = ms_encode(vb, SEC_B_BITS);
    }
  }
  if (reply_zq) return;
  __syncthreads();
  const uint32_t abytes = N * SEC_A_BITS / 8, bbytes = N * SEC_B_BITS / 8;
  uint8_t* out = reply_bytes + (size_t)q * reply_stride + (size_t)part * (abytes + bbytes);
  const uint32_t* ea = sm;
  const uint32_t* eb = sm + N;
  for (uint32_t n = threadIdx.x; n < N; n += blockDim.x) {
    out[n] = (uint8_t)ea[n];
    out[N + n] = (uint8_t)(ea[n] >> 8);
    uint8_t* ob = out + abytes;
    ob[n] = (uint8_t)eb[n];
  }
  for (uint32_t m = threadIdx.x; m < N / 8; m += blockDim.x) {
    uint8_t v = 0;
    for (int u = 0; u < 8; u++) v |= (uint8_t)(((ea[8 * m + u] >> 16) & 1) << (7 - u));
    out[2 * N + m] = v;
  }
  for (uint32_t m = threadIdx.x; m < N / 2; m += blockDim.x) {
    out[abytes + N + m] = (uint8_t)((((eb[2 * m] >> 8) & 0xF) << 4) | ((eb[2 * m + 1] >> 8) & 0xF));
  }
}

}  // namespace

CrtConst host_crt_const();

void launch_decode_query(const uint8_t* bytes, const QDesc* desc, int nq, const PolySpec& spec, uint32_t gk_bytes,
                         uint32_t* qnat, uint32_t* qbrv, size_t q_stride, const uint32_t* sess_nat,
                         const uint32_t* sess_brv, int log2n, const NttTables& T, cudaStream_t st) {
  if (nq <= 0) return;
  dim3 grid(spec.npoly, 2, nq);
  if (log2n == LOG2_N_MAX) {
    decode_query2k_kernel<<<grid, WIRE_NT, 0, st>>>(bytes, desc, spec, gk_bytes, qnat, qbrv, q_stride, sess_nat,
                                                    sess_brv, T);
    return;
  }
  decode_query_kernel<<<grid, 256, (size_t)4 << log2n, st>>>(bytes, desc, spec, gk_bytes, qnat, qbrv, q_stride,
                                                              sess_nat, sess_brv, log2n, T);
}

void launch_ring_to_ntt(const uint64_t* zq, int count, uint32_t* qnat, uint32_t* qbrv, int log2n, const NttTables& T,
                        cudaStream_t st) {
  if (count <= 0) return;
  dim3 grid(count, 2);
  if (log2n == LOG2_N_MAX) {
    ring_to_ntt2k_kernel<<<grid, WIRE_NT, 0, st>>>(zq, qnat, qbrv, T);
    return;
  }
  ring_to_ntt_kernel<<<grid, 256, (size_t)4 << log2n, st>>>(zq, qnat, qbrv, log2n, T);
}

void launch_reply(const uint32_t* chain_out, int nq, int H, uint8_t* reply_bytes, size_t reply_stride,
                  uint64_t* reply_zq, int log2n, const NttTables& T, cudaStream_t st) {
  if (log2n == LOG2_N_MAX) {
    const CrtConst cc = host_crt_const();
    const uint32_t k1 = (uint32_t)((uint64_t)cc.q2inv1 * T.ninv[0][LOG2_N_MAX] % P1);
    const uint32_t k2 = (uint32_t)((uint64_t)cc.q1inv2 * T.ninv[1][LOG2_N_MAX] % P2);
    reply2k_kernel<<<dim3(2 * CTXT_PARTS, nq), REPLY_NT, 0, st>>>(
        chain_out, H, reply_bytes, reply_stride, reply_zq, T, k1, (uint32_t)(((uint64_t)k1 << 32) / P1), k2,
        (uint32_t)(((uint64_t)k2 << 32) / P2));
    return;
  }
  dim3 grid(CTXT_PARTS, nq);
  const size_t smem = (size_t)16 << log2n;
  set_smem(reply_kernel, smem);
  reply_kernel<<<grid, 256, smem, st>>>(chain_out, H, reply_bytes, reply_stride, reply_zq, log2n, T, host_crt_const());
}

}  // namespace dnspir
