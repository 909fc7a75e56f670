// kernels.cuh -- launch wrappers of the device kernels (host side declarations).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <map>
#include <mutex>
#include <utility>

#include "ntt.cuh"

namespace dnspir {

// Raises a kernel's dynamic shared-memory limit when a launch needs more than
// the default 48 KB.  The limit is one value per function and device and is
// only ever raised: kernels launched with several sizes are launched from
// several host threads (fleets, shards, the server), and a thread that set its
// smaller size between another's call and launch would have that launch refused.
inline void raise_smem_limit(const void* kernel, size_t bytes) {
  static std::mutex mu;
  static std::map<std::pair<int, const void*>, size_t> limits;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(mu);
  size_t& limit = limits[{dev, kernel}];
  if (bytes > limit &&
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess)
    limit = bytes;
}
template <class K>
inline void set_smem(K* kernel, size_t bytes) {
  if (bytes > 48 * 1024) raise_smem_limit((const void*)kernel, bytes);
}

// Streaming multiprocessors of the current device.
inline int sm_count() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

// Shape of one PIR database (IndexGroup, base_pir.rs:132-183).
struct Group {
  int log2n;    // ring dimension N = 2^log2n
  uint32_t n;   // N
  uint32_t l;   // group order
  uint32_t L;   // loop_len: l if l < N else N/2
  uint32_t H;   // halves: 2 if l == N (requires_conj) else 1
  uint32_t qbp; // query_base_power = N / 2 / L
  uint32_t na;  // stored arrays per slab row: 2 or 3 (slab_off)
};
Group make_group(int log2n, uint32_t l, uint32_t na = 3);

// Output slots of the scan are ordered by (sign, e): position u = sign * N/2 + e
// holds the slot k with 2k + 1 = (sign ? -1 : 1) 5^e mod 2N.  g[u] is that odd
// residue and uof[k] the position of natural slot k (device tables per N).
struct SlotMaps {
  const uint32_t* g;
  const uint32_t* uof;
};

// Scan-layout offset (in u32 words) of array a of row i, half h, factor p,
// output position u, lane 0 inside one shard slab.  What the arrays hold:
//   na = 2: 0 the chain state a_(i+1) after row i, 1 the high key digit G1
//   na = 3: 0 the entries E, 1 / 2 the key digits G0 / G1
// The reference scans three arrays (base_pir.rs:1085-1247).  They are tied by
// the chain that made them: with t_i = sigma_5(a_i) and G0 = t - 2^26 G1,
//     a_(i+1) = t_i gk_a0 + G1_i (gk_a1 - 2^26 gk_a0) + E_i qry_a   (mod p),
// so where qry_a is invertible at every slot, E_i follows from a_(i+1), a_i
// and G1_i, and t_i[j] = a_i[5 j] is array 0 of the row before at the slot the
// same output reads there.  A scan of two arrays against query vectors that
// carry the relation (launch_scan_vectors) is the same residue, with two
// thirds of the bytes and products.  na = 3 is kept for a-parts with a zero
// among qry_a's slots (about one set in 5500 at N = 2048).
__host__ __device__ __forceinline__ size_t slab_off(const Group& g, int p, int h, uint32_t i, int a, uint32_t k) {
  return (((((size_t)p * g.H + h) * g.L + i) * g.na + a) * g.n + k) * SIMD;
}
__host__ __device__ __forceinline__ size_t slab_words(const Group& g) {
  return (size_t)2 * g.H * g.L * g.na * g.n * SIMD;
}

// Constants of the two-array scan for one a-part set, (sign, e) slot order:
// gk_a0, gk_a1 - 2^26 gk_a0 and the inverses of qry_a of each half.
struct ScanConsts {
  const uint32_t* gka0;   // [p][N]
  const uint32_t* kappa;  // [p][N]
  const uint32_t* qinv;   // [half][p][N]
  uint32_t xscale[2], xinv[2];  // scale of the stored states per factor (chain_state_scale) and its inverse
};
// Query vectors of the scan, [q][half][v][factor][N] in (sign, e) order (12 N
// words a query): na = 2: v = 0, 1 multiply the stored arrays, v = 2 the state
// after the last row once more; na = 3: v = the query, gk0, gk1.  src: decoded
// vectors [slot][factor][N] in natural order, q_stride words apart, at slots
// s_q (conjugate half: s_q + 1), s_gk, s_gk + 1.  Queries nb .. nb_pad - 1 are
// written as zeros.
constexpr int SCAN_VECS = 3;
__host__ __device__ __forceinline__ size_t scan_vec_off(uint32_t n, int h, int v, int p) {
  return ((size_t)(h * SCAN_VECS + v) * 2 + p) * n;
}
void launch_scan_vectors(const uint32_t* src, size_t q_stride, int s_q, int s_gk, int nb, int nb_pad, uint32_t* qv,
                         const Group& g, const ScanConsts& sc, const SlotMaps& maps, cudaStream_t st);

// Limits of the bounded waits inside kernels, wait_ns (0: the default, 2 s; at
// least 0.1 ms, since a block that gave up waits under the same limit for its
// copies in flight, which take microseconds, before its memory is released), and
// the test hooks of the paths they end in (-1: off): the tensor scan's first
// block stops copying before chunk `withhold`, the second block of the first
// paired chain leaves before step `withhold_step`, in groups of `only_group`
// queries (0: in all).
struct WaitLimits {
  uint64_t wait_ns = 0;
  int withhold = -1;
  int withhold_step = -1;
  int only_group = 0;
  uint64_t ns() const { return wait_ns == 0 ? 2000000000ull : wait_ns < 100000 ? 100000 : wait_ns; }
  WaitLimits of_group(int nb) const {
    WaitLimits l = *this;
    if (only_group && only_group != nb) l.withhold = l.withhold_step = -1;
    return l;
  }
};

// ---- DB encoding (set_transformed_entries, base_pir.rs:662-772)
// in: coefficients [t < l_in][lane < nl][n < N] (< t); A: [t][lane][x] (q1, transform
// position x = slot brv(x))
void launch_encode_cols(const uint16_t* in, uint32_t* A, const Group& g, uint32_t l_in, int nl, const NttTables& T,
                        cudaStream_t st);
// A -> Ahat[h][r][lane][x] (q1, position x = slot brv(x)): evaluations of column polys at the Galois orbit
void launch_encode_rows(const uint32_t* A, uint32_t* Ahat, const Group& g, uint32_t l_in, int nl, const NttTables& T,
                        cudaStream_t st);
// Ahat -> transformed entries.  frame 0: scan layout in `slab` (nl == 8);
// frame 1: chain layout out[((p*H + h)*L + r)*nl + lane][pos] in bit-reversed slot order,
// row r for chain step L - 1 - r; out may be Ahat itself (its rows become factor 0).
void launch_encode_lift(const uint32_t* Ahat, uint32_t* out, const Group& g, int nl, int frame, const SlotMaps& maps,
                        const NttTables& T, cudaStream_t st);

// ---- key-switch chain (preprocess / partial_gal, base_pir.rs:496-594, 782-863)
struct ChainConsts {
  const uint32_t* gka;    // [digit][p][pos]  (bit-reversed slot order)
  const uint32_t* qa;     // [half][p][pos]   (qry_a for the database's seed set)
  const uint32_t* galb;   // [pos] -> destination position of sigma_5 (bit-reversed coordinates)
  SlotMaps maps;          // scan-layout slot order
};
// Primary preprocessing chain for `nshards` shards (slabs[s] already hold E);
// writes G0/G1 into the slabs and a_out[s][h][lane][p][pos].
void launch_primary_chain(uint32_t* const* slabs_dev, int nshards, uint32_t* a_out, const Group& g,
                          const ChainConsts& cc, const NttTables& T, cudaStream_t st);
// The same at N = 2048 with two stored arrays (chain_rows_supported): shard s's
// rows (launch_encode_lift, frame 1, nl = 8) lie at rows + s * shard_words and
// take the states, times the factor's CRT constant, in place; the high digits
// go to digits + s * shard_words, the same layout [p][half][r][lane][pos] with
// row r for chain step L - 1 - r (chain_rows_words a shard).  err: one device word
// set to 1 when a bounded wait between the blocks of a chain gave up (here and in
// launch_secondary_chain).
int chain_rows_supported(const Group& g);
size_t chain_rows_words(const Group& g);
void launch_primary_chain_rows(uint32_t* rows, uint32_t* digits, size_t shard_words, int nshards, uint32_t* a_out,
                               uint32_t* err, const WaitLimits& lim, const Group& g, const ChainConsts& cc,
                               const NttTables& T, cudaStream_t st);
// Rows of `words` words in all: bit-reversed positions -> (sign, e) order, in place.
void launch_order_rows(uint32_t* rows, size_t words, const SlotMaps& maps, cudaStream_t st);
// One shard's rows and digits (bit-reversed positions) -> its lane-layout slab.
void launch_lane_rows(const uint32_t* rows, const uint32_t* digits, uint32_t* slab, const Group& g,
                      const SlotMaps& maps, cudaStream_t st);
// Scale that the stored states carry mod factor p, and its inverse (1 where the
// generic chain stores them).
void chain_state_scale(const Group& g, int p, uint32_t* scale, uint32_t* inverse);
// Sums the halves of a_out, returns reply_a as Z_q coefficients (u64) and the
// 17-bit mod-switched a-part (u32) per shard: [s][lane][n].
void launch_primary_finalize(const uint32_t* a_out, int nshards, uint64_t* a_zq, uint32_t* a_ms, const Group& g,
                             const NttTables& T, cudaStream_t st);

// Secondary chain fused with the secondary scan (homomorphic evaluation of
// the secondary database on each query's ciphertext).  E: chain layout from
// launch_encode_lift(frame 1) with nl = 3 * nq lanes; qv: per query decoded
// vectors [q][slot][p][pos] (bit-reversed), slots 0 gk0, 1 gk1, 2 pq, 3 pqc, 4 sq, 5 sqc.
// out: [q][h][part][a/b][p][pos].
// sc: scan_consts of the secondary's a-part set; zeros: one of its query slots is zero.
void launch_secondary_chain(const uint32_t* E, const uint32_t* qv, size_t qv_stride, int nq, uint32_t* out,
                            uint32_t* err, const WaitLimits& lim, const Group& g, const ChainConsts& cc,
                            const ScanConsts& sc, bool zeros, const NttTables& T, cudaStream_t st,
                            bool clustered = false);
// Queries whose chains fill the SMs once.
int secondary_chain_wave(const Group& g, int sms);

// ---- primary scan (main_pir_loop, base_pir.rs:1085-1247)
// B queries (a power of two up to 256) in one launch over all shards, each
// block serving per_block of them (1, 2, 4, 8 or 16; 0: min(B, 8)), the groups
// of one tile in consecutive blocks.  qv: launch_scan_vectors of B queries.  out:
// [b][s][p][u][lane] reduced mod p.
int scan_batch_supported(int B);
int launch_scan_batch(uint32_t* const* slabs_dev, int nshards, const uint32_t* qv, int B, int per_block, uint32_t* out,
                      const Group& g, cudaStream_t st);
// ---- primary scan on the tensor cores (tscan.cu): 8-bit limbs, kind::i8
// Tensor layout: the slab indexed by query slot, bytes in 128 x 128 blocks
// [p][sign][m-tile][k-chunk] (same size as the lane layout).  Needs loop_len
// = N/2 and N >= 256.
struct TScanShape {
  int nq;          // rows of the query operand per CTA (4 limbs x queries)
  int mtpc;        // 128-row m-tiles per CTA
  int stages;      // shared-memory pipeline depth
  int persistent;  // 1: persistent warp-specialised kernel; 2: CTA pair (relayed bulk copies); 3: CTA pair (tensor maps)
};
int tensor_layout_supported(const Group& g);
void tensor_dims(const Group& g, uint32_t* mt_total, uint32_t* kc_total);
void launch_retile(const uint32_t* lane_slab, uint8_t* tensor_slab, const Group& g, cudaStream_t st);
// The same from one shard's rows and digits in (sign, e) order (launch_order_rows).
void launch_retile_rows(const uint32_t* rows, const uint32_t* digits, uint8_t* tensor_slab, const Group& g,
                        cudaStream_t st);
const TScanShape* tscan_shapes(int* count);
size_t tscan_query_bytes(const Group& g, int nb_pad);
// nb queries (qv: launch_scan_vectors) padded to nb_pad (a multiple of
// shape.nq / 4); qb: tscan_query_bytes of workspace; out as
// launch_scan_batch; err: one device word set to 1 when a bounded wait gave
// up.  last: the distinct shards' states after the last row
// (launch_last_rows), distinct_of the distinct shard of each shard (na = 2).
// Returns -1 for a shape that does not fit.
// slab_maps: tscan_slab_maps of the shards (device), required by the
// tensor-map pair shapes (persistent 3), which are refused (-1) without it.
int launch_tscan(uint8_t* const* slabs_dev, int nshards, const uint32_t* qv, int nb, int nb_pad, uint8_t* qb,
                 uint32_t* out, uint32_t* err, const uint32_t* last, const int* distinct_of, const Group& g,
                 const TScanShape& shape, cudaStream_t st, const WaitLimits& lim = WaitLimits(),
                 const void* slab_maps = nullptr);
// A shard's chain state after its last row times 2^32, [p][u][half][lane] (na =
// 2), from its a_out (launch_primary_chain).
size_t last_rows_words(const Group& g);
void launch_last_rows(const uint32_t* a_out, uint32_t* last, const Group& g, const ScanConsts& sc, const SlotMaps& maps,
                      cudaStream_t st);
// Tensor maps of the shards' tensor-layout slabs (host pointers; one map of
// tscan_slab_map_bytes(1) bytes per shard) written to dev_maps; -1 when the
// driver cannot encode them.
size_t tscan_slab_map_bytes(int nshards);
int tscan_slab_maps(uint8_t* const* host_slabs, int nshards, const Group& g, void* dev_maps);
// Per-lane queries (perform_pir_split).  launch_lane_vectors: ring elements zq
// [lane][query, conjugate, gk0, gk1][N] -> the scan vectors of 8 queries, one per
// lane, and sum (scan_lanes_sum_words) cleared; ntt: their transforms' space at N >
// 512.  launch_scan_lanes adds the scan up in sum.
void launch_lane_vectors(const uint64_t* zq, uint32_t* ntt, uint32_t* qv, uint32_t* sum, const Group& g,
                         const ScanConsts& sc, const SlotMaps& maps, const NttTables& T, cudaStream_t st);
constexpr int SCAN_MAX_CHUNKS = 16;  // row chunks per half
size_t scan_lanes_sum_words(const Group& g);
void launch_scan_lanes(const uint32_t* slab, const uint32_t* qv, uint32_t* sum, const Group& g, cudaStream_t st);
// Loads the kernels of launch_lane_vectors, launch_scan_lanes and
// launch_epilogue_zq on the current device (0, or -1 on a CUDA error).
int preload_pir_split_kernels();
// Primary epilogue for nq queries: scan output -> b (iNTT, CRT), mod-switch,
// combine with the shard's a-part, three base-1025 digits -> secondary
// entries.  Queries are grouped in chunks of `chunk`; chunk c starts at
// c * chunk * 3 * nshards * 8 * N and holds [t = s*8+lane][q*3 + part][n].
void launch_primary_epilogue(const uint32_t* fin, int nq, int nshards, const uint32_t* a_ms, const int* distinct_of,
                             uint16_t* sec_in, int chunk, const Group& g, const SlotMaps& maps, const NttTables& T,
                             cudaStream_t st);
// The same for one chunk of nq queries at N = 2048, ending in the encoder's
// column transforms A [t][lane][x] (launch_encode_cols' output) instead of entries.
int epilogue_cols_supported(const Group& g);
void launch_epilogue_cols(const uint32_t* fin, int nq, int nshards, const uint32_t* a_ms, const int* distinct_of,
                          uint32_t* A, const SlotMaps& maps, const NttTables& T, cudaStream_t st);
// Epilogue returning b as Z_q coefficients [lane][n] (shard-level perform_pir_split).
void launch_epilogue_zq(const uint32_t* sum, uint64_t* out, const Group& g, const SlotMaps& maps, const NttTables& T,
                        cudaStream_t st);

// ---- wire codec (pir_wrapper.rs:84-158, 370-408)
// Decodes one query's polynomials: poly_off/poly_bits per polynomial (npoly),
// writes natural-order vectors qnat[poly][p][u] and bit-reversed qbrv[poly][p][pos].
struct PolySpec {
  uint32_t off[6];   // byte offset of each polynomial in the query
  uint32_t bits[6];  // its wire width
  int slot[6];       // destination slot: 0 gk0, 1 gk1, 2 pq, 3 pqc, 4 sq, 5 sqc
  int npoly;
};
// Per query of a group: offset of its bytes, and its session slot (-1: the
// query carries its own Galois keys; otherwise they come from the session
// cache and the bytes omit them, gk_bytes shorter).
struct QDesc {
  uint32_t byte_off;
  int32_t session;
};
// nq queries, outputs at q * q_stride words.
void launch_decode_query(const uint8_t* bytes, const QDesc* desc, int nq, const PolySpec& spec, uint32_t gk_bytes,
                         uint32_t* qnat, uint32_t* qbrv, size_t q_stride, const uint32_t* sess_nat,
                         const uint32_t* sess_brv, int log2n, const NttTables& T, cudaStream_t st);
// Ring elements (Z_q, u64) -> NTT vectors, natural [i][p][u] and bit-reversed [i][p][pos].
void launch_ring_to_ntt(const uint64_t* zq, int count, uint32_t* qnat, uint32_t* qbrv, int log2n, const NttTables& T,
                        cudaStream_t st);
// Secondary chain output -> reply bytes (3 x (17-bit a, 12-bit b)) or Z_q ciphertexts.
void launch_reply(const uint32_t* chain_out, int nq, int H, uint8_t* reply_bytes, size_t reply_stride,
                  uint64_t* reply_zq, int log2n, const NttTables& T, cudaStream_t st);

// Device table of 5^r (inverse: 5^-r) mod 2N for r <= N/2.
const uint32_t* device_pow5(int log2n, bool inverse);

// Read-only view of a shard (api.cu) for the no-allocation entry point (noalloc.cu).
struct DbView {
  int device;
  bool ready;
  Group g;
  const uint32_t* slab;
  NttTables T;
  SlotMaps maps;
  ScanConsts sc;
};

// Payload helpers for synthetic databases (dns/bucket.rs:289-303 packing).
void launch_pack_bytes(const uint8_t* bytes, uint16_t* coeffs, size_t entries, int log2n, cudaStream_t st);

}  // namespace dnspir
