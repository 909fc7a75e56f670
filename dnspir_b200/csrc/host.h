// host.h -- host-side helpers shared by api.cu (device context, shards,
// shape rules) and fleet.cu (fleets and the answer pipeline).
#pragma once
#include <cuda_runtime.h>

#include <mutex>
#include <string>
#include <vector>

#include "dnspir.h"
#include "kernels.cuh"

namespace dnspir {

extern thread_local std::string g_err;
int fail(int code, const std::string& msg);

#define CK(call)                                                                                           \
  do {                                                                                                     \
    cudaError_t e_ = (call);                                                                               \
    if (e_ != cudaSuccess) {                                                                               \
      cudaGetLastError();                                                                                  \
      return fail(e_ == cudaErrorMemoryAllocation ? DNSPIR_ERR_OOM : DNSPIR_ERR_CUDA,                      \
                  std::string(#call) + ": " + cudaGetErrorString(e_));                                     \
    }                                                                                                      \
  } while (0)
#define CKR(expr)             \
  do {                        \
    int r_ = (expr);          \
    if (r_ != DNSPIR_OK) return r_; \
  } while (0)

// Constants of one set of a-parts on a device.  A shard or fleet keeps those that
// it was preprocessed under: dnspir_set_a_parts and the preprocessing of another
// shard may replace the context's at any time, in another thread as well.  The
// buffers live as long as the context.
struct APartConsts {
  uint64_t version = 0;
  const uint32_t* ntt = nullptr;   // a-parts in NTT form: [6][2][N], bit-reversed positions
  const uint32_t* scan = nullptr;  // scan constants: gka0, kappa, then qinv of each a-part set (ScanConsts)
  uint32_t na[2] = {};             // arrays per slab row of each a-part set: 2, or 3 when qry_a has a zero slot (slab_off)
};

struct DeviceCtx {
  int device = -1;
  uint32_t* tables = nullptr;
  NttTables T;
  APartConsts ap[LOG2_N_MAX + 1];  // of the a-parts last in effect
  uint32_t* galb[LOG2_N_MAX + 1] = {};
  uint32_t* gtab[LOG2_N_MAX + 1] = {};  // scan slot order: position -> odd residue
  uint32_t* uof[LOG2_N_MAX + 1] = {};   // natural slot -> position
  std::mutex mu;
};

// RAII device buffer
struct DBuf {
  void* p = nullptr;
  size_t bytes = 0;
  ~DBuf() {
    if (p) cudaFree(p);
  }
  int ensure(size_t b) {
    if (b <= bytes) return DNSPIR_OK;
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
    CK(cudaMalloc(&p, b));
    bytes = b;
    return DNSPIR_OK;
  }
  template <class T>
  T* as() const {
    return (T*)p;
  }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
  }
};

// RAII pinned host buffer (asynchronous copies need page-locked memory)
struct HBuf {
  void* p = nullptr;
  size_t bytes = 0;
  ~HBuf() {
    if (p) cudaFreeHost(p);
  }
  int ensure(size_t b) {
    if (b <= bytes) return DNSPIR_OK;
    if (p) cudaFreeHost(p);
    p = nullptr;
    bytes = 0;
    CK(cudaMallocHost(&p, b));
    bytes = b;
    return DNSPIR_OK;
  }
  template <class T>
  T* as() const {
    return (T*)p;
  }
};

// -------------------------------------------------------------- shard state
// Device buffers shared by set_db and the secondary phase.
struct EncodeWs {
  DBuf A, Ahat, in16, a_out, slab_ptrs;
  DBuf rows;  // chain layout of the shards in flight: entries, then states | digits (chain_rows_supported)
  // At most this much of it outlives a fleet's call: an update of eight half-size
  // or four full shards finds its scratch again (a call that allocates 2 GiB takes
  // 2.5 ms more of 5).
  static constexpr size_t ROWS_KEPT = (size_t)2 << 30;
};

struct DeviceGuard {
  int prev = -1;
  explicit DeviceGuard(int d) {
    cudaGetDevice(&prev);
    cudaSetDevice(d);
  }
  ~DeviceGuard() {
    if (prev >= 0) cudaSetDevice(prev);
  }
};

int get_ctx(int device, DeviceCtx** out);
// Per-dimension constants of a device, and those of the a-parts now in effect.
int ctx_consts(DeviceCtx* c, int log2n, APartConsts* ap);
// The six a-parts in effect for dimension 2^log2n (6 x N coefficients in
// [0, q): gk0, gk1, FirstSet query, its conjugate, SecondSet query, its
// conjugate) and their version.
void a_parts_host(int log2n, uint64_t* out, uint64_t* version);
uint64_t a_parts_version(int log2n);
SlotMaps slot_maps(DeviceCtx* c, int log2n);
ChainConsts chain_consts(DeviceCtx* c, const APartConsts& ap, int log2n, int used_seeds);
ScanConsts scan_consts(const APartConsts& ap, const Group& g, int used_seeds);
int check_group(uint32_t log2n, uint32_t l);
bool reduced(const uint64_t* v, size_t n);
// Encodes `count` shards' entries (device u16, one shard after another), runs
// the preprocessing chains and the a-part finalisation, and writes the slabs:
// lane layout, or tensor layout with `last` rows when last is given (tensor
// engine, chain_rows_supported).  Queued on st; the caller synchronises and
// looks at err (launch_primary_chain_rows).
int preprocess_shards(DeviceCtx* c, const APartConsts& ap, const Group& g, int used_seeds, uint32_t* const* slabs_host,
                      int count, const uint16_t* entries_dev, uint64_t* a_zq, uint32_t* a_ms, EncodeWs& ws,
                      uint32_t* err, const WaitLimits& lim, cudaStream_t st, uint32_t* last = nullptr);
// Whether the encoder may read the caller's entries where they are: on the device
// and on an 8-byte boundary (four coefficients a load); a view that starts on
// another coefficient is copied.
inline bool entries_in_place(const uint16_t* entries, int on_device) {
  return on_device && reinterpret_cast<uintptr_t>(entries) % 8 == 0;
}
// Shards that one call of preprocess_shards may carry, and its scratch for `count`.
uint32_t preprocess_batch(const Group& g);
int preprocess_reserve(const Group& g, uint32_t count, EncodeWs& ws);

}  // namespace dnspir
