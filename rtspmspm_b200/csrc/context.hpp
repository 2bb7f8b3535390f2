// Engine context and host-side helpers shared by the C-ABI implementation.
#pragma once

#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <initializer_list>
#include <string>
#include <vector>

#include "../../include/rtspmspm.h"
#include "common.cuh"
#include "kernels.hpp"
#include "mlp.hpp"

struct spg_ctx {
  int device = 0;
  int sms = 148;
  cudaStream_t own_stream = nullptr;
  cudaStream_t stream = nullptr;
  cudaStream_t copy_stream = nullptr;  // device-to-host copies overlapped with compute (created on first use)
  cudaStream_t upload_stream = nullptr;  // host-to-device copies of input row chunks (created on first use)
  cudaMemPool_t pool = nullptr;     // results (the device's default pool)
  cudaMemPool_t scratch = nullptr;  // a call's work memory (shared by the device's contexts)
  unsigned long long driver_ctx = 0;  // driver_ctx_id() at its creation
  cudaEvent_t ev_start = nullptr, ev_end = nullptr;  // StageTimer's
  std::string last_error;
  std::string gpu_name;
  spg_tuning tuning{};
  // predictor state (device)
  float* mlp_master = nullptr;  // FP32 master weights
  void* mlp_w16 = nullptr;      // BF16 copy used by the kernels
  bool mlp_loaded = false;
  // small device scratch
  int* d_flags = nullptr;
  unsigned long long* d_counter = nullptr;  // tile queue / retry / unit counters (16 words)
  // pinned host staging for small device->host reads
  int64_t* h_stage = nullptr;      // 64 words, mapped
  int64_t* h_stage_dev = nullptr;  // the same words seen from the device
  int launches = 0;
  // batched-launch graph cache
  void* batch_cache = nullptr;
};

namespace spg {

// Records a message on the context and returns `st`.
spg_status fail(spg_ctx* ctx, spg_status st, const char* fmt, ...);

// Converts a CUDA error into a status (and message); SPG_OK on success.
spg_status cuda_status(spg_ctx* ctx, cudaError_t e, const char* what);

#define SPG_CUDA(ctx, call)                                              \
  do {                                                                   \
    cudaError_t _e = (call);                                             \
    if (_e != cudaSuccess) return ::spg::cuda_status((ctx), _e, #call);  \
  } while (0)

#define SPG_TRY(call)                   \
  do {                                  \
    spg_status _s = (call);             \
    if (_s != SPG_OK) return _s;        \
  } while (0)

// Stream-ordered device allocation; released at scope exit (stream-ordered
// free) unless release() is called.  alloc: work memory, from the scratch
// pool; alloc_result: memory that a caller may keep, from the device's default
// pool.  Apart, each call finds the blocks the last one freed: in one pool the
// scratch of a call was cut from the results' blocks and the driver remapped
// gigabytes to make room for the next result (R-MAT 18, 10 GB of C: calls of
// 36 ms took 45 to 3,000 ms).
class DevBuf {
 public:
  DevBuf() = default;
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  ~DevBuf() { reset(); }
  spg_status alloc(spg_ctx* ctx, size_t bytes) { return alloc_from(ctx, bytes, ctx->scratch); }
  spg_status alloc_result(spg_ctx* ctx, size_t bytes) { return alloc_from(ctx, bytes, ctx->pool); }
  void reset();
  void* release() {
    void* p = ptr_;
    ptr_ = nullptr;
    return p;
  }
  template <typename T>
  T* as() const {
    return static_cast<T*>(ptr_);
  }
  void* get() const { return ptr_; }

 private:
  spg_status alloc_from(spg_ctx* ctx, size_t bytes, cudaMemPool_t pool);
  spg_ctx* ctx_ = nullptr;
  void* ptr_ = nullptr;
};

// Part of a DevBuf; several arrays of one call share an allocation.
struct DevSlice {
  void* ptr = nullptr;
  template <typename T>
  T* as() const {
    return static_cast<T*>(ptr);
  }
  void* get() const { return ptr; }
};

// Lays arrays out behind one another, each 256-byte aligned; then one
// allocation holds them all.
class DevLayout {
 public:
  void add(DevSlice* s, size_t bytes) {
    parts_[n_] = s;
    at_[n_++] = size_;
    size_ += (bytes + 255) / 256 * 256;
  }
  spg_status alloc(spg_ctx* ctx, DevBuf& buf) {
    const spg_status st = buf.alloc(ctx, size_);
    if (st == SPG_OK)
      for (int i = 0; i < n_; ++i) parts_[i]->ptr = buf.as<char>() + at_[i];
    return st;
  }

 private:
  static constexpr int kMax = 8;
  DevSlice* parts_[kMax];
  size_t at_[kMax], size_ = 0;
  int n_ = 0;
};

inline LaunchCtx launch_ctx(const spg_ctx* ctx) { return LaunchCtx{ctx->stream, ctx->sms, ctx->device, ctx->driver_ctx}; }

// Smallest product count of an expand-sort-fold row (0: none is folded).
inline int esc_min_products(const spg_tuning& t) {
  return t.esc_min_prod < 0 ? 0 : (t.esc_min_prod == 0 ? kEscMinProd : t.esc_min_prod);
}

// EscArgs::per_margin (0: no capacity below a row's products is folded).
inline float esc_per_margin(const spg_tuning& t) { return t.predict_margin > 0.f ? 1.f / t.predict_margin : 0.f; }

// Enqueues copies of `bytes` (a multiple of 4) device bytes each into the
// mapped staging words at host_dst (inside ctx->h_stage), at most
// StageCopies::kMax in one launch; valid after the next stream
// synchronisation.
struct StageRead {
  void* host_dst;
  const void* dev_src;
  size_t bytes;
};
spg_status stage_reads(spg_ctx* ctx, std::initializer_list<StageRead> reads);
inline spg_status stage_read(spg_ctx* ctx, void* host_dst, const void* dev_src, size_t bytes) {
  return stage_reads(ctx, {{host_dst, dev_src, bytes}});
}

// Device view of an spg_csr already on the device with int64 row pointers.
struct DevMat {
  DCsr view{};
  int64_t nnz = 0;
  DevBuf rp64;      // widened row pointers when the input had int32 ones
  DevBuf rp32;      // narrowed row pointers when the input had int64 ones and nnz < 2^31
  DevBuf upload[3]; // copies of host inputs
  // set while the entries are still being uploaded in row chunks: kernels
  // that read every row (the heavy-row blocked index) wait for it
  cudaEvent_t complete = nullptr;
};

// Prepares `m` for the kernels: uploads host data and widens int32 row
// pointers.  `validate` runs the structure check kernel (flags raised on the
// context's device flag word).
spg_status prepare_matrix(spg_ctx* ctx, const spg_csr* m, DevMat& out, bool validate, bool defer_entries = false);

// A and B describe the same matrix (same storage): prepare it once.
bool same_matrix(const spg_csr* a, const spg_csr* b);

// Reads and clears the device flag word.
spg_status read_flags(spg_ctx* ctx, int* flags);

spg_tuning default_tuning();
BinParams bin_params(const spg_tuning& t);

// Pipelines (api.cu / batched.cu / cusparse_ref.cu).
spg_status multiply_device(spg_ctx* ctx, const DevMat& A, const DevMat& B, spg_csr* C, const spg_opts& o,
                           spg_report* rep);
spg_status multiply_cusparse(spg_ctx* ctx, const DevMat& A, const DevMat& B, spg_csr* C, const spg_opts& o,
                             spg_report* rep);
// Exact per-row nnz of A*B (int64, rows entries) with the plain symbolic pass.
spg_status row_nnz_device(spg_ctx* ctx, const DevMat& A, const DevMat& B, int64_t* d_nnz);
// Heavy-row numeric pass through per-tile staging buckets (heavy.cu);
// *done = false (nothing launched) when it does not apply.
spg_status heavy_staged(spg_ctx* ctx, const DCsr& A, const DCsr& B, const int32_t* heavy_rows, int64_t nheavy,
                        const int32_t* big_slot, const int32_t* tile_cnt, const int32_t* tile_off, int ntiles,
                        const int64_t* c_rp, int32_t* c_col, float* c_val, bool* done);

// Value-only recompute of C's values (C holds the structure of A*B).
spg_status multiply_reuse_device(spg_ctx* ctx, const DevMat& A, const DevMat& B, spg_csr* C, const spg_opts& o,
                                 spg_report* rep);
spg_status ensure_mlp(spg_ctx* ctx);
void free_batch_cache(spg_ctx* ctx);

// Stage timer on the context stream (CUDA events).
class StageTimer {
 public:
  StageTimer(spg_ctx* ctx, bool enabled);
  ~StageTimer();
  void mark(int stage);  // closes the previous stage, opens `stage`
  void finish(spg_report* rep);

 private:
  spg_ctx* ctx_;
  bool on_;
  std::vector<std::pair<int, cudaEvent_t>> marks_;
};

}  // namespace spg
