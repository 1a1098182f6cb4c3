// Shared host-side plumbing of libferrum_cuda: device handle, status/error helpers, launch
// accounting with host-side fault injection, and the packed-weight descriptor every kernel takes.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <string>
#include <vector>

#include "../../include/ferrum_cuda.h"

#define FC_API extern "C" __attribute__((visibility("default")))

constexpr int QK = 32; // elements per quantisation block (ferrum_gguf/src/lib.rs:L55)

struct Workspace { // device scratch and its size
  void* p = nullptr;
  size_t bytes = 0;
};

struct FcDevice {
  int ordinal = 0;
  cudaStream_t stream = nullptr;
  cudaDeviceProp prop{};
  std::string last_error;
  bool lost = false;       // a CUDA call failed: sticky, like the reference's device-lost health
  uint64_t launches = 0;   // kernels launched by this library on this device
  int64_t fail_after = -1; // fault injection: launches left before every launch is refused
  void* pinned = nullptr;  // pinned host staging for results and small inputs
  size_t pinned_bytes = 0;
  // Scratch of the stand-alone products (qweight_scratch), and where it comes from: a pool in the order of `stream` that
  // holds on to at most WORKSPACE_POOL_KEEP bytes, so that a first product finds its memory mapped (mapping took 300 us);
  // null where the device has no memory pools.
  Workspace scratch;
  uint32_t weights = 0; // stand-alone weights alive
  cudaMemPool_t workspaces = nullptr;
  int* d_flag = nullptr;   // device int for kernels that report a status
  int matvec_choice = 0;   // fc_debug_matvec_kernel: which kernel multiplies 1..8 rows (0: the library's rule)
  // per-kernel timing (off by default): one event pair per launch, summed by name on report
  bool profiling = false;
  struct ProfSpan {
    const char* name;
    cudaEvent_t t0, t1;
  };
  std::vector<ProfSpan> spans;
  std::vector<cudaEvent_t> event_pool;
};

constexpr uint64_t WORKSPACE_POOL_KEEP = 512ull << 20;
constexpr uint64_t WORKSPACE_POOL_WARM = 64ull << 20; // mapped when the device is opened
cudaError_t workspace_alloc(FcDevice* dev, void** p, size_t bytes);
void workspace_free(FcDevice* dev, void* p);
// cudaMalloc that gives the scratch and the pool's cached memory back and tries again where there is no room (not under
// capture, nor between asking for scratch and launching with it); and that release by itself.
cudaError_t device_malloc(FcDevice* dev, void** p, size_t bytes);
void release_cached(FcDevice* dev);
bool stream_capturing(FcDevice* dev); // the device's stream is being captured into a graph

// Record a message and hand back the status code.
int fc_fail(FcDevice* dev, int code, const char* fmt, ...);

// Counts one kernel launch; refuses it (before it reaches the device) when the injection hook
// has run out. Every launch in the library goes through FC_LAUNCH.
int fc_pre_launch(FcDevice* dev, const char* what);
int fc_post_launch(FcDevice* dev, const char* what);

#define FC_TRY(expr)            \
  do {                          \
    int _rc = (expr);           \
    if (_rc != FC_OK) return _rc; \
  } while (0)

#define FC_CUDA(dev, expr)                                                                   \
  do {                                                                                       \
    cudaError_t _e = (expr);                                                                 \
    if (_e != cudaSuccess) {                                                                 \
      (dev)->lost = _e != cudaErrorMemoryAllocation;                                         \
      return fc_fail((dev), _e == cudaErrorMemoryAllocation ? FC_ERR_OOM : FC_ERR_DEVICE,    \
                     "%s: %s", #expr, cudaGetErrorString(_e));                               \
    }                                                                                        \
  } while (0)

#define FC_LAUNCH(dev, what, ...)         \
  do {                                    \
    FC_TRY(fc_pre_launch((dev), (what))); \
    __VA_ARGS__;                          \
    FC_TRY(fc_post_launch((dev), (what))); \
  } while (0)

#ifdef __CUDACC__
// A launch on the device's stream; `early`: it may begin while the kernel before it ends (programmatic dependent launch).
// The kernel then has to wait (grid_wait) before it reads what other kernels write, or writes what they read; with that
// first in every kernel of a chain, each begins its waiting while the one before it still works.
template <typename... P, typename... A>
void launch_on(FcDevice* dev, bool early, void (*kern)(P...), dim3 grid, dim3 block, size_t smem, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid, cfg.blockDim = block, cfg.dynamicSmemBytes = smem, cfg.stream = dev->stream;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at, cfg.numAttrs = early ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kern, P(args)...);
}
__device__ __forceinline__ void grid_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
#endif

// A kernel's attributes (dynamic shared memory limit) are set per device: a once-flag per device ordinal, one
// static instance per kernel instantiation.
struct OncePerDevice {
  bool done[64] = {};
  bool first(int ordinal) {
    if (ordinal < 0 || ordinal >= 64) return true; // (out of the table: set the attribute every time)
    if (done[ordinal]) return false;
    done[ordinal] = true;
    return true;
  }
  void again(int ordinal) { // the set-up did not complete: the next call repeats it
    if (ordinal >= 0 && ordinal < 64) done[ordinal] = false;
  }
};

// Pinned staging buffer of at least `bytes` (grown on demand).
int fc_pinned(FcDevice* dev, size_t bytes, void** out);

// A weight matrix as the kernels see it: `n` output rows of `k` inputs.
//  FC_Q8_0: qs = int8 [n][k];            sc = f16 [n][k/32]
//  FC_Q4_0: qs = u8   [n][k/2], 16 bytes (four u32 words) per block; word w holds elements
//           8w..8w+7 of the block, element j in nibble position (j>>1) + 4*(j&1), so that the
//           mask pairs (p, p+4) of one word unpack to consecutive elements; sc as above
//  FC_F32:  qs = f32  [n][k];            sc = nullptr
//  FC_F16:  qs = f16  [n][k];            sc = nullptr
//  FC_FP8_E4M3 / FC_FP8_E5M2: Q8_0's planes, the bytes being FP8 codes instead of int8 quants
//  FC_Q2_K: super-blocks of 256 (k a multiple of 256). qs = u8 [n][k/4], 2 bits per element in element
//           order (64 bytes per super-block; 32-bit word j is sub-block j, 16 elements); sc = 20-byte
//           records [n][k/256]: the 16 scale/min bytes of the sub-blocks in element order, then d and dmin (f16)
//  FC_MXFP4: qs = u8 [n][k/2], 16 bytes per block in element order (byte i: element 2i in the low nibble,
//           2i+1 in the high one), each nibble an E2M1 code; sc = u16 [n][k/32], the bf16 bit pattern
//           of the block's power-of-two scale 2^(e-127) (all 255 scale bytes fit: the smallest is a
//           bf16 subnormal), so a kernel gets the f32 scale with one shift
struct QMat {
  int kind = FC_F32;
  uint32_t k = 0, n = 0;
  const uint8_t* qs = nullptr;
  const __half* sc = nullptr;
};

struct FcQWeight {
  FcDevice* dev = nullptr;
  QMat m;
  void* qs_alloc = nullptr;
  void* sc_alloc = nullptr;
  uint64_t bytes = 0;
  // scratch of products captured into graphs, and what they outgrew (a graph may still hold its address): see qweight_scratch
  Workspace graph_ws;
  std::vector<void*> outgrown;
};

// Scratch for one product of a stand-alone weight. All products of a device handle run one behind the other on its stream
// and share one buffer, as large as the largest of them asked for; it goes back with the last of the weights, or when
// memory is short. (An allocation of the call's own, from the pool and back in stream order, left 2 us between the kernels
// of neighbouring calls: 5 x 1056 x 1500 10.3 us instead of 8.2.) Inside a stream capture the scratch is the weight's own,
// for the graph to replay with on any stream, until the weight is destroyed.
// FC_ERR_OOM: there is no room (a smaller request, or a kernel without scratch, may do).
int qweight_scratch(FcQWeight* w, size_t bytes, Workspace* out);
void release_scratch(FcDevice* dev);

__host__ __device__ constexpr bool kind_is_fp8(int kind) { return kind == FC_FP8_E4M3 || kind == FC_FP8_E5M2; }
// one byte per element and an f16 scale per 32: Q8_0 and the FP8 formats share planes, loads and addressing
__host__ __device__ constexpr bool kind_byte_blocks(int kind) { return kind == FC_Q8_0 || kind_is_fp8(kind); }
// half a byte per element, 16 bytes per block: Q4_0 and MXFP4 share addressing (not the nibble order)
__host__ __device__ constexpr bool kind_nibble_blocks(int kind) { return kind == FC_Q4_0 || kind == FC_MXFP4; }
__host__ __device__ constexpr bool kind_has_scales(int kind) { return kind_byte_blocks(kind) || kind_nibble_blocks(kind); }
static inline bool kind_known(int kind) { return kind >= FC_F32 && kind <= FC_Q2_K; }
constexpr uint32_t QK_K = 256; // elements of a Q2_K super-block
static inline uint32_t kind_block_elems(int kind) { return kind == FC_Q2_K ? QK_K : QK; }
// ops/quant.rs:L134-L144 (`effective`): Q2_K on a width of whole 32s but not whole 256s is stored as Q4_0
static inline int effective_kind(int kind, uint64_t k) {
  return (kind == FC_Q2_K && k % QK_K != 0 && k > 0 && k % QK == 0) ? FC_Q4_0 : kind;
}

static inline size_t qmat_qs_bytes(int kind, size_t k, size_t n) {
  return kind_byte_blocks(kind)     ? k * n
         : kind_nibble_blocks(kind) ? k * n / 2
         : kind == FC_Q2_K          ? k * n / 4
         : kind == FC_F16           ? k * n * 2
                                    : k * n * 4;
}
static inline size_t qmat_sc_bytes(int kind, size_t k, size_t n) {
  return kind == FC_Q2_K ? (k / QK_K) * n * 20 : kind_has_scales(kind) ? (k / QK) * n * 2 : 0;
}

#ifdef __CUDACC__
// Two FP8 codes (the low 16 bits of `two`) as two fp16 values, low byte in the low half. Exact: every
// E4M3 and E5M2 value, infinities and NaNs included, is an fp16 value.
template <int KIND>
__device__ __forceinline__ uint32_t fp8x2_to_f16x2(uint32_t two) {
  uint32_t r;
  const unsigned short v = (unsigned short)two;
  if (KIND == FC_FP8_E4M3)
    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(r) : "h"(v));
  else
    asm("cvt.rn.f16x2.e5m2x2 %0, %1;" : "=r"(r) : "h"(v));
  return r;
}
// The eight E2M1 codes of one word of an MXFP4 block (byte i: elements 2i, 2i+1) as four fp16 pairs in
// element order. Exact: the values are 0, 0.5, 1, 1.5, 2, 3, 4, 6 and their negatives.
__device__ __forceinline__ void e2m1x8_to_f16x2(uint32_t w, uint32_t (&o)[4]) {
  asm("{\n.reg .b8 b0, b1, b2, b3;\nmov.b32 {b0, b1, b2, b3}, %4;\n"
      "cvt.rn.f16x2.e2m1x2 %0, b0;\ncvt.rn.f16x2.e2m1x2 %1, b1;\ncvt.rn.f16x2.e2m1x2 %2, b2;\ncvt.rn.f16x2.e2m1x2 %3, b3;\n}"
      : "=r"(o[0]), "=r"(o[1]), "=r"(o[2]), "=r"(o[3])
      : "r"(w));
}
// The f32 scale of a block from its 16-bit slot: an f16 for the GGUF integer / FP8 formats, the bf16 bits
// of a power of two for MXFP4.
template <int KIND>
__device__ __forceinline__ float block_scale_f32(__half raw) {
  return KIND == FC_MXFP4 ? __uint_as_float((uint32_t)__half_as_ushort(raw) << 16) : __half2float(raw);
}
// One code as f32 (exact).
template <int KIND>
__device__ __forceinline__ float fp8_to_f32(uint32_t code) {
  const uint32_t h2 = fp8x2_to_f16x2<KIND>(code & 0xffu);
  return __half2float(__ushort_as_half((unsigned short)(h2 & 0xffffu)));
}
// Elements i .. i + 7 (i a multiple of 8) of weight row `row`, d * q rounded as the decoder rounds it.
template <int KIND>
__device__ __forceinline__ void qmat_eight(const QMat& w, uint32_t row, uint32_t i, float (&v)[8]) {
  const uint32_t k = w.k;
  if (KIND == FC_Q8_0) {
    const uint2 q = *reinterpret_cast<const uint2*>(w.qs + (size_t)row * k + i);
    const float d = __half2float(w.sc[(size_t)row * (k / QK) + i / QK]);
    const uint32_t qw[2] = {q.x, q.y};
#pragma unroll
    for (int j = 0; j < 8; j++) v[j] = __fmul_rn(d, (float)(int8_t)((qw[j >> 2] >> (8 * (j & 3))) & 0xff));
  } else if (KIND == FC_Q2_K) { // (d * sc) * q - dmin * m, as the decoder rounds it
    const uint32_t sub = i / 16;
    const uint8_t* rec = reinterpret_cast<const uint8_t*>(w.sc) + ((size_t)row * (k / QK_K) + i / QK_K) * 20;
    const uint32_t word = reinterpret_cast<const uint32_t*>(w.qs)[(size_t)row * (k / 16) + sub] >> (2 * (i % 16));
    const uint8_t sc = rec[sub % 16];
    const float dl = __fmul_rn(__half2float(*reinterpret_cast<const __half*>(rec + 16)), (float)(sc & 15));
    const float ml = __fmul_rn(__half2float(*reinterpret_cast<const __half*>(rec + 18)), (float)(sc >> 4));
#pragma unroll
    for (int j = 0; j < 8; j++) v[j] = __fsub_rn(__fmul_rn(dl, (float)((word >> (2 * j)) & 3)), ml);
  } else if (KIND == FC_MXFP4) {
    const uint32_t q = *reinterpret_cast<const uint32_t*>(w.qs + (size_t)row * (k / 2) + i / 2);
    const float d = block_scale_f32<KIND>(w.sc[(size_t)row * (k / QK) + i / QK]);
    uint32_t h[4];
    e2m1x8_to_f16x2(q, h);
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h[j]));
      v[2 * j] = __fmul_rn(d, f.x);
      v[2 * j + 1] = __fmul_rn(d, f.y);
    }
  } else if (kind_is_fp8(KIND)) {
    const uint2 q = *reinterpret_cast<const uint2*>(w.qs + (size_t)row * k + i);
    const float d = __half2float(w.sc[(size_t)row * (k / QK) + i / QK]);
    const uint32_t qw[2] = {q.x, q.y};
#pragma unroll
    for (int j = 0; j < 8; j++) v[j] = __fmul_rn(d, fp8_to_f32<KIND>(qw[j >> 2] >> (8 * (j & 3))));
  } else if (KIND == FC_Q4_0) {
    const uint32_t q = *reinterpret_cast<const uint32_t*>(w.qs + (size_t)row * (k / 2) + i / 2);
    const float d = __half2float(w.sc[(size_t)row * (k / QK) + i / QK]);
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int pos = (j >> 1) + 4 * (j & 1);
      v[j] = __fmul_rn(d, (float)((q >> (4 * pos)) & 0xf) - 8.0f);
    }
  } else if (KIND == FC_F16) {
    const uint4 q = *reinterpret_cast<const uint4*>(w.qs + ((size_t)row * k + i) * 2);
    const uint32_t qw[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&qw[j]));
      v[2 * j] = f.x;
      v[2 * j + 1] = f.y;
    }
  } else {
    const float* src = reinterpret_cast<const float*>(w.qs) + (size_t)row * k;
#pragma unroll
    for (int j = 0; j < 8; j++) v[j] = i + j < k ? src[i + j] : 0.0f;
  }
}
// One output (or its part over [i0, i1), whole blocks) by an f32 chain in ascending k: what the products on fp16 terms of x
// do with rows that such terms cannot hold.
template <int KIND>
__device__ __noinline__ float exact_dot(const float* x, const uint8_t* qs, const __half* sc, uint32_t k, uint32_t row, uint32_t i0,
                                        uint32_t i1) {
  const QMat w{KIND, k, 0, qs, sc}; // (by reference, a kernel's whole argument block would be copied to the stack)
  float acc = 0.0f;
#pragma unroll 4
  for (uint32_t i = i0; i < i1; i += 8) {
    float v[8];
    qmat_eight<KIND>(w, row, i, v);
#pragma unroll
    for (int j = 0; j < 8; j++) acc = fmaf(x[i + j], v[j], acc); // (x: a caller's pointer, aligned to nothing but floats)
  }
  return acc;
}
#endif

// Epilogue of a matrix product: y = act(x W + bias) (+ resid). All pointers device, nullable.
enum { ACT_NONE = 0, ACT_GELU = 1 };
// A 9..64-row product whose split-K partial sums have not been combined yet: the consumer of its result
// (the norm + split launch of the next product) adds them up, applies bias and residual, writes y and
// carries on - one launch instead of two on a step that is bound by its launch chain.
struct DeferredReduce {
  const float* partial = nullptr; // [splits][m][n]
  uint32_t splits = 0;            // 0: nothing pending
  uint32_t m = 0, n = 0;
  const float* bias = nullptr;
  const float* resid = nullptr;
  float* y = nullptr;
};

struct Epilogue {
  const float* bias = nullptr;  // [n]
  const float* resid = nullptr; // [m][n]; may alias y
  int act = ACT_NONE;
  // device scratch of at least qmatvec_mma_scratch_bytes(k, n): lets products of 9..64 rows run on the
  // tensor-core batched-decode kernel; without it they take the tiled f32 kernel
  void* scratch = nullptr;
  // a stand-alone product (no norm, nothing pending or deferred) whose width need not be whole 128s: the scratch also
  // serves qmatvec_mma_ragged_supports
  bool ragged = false;
  // device scratch that lets products of more than 64 rows of Q8_0 / Q4_0 weights run on the tensor cores (gemm_pair.cu;
  // qgemm_pair_scratch_bytes is what the best cut takes); without it, or where it is too small, they take the
  // tiled f32 kernel. (One pointer, read by host code only: the decode kernels take this struct as an
  // argument, and with eight bytes more a decode step of 12 layers took 445 us instead of 433.)
  const Workspace* wide = nullptr;
  // "x is the raw residual stream: normalise each row first" (NORM_RMS: y = x / sqrt(mean(x^2) + eps) * g,
  // NORM_LAYER: (x - mean) / sqrt(var + 1e-5) * g + b). The one-row FMA matvec does it while it stages x
  // in shared memory (one launch less per product); the other kernels run the norm kernel into
  // `norm_tmp` ([m][k] floats) first.
  int norm = 0;
  const float* norm_g = nullptr;
  const float* norm_b = nullptr;
  float norm_eps = 0.0f;
  float* norm_tmp = nullptr;
  // x is the fused gate / up row (2 k wide, the layout of k_swiglu's `group`) and the product is fed silu(gate) * up: only
  // where qlinear_takes_swiglu says so
  bool swiglu = false;
  uint32_t swiglu_group = 0;
  // the producer of x has already written its two fp16 terms where the 9..64-row tensor-core product
  // stages them (qmatvec_mma_split_ptrs): the product skips its split launch and ignores `x`
  bool presplit = false;
  // leave this product's split-K reduce to the consumer (filled in when the product did split)
  DeferredReduce* defer_out = nullptr;
  // where a deferring product puts its partial sums, when the place behind its own x terms would be
  // overwritten by the consumer (nullable: that default place)
  float* partial_at = nullptr;
  // finish this pending reduce first: its y is this product's x (same buffer, raw residual stream)
  const DeferredReduce* pending = nullptr;
};
enum { NORM_NONE = 0, NORM_RMS = 1, NORM_LAYER = 2 };

// matvec_mma.cu: 9 <= m <= 64 rows at f32-class accuracy on mma.sync
bool qmatvec_mma_supports(const QMat& w, uint32_t m);
bool qmatvec_mma_ragged_supports(const QMat& w, uint32_t m); // 2..64 rows, other whole-block widths (Epilogue::ragged)
size_t qmatvec_mma_scratch_bytes(uint32_t k, uint32_t n);
int k_qmatvec_mma(FcDevice* dev, const QMat& w, const float* x, uint32_t m, float* y, const Epilogue& ep, void* scratch);
// Whether k_qlinear_f32 will take the 9..64-row tensor-core product for (w, m) with this scratch, and where
// that product expects the two fp16 terms of x ([mp][k] each, rows >= m zero).
bool qlinear_takes_swiglu(const FcDevice* dev, const QMat& w); // one row, the streamed product (matvec1.cu)
bool qlinear_takes_wide_mma(const QMat& w, uint32_t m, const void* scratch);
int k_flush_deferred(FcDevice* dev, const DeferredReduce& d);
int k_norm_pending(FcDevice* dev, const DeferredReduce& d, int norm, const float* g, const float* b, float eps, float* h);
void qmatvec_mma_split_ptrs(void* scratch, uint32_t m, uint32_t k, __half** xh, __half** xl, uint32_t* mp);

// ---- kernels' host entry points (each enqueues on dev->stream) --------------------------------
// codec.cu
int k_quantise_kn(FcDevice* dev, int kind, const float* w_kn_dev, uint32_t k, uint32_t n, uint8_t* qs, __half* sc);
int k_transpose_kn(FcDevice* dev, const float* w_kn_dev, uint32_t k, uint32_t n, float* out_nk);
int k_repack_blocks(FcDevice* dev, int kind, const uint8_t* blocks_dev, uint32_t k, uint32_t n, uint8_t* qs, __half* sc);
int k_export_blocks(FcDevice* dev, const QMat& m, uint8_t* blocks_dev);
int k_dequant(FcDevice* dev, const QMat& m, float* out_nk_dev);
// matvec.cu: m <= 8 rows
int k_qmatvec(FcDevice* dev, const QMat& w, const float* x, uint32_t m, float* y, const Epilogue& ep);
// matvec1.cu: one row of a block format, streamed through shared memory onto mma.sync
// gemm_tc.cu: the exact-class tcgen05 product of 2..64 rows of x (x as its two fp16 terms)
bool qgemm_tx_takes(const FcDevice* dev, const QMat& w, uint32_t m, bool deferring);
int k_qgemm_tx(FcDevice* dev, const QMat& w, const __half* xh, const __half* xl, uint32_t mp, uint32_t m, float* y,
               const Epilogue& ep);
bool qmatvec1_supports(const FcDevice* dev, const QMat& w);
int k_qmatvec1(FcDevice* dev, const QMat& w, const float* x, float* y, const Epilogue& ep);
// gemm_f32.cu: any m
int k_qgemm_f32(FcDevice* dev, const QMat& w, const float* x, uint32_t m, float* y, const Epilogue& ep);
// The exact-f32 product of any m: picks matvec or tiled GEMM.
int k_qlinear_f32(FcDevice* dev, const QMat& w, const float* x, uint32_t m, float* y, const Epilogue& ep);

// Upload helpers (runtime.cu)
// One host tensor of a weight: kind FC_F32 = an f32 `[in, out]` matrix (the reference's host layout), a block kind =
// the GGUF bytes of the `[out, in]` tensor.
struct WeightSrc {
  const void* p;
  int kind;
};
int qweight_from_parts(FcDevice* dev, int kind, const WeightSrc* parts, const uint32_t* ns, int count, uint32_t k,
                       FcQWeight** out);
int qweight_from_f32(FcDevice* dev, int kind, const float* w_in_out_host, uint32_t k, uint32_t n, FcQWeight** out);
int qweight_from_f32_concat(FcDevice* dev, int kind, const float* const* mats_host, const uint32_t* ns, int count,
                            uint32_t k, FcQWeight** out);
void qweight_free(FcQWeight* w);
