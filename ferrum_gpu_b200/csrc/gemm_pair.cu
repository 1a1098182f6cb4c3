// The exact-class product of many rows (more than the 64 of batched decode) on CTA pairs:
//
//   y[r, n] = sum_k x[r, k] * d[n, k / 32] * q[n, k]
//
// Both factors become two fp16 terms, written once per call by two preparation kernels (gemm_pair.cu: rows_split,
// weights_split) and read by TMA: x 2^s = xh + xl 2^-11, d q 2^t = wh + wl 2^-11, s per row of x and t per weight row,
// powers of two that put the row's largest magnitude next to the top of the fp16 range; the epilogue takes 2^-s 2^-t back.
// The low terms are kept 2^11 larger than what they stand for, at the magnitude of the high ones, so that they are as far
// from fp16's subnormals: an element of x has 22 bits down to 2^-28 of its row's largest, and d q (19 bits, and no f16
// scale is below 2^-24) is always exact. A row that reaches further down with a part of its sum that counts is multiplied
// by the f32 chain instead, as are rows with infinities and NaNs (row_is_wide). Three of the four cross terms are
// multiplied (wl . xl is below 2^-22 of the product, a quarter of an f32 rounding), all into one f32 accumulator, the small
// ones first; the first large one brings their sum down by 2^-11 (the MMA's own scaling of D). The tensor cores' f32
// accumulation rounds toward zero, so tensor memory only ever holds the sum of 128 k (64 k at short widths): then the
// epilogue warps add the finished sum into f32 registers.
//
// The pair: two CTAs on neighbouring SMs work on one tile of 256 weight rows x 128 or 64 rows of x
// (tcgen05.mma.cta_group::2): each holds its 128 weight rows (tensor-memory lanes) and half of the x rows in shared
// memory, so a K step reads 16 KB + 64 BN bytes per CTA and term for 128 x BN x 64 multiply-adds each - half the L2
// traffic of two single CTAs with the same tile, which is what bounds a 128 x 128 tile here.
//
//   warp 0        TMA: this CTA's boxes of a K step (wh, wl, xh, xl) into the ring; bytes are counted on the LEADER's
//                 barrier (even CTA of the pair)
//   warp 1        tensor-memory owner; in the leader one thread issues the MMAs of both CTAs
//   warps 4-11    epilogue: warp w owns lane quadrant w % 4 (32 weight rows) and half of the x rows, accumulators
//                 in registers; stores are 128 contiguous bytes per row of y
//
// Barriers: full[s] (leader: the bytes of both CTAs), empty[s] and acc_full[b] (MMA commit, multicast to both CTAs),
// acc_empty[b] (leader: 16 epilogue warps). Every wait is bounded and polls the CTA's abort word.
#include "gemm_pair.cuh"

#include "tc_ptx.cuh"
#include "tensor_map.cuh"

namespace {

constexpr uint32_t BK = 64;                        // k per stage: one 128-byte swizzle row of fp16
constexpr int PAIR_THREADS = 384;
constexpr uint32_t A_TERM = 128 * BK * 2;          // 16 KB: this CTA's 128 weight rows, one term
constexpr uint32_t NACC = 4;                       // accumulator buffers: the hand-over between SMs takes about a chunk's MMA time
template <int BN>
struct Shape {
  static constexpr uint32_t B_TERM = (BN / 2) * BK * 2; // this CTA's half of the x rows, one term
  static constexpr uint32_t STAGE = 2 * (A_TERM + B_TERM);
  static constexpr int STAGES = BN == 128 ? 4 : 5;
  static_assert(NACC * BN <= 512, "tensor memory has 512 columns");
  static constexpr uint32_t SMEM = STAGES * STAGE + 256 /*barriers*/ + 1024 /*alignment slack*/;
};
enum { ERR_PAIR_EMPTY = 11, ERR_PAIR_FULL = 12, ERR_PAIR_ACC = 13 };

__device__ __forceinline__ float gelu_f(float x) {
  const float K = 0.7978846f;
  return 0.5f * x * (1.0f + tanhf(K * (x + 0.044715f * x * x * x)));
}

// Bounded wait with suspended tries of up to 20 us each (about 1.3 s in all); polls the CTA's abort word.
__device__ __forceinline__ bool wait_bounded(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_word) {
  for (uint32_t i = 0; i < (1u << 16); i++) {
    if (tc::mbar_try_wait_for(bar, parity, 20000u)) return true;
    if (*abort_word) return false;
  }
  *abort_word = 1;
  return false;
}
// The same for the MMA thread, which must not sleep.
__device__ __forceinline__ bool wait_spin(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_word) {
  for (uint32_t i = 0; i < tc::WAIT_LIMIT; i++) {
    if (tc::mbar_try_wait(bar, parity)) return true;
    if ((i & 1023u) == 1023u && *abort_word) return false;
  }
  *abort_word = 1;
  return false;
}

struct PairArgs {
  QMat w;                       // the weight rows of this launch (the exact dot of rows that fp16 terms cannot hold)
  const float* x = nullptr;     // [m][w.k] (normalised)
  uint32_t m = 0;               // rows of x
  uint32_t steps = 0;           // K steps of 64
  uint32_t steps_per_split = 0, splits = 1;
  uint32_t chunk = 1;           // stages that one accumulator buffer sums (at most STAGES / 2)
  float* y = nullptr;           // [m][ldy]
  uint32_t ldy = 0;
  const float* bias = nullptr;  // [w.n]
  const float* resid = nullptr; // [m][ldy]; may alias y
  const float* x_scale = nullptr; // [m] 2^-s; 0: the fp16 terms do not hold the row
  const float* w_scale = nullptr; // [w.n] 2^-t; 0: a block scale of the row is not finite
  float* partial = nullptr;       // [splits][m][w.n]: the sums without bias, activation and residual
  int* err_flag = nullptr;
};

template <int KIND, int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PAIR_THREADS, 1)
    qgemm_pair_kernel(const __grid_constant__ CUtensorMap t_wh, const __grid_constant__ CUtensorMap t_wl,
                      const __grid_constant__ CUtensorMap t_xh, const __grid_constant__ CUtensorMap t_xl, const PairArgs a) {
  using S = Shape<BN>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (tc::smem_u32(smem_raw) + 1023u) & ~1023u; // (the 128B swizzle is a function of the address)
  uint8_t* smem = smem_raw + (base - tc::smem_u32(smem_raw));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + S::STAGES * S::STAGE);
  uint64_t* empty = full + S::STAGES;
  uint64_t* acc_full = empty + S::STAGES;
  uint64_t* acc_empty = acc_full + NACC;
  uint64_t* done = acc_empty + NACC;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile uint32_t* abort_word = tmem_slot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = blockIdx.x & 1u; // (clusters are two consecutive blocks)
  const uint32_t tiles_n = (a.w.n + 255) / 256, tiles_x = (a.m + BN - 1) / BN;
  const uint32_t items = tiles_n * tiles_x * a.splits;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S::STAGES; s++) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    for (uint32_t b = 0; b < NACC; b++) {
      tc::mbar_init(&acc_full[b], 1);
      tc::mbar_init(&acc_empty[b], 16);
    }
    tc::mbar_init(done, 1);
    *abort_word = 0;
    tc::fence_barrier_init();
    tc::prefetch_tmap(&t_wh);
    tc::prefetch_tmap(&t_wl);
    tc::prefetch_tmap(&t_xh);
    tc::prefetch_tmap(&t_xl);
  }
  if (warp == 1) {
    tc::tmem_alloc_pair(tmem_slot, 512);
    tc::tmem_relinquish_pair();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::cluster_sync(); // both CTAs' barriers are initialised and both tensor memories allocated
  tc::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  // work item -> (weight tile, x tile, split); the weight tiles run fastest, so that the pairs at work share x tiles
  auto decode = [&](uint32_t item, uint32_t& n0, uint32_t& x0, uint32_t& k0, uint32_t& k1) {
    const uint32_t tn = item % tiles_n, rest = item / tiles_n;
    n0 = tn * 256, x0 = (rest % tiles_x) * BN;
    k0 = (rest / tiles_x) * a.steps_per_split;
    k1 = min(k0 + a.steps_per_split, a.steps);
  };

  if (warp == 0) {
    // ---- TMA ----
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (uint32_t item = blockIdx.x >> 1; item < items && ok; item += gridDim.x >> 1) {
        uint32_t n0, x0, k0, k1;
        decode(item, n0, x0, k0, k1);
        for (uint32_t kk = k0; kk < k1; kk++, it++) {
          const uint32_t s = it % S::STAGES, ph = (it / S::STAGES) & 1;
          if (!wait_bounded(&empty[s], ph ^ 1, abort_word)) {
            atomicExch(a.err_flag, ERR_PAIR_EMPTY);
            ok = false;
            break;
          }
          uint8_t* st = smem + s * S::STAGE;
          const uint32_t bar = tc::leader_addr(&full[s]);
          if (rank == 0) tc::mbar_arrive_expect_tx(&full[s], 2 * S::STAGE);
          const int32_t kx = (int32_t)(kk * BK), ny = (int32_t)(n0 + rank * 128), xy = (int32_t)(x0 + rank * (BN / 2));
          tc::tma_load_2d_pair(st, &t_wh, bar, kx, ny);
          tc::tma_load_2d_pair(st + A_TERM, &t_wl, bar, kx, ny);
          tc::tma_load_2d_pair(st + 2 * A_TERM, &t_xh, bar, kx, xy);
          tc::tma_load_2d_pair(st + 2 * A_TERM + S::B_TERM, &t_xl, bar, kx, xy);
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer: one thread of the leader, for both CTAs ----
    if (rank == 0 && tc::elect_one()) {
      constexpr uint32_t idesc = tc::idesc_f16_f32(256, BN);
      constexpr uint32_t desc_hi = (1024u >> 4) | (1u << 14) | (2u << 29); // stride 1024 B, version 1, 128B swizzle
      uint32_t it = 0, ch = 0; // stages and chunks issued so far
      bool ok = true;
      for (uint32_t item = blockIdx.x >> 1; item < items && ok; item += gridDim.x >> 1) {
        uint32_t n0, x0, k0, k1;
        decode(item, n0, x0, k0, k1);
        for (uint32_t kc = k0; kc < k1 && ok; kc += a.chunk, ch++) {
          const uint32_t buf = ch % NACC;
          if (!wait_spin(&acc_empty[buf], ((ch / NACC) & 1) ^ 1, abort_word)) { // both CTAs have taken the buffer's last sum
            atomicExch(a.err_flag, ERR_PAIR_ACC);
            ok = false;
            break;
          }
          const uint32_t d = tmem_base + buf * BN, n_st = min(a.chunk, k1 - kc);
          constexpr uint64_t hi = (uint64_t)desc_hi << 32;
          // the small cross terms of the whole chunk first, then the large ones: the accumulator rounds each addition
          // toward zero at its own magnitude, so only the last four MMAs per stage cost accuracy
          for (uint32_t c = 0; c < n_st; c++) {
            const uint32_t s = (it + c) % S::STAGES;
            if (!wait_spin(&full[s], ((it + c) / S::STAGES) & 1, abort_word)) {
              atomicExch(a.err_flag, ERR_PAIR_FULL);
              ok = false;
              break;
            }
            tc::tc_fence_after();
            const uint32_t st = base + s * S::STAGE;
            const uint64_t dwh = hi | (st >> 4), dwl = hi | ((st + A_TERM) >> 4);
            const uint64_t dxh = hi | ((st + 2 * A_TERM) >> 4), dxl = hi | ((st + 2 * A_TERM + S::B_TERM) >> 4);
#pragma unroll
            for (uint32_t ks = 0; ks < BK / 16; ks++)
              tc::mma_f16_pair(d, dwl + 2 * ks, dxh + 2 * ks, idesc, (c | ks) ? 1u : 0u); // a chunk starts from zero
#pragma unroll
            for (uint32_t ks = 0; ks < BK / 16; ks++) tc::mma_f16_pair(d, dwh + 2 * ks, dxl + 2 * ks, idesc, 1u);
          }
          if (!ok) break;
          for (uint32_t c = 0; c < n_st; c++) {
            const uint32_t s = (it + c) % S::STAGES, st = base + s * S::STAGE;
            const uint64_t dwh = hi | (st >> 4), dxh = hi | ((st + 2 * A_TERM) >> 4);
#pragma unroll
            for (uint32_t ks = 0; ks < BK / 16; ks++) {
              if (ks == 0 && c == 0)
                tc::mma_f16_pair_shifted<LOW_SHIFT>(d, dwh, dxh, idesc); // what is there so far are the low terms' products
              else
                tc::mma_f16_pair(d, dwh + 2 * ks, dxh + 2 * ks, idesc, 1u);
            }
            tc::mma_commit_pair(&empty[s]);
          }
          it += n_st;
          tc::mma_commit_pair(&acc_full[buf]);
        }
      }
      // every MMA has finished before the tensor memory goes back (also after a wait that gave up)
      tc::mma_commit_pair(done);
    }
    __syncwarp();
    if (lane == 0) {
      volatile uint32_t never = 0;
      if (!wait_bounded(done, 0, &never)) atomicExch(a.err_flag, ERR_PAIR_ACC);
    }
    __syncwarp();
  } else if (warp >= 4) {
    // ---- epilogue ----
    const uint32_t quad = (uint32_t)warp & 3u, half = (uint32_t)(warp - 4) >> 2;
    constexpr int COLS = BN / 2; // rows of x of this warp
    uint32_t ch = 0;
    bool ok = true;
    for (uint32_t item = blockIdx.x >> 1; item < items && ok; item += gridDim.x >> 1) {
      uint32_t n0, x0, k0, k1;
      decode(item, n0, x0, k0, k1);
      float acc[COLS];
#pragma unroll
      for (int j = 0; j < COLS; j++) acc[j] = 0.0f;
      for (uint32_t kc = k0; kc < k1; kc += a.chunk, ch++) {
        const uint32_t buf = ch % NACC;
        ok = wait_spin(&acc_full[buf], (ch / NACC) & 1, abort_word);
        if (!ok) atomicExch(a.err_flag, ERR_PAIR_ACC);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc::tc_fence_after();
        const uint32_t taddr = tmem_base + ((quad * 32u) << 16) + buf * BN + half * COLS;
        uint32_t v[COLS]; // (all loads in flight at once: one by one, their latencies add up to more than the MMAs take)
#pragma unroll
        for (int c = 0; c < COLS; c += 32) tc::tmem_ld_32x32(taddr + c, v + c);
        tc::tmem_ld_wait();
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive_cluster(tc::leader_addr(&acc_empty[buf]));
#pragma unroll
        for (int j = 0; j < COLS; j++) acc[j] += __uint_as_float(v[j]);
      }
      if (!ok) break;
      const uint32_t n = n0 + rank * 128 + quad * 32 + lane, xr = x0 + half * COLS;
      if (n < a.w.n && xr < a.m) {
        const float ws = a.w_scale[n];
        const float bias = a.bias ? a.bias[n] : 0.0f;
        float* out = a.partial ? a.partial + (size_t)(k0 / a.steps_per_split) * a.m * a.w.n : a.y;
        const uint32_t ldo = a.partial ? a.w.n : a.ldy;
        const float* res = a.partial ? nullptr : a.resid;
        bool bad = ws == 0.0f;
        // (this code is unrolled over the registers that hold the sums and runs once per tile, from a cold instruction
        // cache: it is kept short. The activation runs in pair_reduce_kernel, rows that fp16 terms cannot hold below.)
#pragma unroll
        for (int c = 0; c < COLS; c += 8) {
          float xs[8], rs[8];
#pragma unroll
          for (int j = 0; j < 8; j++) {
            const bool in = xr + c + j < a.m;
            xs[j] = in ? a.x_scale[xr + c + j] : 1.0f;
            rs[j] = (res && in) ? res[(size_t)(xr + c + j) * ldo + n] : 0.0f;
            bad |= xs[j] == 0.0f;
          }
#pragma unroll
          for (int j = 0; j < 8; j++) {
            float v = (acc[c + j] * ws) * xs[j];
            if (!a.partial) v += bias;
            if (res) v = rs[j] + v;
            if (xr + c + j < a.m && ws != 0.0f && xs[j] != 0.0f) out[(size_t)(xr + c + j) * ldo + n] = v;
          }
        }
        if (bad) {
#pragma unroll 1
          for (uint32_t row = xr; row < min(xr + COLS, a.m); row++) {
            if (ws != 0.0f && a.x_scale[row] != 0.0f) continue;
            float v = 0.0f; // (of several splits the first has the whole sum)
            if (k0 == 0) v = exact_dot<KIND>(a.x + (size_t)row * a.w.k, a.w.qs, a.w.sc, a.w.k, n, 0, a.w.k);
            if (!a.partial) v += bias;
            if (res) v = res[(size_t)row * ldo + n] + v;
            out[(size_t)row * ldo + n] = v;
          }
        }
      }
      __syncwarp();
    }
  }
  // A wait that gave up leaves copies in flight: they land within microseconds, long before this runs out.
  if (*abort_word)
    for (int i = 0; i < 1000; i++) __nanosleep(1000);
  tc::tc_fence_before();
  __syncthreads();
  __syncwarp();
  tc::cluster_sync(); // nobody leaves while the partner may still signal it or read its operands
  if (warp == 1) tc::tmem_dealloc_pair(tmem_base, 512);
}

// y = epilogue(sum over splits, ascending split index)
__global__ void __launch_bounds__(256)
    pair_reduce_kernel(const float* __restrict__ partial, uint32_t splits, uint32_t m, uint32_t n, float* y, uint32_t ldy,
                       const float* __restrict__ bias, const float* resid, int act) {
  const uint32_t col = blockIdx.x * 256 + threadIdx.x;
  if (col >= n) return;
  for (uint32_t row = blockIdx.y; row < m; row += gridDim.y) {
    const size_t i = (size_t)row * n + col, o = (size_t)row * ldy + col;
    float v = 0.0f;
    for (uint32_t s = 0; s < splits; s++) v += partial[(size_t)s * m * n + i];
    if (bias) v += bias[col];
    if (act == ACT_GELU) v = gelu_f(v);
    if (resid) v = resid[o] + v;
    y[o] = v;
  }
}

// ---- preparation -------------------------------------------------------------------------------------------------

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  return warp_sum(lane < nw ? red[lane] : 0.0f);
}
// the power of two that puts a magnitude `mx` into [2^e, 2^(e+1)), as (multiplier, its inverse); both stay normal floats
__device__ __forceinline__ void pow2_to(float mx, int e, float& mul, float& inv) {
  int s = mx > 0.0f ? e - ((int)((__float_as_uint(mx) >> 23) & 0xffu) - 127) : 0;
  s = max(-126, min(126, s));
  mul = __uint_as_float((uint32_t)(127 + s) << 23);
  inv = __uint_as_float((uint32_t)(127 - s) << 23);
}

// Whether the two terms of a row lose what an f32 sum would keep. `lost` is what this thread's elements lose beyond 2^-22
// of themselves (elements below 2^-28 of the row's largest: their low terms are subnormal, or both terms are zero), `sum`
// the sum of its elements' magnitudes. One such element among ordinary ones is far below a rounding of the result; it
// counts where the row's large elements meet weights of zero and only small ones remain. So the row is held as long as
// 2^-22 of what is left covers the loss even without any `few` threads' parts (so many large elements at least): where
// few + 1 threads each have as much, or few + a quarter of the threads their share of it. No element loses more than 2^-50
// of the row's largest: ordinary rows, whose other elements sum to far more than k 2^-28 of it, are never refused.
__device__ __forceinline__ bool row_is_wide(float lost, float sum, uint32_t k, float* red) {
  if (!__syncthreads_or(lost > 0.0f)) return false;
  const float covered = block_sum(lost, red) * 0x1p22f;
  const int few = (int)min(15u, k / 8 - 1), quarter = (int)min(256u, k / 2) / 4;
  const int have = __syncthreads_count(sum >= covered), share = __syncthreads_count(sum * (float)quarter >= covered);
  return have < few + 1 && share < few + quarter;
}

// One CTA per row: norm (the sums in the order of the stand-alone norm kernels: the same bits), the row's power of
// two, the two fp16 terms, zeros up to the padded width. `normed` (with a norm) gets the f32 row.
__global__ void __launch_bounds__(256)
    rows_split_kernel(const float* __restrict__ x, uint32_t m, uint32_t k, uint32_t kp, int norm, const float* __restrict__ g,
                      const float* __restrict__ b, float eps, float* __restrict__ normed, __half* __restrict__ xh,
                      __half* __restrict__ xl, float* __restrict__ x_scale) {
  __shared__ float red[32];
  __shared__ uint32_t s_max;
  const uint32_t r = blockIdx.x;
  if (r >= m) { // padding rows
    for (uint32_t i = threadIdx.x * 2; i < kp; i += blockDim.x * 2)
      *reinterpret_cast<__half2*>(xh + (size_t)r * kp + i) = *reinterpret_cast<__half2*>(xl + (size_t)r * kp + i) = __floats2half2_rn(0.0f, 0.0f);
    if (threadIdx.x == 0) x_scale[r] = 1.0f;
    return;
  }
  const float* row = x + (size_t)r * k;
  if (threadIdx.x == 0) s_max = 0;
  float mean = 0.0f, inv = 1.0f;
  if (norm == NORM_RMS) {
    float ss = 0.0f;
    for (uint32_t i = threadIdx.x; i < k; i += blockDim.x) ss = fmaf(row[i], row[i], ss);
    inv = 1.0f / sqrtf(block_sum(ss, red) / (float)k + eps);
  } else if (norm == NORM_LAYER) {
    float s = 0.0f;
    for (uint32_t i = threadIdx.x; i < k; i += blockDim.x) s += row[i];
    mean = block_sum(s, red) / (float)k;
    float vs = 0.0f;
    for (uint32_t i = threadIdx.x; i < k; i += blockDim.x) {
      const float dl = row[i] - mean;
      vs = fmaf(dl, dl, vs);
    }
    inv = 1.0f / sqrtf(block_sum(vs, red) / (float)k + 1e-5f);
  }
  auto value = [&](uint32_t i) {
    return norm == NORM_RMS ? row[i] * inv * g[i] : norm == NORM_LAYER ? (row[i] - mean) * inv * g[i] + b[i] : row[i];
  };
  uint32_t mx = 0; // magnitudes order as their bits do; an infinity or NaN is above every finite value
  for (uint32_t i = threadIdx.x; i < k; i += blockDim.x) {
    const float v = value(i);
    mx = max(mx, __float_as_uint(v) & 0x7fffffffu);
    if (norm) normed[(size_t)r * k + i] = v;
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) atomicMax(&s_max, mx);
  __syncthreads();
  const bool finite = s_max < 0x7f800000u;
  float mul, back;
  pow2_to(__uint_as_float(s_max), 14, mul, back);
  constexpr float UP = (float)(1 << LOW_SHIFT);
  float lost = 0.0f, sum = 0.0f;
  for (uint32_t i = threadIdx.x * 2; i < kp; i += blockDim.x * 2) { // (k and kp are even)
    float v0 = 0.0f, v1 = 0.0f;
    if (finite && i < k) v0 = value(i) * mul, v1 = value(i + 1) * mul;
    const __half2 h = __floats2half2_rn(v0, v1);
    float2 f = __half22float2(h);
    *reinterpret_cast<__half2*>(xh + (size_t)r * kp + i) = h;
    const float l0 = (v0 - f.x) * UP, l1 = (v1 - f.y) * UP;
    const __half2 l = __floats2half2_rn(l0, l1);
    *reinterpret_cast<__half2*>(xl + (size_t)r * kp + i) = l;
    const float a0 = fabsf(v0), a1 = fabsf(v1);
    if (fminf(a0, a1) < 0x1p-14f) { // (only there can the terms be short)
      const float2 lf = __half22float2(l);
      const float e0 = fabsf(l0 - lf.x), e1 = fabsf(l1 - lf.y); // the errors, times 2^11
      if (e0 > a0 * 0x1p-11f) lost += e0 * 0x1p-11f;
      if (e1 > a1 * 0x1p-11f) lost += e1 * 0x1p-11f;
    }
    sum += a0 + a1;
  }
  const bool held = finite && !row_is_wide(lost, sum, k, red); // (else: the product's own f32 chain)
  if (threadIdx.x == 0) x_scale[r] = held ? back : 0.0f;
}

// One warp per weight row: the row's power of two from its block scales, then eight elements per lane and step: the
// f32 product d q 2^t (exact: 19 bits) and its two fp16 terms, 16 bytes of each per lane.
template <int KIND>
__global__ void __launch_bounds__(256)
    weights_split_kernel(QMat w, uint32_t kp, __half* __restrict__ wh, __half* __restrict__ wl, float* __restrict__ w_scale) {
  const uint32_t n = blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (n >= w.n) return;
  const uint32_t nb = w.k / QK;
  const __half* sc = w.sc + (size_t)n * nb;
  uint32_t mx = 0;
  for (uint32_t i = lane; i < nb; i += 32) mx = max(mx, (uint32_t)__half_as_ushort(sc[i]) & 0x7fffu);
  mx = __reduce_max_sync(0xffffffffu, mx);
  const bool finite = mx < 0x7c00u;
  float mul, back;
  pow2_to(__half2float(__ushort_as_half((unsigned short)mx)), 7, mul, back);
  if (lane == 0) w_scale[n] = finite ? back : 0.0f;
  for (uint32_t i = lane; i < kp / 8; i += 32) {
    float v[8];
    if (i * 8 < w.k && finite) {
      const float d = __half2float(sc[i / 4]) * mul;
      if (KIND == FC_Q8_0) {
        const uint2 q = *reinterpret_cast<const uint2*>(w.qs + (size_t)n * w.k + i * 8);
        const uint32_t qw[2] = {q.x, q.y};
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = d * (float)(int8_t)((qw[j >> 2] >> (8 * (j & 3))) & 0xffu);
      } else {
        const uint32_t q = *reinterpret_cast<const uint32_t*>(w.qs + (size_t)n * (w.k / 2) + i * 4);
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = d * ((float)((q >> (4 * ((j >> 1) + 4 * (j & 1)))) & 15u) - 8.0f);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; j++) v[j] = 0.0f;
    }
    uint32_t h[4], l[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const __half2 hh = __floats2half2_rn(v[2 * j], v[2 * j + 1]);
      const float2 f = __half22float2(hh);
      const __half2 ll = __floats2half2_rn((v[2 * j] - f.x) * (float)(1 << LOW_SHIFT), (v[2 * j + 1] - f.y) * (float)(1 << LOW_SHIFT));
      h[j] = *reinterpret_cast<const uint32_t*>(&hh);
      l[j] = *reinterpret_cast<const uint32_t*>(&ll);
    }
    const size_t at = (size_t)n * kp + i * 8;
    *reinterpret_cast<uint4*>(wh + at) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4*>(wl + at) = make_uint4(l[0], l[1], l[2], l[3]);
  }
}

// [rows][kp] fp16, boxes of `box` rows x 64 k under the 128-byte swizzle; rows past the end read as zeros
int make_map(FcDevice* dev, CUtensorMap* map, const __half* p, uint32_t rows, uint32_t kp, uint32_t box_rows) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return fc_fail(dev, FC_ERR_DEVICE, "cuTensorMapEncodeTiled is not available from this driver");
  const cuuint64_t dims[2] = {kp, rows};
  const cuuint64_t strides[1] = {(cuuint64_t)kp * 2};
  const cuuint32_t box[2] = {BK, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult cr = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (void*)p, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (cr != CUDA_SUCCESS) return fc_fail(dev, FC_ERR_DEVICE, "cuTensorMapEncodeTiled failed with %d", (int)cr);
  return FC_OK;
}

// Widths up to this many K steps add every 64 k in f32: a short f32 chain is accurate itself (K 96: 1.75e-7 of the
// result's norm), and there are too few steps for the epilogue to hold the MMAs up.
constexpr uint32_t SHORT_STEPS = 4;

// The tiled f32 kernel takes about 4 us and 57 ns per k while its 64 x 64 tiles are at most 174 or so, in proportion to
// them beyond; the pair's three launches take 17 us at least: k x max(tiles, 174) up to which the tiled kernel is ahead.
constexpr uint64_t TILED_WAVE = 174, TILED_KEEPS = 228 * TILED_WAVE;

// How a launch is cut: rows of x per tile and the split of K.
struct Plan {
  uint32_t kp, steps, bn, splits, per_split, slice; // slice: weight rows whose terms are in the workspace at once
};
constexpr size_t W_TERMS_BYTES = (size_t)64 << 20;
size_t al(size_t v) { return (v + 1023) & ~(size_t)1023; }
// sums: the result leaves through pair_reduce_kernel even without a split of K (an activation)
size_t plan_bytes(const Plan& p, uint32_t m, bool sums) {
  return 2 * al((size_t)m * p.kp * 2) + 2 * al((size_t)p.slice * p.kp * 2) + al((size_t)m * 4) + al((size_t)p.slice * 4) +
         (p.splits > 1 || sums ? al((size_t)p.splits * m * p.slice * 4) : 0) + 1024;
}
// The best cut whose workspace fits into `limit` bytes; splits == 0 where not even the smallest does. (Fewer rows may ask
// for more than many: they leave the chip idle without a split of K, and every split has sums of its own.)
Plan make_plan(uint32_t sms, uint32_t k, uint32_t n, uint32_t m, bool sums, size_t limit) {
  Plan p;
  p.kp = (k + BK - 1) / BK * BK;
  p.steps = p.kp / BK;
  const size_t fit = W_TERMS_BYTES / ((size_t)p.kp * 4) / 256 * 256;
  p.slice = (uint32_t)(fit < 256 ? 256 : fit);
  if (p.slice >= n) p.slice = n;
  // The cut with the least estimated time: whole waves of pairs, K steps of one pair at about 1000 (128 rows of x) or
  // 700 (64 rows) cycles each, and for a split of K its second launch and the sums' way through L2 (2 KB a cycle).
  const uint64_t pairs = sms / 2, tiles_n = (p.slice + 255) / 256;
  uint64_t best = ~0ull;
  p.bn = p.splits = p.per_split = 0;
  for (uint32_t bn : {128u, 64u})
    for (uint32_t c = 1; c <= 8 && c <= p.steps; c++) {
      const uint64_t items = tiles_n * ((m + bn - 1) / bn) * c, per = (p.steps + c - 1) / c;
      const uint64_t cost = (items + pairs - 1) / pairs * (per * (bn == 128 ? 1000 : 700) + 3000) +
                            (c > 1 ? 5000 + (uint64_t)m * p.slice * 4 * (2 * c + 1) / 2048 : 0);
      if (cost >= best) continue;
      Plan q = p;
      q.bn = bn, q.per_split = (uint32_t)per, q.splits = (uint32_t)((p.steps + per - 1) / per);
      if (plan_bytes(q, m, sums) <= limit) best = cost, p = q;
    }
  return p;
}

template <int KIND, int BN>
int launch(FcDevice* dev, const CUtensorMap* maps, const PairArgs& a) {
  auto kern = qgemm_pair_kernel<KIND, BN>;
  static OncePerDevice attr;
  if (attr.first(dev->ordinal)) {
    FC_CUDA(dev, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Shape<BN>::SMEM));
  }
  const uint32_t items = ((a.w.n + 255) / 256) * ((a.m + BN - 1) / BN) * a.splits;
  const uint32_t pairs = (uint32_t)dev->prop.multiProcessorCount / 2;
  FC_LAUNCH(dev, "qgemm_pair",
            kern<<<2 * (items < pairs ? items : pairs), PAIR_THREADS, Shape<BN>::SMEM, dev->stream>>>(maps[0], maps[1], maps[2], maps[3], a));
  return FC_OK;
}

} // namespace

// Every product of more than 64 rows of the integer formats (up to 64 the weights are streamed packed: matvec_mma.cu).
// Against the tiled f32 kernel: 512 x 2048 x 32000 Q8_0 294 us instead of 2523, 1536 x 1024 x 5632 Q8_0 69 instead of 677,
// 100 x 768 x 1280 Q4_0 21 instead of 46, 65 x 512 x 512 19 instead of 33, 128 x 320 x 1000 19 instead of 21; short widths
// with few tiles, where three launches cost more than they save (128 x 64 x 512: 17.5 instead of 7.8, 333 x 96 x 1000: 17
// instead of 10), keep the tiled kernel (TILED_KEEPS). At 1536 x 1024 x 5632 the tensor pipe is
// active 47 %, L2 33 %: 264 tiles take 4 waves of pairs (3.6 full), and every 128 k the accumulator changes hands between
// the MMA thread and the epilogues of two SMs.
// Error against f64 on N(0, 1) x N(0, 0.02), of the result's norm: 1.2e-7 (K 96) to 2.2e-7 (K 4096); the f32 chain
// 1.8e-7 to 1.15e-6. With two elements of 2^20 or 2^26 in every row, the largest error of an output against its own
// sum |x w|: 0.9e-6..1.3e-6 (the chain 2.3e-6..7.7e-6; with low terms at their own magnitude 2^26 came to 1e-5, beyond 2^34
// to a thousandth and more). The check of the rows costs 1 us a call.
bool qgemm_pair_takes(const QMat& w, uint32_t m) {
  const uint64_t tiles = (uint64_t)((w.n + 63) / 64) * ((m + 63) / 64); // the tiled kernel's CTAs
  if (w.k * (tiles > TILED_WAVE ? tiles : TILED_WAVE) < TILED_KEEPS) return false;
  return (w.kind == FC_Q8_0 || w.kind == FC_Q4_0) && m > 64 && w.k % QK == 0 && w.k > 0 && w.n > 0;
}

size_t qgemm_pair_scratch_bytes(const FcDevice* dev, uint32_t k, uint32_t n, uint32_t m, int act) {
  return plan_bytes(make_plan((uint32_t)dev->prop.multiProcessorCount, k, n, m, act != ACT_NONE, SIZE_MAX), m, act != ACT_NONE);
}
bool qgemm_pair_fits(const FcDevice* dev, uint32_t k, uint32_t n, uint32_t m, int act, size_t bytes) {
  return make_plan((uint32_t)dev->prop.multiProcessorCount, k, n, m, act != ACT_NONE, bytes).splits != 0;
}
FC_API uint64_t fc_debug_pair_bytes(uint32_t sm_count, uint32_t k, uint32_t n, uint32_t m, int gelu, uint64_t limit) {
  if (sm_count < 2 || !k || k % QK || !n || !m) return 0;
  const Plan p = make_plan(sm_count, k, n, m, gelu != 0, (size_t)limit);
  return p.splits ? plan_bytes(p, m, gelu != 0) : 0;
}

int k_qgemm_pair(FcDevice* dev, const QMat& w, const float* x, uint32_t m, float* y, const Epilogue& ep, const Workspace& space) {
  if (m == 0) return FC_OK;
  const Plan p = make_plan((uint32_t)dev->prop.multiProcessorCount, w.k, w.n, m, ep.act != ACT_NONE, space.bytes);
  if (!p.splits) return fc_fail(dev, FC_ERR_ARG, "a %zu-byte workspace is too small for this product", space.bytes);
  uint8_t* at = (uint8_t*)(((uintptr_t)space.p + 1023) & ~(uintptr_t)1023);
  auto take = [&](size_t bytes) {
    uint8_t* r = at;
    at += al(bytes);
    return r;
  };
  __half* xh = (__half*)take((size_t)m * p.kp * 2);
  __half* xl = (__half*)take((size_t)m * p.kp * 2);
  __half* wh = (__half*)take((size_t)p.slice * p.kp * 2);
  __half* wl = (__half*)take((size_t)p.slice * p.kp * 2);
  float* xs = (float*)take((size_t)m * 4);
  float* ws = (float*)take((size_t)p.slice * 4);
  float* partial = p.splits > 1 || ep.act != ACT_NONE ? (float*)take((size_t)p.splits * m * p.slice * 4) : nullptr;
  if (ep.norm != NORM_NONE && !ep.norm_tmp) return fc_fail(dev, FC_ERR_ARG, "a fused norm needs a temporary");
  FC_LAUNCH(dev, "rows_split",
            rows_split_kernel<<<m, 256, 0, dev->stream>>>(x, m, w.k, p.kp, ep.norm, ep.norm_g, ep.norm_b, ep.norm_eps, ep.norm_tmp, xh, xl, xs));
  if (ep.norm != NORM_NONE) x = ep.norm_tmp;
  CUtensorMap maps[4];
  FC_TRY(make_map(dev, &maps[2], xh, m, p.kp, p.bn / 2));
  FC_TRY(make_map(dev, &maps[3], xl, m, p.kp, p.bn / 2));
  for (uint32_t n0 = 0; n0 < w.n; n0 += p.slice) {
    PairArgs a;
    a.w = w;
    a.w.n = w.n - n0 < p.slice ? w.n - n0 : p.slice;
    a.w.qs = w.qs + qmat_qs_bytes(w.kind, w.k, n0);
    a.w.sc = (const __half*)((const uint8_t*)w.sc + qmat_sc_bytes(w.kind, w.k, n0));
    if (w.kind == FC_Q8_0)
      FC_LAUNCH(dev, "weights_split", weights_split_kernel<FC_Q8_0><<<(a.w.n + 7) / 8, 256, 0, dev->stream>>>(a.w, p.kp, wh, wl, ws));
    else
      FC_LAUNCH(dev, "weights_split", weights_split_kernel<FC_Q4_0><<<(a.w.n + 7) / 8, 256, 0, dev->stream>>>(a.w, p.kp, wh, wl, ws));
    FC_TRY(make_map(dev, &maps[0], wh, a.w.n, p.kp, 128));
    FC_TRY(make_map(dev, &maps[1], wl, a.w.n, p.kp, 128));
    a.x = x, a.m = m, a.steps = p.steps, a.steps_per_split = p.per_split, a.splits = p.splits;
    a.chunk = p.steps <= SHORT_STEPS ? 1 : 2;
    a.y = y + n0, a.ldy = w.n;
    a.bias = ep.bias ? ep.bias + n0 : nullptr;
    a.resid = ep.resid ? ep.resid + n0 : nullptr;
    a.x_scale = xs, a.w_scale = ws, a.partial = partial, a.err_flag = dev->d_flag;
    if (w.kind == FC_Q8_0)
      FC_TRY(p.bn == 128 ? (launch<FC_Q8_0, 128>(dev, maps, a)) : (launch<FC_Q8_0, 64>(dev, maps, a)));
    else
      FC_TRY(p.bn == 128 ? (launch<FC_Q4_0, 128>(dev, maps, a)) : (launch<FC_Q4_0, 64>(dev, maps, a)));
    if (partial)
      FC_LAUNCH(dev, "pair_reduce",
                pair_reduce_kernel<<<dim3((a.w.n + 255) / 256, m < 65535 ? m : 65535), 256, 0, dev->stream>>>(
                    partial, p.splits, m, a.w.n, a.y, a.ldy, a.bias, a.resid, ep.act));
  }
  return FC_OK;
}

int k_rows_split(FcDevice* dev, const float* x, uint32_t m, uint32_t mp, uint32_t k, __half* xh, __half* xl, float* x_scale) {
  FC_LAUNCH(dev, "rows_split", rows_split_kernel<<<mp, 256, 0, dev->stream>>>(x, m, k, k, NORM_NONE, nullptr, nullptr, 0.0f,
                                                                              nullptr, xh, xl, x_scale));
  return FC_OK;
}
