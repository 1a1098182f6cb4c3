// Decode steps of one to 64 streams as ONE persistent kernel over all SMs, a chain of greedy ones without leaving it: embedding, every layer (norm, q/k/v
// product, rotation and cache append, attention, output product, norm, gate/up or fc product, activation, down product),
// final norm, head and the greedy pick. Op order of GpuLlama::feed / GpuGpt2::feed
// (ferrum_wgpu/src/models/llama/forward.rs:L18-L72, models/gpt2.rs:L192-L265).
//
// What bounds such a step: neither bytes nor flops but the chain of dependent stages, five per layer. As launches each
// stage pays launch, drain and a cold start of its weight stream: 6-8 us. Here a stage costs one trip of its input through
// L2 and the multiply-adds of a few 16-row tiles:
//
//   * No barrier separates stages. Every activation travels as a 64-bit word, the f32 value beside a 32-bit tag of
//     (launch, layer); consumers poll the very words they need (a 64-bit access is single, so a matching tag vouches for
//     its value). Producer and consumer are one store and one load apart.
//   * The weight stream never waits for activations: one producer warp per CTA runs ahead through the CTA's tiles of all
//     stages and fills a ring in shared memory; the K/V tiles of the CTA's attention items likewise. What a stage needs is
//     there when its input arrives. A slot is one TMA box of 16 rows x up to 1024 bytes, 128-byte swizzled so that the lanes'
//     reads fall into different banks (a bulk copy per row, to a padded pitch, took 110 cycles each: 1900 per tile).
//   * A product gives every CTA tiles of 16 weight rows. Its warps poll x, eight elements per lane, and leave it in shared
//     memory as two fp16 terms (22 bits, every 32-block at a power of two of its own); then they share out the tiles' units
//     of 128 k (mma.sync m16n8k16, the block scale applied to the f32 sum of a block), and the units' sums meet in shared
//     memory. What counts is the length of this chain for some 100 KB of weights: no divisions, the codes of a warp's first
//     unit in registers before x arrives, the factor of RMSNorm applied to the sums.
//     One row uses the eight MMA columns as (block, term) pairs, four blocks at a time: a lane's k slots all come from one
//     block, and its column pair carries that block's x and zeros elsewhere. More rows take a column each (up to four rows:
//     two, one per term).
//   * More than eight rows: the SMs split into as many grids as there are groups of eight rows, each a whole step of its own
//     over all weights, which come from L2 once per group.
//   * Attention: an item is (row, heads of a group, part of the positions); parts merge through the same tagged words.
//
// The code of a layer has to stay below the 32 KB or so that an SM's instruction cache holds: beyond it straight-line code
// takes 6 cycles an instruction, whatever the number of warps (measured; 3 below). Hence one copy of the product for every
// stage and of what it does, a kernel per (format, rows, architecture, heads of an item), and descriptors that spare address
// arithmetic.
//
// A step of a chain ends like a grid barrier: the last CTA to arrive takes the picks and publishes them as tagged words, which
// start the next step; by then every cache append of the step before is visible.
//
// A value is overwritten one layer later at the earliest (a token one step later); its writer then depends, through the tags,
// on every reader of the old one having finished its stage. A word belongs to one group of CTAs for good: tags count per group,
// and only one that never comes round again tells a word from what an earlier launch left there. All CTAs are resident (cooperative launch) and every wait is bounded: one
// that gives up raises the device's status word and ends its CTA's other waits; the other CTAs, which miss what that one had to
// send, run into their own limits (1.5 s) at about the same time, and the step reports it. A word raised before the launch ends all
// waits at once.
#include <algorithm>
#include <cstring>

#include "model.cuh"
#include "tc_ptx.cuh"
#include "tensor_map.cuh"

namespace {

// 12 consumer warps and a warpgroup for the producer: 128 registers a thread. (20 warps at 96 spilled 90 of them, and next to
// 227 KB of shared memory there is no L1 to hold spills: every stage took three times as long.)
constexpr int WARPS = 12;
constexpr int AWARPS = 8;               // those that an attention item needs
constexpr int CONS = WARPS * 32;
constexpr int THREADS = CONS + 128;
constexpr uint32_t MAX_K = 3072;
constexpr uint32_t TASKS = MAX_K / 256; // 256-element parts of a row of x
constexpr uint32_t MAX_GROUPS = 8;      // groups of eight rows
// 128-byte lines of a weight row per ring slot, at most
__host__ __device__ constexpr uint32_t slot_lines(int mt) { return mt == 8 ? 4 : 8; }
// tiles between two barriers, at most: their 16 x mt results take a thread each
__host__ __device__ constexpr uint32_t tile_group(int mt) { return mt == 8 ? 3 : 4; }
constexpr uint32_t SLOTS = 16;          // ring slots outstanding, at most
constexpr uint32_t KV_POS = 64;         // positions of a K/V tile
constexpr uint32_t KV_TILE = KV_POS * 64 * 4;
constexpr uint32_t MAX_KV = 4;          // K/V tiles in flight
constexpr uint32_t MAX_SPLITS = 16;
constexpr uint32_t MAX_ITEMS = 24;      // attention items per CTA
constexpr uint32_t MAX_RESID = 11;      // 16-row tiles of the residual stream per CTA
constexpr uint32_t ITEM_HEADS = 4;      // heads of an attention item, at most
constexpr uint32_t PART = 66;           // max, sum, 64 channels
constexpr uint32_t SMEM_MAX = 227 * 1024;
constexpr uint32_t POLL_LIMIT = 1u << 21; // tries of a poll (about 0.7 us each)

struct DgMat {
  const void *map_w, *map_s; // tensor maps of the codes, [line][row][128 bytes], and of the scales
  const __half* sc;
  const float *bias, *gain, *beta; // (gain: its input is normed)
};
struct DgLayer {
  DgMat m[4]; // qkv, wo, ff1, ff2
  float *kc, *vc;
};
// What the four matrices have in common over the layers (the fifth is the head), derived so that no stage divides:
// 256-element parts of a row of x and 2^16 / that, 128-element units, ring slots per tile; of a slot the place of the scales,
// their pitch (halves) and bytes, its size; tiles between two barriers.
struct DgShape {
  const unsigned long long* src; // tagged words of its input and its result
  unsigned long long* dst;
  uint32_t k, n, tpr, tpr_inv, nu, nch, sc_off, sc_pitch, sc_bytes, size, group, dst_stride;
  float k_inv;
};
struct DgArgs {
  DgShape sh[5];
  const DgLayer* layers;
  DgMat head;
  const float *tok, *pos_table, *cos, *sin;
  uint32_t rope_dim, rope_type, n_layers, dim, heads, kv_heads, ctx;
  uint32_t heads_inv; // 2^16 / heads, rounded up
  float eps;
  // tagged words: b_qkv [row][width]; the others, inputs of a product, [row][width in whole 256s] with the words of 256
  // elements in the order of ll_at; partial attention results per (row, head): [8 channels][split][8], then max and sum of
  // every split
  unsigned long long *b_qkv, *b_attn, *b_x1, *b_x2, *b_act, *b_part;
  uint32_t x_stride, attn_stride, act_stride; // words of a row
  uint32_t group_words;     // (of one group of rows)
  uint32_t* state;          // per group: [0] the last tag of the launches before, [1] CTAs that are through
  unsigned long long* keys; // [64] best (logit, index) of a row; zero between launches
  int32_t* out;             // [64] picks, [8] the groups' status words
  float* logits;
  int* err_flag;
  // tagged words: [group][8] the tokens of a chain's next step. By group and not by row of the batch: tags count per group, and
  // the group of a row depends on how many rows there are (row 5 of 8 is in group 0, of 10 in group 1).
  unsigned long long* toks;
  int32_t* log;             // [step][row] the tokens that a chain consumes
  int32_t tok_in[64], pos[64], stream[64];
  uint32_t rows, group_rows, sub; // rows of a group, CTAs of a group
  uint32_t steps, chained, splits, item_heads, kv_log; // (2^kv_log K/V tiles in flight)
  uint32_t off_desc, off_red, off_x, off_ys, off_kv, off_ring, ring_bytes;
};

struct Misc { // small per-CTA state
  uint64_t full[SLOTS], empty[SLOTS], kv_full[MAX_KV], kv_empty[MAX_KV];
  uint32_t slot_at[SLOTS];     // where in the ring the producer put a slot
  float redss[2][8][TASKS], ln1[8][TASKS], ln2[8][TASKS];
  float resid[MAX_RESID * 8 * 16];
  float slice[(ITEM_HEADS + 2) * 64]; // q heads (scaled), k, v of the attention item's own position
  float pw[AWARPS][8][ITEM_HEADS], cw[AWARPS][ITEM_HEADS];
  float wm[AWARPS][ITEM_HEADS], wl[AWARPS][ITEM_HEADS];
  int32_t ids[8], next[8], pos[8], stream[8];
  uint32_t used[8];            // parts that a row's positions are in
  struct Item {
    uint32_t r, h0, kvh, s, c0, c1, append; // row, first head, split, its K/V tiles; whether it appends k and v to the cache
  } items[MAX_ITEMS];
  uint32_t n_items, tiles[5], first[5]; // the CTA's attention items; its tiles of qkv, wo, ff1, ff2, head: T = first, + grid, ..
  uint32_t planned, seen;      // steps whose items and positions are there; steps whose the producer has no more use for
  int dead, stop;
};

__device__ __forceinline__ unsigned long long ll_ld(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void ll_ld2(const unsigned long long* p, unsigned long long& v, unsigned long long& w) {
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v), "=l"(w) : "l"(p) : "memory");
}
__device__ __forceinline__ void ll_st(unsigned long long* p, float v, uint32_t tag) {
  const unsigned long long w = ((unsigned long long)tag << 32) | __float_as_uint(v);
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ float ll_val(unsigned long long w) { return __uint_as_float((uint32_t)w); }
__device__ __forceinline__ bool ll_ok(unsigned long long w, uint32_t tag) { return (uint32_t)(w >> 32) == tag; }

// Where element e of a product's input has its word. A warp polls 256 elements, eight consecutive ones per lane: pair i of
// all lanes lies together, so that a request is four lines and not sixteen (the polls share the load pipe with everything
// that the other warps do in shared memory).
__device__ __forceinline__ uint32_t ll_at(uint32_t e) { return (e & ~255u) | ((e >> 1) & 3u) << 6 | ((e >> 3) & 31u) << 1 | (e & 1u); }

__device__ __forceinline__ void cons_sync() { asm volatile("bar.sync 1, 384;" ::: "memory"); }

__device__ __forceinline__ float dg_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 1 / sqrt(x) by one Newton step on the approximation, to the last bit or so (x a mean square plus eps: normal)
__device__ __forceinline__ float dg_rsqrt(float x) {
  const float y = rsqrtf(x);
  return fmaf(0.5f * y, fmaf(-x * y, y, 1.0f), y);
}
__device__ __forceinline__ float dg_gelu(float x) {
  const float K = 0.7978846f; // ferrum_ref/src/kernels/nn.rs:L12-L15
  return 0.5f * x * (1.0f + tanhf(K * (x + 0.044715f * x * x * x)));
}
__device__ __forceinline__ void dg_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t h2sub(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t h2fma(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t r;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
}
// Eight consecutive weights of a row as four fp16 pairs in element order: the integer codes, exactly.
// Q8_0 (two words): byte b as 1024 + (b + 128) in the mantissa, minus 1152. Q4_0 (one): the nibble as 1024 + n (minus
// 1032), or one place up as 1024 + 16 n (times 1/16, minus 72).
template <bool Q8>
__device__ __forceinline__ void codes8(uint32_t w, uint32_t w2, uint32_t (&p)[4]) {
  if (Q8) {
    const uint32_t u0 = w ^ 0x80808080u, u1 = w2 ^ 0x80808080u, c = 0x64806480u;
    p[0] = h2sub(__byte_perm(u0, 0x64646464u, 0x4140), c);
    p[1] = h2sub(__byte_perm(u0, 0x64646464u, 0x4342), c);
    p[2] = h2sub(__byte_perm(u1, 0x64646464u, 0x4140), c);
    p[3] = h2sub(__byte_perm(u1, 0x64646464u, 0x4342), c);
  } else {
    const uint32_t w8 = w >> 8;
    p[0] = h2sub((w & 0x000f000fu) | 0x64006400u, 0x64086408u);
    p[1] = h2fma((w & 0x00f000f0u) | 0x64006400u, 0x2c002c00u, 0xd480d480u);
    p[2] = h2sub((w8 & 0x000f000fu) | 0x64006400u, 0x64086408u);
    p[3] = h2fma((w8 & 0x00f000f0u) | 0x64006400u, 0x2c002c00u, 0xd480d480u);
  }
}

// Bounded waits that end early once somebody in the CTA gave up; other CTAs run into their own limit at about the same time. Who
// gave up goes on with whatever is there: values may be anything, addresses may not come from words that the wait vouches for.
// (Nor does a barrier's parity vouch for them then: a whole ring past the producer it counts as complete.)
struct Ctl {
  volatile int* dead;
  int* err;
  __device__ __forceinline__ bool give_up(uint32_t tries, uint32_t every = 256) { // by a polling thread, after every try
    if (tries & (every - 1)) return false;
    if (tries >= POLL_LIMIT) *dead = 1, *(volatile int*)err = 1;
    return *dead != 0;
  }
  __device__ __forceinline__ void mbar(uint64_t* bar, uint32_t parity) {
    uint32_t tries = 0;
    while (!tc::mbar_try_wait(bar, parity))
      if (give_up(++tries, 8)) break;
  }
};

// Positions of an item: its part of the row's 64-position tiles, cut evenly over the splits.
__device__ __forceinline__ void item_range(uint32_t len, uint32_t splits, uint32_t s, uint32_t& c0, uint32_t& c1, uint32_t& used) {
  const uint32_t tiles = (len + KV_POS - 1) / KV_POS, per = (tiles + splits - 1) / splits;
  c0 = min(tiles, s * per), c1 = min(tiles, c0 + per);
  used = (tiles + per - 1) / per;
}

// One attention item. GP: its heads, padded to 1 or 4. A warp takes eight positions of every 64-position tile: two per
// eight lanes for the scores (a lane has 8 channels of every head; the sums are exchanged so that a lane ends up with one
// head's score), then the 16 four-channel columns x two halves of the positions for the weighted sum of V.
template <int GP>
__device__ __forceinline__ void attn_item(const DgArgs& a, const DgLayer& L, Misc& ms, float* wpart, float* kv_tiles, uint32_t& kvn,
                                          Ctl ctl, uint32_t tag, uint32_t words, const Misc::Item& im) {
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), grp = lane >> 3, sub = lane & 7;
  const uint32_t r = im.r, h0 = im.h0, kvh = im.kvh, c0 = im.c0, c1 = im.c1;
  const uint32_t G = GP == 1 ? 1u : a.item_heads, len = (uint32_t)ms.pos[r] + 1;
  // q, k, v of the row's own position: two channels per thread, rotated on the way in
  if (tid < (int)(G + 2) * 32) {
    const uint32_t hs = tid >> 5, pp = tid & 31, half = a.rope_dim / 2, p = len - 1;
    const bool rot = a.cos && hs <= G && pp < half;
    const bool neox = rot && a.rope_type != FC_ROPE_NORM;
    const uint32_t ia = neox ? pp : 2 * pp, ib = neox ? pp + half : 2 * pp + 1;
    const float cs = rot ? a.cos[(size_t)p * half + pp] : 1.0f, sn = rot ? a.sin[(size_t)p * half + pp] : 0.0f;
    const uint32_t col = (hs < G ? h0 + hs : a.heads + kvh + (hs == G ? 0u : a.kv_heads)) * 64;
    const unsigned long long* src = a.b_qkv + words + r * a.sh[0].dst_stride + col;
    unsigned long long w0, w1;
    uint32_t tries = 0;
    do {
      w0 = ll_ld(src + ia), w1 = ll_ld(src + ib);
    } while (!(ll_ok(w0, tag) && ll_ok(w1, tag)) && !ctl.give_up(++tries));
    float x = ll_val(w0), y = ll_val(w1);
    if (rot) {
      const float xr = x * cs - y * sn, yr = x * sn + y * cs;
      x = xr, y = yr;
    }
    const float qs = hs < G ? 0.125f * 1.4426950408889634f : 1.0f; // (scores in the log2 domain)
    ms.slice[hs * 64 + ia] = x * qs;
    ms.slice[hs * 64 + ib] = y * qs;
    if (hs >= G && im.append) {
      float* dst = (hs == G ? L.kc : L.vc) + (((size_t)ms.stream[r] * a.kv_heads + kvh) * a.ctx + p) * 64;
      dst[ia] = x, dst[ib] = y;
    }
  }
  cons_sync();
  const uint32_t hh = GP == 4 ? sub >> 1 : 0; // the head whose score this lane ends up with
  const int ch4 = lane & 15, half = lane >> 4;
  if (warp < AWARPS) {
    float m_run = -INFINITY, l_run = 0.0f, acc[GP][4];
#pragma unroll
    for (int h = 0; h < GP; h++) acc[h][0] = acc[h][1] = acc[h][2] = acc[h][3] = 0.0f;
#pragma unroll 1
    for (uint32_t c = c0; c < c1; c++, kvn++) {
      const uint32_t buf = kvn & ((1u << a.kv_log) - 1), base = c * KV_POS + warp * 8;
      float* kt = kv_tiles + buf * 2 * (KV_TILE / 4) + warp * 8 * 64;
      const float* vt = kt + KV_TILE / 4;
      ctl.mbar(&ms.kv_full[buf], (kvn >> a.kv_log) & 1);
      if (base < len) { // (uniform in the warp)
        if (base + 8 >= len) { // the row's own position, which the cache did not hold when the tile was fetched
          const uint32_t at = (half ? KV_TILE / 4 : 0u) + (len - 1 - base) * 64 + ch4 * 4;
          *reinterpret_cast<float4*>(kt + at) = *reinterpret_cast<const float4*>(ms.slice + (G + half) * 64 + ch4 * 4);
          tc::fence_async_smem(); // (the tile's next contents come by the async proxy)
          __syncwarp();
        }
        float sc[2];
#pragma unroll
        for (int i = 0; i < 2; i++) {
          const uint32_t pos = base + i * 4 + grp;
          const bool valid = pos < len;
          const float* kp = kt + (i * 4 + grp) * 64 + sub * 4; // (past the end: anything, the score is not used)
          const float4 k0 = *reinterpret_cast<const float4*>(kp), k1 = *reinterpret_cast<const float4*>(kp + 32);
          float d[GP];
#pragma unroll
          for (int h = 0; h < GP; h++) {
            d[h] = 0.0f;
            if (GP == 1 || h < (int)G) {
              const float4 q0 = *reinterpret_cast<const float4*>(ms.slice + h * 64 + sub * 4);
              const float4 q1 = *reinterpret_cast<const float4*>(ms.slice + h * 64 + 32 + sub * 4);
              float v = q0.x * k0.x, w = q1.x * k1.x;
              v = fmaf(q0.y, k0.y, v), w = fmaf(q1.y, k1.y, w);
              v = fmaf(q0.z, k0.z, v), w = fmaf(q1.z, k1.z, w);
              v = fmaf(q0.w, k0.w, v), w = fmaf(q1.w, k1.w, w);
              d[h] = v + w;
            }
          }
          if (GP == 4) {
            const bool u4 = sub & 4, u2 = sub & 2;
            float e[2];
#pragma unroll
            for (int j = 0; j < 2; j++)
              e[j] = (u4 ? d[(j + 2) % GP] : d[j % GP]) + __shfl_xor_sync(0xffffffffu, u4 ? d[j % GP] : d[(j + 2) % GP], 4);
            sc[i] = (u2 ? e[1] : e[0]) + __shfl_xor_sync(0xffffffffu, u2 ? e[0] : e[1], 2);
            sc[i] += __shfl_xor_sync(0xffffffffu, sc[i], 1);
          } else {
            sc[i] = d[0];
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) sc[i] += __shfl_xor_sync(0xffffffffu, sc[i], o);
          }
          if (!valid) sc[i] = -INFINITY;
        }
        float mn = fmaxf(sc[0], sc[1]);
        mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 8));
        mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 16));
        mn = fmaxf(mn, m_run);
        const bool any = mn != -INFINITY;
        const float corr = any ? dg_ex2(m_run - mn) : 1.0f;
        m_run = mn;
        float ps = 0.0f;
#pragma unroll
        for (int i = 0; i < 2; i++) {
          const float p = any ? dg_ex2(sc[i] - mn) : 0.0f;
          ms.pw[warp][i * 4 + grp][hh] = p;
          ps += p;
        }
        if (grp == 0) ms.cw[warp][hh] = corr;
        __syncwarp();
        ps += __shfl_xor_sync(0xffffffffu, ps, 8);
        ps += __shfl_xor_sync(0xffffffffu, ps, 16);
        l_run = fmaf(l_run, corr, ps);
#pragma unroll
        for (int h = 0; h < GP; h++) {
          const float cf = ms.cw[warp][h];
          acc[h][0] *= cf, acc[h][1] *= cf, acc[h][2] *= cf, acc[h][3] *= cf;
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const uint32_t g = 2 * i + half, pv = base + g;
          if (pv < len) {
            const float4 v = *reinterpret_cast<const float4*>(vt + g * 64 + ch4 * 4);
#pragma unroll
            for (int h = 0; h < GP; h++) {
              const float w = ms.pw[warp][g][h];
              acc[h][0] = fmaf(w, v.x, acc[h][0]);
              acc[h][1] = fmaf(w, v.y, acc[h][1]);
              acc[h][2] = fmaf(w, v.z, acc[h][2]);
              acc[h][3] = fmaf(w, v.w, acc[h][3]);
            }
          }
        }
      }
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&ms.kv_empty[buf]);
    }
    // the warp's part, then the merge over the warps
#pragma unroll
    for (int h = 0; h < GP; h++) {
#pragma unroll
      for (int i = 0; i < 4; i++) acc[h][i] += __shfl_xor_sync(0xffffffffu, acc[h][i], 16);
      if (half == 0)
        *reinterpret_cast<float4*>(wpart + ((size_t)warp * GP + h) * 64 + ch4 * 4) = make_float4(acc[h][0], acc[h][1], acc[h][2], acc[h][3]);
    }
    if (grp == 0) ms.wm[warp][hh] = m_run, ms.wl[warp][hh] = l_run;
  }
  cons_sync();
  if (warp < (int)G * 2) {
    const int h = tid >> 6, ch = tid & 63, w = lane & 7;
    const float mm = ms.wm[w][h];
    float M = mm;
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
    const float f = mm == -INFINITY ? 0.0f : dg_ex2(mm - M);
    float l = f * ms.wl[w][h];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    float o = 0.0f;
#pragma unroll
    for (int i = 0; i < AWARPS; i++) o = fmaf(__shfl_sync(0xffffffffu, f, i), wpart[((size_t)i * GP + h) * 64 + ch], o);
    if (ms.used[r] == 1) {
      ll_st(a.b_attn + words + r * a.attn_stride + ll_at((h0 + h) * 64 + ch), o / l, tag);
    } else {
      unsigned long long* dst = a.b_part + words + (r * a.heads + h0 + h) * a.splits * PART;
      ll_st(dst + ((ch >> 3) * a.splits + im.s) * 8 + (ch & 7), o, tag);
      if (ch < 2) ll_st(dst + a.splits * 64 + 2 * im.s + ch, ch ? l : M, tag);
    }
  }
  cons_sync(); // (the slice and the warps' parts may be overwritten)
}

__host__ __device__ constexpr uint32_t al(uint32_t v, uint32_t a) { return (v + a - 1) / a * a; }
// MT: rows, padded to 1, 2, 4 or 8. GP: heads of an attention item, 1 or up to 4.
template <int KIND, int MT, bool LLAMA, int GP>
__global__ void __launch_bounds__(THREADS, 1) decode_grid_kernel(const __grid_constant__ DgArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  constexpr bool Q8 = KIND == FC_Q8_0, ONE = MT == 1;
  constexpr bool WIDE = MT == 8;           // (else the low terms of x take columns 4 .. 7)
  constexpr uint32_t BLK = Q8 ? 32 : 16;   // bytes of a block's codes
  constexpr uint32_t UPC = slot_lines(MT) * 128 / (4 * BLK); // units of a full slot
  constexpr uint32_t XBLK = 2 * MT * 64;   // bytes of a block of x: both terms of every row
  constexpr uint32_t PIECE = MT * 16;      // floats of a piece: a warp's sums of a tile
  uint8_t* smem = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u); // (the swizzle is a function of the address)
  Misc& ms = *reinterpret_cast<Misc*>(smem);
  DgLayer* layers = reinterpret_cast<DgLayer*>(smem + a.off_desc);
  float* red = reinterpret_cast<float*>(smem + a.off_red);
  uint8_t* xs = smem + a.off_x;
  float* ysm = reinterpret_cast<float*>(smem + a.off_ys);
  float* kv_tiles = reinterpret_cast<float*>(smem + a.off_kv);
  uint8_t* ring = smem + a.off_ring;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31; // (uniform, and known to be)
  // this CTA's group of rows, and the grid that works on it
  const uint32_t grp = WIDE ? blockIdx.x / a.sub : 0, grid = a.sub, cta = blockIdx.x - grp * grid, r0 = grp * a.group_rows;
  const uint32_t M = ONE ? 1 : min(a.group_rows, a.rows - r0), words = grp * a.group_words;
  Ctl ctl{&ms.dead, a.err_flag};

  if (tid == 0) {
    ms.dead = *(volatile int*)a.err_flag != 0; // an earlier launch gave up: do not wait again
#pragma unroll 1
    for (uint32_t i = 0; i < SLOTS; i++) tc::mbar_init(&ms.full[i], 1), tc::mbar_init(&ms.empty[i], 1), ms.slot_at[i] = 0;
#pragma unroll 1
    for (uint32_t i = 0; i < MAX_KV; i++) tc::mbar_init(&ms.kv_full[i], 1), tc::mbar_init(&ms.kv_empty[i], AWARPS);
    ms.planned = ms.seen = 0;
    tc::fence_barrier_init();
  }
  if (tid < (int)M) {
    ms.ids[tid] = a.chained ? *(volatile int32_t*)(a.out + r0 + tid) : a.tok_in[r0 + tid];
    ms.stream[tid] = a.stream[r0 + tid];
  }
  // (the descriptors are read at every stage: from global memory each would be a trip to L2 in the stage's chain)
#pragma unroll 1
  for (uint32_t i = tid; i < a.n_layers * (uint32_t)(sizeof(DgLayer) / 8); i += THREADS)
    reinterpret_cast<uint64_t*>(layers)[i] = reinterpret_cast<const uint64_t*>(a.layers)[i];
  uint32_t tag0 = *(volatile uint32_t*)(a.state + 2 * grp) + 1; // (words start out as zeros: 0 is no tag)
  // Tile T of a stage belongs to CTA (T + start) mod grid; the starts follow one another so that the small stages land on
  // different CTAs. wo and ff2 share theirs: the CTA of a tile keeps its rows of the residual stream.
  if (tid < 5) {
    auto tiles_of = [](uint32_t n) { return (n + 15) / 16; };
    const uint32_t start = tid == 0 ? tiles_of(a.dim) % grid : tid == 2 ? (tiles_of(a.dim) + tiles_of(a.sh[0].n)) % grid : 0u;
    const uint32_t T = cta >= start ? cta - start : cta + grid - start, n = tiles_of(a.sh[tid].n);
    ms.first[tid] = T;
    ms.tiles[tid] = T < n ? (n - T + grid - 1) / grid : 0u;
  }
  __syncthreads();

  // 512 threads x 128 registers: the consumers take 144, the producer's warpgroup keeps 80
  if (warp >= WARPS) { // ---- the producer warp ----
    asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
    if (warp > WARPS) return;
    if (lane != 0) return; // (one thread issues all copies)
    // The ring: slots of the sizes that their matrices need, one behind the other, freed in the same order.
    uint32_t it = 0, tail = 0, head = 0, kvn = 0;
    bool on = true; // (nothing is requested any more once somebody gave up: a slot may still be in flight)
    auto copy = [&](uint32_t to, const void* from, uint32_t bytes, uint64_t* bar) {
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(to), "l"(from),
                   "r"(bytes), "r"(tc::smem_u32(bar))
                   : "memory");
    };
    uint32_t n_items = 0;
    auto kv_tiles_of = [&](const DgLayer& L) {
#pragma unroll 1
      for (uint32_t i = 0; i < n_items; i++) {
        const Misc::Item& im = ms.items[i];
        const uint32_t len = (uint32_t)ms.pos[im.r] + 1;
        const size_t at = ((size_t)ms.stream[im.r] * a.kv_heads + im.kvh) * a.ctx * 64;
#pragma unroll 1
        for (uint32_t c = im.c0; c < im.c1; c++, kvn++) {
          const uint32_t buf = kvn & ((1u << a.kv_log) - 1), p0 = c * KV_POS, cnt = min(KV_POS, len - 1 - p0); // (the new position is not in the cache yet)
          if (kvn >> a.kv_log) ctl.mbar(&ms.kv_empty[buf], ((kvn >> a.kv_log) - 1) & 1);
          on = *ctl.dead == 0;
          if (!on) return;
          tc::mbar_arrive_expect_tx(&ms.kv_full[buf], cnt * 512);
          const uint32_t to = tc::smem_u32(kv_tiles) + buf * 2 * KV_TILE;
          if (cnt) {
            copy(to, L.kc + at + (size_t)p0 * 64, cnt * 256, &ms.kv_full[buf]);
            copy(to + KV_TILE, L.vc + at + (size_t)p0 * 64, cnt * 256, &ms.kv_full[buf]);
          }
        }
      }
    };
    uint32_t step = 0, si = 0;
#pragma unroll 1
    for (; step < a.steps && on; si = si == 4 * a.n_layers ? 0 : si + 1, step += si == 0) { // qkv, wo, ff1, ff2 of every layer, the head
      const uint32_t mi = si == 4 * a.n_layers ? 4 : si & 3;
      const DgMat& W = mi == 4 ? a.head : layers[si >> 2].m[mi];
      const DgShape& sh = a.sh[mi];
      const uint32_t nch = sh.nch, size = sh.size;
      uint32_t T = ms.first[mi];
#pragma unroll 1
      for (uint32_t left = ms.tiles[mi]; left && on; left--, T += grid)
#pragma unroll 1
        for (uint32_t c = 0; c < nch; c++, it++) {
          uint32_t at;
#pragma unroll 1
          for (;;) {
            const uint32_t oldest = tail < it ? ms.slot_at[tail % SLOTS] : 0;
            bool fits;
            if (tail == it) {
              at = 0, fits = true;
            } else if (head > oldest) { // [oldest, head) is taken
              at = head + size <= a.ring_bytes ? head : 0;
              fits = at == head || size < oldest;
            } else { // it has wrapped: [head, oldest) is free
              at = head, fits = head + size < oldest;
            }
            if (fits && it - tail < SLOTS) break;
            ctl.mbar(&ms.empty[tail % SLOTS], (tail / SLOTS) & 1);
            tail++;
            on = *ctl.dead == 0;
            if (!on) break;
          }
          if (!on) break;
          head = at + size;
          uint64_t* bar = &ms.full[it % SLOTS];
          ms.slot_at[it % SLOTS] = at;
          // (a box counts in full, rows and lines past the matrix's end are zeros; scales in one piece: valid rows only)
          const uint32_t sb = nch == 1 ? min(16u, sh.n - T * 16) * sh.sc_pitch * 2 : sh.sc_bytes;
          tc::mbar_arrive_expect_tx(bar, sh.sc_off + sb);
          const uint32_t to = tc::smem_u32(ring) + at;
          asm volatile(
              "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(to),
              "l"(W.map_w), "r"(tc::smem_u32(bar)), "r"(0), "r"((int32_t)(T * 16)), "r"((int32_t)(c * slot_lines(MT)))
              : "memory");
          if (nch == 1)
            copy(to + sh.sc_off, W.sc + (size_t)T * 16 * sh.sc_pitch, sb, bar);
          else
            asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
                             to + sh.sc_off),
                         "l"(W.map_s), "r"(tc::smem_u32(bar)), "r"((int32_t)(c * sh.sc_pitch)), "r"((int32_t)(T * 16))
                         : "memory");
        }
      if (si == 0 && on) { // (the items of a step, and the caches it reads, are there once its tokens are)
        for (uint32_t tries = 1; *(volatile uint32_t*)&ms.planned <= step && !ctl.give_up(tries, 8); tries++) __nanosleep(20);
        __threadfence_block();
        // (no plan: somebody gave up before there was one, and what lies in its place is anything)
        on = *(volatile uint32_t*)&ms.planned > step && *ctl.dead == 0;
        n_items = on ? *(volatile uint32_t*)&ms.n_items : 0;
        asm volatile("fence.proxy.async;" ::: "memory");
      }
      if (mi == 0 && on) {
        kv_tiles_of(layers[si >> 2]);
        if (on && (si >> 2) + 1 == a.n_layers) { // (behind the last read of the step's items: the consumers write the next step's over them)
          __threadfence_block();
          *(volatile uint32_t*)&ms.seen = step + 1;
        }
      }
    }
    // the CTA may not end under a copy in flight: the last use of every slot has landed
#pragma unroll 1
    for (uint32_t s = 0; s < SLOTS; s++)
      if (it > s)
        for (uint32_t i = 0; i < POLL_LIMIT && !tc::mbar_try_wait(&ms.full[s], ((it - 1 - s) / SLOTS) & 1); i++) {}
#pragma unroll 1
    for (uint32_t b = 0; b < (1u << a.kv_log); b++)
      if (kvn > b)
        for (uint32_t i = 0; i < POLL_LIMIT && !tc::mbar_try_wait(&ms.kv_full[b], ((kvn - 1 - b) >> a.kv_log) & 1); i++) {}
    return;
  }

  // ---- the consumer warps ----
  asm volatile("setmaxnreg.inc.sync.aligned.u32 144;");
  // The epilogue of a group of tiles falls to the last warps (short groups keep the first ones busy with units). One row: a
  // warp per tile, whose halves share the pieces; more: 16 MT threads per tile.
  const uint32_t ewarp = (uint32_t)(WARPS - 1 - warp), etid = ewarp * 32 + lane, e_row = lane & 15;
  const uint32_t e_ti = ONE ? ewarp : etid / PIECE, e_col = ONE ? 0 : (etid >> 4) & (MT - 1);
  const int g = lane >> 2, t = lane & 3;
  // Fragment row g is tile row rho: a row's 16-byte chunks are XORed with its low three bits, and the rows whose lanes read
  // together are to differ where their chunks then do (one row, Q8_0: two rows, every second chunk; Q4_0: two rows, four
  // neighbouring chunks; more rows, Q8_0: four rows, two neighbouring chunks; Q4_0: eight rows, one chunk).
  const uint32_t rho = ONE ? (Q8 ? g : (g >> 1) | ((g & 1) << 2)) : (Q8 ? ((g & 3) << 1) | (g >> 2) : g);
  uint32_t it = 0, kvn = 0, red_par = 0;
#pragma unroll 1
  for (uint32_t step = 0;; step++, tag0 += a.n_layers + 1) {
  // The step's tokens (a chain's: picks of the step before), positions and attention items.
  if (tid < (int)M) {
    if (step) {
      unsigned long long w;
      uint32_t tries = 0;
      do {
        w = ll_ld(a.toks + grp * 8 + tid);
      } while (!ll_ok(w, tag0) && !ctl.give_up(++tries));
      __threadfence();
      ms.ids[tid] = ll_ok(w, tag0) ? (int32_t)(uint32_t)w : 0;
    }
    ms.pos[tid] = a.pos[r0 + tid] + step;
    uint32_t c0, c1;
    item_range((uint32_t)a.pos[r0 + tid] + step + 1, a.splits, 0, c0, c1, ms.used[tid]);
  } else if (tid == 32) {
    const uint32_t head_groups = a.heads / a.item_heads, group = a.heads / a.kv_heads;
    uint32_t n = 0;
#pragma unroll 1
    for (uint32_t item = cta; item < M * head_groups * a.splits; item += grid) {
      const uint32_t s = item % a.splits, hg = item / a.splits % head_groups, r = item / (a.splits * head_groups);
      const uint32_t h0 = hg * a.item_heads, len = (uint32_t)a.pos[r0 + r] + step + 1;
      uint32_t c0, c1, used;
      item_range(len, a.splits, s, c0, c1, used);
      // (one of the items that hold the row's own position appends it)
      if (c0 < c1) ms.items[n++] = Misc::Item{r, h0, h0 / group, s, c0, c1, c1 * KV_POS >= len && h0 % group == 0};
    }
    ms.n_items = n;
  }
  cons_sync();
  if (tid == 0) {
    __threadfence_block();
    *(volatile uint32_t*)&ms.planned = step + 1;
  }
  // the embedding, by the CTAs that keep the residual stream: its words carry the tag before the first layer's
  static_assert(tile_group(MT) * (ONE ? 32 : PIECE) <= CONS, "a thread per result of a group");
#pragma unroll 1
  for (uint32_t li = e_ti; li < MAX_RESID && e_ti < tile_group(MT); li += tile_group(MT)) {
    const uint32_t o = (cta + li * grid) * 16 + e_row;
    if (o < a.dim && e_col < M) {
      float v = a.tok[(size_t)ms.ids[e_col] * a.dim + o];
      if (a.pos_table) v += a.pos_table[(size_t)ms.pos[e_col] * a.dim + o];
      ms.resid[(li * MT + e_col) * 16 + e_row] = v;
      ll_st(a.b_x2 + words + e_col * a.x_stride + ll_at(o), v, tag0);
    }
  }

  unsigned long long best = 0; // head: the best (logit, index) of this thread's row
  uint32_t mi = 0, l = 0;      // matrix 0 .. 3 of layer l; 4: the head
#pragma unroll 1
  for (;;) {
    const uint32_t tag = tag0 + l + 1; // of this layer's words; the stream that enters it carries tag - 1
    uint32_t left = ms.tiles[mi];
    if (left) { // ---- a product ----
      const DgMat& W = mi == 4 ? a.head : layers[l].m[mi];
      const DgShape& sh = a.sh[mi];
      const uint32_t k = sh.k, tpr = sh.tpr, nu = sh.nu;
      const float* ng = W.gain;
      float(*redss)[TASKS] = ms.redss[mi == 2];
      uint32_t T = ms.first[mi], li0 = 0; // (tiles before the group)
      bool staged = false;
#pragma unroll 1
      do { // the tiles, in groups
        // `per` warps to a tile: warp i * per + j takes the units (128 k) j, j + per, .. of tile i
        const uint32_t ntg = min(sh.group, left), per = ntg == 1 ? 12u : ntg == 2 ? 6u : ntg == 3 ? 4u : 3u;
        const uint32_t u_ti = ntg == 1 ? 0u : ntg == 2 ? (uint32_t)(warp >= 6) : ntg == 3 ? warp >> 2 : (warp * 11) >> 5;
        uint32_t kg = u_ti < ntg ? warp - u_ti * per : nu;
        const bool works = kg < nu;
        const uint32_t o = (T + e_ti * grid) * 16 + e_row;
        const bool mine = e_ti < ntg && o < sh.n && e_col < M && (!ONE || lane < 16);
        const float bias = mine && W.bias ? W.bias[o] : 0.0f;
        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 1
        do {
          // a unit's codes and scales, raw: on their way before x arrives
          constexpr int NW = Q8 ? 16 : 8;
          uint32_t wraw[NW], sraw[4]; // one row: rows g, g + 8 of the lane's block; more: of its quarter of four blocks
          if (works) {
            const uint32_t c = kg / UPC, si = it + u_ti * sh.nch + c, b0 = (kg - c * UPC) * 4; // (first block, within the slot)
            ctl.mbar(&ms.full[si % SLOTS], (si / SLOTS) & 1);
            // (once somebody gave up, the place may be that of an earlier, smaller slot, or the first zero: inside the ring either way)
            const uint8_t* slot = ring + min(ms.slot_at[si % SLOTS], a.ring_bytes - sh.size);
            const uint32_t sc_pitch = sh.sc_pitch;
            const __half* sp = reinterpret_cast<const __half*>(slot + sh.sc_off) + rho * sc_pitch + b0;
            const uint8_t* wp = slot + (b0 / (128 / BLK)) * 2048 + rho * 128; // the unit's line (Q4_0: half a line) of row rho
            const uint32_t h4 = Q8 ? 0 : b0 & 4;
            if (ONE) {
#pragma unroll
              for (int h = 0; h < (Q8 ? 2 : 1); h++) {
                const uint8_t* p = wp + ((Q8 ? 2 * t + h : h4 + t) ^ (rho & 7)) * 16;
                const uint4 va = *reinterpret_cast<const uint4*>(p), vb = *reinterpret_cast<const uint4*>(p + 1024);
                wraw[h * 8] = va.x, wraw[h * 8 + 1] = va.y, wraw[h * 8 + 2] = va.z, wraw[h * 8 + 3] = va.w;
                wraw[h * 8 + 4] = vb.x, wraw[h * 8 + 5] = vb.y, wraw[h * 8 + 6] = vb.z, wraw[h * 8 + 7] = vb.w;
              }
              sraw[0] = __half_as_ushort(sp[t]), sraw[1] = __half_as_ushort(sp[8 * sc_pitch + t]);
            } else {
#pragma unroll
              for (int bb = 0; bb < 4; bb++) {
                if (Q8) {
                  const uint8_t* p = wp + ((2 * bb + (t >> 1)) ^ (rho & 7)) * 16 + (t & 1) * 8;
                  const uint2 va = *reinterpret_cast<const uint2*>(p), vb = *reinterpret_cast<const uint2*>(p + 1024);
                  wraw[(bb * 4) % NW] = va.x, wraw[(bb * 4 + 1) % NW] = va.y, wraw[(bb * 4 + 2) % NW] = vb.x, wraw[(bb * 4 + 3) % NW] = vb.y;
                } else {
                  const uint8_t* p = wp + ((h4 + bb) ^ (rho & 7)) * 16 + t * 4;
                  wraw[bb * 2] = *reinterpret_cast<const uint32_t*>(p);
                  wraw[bb * 2 + 1] = *reinterpret_cast<const uint32_t*>(p + 1024);
                }
              }
              const uint2 sa = *reinterpret_cast<const uint2*>(sp), sb = *reinterpret_cast<const uint2*>(sp + 8 * sc_pitch);
              sraw[0] = sa.x, sraw[1] = sa.y, sraw[2] = sb.x, sraw[3] = sb.y;
            }
          }

          if (!staged) { // -- x: a task is 256 elements of a row, eight per lane --
            staged = true;
            const uint32_t n_tasks = M * tpr, want = mi == 0 || mi == 4 ? tag - 1 : tag;
            auto row_of = [&](uint32_t task) { return ONE ? 0u : (task * sh.tpr_inv) >> 16; };
            const unsigned long long* src = sh.src + words + lane * 2;
            unsigned long long q[8];
            auto request = [&](uint32_t task) {
              const unsigned long long* p = src + task * 256; // (a row is whole tasks)
#pragma unroll
              for (int i = 0; i < 4; i++) ll_ld2(p + 64 * i, q[2 * i], q[2 * i + 1]);
            };
            auto arrive = [&](uint32_t task, float (&x)[8]) { // (the words past the end of a row: never written, not waited for)
              const bool in = (task - row_of(task) * tpr) * 256 + lane * 8 < k;
              uint32_t tries = 0;
              for (;;) {
                uint32_t bad = 0;
#pragma unroll
                for (int i = 0; i < 8; i++) bad |= (uint32_t)(q[i] >> 32) ^ want;
                if (__all_sync(0xffffffffu, bad == 0 || !in)) break;
                if (__any_sync(0xffffffffu, ctl.give_up(++tries))) break;
                request(task);
              }
#pragma unroll
              for (int i = 0; i < 8; i++) x[i] = in ? ll_val(q[i]) : 0.0f;
            };
            auto load8 = [&](const float* p, uint32_t task, float (&v)[8]) {
              const uint32_t e = (task - row_of(task) * tpr) * 256 + lane * 8;
              float4 u = make_float4(0, 0, 0, 0), w = u;
              if (e < k) u = *reinterpret_cast<const float4*>(p + e), w = *reinterpret_cast<const float4*>(p + e + 4);
              v[0] = u.x, v[1] = u.y, v[2] = u.z, v[3] = u.w, v[4] = w.x, v[5] = w.y, v[6] = w.z, v[7] = w.w;
            };
            // Two fp16 terms of every element, at the power of two that brings its 32-block's largest into [2^14, 2^15). One row keeps
            // the low terms 2^11 larger: 22 bits of every element down to 2^-28 of the largest. A block with a smaller one that is
            // not zero, with one that is not finite, or of magnitudes whose scale would leave the normal floats goes as it is (its
            // scale says so) and is multiplied in f32. (Terms alone put the logits of a model with a constant 2^30 beside its
            // activations off by 1e-3. The check and the factor cost 0.2 to 1.1 % of a step: 60.3 -> 60.8 us, 384 wide; asking for
            // the smallest element first and looking closer behind a vote cost 2.4 %.)
            auto stage = [&](uint32_t task, const float (&x)[8]) {
              const uint32_t r = row_of(task), b = (task - r * tpr) * 8 + g; // (lane = block, quarter)
              uint32_t mx = 0, mn = 0xffffffffu; // (of the bits; a zero is not the smallest)
#pragma unroll
              for (int i = 0; i < 8; i++) {
                const uint32_t u = __float_as_uint(x[i]) & 0x7fffffffu;
                mx = max(mx, u);
                if (ONE) mn = min(mn, u - 1);
              }
              mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
              mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
              const uint32_t ex = min(max(mx & 0x7f800000u, 15u << 23), 254u << 23);
              const float up = __uint_as_float((268u << 23) - ex);
              bool held = true;
              if (ONE) {
                const bool bad = (mx != 0 && mx - (63u << 23) >= (161u << 23)) || mn < ex - (28u << 23) - 1;
                held = (__ballot_sync(0xffffffffu, bad) >> (lane & 28) & 15u) == 0;
              }
              uint32_t hi[4], lo[4];
#pragma unroll
              for (int i = 0; i < 4; i++) {
                const float v0 = x[2 * i] * up, v1 = x[2 * i + 1] * up;
                const __half2 h = __floats2half2_rn(v0, v1);
                const float2 f = __half22float2(h);
                const __half2 d = ONE ? __floats2half2_rn((v0 - f.x) * 2048.0f, (v1 - f.y) * 2048.0f) : __floats2half2_rn(v0 - f.x, v1 - f.y);
                hi[i] = *reinterpret_cast<const uint32_t*>(&h), lo[i] = *reinterpret_cast<const uint32_t*>(&d);
              }
              if (b * 32 < k) {
                // one row: [four blocks][quarter][term][block]; more: [block][term][row][quarter], 16 bytes each
                uint8_t* at = ONE ? xs + (b >> 2) * (4 * XBLK) + t * 128 + (b & 3) * 16 : xs + b * XBLK + r * 64 + t * 16;
                *reinterpret_cast<uint4*>(at) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<uint4*>(at + (ONE ? 64 : MT * 64)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
                if (t == 0) ysm[b * MT + r] = __uint_as_float(ex - (14u << 23));
                if (ONE && !held) {
                  *reinterpret_cast<float4*>(at) = make_float4(x[0], x[1], x[2], x[3]);
                  *reinterpret_cast<float4*>(at + 64) = make_float4(x[4], x[5], x[6], x[7]);
                  if (t == 0) ysm[b] = __uint_as_float(0x7fffffffu);
                }
              }
            };
            auto warp_sum = [&](float v) {
#pragma unroll
              for (int s = 16; s > 0; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
              return v;
            };
            if (LLAMA || !ng) {
              uint32_t task = warp;
              if (task < n_tasks) request(task);
#pragma unroll 1
              while (task < n_tasks) {
                float x[8], ss = 0.0f;
                float gain[8];
                if (LLAMA && ng) load8(ng, task, gain);
                arrive(task, x);
                const uint32_t done = task;
                task += WARPS;
                if (!ONE && task < n_tasks) request(task); // (the next task's words travel while this one is converted)
                if (LLAMA && ng) { // the gain here; 1 / rms multiplies the sums at the end
#pragma unroll
                  for (int i = 0; i < 8; i++) ss = fmaf(x[i], x[i], ss), x[i] *= gain[i];
                }
                stage(done, x);
                if (LLAMA && ng) {
                  ss = warp_sum(ss);
                  const uint32_t r = row_of(done);
                  if (lane == 0) redss[r][done - r * tpr] = ss;
                }
                if (ONE) break; // (at most 12 tasks)
              }
            } else { // LayerNorm: at most two tasks per warp (decode_grid_ready); two passes, ferrum_ref/src/kernels/nn.rs:L31-L43
              constexpr int NT = ONE ? 1 : 2;
              float x[NT][8], mean[NT];
#pragma unroll
              for (int i = 0; i < NT; i++) {
                const uint32_t task = warp + i * WARPS;
                mean[i] = 0.0f;
                if (task < n_tasks) request(task), arrive(task, x[i]);
              }
#pragma unroll
              for (int pass = 0; pass < 2; pass++) {
                float(*part)[TASKS] = pass ? ms.ln2 : ms.ln1;
#pragma unroll
                for (int i = 0; i < NT; i++) {
                  const uint32_t task = warp + i * WARPS, r = row_of(task);
                  if (task < n_tasks) {
                    float s = 0.0f;
                    if ((task - r * tpr) * 256 + lane * 8 < k) {
#pragma unroll
                      for (int j = 0; j < 8; j++) s = pass ? fmaf(x[i][j] - mean[i], x[i][j] - mean[i], s) : s + x[i][j];
                    }
                    s = warp_sum(s);
                    if (lane == 0) part[r][task - r * tpr] = s;
                  }
                }
                cons_sync();
#pragma unroll
                for (int i = 0; i < NT; i++) {
                  const uint32_t task = warp + i * WARPS;
                  if (task < n_tasks) {
                    float s = 0.0f;
#pragma unroll 1
                    for (uint32_t j = 0; j < tpr; j++) s += part[row_of(task)][j];
                    if (pass == 0) {
                      mean[i] = s * sh.k_inv;
                    } else {
                      const float inv = dg_rsqrt(s * sh.k_inv + 1e-5f);
                      float gain[8], beta[8];
                      load8(ng, task, gain);
                      load8(W.beta, task, beta);
#pragma unroll
                      for (int j = 0; j < 8; j++) x[i][j] = (x[i][j] - mean[i]) * inv * gain[j] + beta[j];
                      stage(task, x[i]);
                    }
                  }
                }
              }
            }
            cons_sync();
          }

          if (works) {
            if (ONE) {
              uint4 xb[4];
#pragma unroll
              for (int j = 0; j < 4; j++) {
                xb[j] = make_uint4(0, 0, 0, 0);
                if (t == (g >> 1)) xb[j] = *reinterpret_cast<const uint4*>(xs + kg * (4 * XBLK) + j * 128 + (g & 1) * 64 + t * 16);
              }
              const float ys = ysm[kg * 4 + t];
              const bool plain = __any_sync(0xffffffffu, ys != ys); // a block of the unit is multiplied in f32
              float cc[2][4];
#pragma unroll
              for (int j = 0; j < 2; j++) cc[j][0] = cc[j][1] = cc[j][2] = cc[j][3] = 0.0f;
#pragma unroll
              for (int j = 0; j < 4; j++) { // quarter j: eight elements of every lane's block
                uint32_t pa[4], pb[4];
                if (Q8) {
                  const int at = (j >> 1) * 8 + (j & 1) * 2;
                  codes8<Q8>(wraw[at % NW], wraw[(at + 1) % NW], pa);
                  codes8<Q8>(wraw[(at + 4) % NW], wraw[(at + 5) % NW], pb);
                } else {
                  codes8<Q8>(wraw[j], 0, pa);
                  codes8<Q8>(wraw[4 + j], 0, pb);
                }
                dg_mma(cc[0], pa[0], pb[0], pa[1], pb[1], xb[j].x, xb[j].y);
                dg_mma(cc[1], pa[2], pb[2], pa[3], pb[3], xb[j].z, xb[j].w);
              }
              float d = __half2float(__ushort_as_half((unsigned short)sraw[0])), d8 = __half2float(__ushort_as_half((unsigned short)sraw[1]));
              float s = fmaf(cc[0][1] + cc[1][1], 0x1p-11f, cc[0][0] + cc[1][0]), s8 = fmaf(cc[0][3] + cc[1][3], 0x1p-11f, cc[0][2] + cc[1][2]);
              if (!plain) {
                d *= ys, d8 *= ys;
              } else if (ys == ys) {
                d *= ys, d8 *= ys;
              } else { // this lane's block lies there as it is (of the sums above only the block's own columns saw it)
                const uint32_t c = kg / UPC, si = it + u_ti * sh.nch + c, b0 = (kg - c * UPC) * 4;
                const uint8_t* wp = ring + min(ms.slot_at[si % SLOTS], a.ring_bytes - sh.size) + (b0 / (128 / BLK)) * 2048 + rho * 128;
                const uint8_t* xp = xs + kg * (4 * XBLK) + t * 16;
                constexpr int PER = Q8 ? 4 : 8; // codes of a word
                s = s8 = 0.0f;
#pragma unroll 1
                for (uint32_t e = 0; e < 32; e += PER) {
                  const uint32_t chunk = Q8 ? 2 * t + (e >> 4) : (b0 & 4) + t, word = Q8 ? (e >> 2) & 3 : e >> 3;
                  const uint32_t* p = reinterpret_cast<const uint32_t*>(wp + (chunk ^ (rho & 7)) * 16) + word;
                  const uint32_t w = p[0], w8 = p[256];
#pragma unroll
                  for (uint32_t j = 0; j < PER; j++) {
                    const float xe = *reinterpret_cast<const float*>(xp + (e >> 3) * 128 + ((e + j) & 4) * 16 + (j & 3) * 4);
                    // (Q4_0: element j of a word's eight at nibble (j >> 1) + 4 (j & 1))
                    const uint32_t sft = Q8 ? 8 * j : 4 * (j >> 1) + 16 * (j & 1);
                    s = fmaf(xe, Q8 ? (float)(int8_t)(w >> sft) : (float)(int)(w >> sft & 15) - 8.0f, s);
                    s8 = fmaf(xe, Q8 ? (float)(int8_t)(w8 >> sft) : (float)(int)(w8 >> sft & 15) - 8.0f, s8);
                  }
                }
              }
              acc[0] = fmaf(s, d, acc[0]);
              acc[2] = fmaf(s8, d8, acc[2]);
            } else {
              const uint8_t* xp = xs + kg * (4 * XBLK) + (WIDE ? g : (g >> 2) * MT + (g & (MT - 1))) * 64 + t * 16;
              const float* yp = ysm + kg * 4 * MT + ((2 * t) & (MT - 1));
#pragma unroll
              for (int bb = 0; bb < 4; bb++) {
                const __half2 sa = *reinterpret_cast<const __half2*>(&sraw[bb >> 1]), sb = *reinterpret_cast<const __half2*>(&sraw[2 + (bb >> 1)]);
                const float dg = (bb & 1) ? __high2float(sa) : __low2float(sa), dg8 = (bb & 1) ? __high2float(sb) : __low2float(sb);
                uint32_t pa[4], pb[4];
                if (Q8) {
                  codes8<Q8>(wraw[(bb * 4) % NW], wraw[(bb * 4 + 1) % NW], pa);
                  codes8<Q8>(wraw[(bb * 4 + 2) % NW], wraw[(bb * 4 + 3) % NW], pb);
                } else {
                  codes8<Q8>(wraw[(bb * 2) % NW], 0, pa);
                  codes8<Q8>(wraw[(bb * 2 + 1) % NW], 0, pb);
                }
                // (two rows: columns 2, 3, 6, 7 repeat them and are not read)
                const uint4 x0 = *reinterpret_cast<const uint4*>(xp + bb * XBLK);
                const float2 ys = *reinterpret_cast<const float2*>(yp + bb * MT);
                float c4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                if (WIDE) { // the small terms first
                  const uint4 x1 = *reinterpret_cast<const uint4*>(xp + bb * XBLK + MT * 64);
                  dg_mma(c4, pa[0], pb[0], pa[1], pb[1], x1.x, x1.y);
                  dg_mma(c4, pa[2], pb[2], pa[3], pb[3], x1.z, x1.w);
                }
                dg_mma(c4, pa[0], pb[0], pa[1], pb[1], x0.x, x0.y);
                dg_mma(c4, pa[2], pb[2], pa[3], pb[3], x0.z, x0.w);
                acc[0] = fmaf(c4[0], dg * ys.x, acc[0]);
                acc[1] = fmaf(c4[1], dg * ys.y, acc[1]);
                acc[2] = fmaf(c4[2], dg8 * ys.x, acc[2]);
                acc[3] = fmaf(c4[3], dg8 * ys.y, acc[3]);
              }
            }
          }
          kg += per;
        } while (kg < nu);
        float* redp = red + red_par * WARPS * PIECE;
        if (works) {
          float* rw = redp + warp * PIECE;
          if (ONE) {
#pragma unroll
            for (int s = 1; s < 4; s <<= 1)
              acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], s), acc[2] += __shfl_xor_sync(0xffffffffu, acc[2], s);
            if (t == 0) rw[rho] = acc[0], rw[rho + 8] = acc[2];
          } else {
            if (!WIDE) { // columns 4 .. 7 are the low terms of columns 0 .. 3
#pragma unroll
              for (int s = 0; s < 4; s++) acc[s] += __shfl_xor_sync(0xffffffffu, acc[s], 2);
            }
            if (2 * t < MT) rw[2 * t * 16 + rho] = acc[0], rw[2 * t * 16 + rho + 8] = acc[2];
            if (2 * t + 1 < MT) rw[(2 * t + 1) * 16 + rho] = acc[1], rw[(2 * t + 1) * 16 + rho + 8] = acc[3];
          }
        }
        const bool busy = (ONE ? ewarp : (etid & ~31u) / PIECE) < ntg; // (uniform in the warp)
        float inv = 1.0f;
        if (LLAMA && busy && ng) {
          float s = e_row < tpr ? redss[e_col][e_row] : 0.0f;
#pragma unroll
          for (int i = 8; i > 0; i >>= 1) s += __shfl_xor_sync(0xffffffffu, s, i);
          inv = dg_rsqrt(s * sh.k_inv + a.eps);
        }
        cons_sync();
        if (warp == 0 && lane < (int)(ntg * sh.nch)) tc::mbar_arrive(&ms.empty[(it + lane) % SLOTS]);
        if (busy) {
          const uint32_t np = min(per, nu);
          float v = 0.0f;
          if (ONE) {
            const float* rp = redp + (e_ti * per + (lane >> 4)) * PIECE + e_row;
#pragma unroll
            for (uint32_t w = 0; w < 12; w += 2)
              if (w + (lane >> 4) < np) v += rp[w * PIECE];
            v += __shfl_xor_sync(0xffffffffu, v, 16);
          } else {
            const float* rp = redp + e_ti * per * PIECE + e_col * 16 + e_row;
            float w4[2] = {0.0f, 0.0f};
#pragma unroll
            for (uint32_t w = 0; w < 12; w++)
              if (w < np) w4[w & 1] += rp[w * PIECE];
            v = w4[0] + w4[1];
          }
          v = v * inv + bias;
          uint32_t at = o;
          if (mi == 2) {
            if (LLAMA) { // gate and up rows alternate
              const float up = __shfl_down_sync(0xffffffffu, v, 1);
              v = v / (1.0f + expf(-v)) * up;
              at = o >> 1;
            } else {
              v = dg_gelu(v);
            }
          }
          if (mine) {
            if (mi == 4) {
              a.logits[(size_t)(r0 + e_col) * sh.n + o] = v;
              // first maximum; NaN and -inf never win; -0 equals 0
              if (v > -INFINITY) {
                const uint32_t b = __float_as_uint(v + 0.0f), ord = (b & 0x80000000u) ? ~b : b | 0x80000000u;
                const unsigned long long key = ((unsigned long long)ord << 32) | (0xffffffffu - o);
                best = key > best ? key : best;
              }
            } else if (!(LLAMA && mi == 2 && (e_row & 1))) {
              if (mi & 1) { // wo, ff2: the residual stream
                float* rs = &ms.resid[((li0 + e_ti) * MT + e_col) * 16 + e_row];
                v = *rs + v;
                *rs = v;
              }
              if (mi) at = ll_at(at);
              ll_st(sh.dst + words + e_col * sh.dst_stride + at, v, tag);
            }
          }
        }
        it += ntg * sh.nch, li0 += ntg, left -= ntg, T += ntg * grid, red_par ^= 1;
      } while (left);
    }
    if (mi == 4) break;
    if (mi == 0) { // ---- attention ----
#pragma unroll 1
      for (uint32_t i = 0; i < ms.n_items; i++) attn_item<GP>(a, layers[l], ms, red, kv_tiles, kvn, ctl, tag, words, ms.items[i]);
      if (a.splits > 1) {
        // rows in several parts: a warp merges eight channels of a (row, head), eight splits at a time with four lanes each
#pragma unroll 1
        for (uint32_t p = (grid - 1 - cta) + grid * warp; p < M * a.heads * 8; p += grid * WARPS) {
          const uint32_t rh = p >> 3, r = (rh * a.heads_inv) >> 16, used = ms.used[r];
          if (used == 1) continue;
          const unsigned long long* src = a.b_part + words + rh * a.splits * PART;
          const unsigned long long *col = src + (p & 7) * 8 * a.splits + 2 * t, *mls = src + a.splits * 64 + 2 * min((uint32_t)lane, used - 1);
          const uint32_t s0 = 8 * min((uint32_t)g, used - 1), s1 = 8 * min(g + 8u, used - 1);
          unsigned long long w[6];
          uint32_t tries = 0, bad;
          do {
            ll_ld2(mls, w[0], w[1]);
            ll_ld2(col + s0, w[2], w[3]);
            ll_ld2(col + s1, w[4], w[5]);
            bad = 0;
#pragma unroll
            for (int i = 0; i < 6; i++) bad |= (uint32_t)(w[i] >> 32) ^ tag;
          } while (!__all_sync(0xffffffffu, bad == 0) && !__any_sync(0xffffffffu, ctl.give_up(++tries)));
          const bool in = lane < (int)used;
          float mx = in ? ll_val(w[0]) : -INFINITY;
#pragma unroll
          for (int i = 8; i > 0; i >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, i)); // (of lanes 0 .. 15)
          const float f = in ? dg_ex2(ll_val(w[0]) - mx) : 0.0f;
          float den = in ? f * ll_val(w[1]) : 0.0f;
#pragma unroll
          for (int i = 8; i > 0; i >>= 1) den += __shfl_xor_sync(0xffffffffu, den, i);
          den = __shfl_sync(0xffffffffu, den, 0);
          const float f0 = __shfl_sync(0xffffffffu, f, g), f1 = __shfl_sync(0xffffffffu, f, g + 8); // (0 past the last split)
          float o0 = fmaf(f0, ll_val(w[2]), f1 * ll_val(w[4])), o1 = fmaf(f0, ll_val(w[3]), f1 * ll_val(w[5]));
#pragma unroll
          for (int i = 4; i < 32; i <<= 1) o0 += __shfl_xor_sync(0xffffffffu, o0, i), o1 += __shfl_xor_sync(0xffffffffu, o1, i);
          if (g == 0) {
            unsigned long long* dst = a.b_attn + words + r * a.attn_stride + ll_at((rh - r * a.heads) * 64 + (p & 7) * 8 + 2 * t);
            ll_st(dst, o0 / den, tag);
            ll_st(dst + 1, o1 / den, tag);
          }
        }
      }
    }
    if (++mi == 4) mi = ++l == a.n_layers ? 4 : 0;
  }

  // the picks: every warp's best of a row, then the last CTA to arrive writes the step's results
#pragma unroll
  for (int o = 1; o < (ONE ? 32 : 16); o <<= 1) {
    const unsigned long long ov = __shfl_xor_sync(0xffffffffu, best, o);
    best = ov > best ? ov : best;
  }
  if ((lane & (ONE ? 31 : 15)) == 0 && best && e_col < M) atomicMax(&a.keys[r0 + e_col], best);
  asm volatile("fence.proxy.async;" ::: "memory"); // (the cache appends, which bulk copies will read)
  cons_sync();
  const bool last = step + 1 == a.steps;
  if (tid == 0) {
    __threadfence(); // (behind the barrier: it orders what every thread of the CTA wrote before the count)
    const uint32_t n = atomicAdd(&a.state[2 * grp + 1], 1u);
    if (n + 1 == grid) {
      __threadfence();
#pragma unroll 1
      for (uint32_t r = 0; r < M; r++) {
        const unsigned long long key = atomicExch(&a.keys[r0 + r], 0ull);
        const uint32_t pick = key ? 0xffffffffu - (uint32_t)key : 0u;
        if (a.log) a.log[(size_t)step * a.rows + r0 + r] = ms.ids[r];
        if (last)
          a.out[r0 + r] = (int32_t)pick;
        else
          ms.next[r] = (int32_t)pick;
      }
      a.state[2 * grp + 1] = 0;
      if (last) {
        a.state[2 * grp] = tag0 + a.n_layers;
        a.out[64 + grp] = *(volatile int*)a.err_flag;
      }
      __threadfence();
      if (!last)
#pragma unroll 1
        for (uint32_t r = 0; r < M; r++) ll_st(a.toks + grp * 8 + r, __int_as_float(ms.next[r]), tag0 + a.n_layers + 1);
    }
    for (uint32_t tries = 1; *(volatile uint32_t*)&ms.seen <= step && !ctl.give_up(tries, 8); tries++) __nanosleep(20); // (at once)
    ms.stop = last || *ctl.dead;
    if (!last && ms.stop) a.out[64 + grp] = 1; // (this CTA does not go on, the others' waits will run out)
  }
  cons_sync();
  if (ms.stop) return;
  }
}

enum { DG_UNTRIED, DG_READY, DG_NO_ROOM, DG_UNFIT };
struct DgState {
  int set_up = DG_UNTRIED;
  uint32_t asked = 0, retry = 64; // without room: questions since the last try, and after how many the next one is
  DgArgs args[4];              // for 1, 2, 4 and 8 padded rows
  void* d_layers = nullptr;    // the tensor maps and the layers' descriptors, for slots of 8 and of 4 lines
  void* words = nullptr;
  uint64_t tags = 0;           // used since the words were cleared
  double units = 0.0;          // of 16 rows x 128 k, in all matrices
  int kind = 0;
};

// A matrix's slots: 16 rows of up to `slot_lines` lines, then their scales.
void slot_shape(DgShape& d, bool q8, int mt) {
  const uint32_t lines = (q8 ? d.k : d.k / 2) / 128, box = std::min(lines, slot_lines(mt));
  d.nch = (lines + box - 1) / box;
  d.sc_off = box * 2048;
  d.sc_pitch = d.nch == 1 ? d.k / 32 : box * (q8 ? 4 : 8);
  d.sc_bytes = 16 * d.sc_pitch * 2;
  d.size = al(d.sc_off + d.sc_bytes, 1024); // (the swizzle is a function of the address)
}

// Shared memory for `mt` padded rows; false where the ring cannot hold a tile of the longest K and one slot more.
bool layout(DgArgs& a, int kind, int mt, uint32_t max_k) {
  const uint32_t gp = a.heads == a.kv_heads ? 1 : ITEM_HEADS;
  DgShape d{};
  d.k = max_k;
  slot_shape(d, kind == FC_Q8_0, mt);
  a.off_desc = al((uint32_t)sizeof(Misc), 128);
  a.off_red = al(a.off_desc + a.n_layers * (uint32_t)sizeof(DgLayer), 128);
  // sums of the warps (two groups of tiles), x and its scales; the attention's per-warp parts lie over all of them
  a.off_x = a.off_red + 2 * WARPS * mt * 16 * 4;
  a.off_ys = a.off_x + max_k * 4 * mt;
  a.off_kv = al(std::max(a.off_ys + max_k / 32 * mt * 4, a.off_red + AWARPS * gp * 64 * 4), 128);
  for (a.kv_log = mt <= 2 ? 2 : 1;; a.kv_log--) {
    a.off_ring = al(a.off_kv + (2 * KV_TILE << a.kv_log), 1024);
    a.ring_bytes = a.off_ring + 1024 < SMEM_MAX ? (SMEM_MAX - 1024 - a.off_ring) / 1024 * 1024 : 0;
    if (a.ring_bytes >= std::max(2 * d.nch + 1, 4u) * d.size) return true;
    if (a.kv_log == 0) return a.ring_bytes >= (d.nch + 1) * d.size;
  }
}

template <int KIND, int MT, bool LLAMA, int GP>
int launch(FcDevice* dev, DgArgs& a) {
  auto kern = decode_grid_kernel<KIND, MT, LLAMA, GP>;
  static OncePerDevice attr;
  if (attr.first(dev->ordinal)) FC_CUDA(dev, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_MAX));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(a.sub * ((a.rows + a.group_rows - 1) / a.group_rows)), cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = a.off_ring + a.ring_bytes + 1024, cfg.stream = dev->stream;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeCooperative; // (CTAs wait for one another: all must be resident)
  at.val.cooperative = 1;
  cfg.attrs = &at, cfg.numAttrs = 1;
  FC_LAUNCH(dev, "decode_grid", cudaLaunchKernelEx(&cfg, kern, a));
  return FC_OK;
}

template <int KIND, int MT>
int launch_arch(FcDevice* dev, DgArgs& a, bool llama) {
  if (!llama) return launch<KIND, MT, false, 1>(dev, a);
  return a.item_heads == 1 ? launch<KIND, MT, true, 1>(dev, a) : launch<KIND, MT, true, ITEM_HEADS>(dev, a);
}
template <int KIND>
int launch_rows(FcDevice* dev, DgArgs& a, bool llama) {
  return a.rows == 1   ? launch_arch<KIND, 1>(dev, a, llama)
         : a.rows == 2 ? launch_arch<KIND, 2>(dev, a, llama)
         : a.rows <= 4 ? launch_arch<KIND, 4>(dev, a, llama)
                       : launch_arch<KIND, 8>(dev, a, llama);
}

} // namespace

void decode_grid_free(FcModel* m) {
  DgState* st = (DgState*)m->dg;
  if (!st) return;
  if (st->d_layers) cudaFree(st->d_layers);
  if (st->words) cudaFree(st->words);
  delete st;
  m->dg = nullptr;
}

// CTAs of a group of a step of `rows` rows.
static uint32_t group_ctas(const FcModel* m, uint32_t rows) {
  return (uint32_t)m->dev->prop.multiProcessorCount / ((rows + 7) / 8);
}

// The set-up. On failure the caller frees what it had taken.
static int decode_grid_set_up(FcModel* m, DgState* st) {
  const int kind = m->head.w->m.kind;
  const bool q8 = kind == FC_Q8_0;
  if (!q8 && kind != FC_Q4_0) return DG_UNFIT;
  auto mat_ok = [&](const Linear& l) {
    const QMat& q = l.w->m;
    if (q.kind != kind || q.k % (q8 ? 128 : 256) || q.k > MAX_K) return false; // (whole lines)
    // (copies are whole 16 bytes: a row's scales as a tensor map has them, or those of a 16-row tile where a slot holds the row)
    if (q.k % 256 && (q.k > slot_lines(8) * 128 || q.n % 16)) return false;
    return (((uintptr_t)q.qs | (uintptr_t)q.sc) & 15) == 0;
  };
  if (m->hd != 64 || m->heads % m->kv_heads || m->rope.rope_dim > 64) return DG_UNFIT;
  if (m->dim > MAX_K || m->hidden > MAX_K || m->qd() > MAX_K) return DG_UNFIT;
  if (m->arch == ARCH_LLAMA && m->gu_group != 1) return DG_UNFIT;
  if (!mat_ok(m->head)) return DG_UNFIT;
  for (auto& l : m->layers)
    if (!mat_ok(l.qkv) || !mat_ok(l.wo) || !mat_ok(l.ff1) || !mat_ok(l.ff2)) return DG_UNFIT;
  int coop = 0;
  if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, m->dev->ordinal) != cudaSuccess || !coop) return DG_UNFIT;
  EncodeTiledFn enc = encode_fn();
  if (!enc) return DG_UNFIT;
  const uint32_t grid = (uint32_t)m->dev->prop.multiProcessorCount, max_k = std::max(m->dim, std::max(m->hidden, m->qd()));
  DgArgs a = DgArgs();
  a.n_layers = m->n_layers, a.dim = m->dim, a.heads = m->heads, a.kv_heads = m->kv_heads, a.ctx = m->ctx;
  a.heads_inv = 65536 / m->heads + 1;
  a.x_stride = al(m->dim, 256), a.attn_stride = al(m->qd(), 256), a.act_stride = al(m->hidden, 256);
  a.tok = m->tok, a.pos_table = m->pos_table;
  a.cos = m->rope.cos, a.sin = m->rope.sin, a.rope_dim = m->rope.rope_dim, a.rope_type = m->rope.type;
  a.eps = m->eps, a.logits = m->logits, a.err_flag = m->dev->d_flag;
  for (int v = 0; v < 4; v++)
    if (!layout(a, kind, 1 << v, max_k)) return DG_UNFIT;
  // The tagged words, outside the model's plan: a model that fits without them decodes as launches.
  const uint32_t groups = (std::min<uint32_t>(8 * MAX_GROUPS, m->max_streams) + 7) / 8, rows_max = std::min<uint32_t>(8, m->max_streams);
  const size_t w_part = (size_t)grid * ITEM_HEADS * PART;
  const size_t g_words = rows_max * (m->qkv_w() + a.attn_stride + 2 * (size_t)a.x_stride + a.act_stride) + w_part;
  const size_t n_words = groups * g_words + 64 + 64 + 8 + 40; // next tokens, keys, state, out
  // descriptors: per variant of the slots two tensor maps per matrix, then the layers
  const size_t n_mats = 4 * (size_t)m->n_layers + 1, maps_bytes = n_mats * 2 * sizeof(CUtensorMap);
  const size_t var_bytes = (maps_bytes + m->n_layers * sizeof(DgLayer) + 255) & ~(size_t)255;
  if (device_malloc(m->dev, &st->d_layers, 2 * var_bytes) != cudaSuccess || device_malloc(m->dev, &st->words, n_words * 8) != cudaSuccess) {
    cudaGetLastError();
    return DG_NO_ROOM;
  }
  std::vector<uint8_t> host(2 * var_bytes);
  DgMat heads[2];
  for (int var = 0; var < 2; var++) {
    uint8_t* at = host.data() + var * var_bytes;
    const uint8_t* dev_at = (const uint8_t*)st->d_layers + var * var_bytes;
    size_t next = 0;
    bool ok = true;
    auto mat = [&](const Linear& l, const float* gain, const float* beta) {
      const QMat& q = l.w->m;
      DgShape d{};
      d.k = q.k;
      slot_shape(d, q8, var ? 8 : 1);
      CUtensorMap tw, ts;
      memset(&ts, 0, sizeof(ts));
      const uint32_t row_bytes = q8 ? q.k : q.k / 2;
      {
        const cuuint64_t dims[3] = {128, q.n, row_bytes / 128}, strides[2] = {row_bytes, 128};
        const cuuint32_t box[3] = {128, 16, d.sc_off / 2048}, estr[3] = {1, 1, 1};
        ok = ok && enc(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, (void*)q.qs, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                       CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
      }
      if (d.nch > 1) {
        const cuuint64_t dims[2] = {q.k / 32, q.n}, strides[1] = {q.k / 32 * 2};
        const cuuint32_t box[2] = {d.sc_pitch, 16}, estr[2] = {1, 1};
        ok = ok && enc(&ts, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, (void*)q.sc, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                       CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
      }
      memcpy(at + next, &tw, sizeof(tw));
      memcpy(at + next + sizeof(tw), &ts, sizeof(ts));
      const DgMat r{dev_at + next, dev_at + next + sizeof(tw), q.sc, l.bias, gain, beta};
      next += 2 * sizeof(tw);
      return r;
    };
    heads[var] = mat(m->head, m->normf_g, m->normf_b);
    heads[var].bias = nullptr;
    std::vector<DgLayer> hl(m->n_layers);
    for (uint32_t i = 0; i < m->n_layers; i++) {
      const Layer& l = m->layers[i];
      hl[i] = DgLayer{{mat(l.qkv, l.norm1_g, l.norm1_b), mat(l.wo, nullptr, nullptr), mat(l.ff1, l.norm2_g, l.norm2_b), mat(l.ff2, nullptr, nullptr)},
                      l.kv.k,
                      l.kv.v};
    }
    memcpy(at + maps_bytes, hl.data(), hl.size() * sizeof(DgLayer));
    if (!ok) return DG_UNFIT;
  }
  if (cudaMemcpyAsync(st->d_layers, host.data(), host.size(), cudaMemcpyHostToDevice, m->dev->stream) != cudaSuccess ||
      cudaMemsetAsync(st->words, 0, n_words * 8, m->dev->stream) != cudaSuccess || cudaStreamSynchronize(m->dev->stream) != cudaSuccess) {
    cudaGetLastError();
    return DG_UNFIT;
  }
  unsigned long long* w = (unsigned long long*)st->words;
  a.group_words = (uint32_t)g_words;
  a.b_part = w, w += w_part;
  a.b_attn = w, w += rows_max * a.attn_stride;
  a.b_x1 = w, w += rows_max * a.x_stride;
  a.b_x2 = w, w += rows_max * a.x_stride;
  a.b_act = w, w += rows_max * a.act_stride;
  a.b_qkv = w;
  w = (unsigned long long*)st->words + groups * g_words;
  a.toks = w, w += 64;
  a.keys = w, w += 64;
  a.state = (uint32_t*)w, w += 8;
  a.out = (int32_t*)w;
  for (int v = 0; v < 4; v++) {
    DgArgs& b = st->args[v];
    b = a;
    layout(b, kind, 1 << v, max_k);
    b.layers = (const DgLayer*)((uint8_t*)st->d_layers + (v == 3) * var_bytes + maps_bytes);
    b.head = heads[v == 3];
    auto shape = [&](const Linear& l, const unsigned long long* src, unsigned long long* dst, uint32_t dst_stride) {
      const QMat& q = l.w->m;
      DgShape d{src, dst, q.k, q.n};
      slot_shape(d, q8, 1 << v);
      d.tpr = (q.k + 255) / 256, d.tpr_inv = 65536 / d.tpr + 1, d.nu = q.k / 128;
      // (a group's slots, and where it can be the next group's as well: a ring of one tile and a slot holds one tile's)
      d.group = std::max(1u, std::min(tile_group(1 << v), std::min(SLOTS, b.ring_bytes / d.size) / (2 * d.nch)));
      d.k_inv = 1.0f / (float)q.k, d.dst_stride = dst_stride;
      return d;
    };
    const Layer& l = m->layers[0];
    b.sh[0] = shape(l.qkv, a.b_x2, a.b_qkv, m->qkv_w());
    b.sh[1] = shape(l.wo, a.b_attn, a.b_x1, a.x_stride);
    b.sh[2] = shape(l.ff1, a.b_x1, a.b_act, a.act_stride);
    b.sh[3] = shape(l.ff2, a.b_act, a.b_x2, a.x_stride);
    b.sh[4] = shape(m->head, a.b_x2, nullptr, 0);
  }
  st->kind = kind;
  auto add = [&](const Linear& l) { st->units += (l.w->m.n + 15) / 16 * (l.w->m.k / 128); };
  for (const auto& l : m->layers) add(l.qkv), add(l.wo), add(l.ff1), add(l.ff2);
  add(m->head);
  return DG_READY;
}

// Whether a step of `rows` rows can run as this kernel. The set-up is made on first use, and tried again now and then where there
// was no room for it (a try gives back what the scratch pool holds and waits for the stream).
bool decode_grid_ready(FcModel* m, uint32_t rows) {
  if (rows == 0 || rows > 8 * MAX_GROUPS || m->n_shards != 1) return false;
  DgState* st = (DgState*)m->dg;
  if (!st) m->dg = st = new DgState();
  if (st->set_up == DG_UNTRIED || (st->set_up == DG_NO_ROOM && ++st->asked == st->retry)) {
    st->asked = 0;
    if (st->set_up == DG_NO_ROOM) st->retry = std::min(2 * st->retry, 4096u);
    st->set_up = decode_grid_set_up(m, st);
    if (st->set_up != DG_READY) {
      if (st->d_layers) cudaFree(st->d_layers);
      if (st->words) cudaFree(st->words);
      st->d_layers = st->words = nullptr;
    }
  }
  if (st->set_up != DG_READY) return false;
  const uint32_t sub = group_ctas(m, rows), group_rows = std::min(rows, 8u);
  // (LayerNorm keeps its input in registers: two 256-element parts per warp)
  return (m->arch == ARCH_LLAMA || group_rows * ((m->dim + 255) / 256) <= 2 * WARPS) && (m->dim + 15) / 16 <= MAX_RESID * sub &&
         group_rows * m->heads <= MAX_ITEMS * sub;
}

// How the attention of steps that reach `longest` positions is cut into items: as few heads of a group each as the CTAs allow. A
// row's positions are split only where one CTA would work through more than four 64-position tiles: the merge costs another trip
// through L2.
struct DgPlan {
  uint32_t splits, item_heads;
};
static DgPlan decode_grid_plan(const FcModel* m, uint32_t group_rows, uint32_t sub, uint32_t longest) {
  const uint32_t tiles = (longest + KV_POS - 1) / KV_POS, group = m->heads / m->kv_heads;
  DgPlan p{tiles <= 4 ? 1 : std::min(tiles, MAX_SPLITS), 0};
  uint32_t widest = 1;
  for (uint32_t h = 1; h <= std::min(group, ITEM_HEADS); h++)
    if (group % h == 0) {
      widest = h;
      if (!p.item_heads && group_rows * (m->heads / h) * p.splits <= sub) p.item_heads = h;
    }
  if (!p.item_heads) {
    p.item_heads = widest;
    p.splits = std::max(1u, std::min(p.splits, sub / (group_rows * (m->heads / widest))));
  }
  return p;
}

// Whether a step of these rows is faster as this kernel than as launches; figures in us, measured through decode_greedy. One row
// always was (MHA of 48 heads at 3900 positions: 56 a layer here, 87 as launches; 12 heads: 21 and 169).
//
// Two to eight rows: the launches are a chain of some 33 per layer whose attention reads the caches at 5 TB/s with all SMs; here a
// CTA works through its items' tiles one after the other (0.73 per 64-position tile, 0.95 for heads of a group together; from three
// rows on twice that where the widths leave room for one tile in flight), so long caches of many heads go as launches. Per layer, here
// and as launches: 48 heads of 48 as Q8_0, 8 rows at 0 positions 80 and 82, at 500 111 and 102, at 3900 328 and 235, 4 rows at 1000
// 89 and 103, at 2000 132 and 123; 12 of 12 as Q4_0, 8 rows at 1000 45 and 48, at 2000 66 and 59; 16 of 2 as Q8_0, 8 rows at 2000
// 44 and 49, at 3900 58 and 53; 32 of 8 as Q4_0, 8 rows at 1000 56 and 62, at 2000 71 and 68. Of 172 such pairs (2 to 8 rows, 0 to
// 3900 positions, seven models) the estimates below pick the slower side of two, which differ by 1 %.
//
// More rows: every group of eight reads all weights (a unit of 16 rows x 128 k costs an SM 0.15 us as Q4_0, 0.17 as Q8_0) and works through
// its caches on its share of the SMs (2 us per 64-position tile and item), where the launches' step is a chain of some 40 us
// per layer whatever it holds. Steps at 0 .. 60 positions, us as launches and here: Qwen2-style 24 layers Q8_0, 16 rows 1197 and
// 712, 32 rows 1316 and 1116, 48 rows 1555 and 1599, 64 rows 1450 and 2017; Llama-style 12 layers Q4_0, 16 rows 464 and 245, 64
// rows 575 and 503; GPT-2-124M-style Q4_0, 64 rows 732 and 616. At 950 positions: Qwen2-style 16 rows 1177 and 1117, 24 rows
// 1348 and 1612; GPT-2-124M-style 24 rows 858 and 811, 32 rows 1014 and 1109.
bool decode_grid_takes(FcModel* m, uint32_t rows, const uint32_t* positions) {
  if (!decode_grid_ready(m, rows)) return false;
  if (rows == 1) return true;
  const double sms = m->dev->prop.multiProcessorCount, layers = m->n_layers, groups = (rows + 7) / 8;
  const double units = ((DgState*)m->dg)->units;
  double tiles = 0.0, bytes = 0.0;
  uint32_t longest = 0;
  for (uint32_t r = 0; r < rows; r++) {
    tiles += positions[r] / KV_POS + 1;
    bytes += (positions[r] + 1.0) * m->kv_heads * 512;
    longest = std::max(longest, positions[r] + 1);
  }
  if (rows <= 8) {
    const uint32_t sub = group_ctas(m, rows), longest_tiles = (longest + KV_POS - 1) / KV_POS;
    const DgPlan p = decode_grid_plan(m, rows, sub, longest);
    const uint32_t items = rows * (m->heads / p.item_heads) * p.splits, each = (longest_tiles + p.splits - 1) / p.splits;
    const bool one_tile = rows > 2 && ((DgState*)m->dg)->args[rows <= 4 ? 2 : 3].kv_log == 0;
    const double tile = (p.item_heads == 1 ? 0.73 : 0.95) * (one_tile ? 1.9 : 1.0);
    const double here = layers * (10.0 + (items + sub - 1) / sub * each * tile + (p.splits > 1 ? 5.0 : 0.0)) + (rows <= 4 ? 0.12 : 0.25) * units / sms;
    const double launches = layers * (33.0 + 1.5e-3 * longest + bytes / 5.3e6) + 1.2e-3 * units;
    return here < launches;
  }
  uint32_t item = 1;
  for (uint32_t h = 1; h <= ITEM_HEADS; h++)
    if (m->heads / m->kv_heads % h == 0) item = h;
  const double here = layers * (10.0 + 2.0 * tiles * (m->heads / item) / sms) + (((DgState*)m->dg)->kind == FC_Q8_0 ? 0.17 : 0.15) * groups * units / sms;
  const double launches = layers * ((rows <= 16 ? 38.0 : rows <= 32 ? 42.0 : 50.0) + bytes / 4e6) + 1.3e-3 * units;
  return here < launches;
}

// Of `steps` steps that follow one another, the first of them at `positions`: how many go the way the first one goes, in one kernel or
// as launches; and, in one kernel, how many have its cut of the attention. A chain is cut there, so that it is its single steps bit for bit.
uint32_t decode_grid_steps(FcModel* m, uint32_t rows, const uint32_t* positions, uint32_t steps, bool* takes) {
  uint32_t at[8 * MAX_GROUPS], n = 0;
  *takes = rows <= 8 * MAX_GROUPS && decode_grid_takes(m, rows, positions);
  if (rows == 1 || rows > 8 * MAX_GROUPS || !decode_grid_ready(m, rows)) return steps;
  for (bool same = true; same && ++n < steps;) {
    for (uint32_t r = 0; r < rows; r++) at[r] = positions[r] + n;
    same = decode_grid_takes(m, rows, at) == *takes;
  }
  return n;
}
static uint32_t decode_grid_same_plan(const FcModel* m, uint32_t group_rows, uint32_t sub, uint32_t longest, uint32_t steps) {
  const DgPlan first = decode_grid_plan(m, group_rows, sub, longest);
  uint32_t n = 0;
  do {
    n += KV_POS - (longest + n - 1) % KV_POS; // (a plan holds for whole tiles)
    const DgPlan p = decode_grid_plan(m, group_rows, sub, longest + n);
    if (p.splits != first.splits || p.item_heads != first.item_heads) break;
  } while (n < steps);
  return std::min(n, steps);
}

const int32_t* decode_grid_out(const FcModel* m) { return ((DgState*)m->dg)->args[0].out; }

// After a step that reported a wait that gave up: as before the first one.
int decode_grid_clear(FcModel* m) {
  DgState* st = (DgState*)m->dg;
  FC_CUDA(m->dev, cudaMemsetAsync(st->words, 0, (size_t)((uint8_t*)(st->args[0].out + 72) - (uint8_t*)st->words), m->dev->stream));
  st->tags = 0;
  return FC_OK;
}

int k_decode_grid(FcModel* m, uint32_t rows, const uint32_t* streams, const uint32_t* positions, const int32_t* tokens, uint32_t steps, int32_t* log) {
  DgState* st = (DgState*)m->dg;
  FcDevice* dev = m->dev;
  const int v = rows == 1 ? 0 : rows == 2 ? 1 : rows <= 4 ? 2 : 3;
  DgArgs a = st->args[v];
  const uint32_t groups = (rows + 7) / 8;
  a.rows = rows, a.group_rows = (rows + groups - 1) / groups, a.sub = group_ctas(m, rows);
  uint32_t longest = 0;
  for (uint32_t r = 0; r < rows; r++) {
    a.tok_in[r] = tokens ? tokens[r] : 0;
    a.stream[r] = (int32_t)streams[r];
    longest = std::max(longest, positions[r] + 1);
  }
  const bool llama = m->arch == ARCH_LLAMA;
  for (uint32_t s = 0; s < steps; s += a.steps) { // a launch for as long as the cut of the attention holds, up to 256 steps
    a.steps = std::min(256u, decode_grid_same_plan(m, a.group_rows, a.sub, longest + s, steps - s));
    st->tags += (uint64_t)a.steps * (m->n_layers + 1);
    if (st->tags >= 1ull << 31) { // (before a tag could come round again)
      FC_CUDA(dev, cudaMemsetAsync(st->words, 0, (size_t)((uint8_t*)st->args[0].out - (uint8_t*)st->words), dev->stream));
      st->tags = (uint64_t)a.steps * (m->n_layers + 1);
    }
    for (uint32_t r = 0; r < rows; r++) a.pos[r] = (int32_t)(positions[r] + s);
    a.chained = tokens && s == 0 ? 0 : 1, a.log = log ? log + (size_t)s * rows : nullptr;
    const DgPlan plan = decode_grid_plan(m, a.group_rows, a.sub, longest + s);
    a.splits = plan.splits, a.item_heads = plan.item_heads;
    FC_TRY(st->kind == FC_Q8_0 ? launch_rows<FC_Q8_0>(dev, a, llama) : launch_rows<FC_Q4_0>(dev, a, llama));
  }
  return FC_OK;
}
