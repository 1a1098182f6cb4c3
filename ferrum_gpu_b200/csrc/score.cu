// Scoring on the device: batched GpuLlama::score (ferrum_wgpu/src/models/llama/forward.rs:L74-L88)
// over many sequences, in chunks that bound the workspace, plus the pieces of the
// vocabulary-split head (trunk / head partials / combine) that the multi-GPU driver strings
// together around its collectives.
#include <algorithm>
#include <cstring>

#include "gemm_tc.cuh"
#include "model.cuh"

namespace {

// in_ids[s][i] = ids[s][i], targets[s][i] = ids[s][i+1], positions[s][i] = i, for i < seq_len-1
__global__ void score_prep_kernel(const int32_t* __restrict__ ids, uint32_t n_seqs, uint32_t seq_len,
                                  int32_t* __restrict__ in_ids, int32_t* __restrict__ targets,
                                  int32_t* __restrict__ positions) {
  const uint32_t t = seq_len - 1;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)n_seqs * t) return;
  const size_t s = i / t, p = i % t;
  in_ids[i] = ids[s * seq_len + p];
  targets[i] = ids[s * seq_len + p + 1];
  positions[i] = (int32_t)p;
}

size_t al(size_t v) { return (v + 255) & ~(size_t)255; }

// Workspace bytes of one chunk of `rows` rows (trunk buffers + ids + head scratch).
size_t chunk_bytes(const FcModel* m, size_t rows, int mode) {
  const size_t vs = m->v1 - m->v0;
  size_t b = al(rows * m->dim * 4) * 2 + al(rows * m->qkv_w() * 4) + al(rows * m->qd() * 4) + al(rows * m->ff1_w() * 4) +
             al(rows * m->hidden * 4) + 3 * al(rows * 4) + al(rows * 16) + al(rows * m->dim * 2) + 8192;
  if (mode == FC_EXACT_F32) b += al(rows * vs * 4); // materialised logits of the chunk
  else b += model_tc_head_bytes(m, rows);           // per-tile log-sum-exp partials
  return b;
}

// What one pass may take: whole sequences as long as it fits (2 GiB exact, 6 GiB tensor path).
size_t pass_cap(const FcModel* m, int mode) { return m->pass_bytes ? m->pass_bytes : (size_t)(mode == FC_EXACT_F32 ? 2 : 6) << 30; }

} // namespace

FC_API int fc_debug_score_pass_bytes(FcModel* m, uint64_t bytes) {
  if (!m) return FC_ERR_ARG;
  m->pass_bytes = (size_t)bytes;
  return FC_OK;
}

// Exact-f32 head over this rank's vocabulary rows: logits of the chunk are materialised, then
// reduced to per-row partials.
static int head_partial_f32(FcModel* m, const float* hidden, const int32_t* targets, uint32_t rows, float* logits_ws,
                            float* partial) {
  Epilogue ep;
  ep.wide = &m->wide;
  FC_TRY(k_qlinear_f32(m->dev, m->head_view, hidden, rows, logits_ws, ep));
  return k_score_partial(m->dev, logits_ws, targets, rows, m->v1 - m->v0, m->v0, partial);
}

FC_API int fc_model_score_dev(FcModel* m, const int32_t* ids_dev, uint32_t n_seqs, uint32_t seq_len, int mode,
                              float* logprob_dev, uint8_t* greedy_dev, double* nll_sum_dev) {
  if (!m || !ids_dev) return FC_ERR_ARG;
  FcDevice* dev = m->dev;
  cudaSetDevice(dev->ordinal);
  if (seq_len < 2) return fc_fail(dev, FC_ERR_SHAPE, "scoring needs at least 2 tokens");
  if (seq_len - 1 > m->ctx) return fc_fail(dev, FC_ERR_SHAPE, "sequence length %u must be in 1..=%u", seq_len - 1, m->ctx);
  if (mode != FC_EXACT_F32 && mode != FC_TENSOR_F16) return fc_fail(dev, FC_ERR_ARG, "unknown arithmetic mode %d", mode);
  if (m->n_shards != 1)
    return fc_fail(dev, FC_ERR_UNSUPPORTED, "this model holds one vocabulary shard: use the trunk / head_partial / combine calls");
  if (n_seqs == 0) return FC_OK;
  const uint32_t t = seq_len - 1;
  const size_t cap = pass_cap(m, mode);
  uint32_t per = n_seqs;
  while (per > 1 && chunk_bytes(m, (size_t)per * t, mode) > cap) per = (per + 1) / 2;
  const size_t rows_max = (size_t)per * t;
  const size_t lp_bytes = logprob_dev ? 0 : al((size_t)n_seqs * t * 4);
  FC_TRY(arena_reserve_wide(m, chunk_bytes(m, rows_max, mode) + lp_bytes, rows_max, mode));
  float* lp_all = logprob_dev ? logprob_dev : (float*)arena_take(m, (size_t)n_seqs * t * 4);
  int32_t* in_ids = (int32_t*)arena_take(m, rows_max * 4);
  int32_t* targets = (int32_t*)arena_take(m, rows_max * 4);
  int32_t* positions = (int32_t*)arena_take(m, rows_max * 4);
  float* partial = (float*)arena_take(m, rows_max * 16);
  float* logits_ws = mode == FC_EXACT_F32 ? (float*)arena_take(m, rows_max * (m->v1 - m->v0) * 4) : nullptr;
  void* hidden = arena_take(m, rows_max * m->dim * 4); // f32 (exact) or bf16 (tensor)
  const size_t mark = m->arena.off;
  for (uint32_t s0 = 0; s0 < n_seqs; s0 += per) {
    const uint32_t ns = n_seqs - s0 < per ? n_seqs - s0 : per;
    const uint32_t rows = ns * t;
    m->arena.off = mark;
    FC_LAUNCH(dev, "score_prep",
              score_prep_kernel<<<(rows + 255) / 256, 256, 0, dev->stream>>>(ids_dev + (size_t)s0 * seq_len, ns, seq_len,
                                                                             in_ids, targets, positions));
    float* lp = lp_all + (size_t)s0 * t;
    uint8_t* gr = greedy_dev ? greedy_dev + (size_t)s0 * t : nullptr;
    if (mode == FC_EXACT_F32) {
      FC_TRY(model_trunk_f32(m, in_ids, positions, ns, t, (float*)hidden));
      FC_TRY(head_partial_f32(m, (const float*)hidden, targets, rows, logits_ws, partial));
    } else {
      FC_TRY(model_trunk_tc(m, in_ids, positions, ns, t, (__half*)hidden));
      FC_TRY(model_head_partial_tc(m, (const __half*)hidden, targets, rows, partial));
    }
    FC_TRY(k_score_combine(dev, partial, 1, rows, targets, lp, gr));
  }
  if (nll_sum_dev) FC_TRY(k_nll_sums(dev, lp_all, n_seqs, t, nll_sum_dev));
  return FC_OK;
}

// ---- vocabulary-split head ------------------------------------------------------------------------

FC_API int fc_model_set_head_shard(FcModel* m, uint32_t shard, uint32_t n_shards) {
  if (!m) return FC_ERR_ARG;
  if (n_shards == 0 || shard >= n_shards) return fc_fail(m->dev, FC_ERR_ARG, "shard %u of %u", shard, n_shards);
  const uint32_t per = (m->vocab + n_shards - 1) / n_shards;
  const uint32_t v0 = per * shard < m->vocab ? per * shard : m->vocab;
  const uint32_t v1 = v0 + per < m->vocab ? v0 + per : m->vocab;
  if (v1 <= v0) return fc_fail(m->dev, FC_ERR_SHAPE, "shard %u of %u holds no vocabulary rows", shard, n_shards);
  const QMat& full = m->head.w->m;
  QMat v = full;
  v.n = v1 - v0;
  v.qs = full.qs + qmat_qs_bytes(full.kind, full.k, v0);
  v.sc = full.sc ? (const __half*)((const uint8_t*)full.sc + qmat_sc_bytes(full.kind, full.k, v0)) : nullptr;
  m->head_view = v;
  m->shard = shard, m->n_shards = n_shards, m->v0 = v0, m->v1 = v1;
  return FC_OK;
}

FC_API int fc_model_trunk_dev(FcModel* m, const int32_t* ids_dev, uint32_t n_seqs, uint32_t seq_len, int mode,
                              void* hidden_dev) {
  if (!m || !ids_dev || !hidden_dev) return FC_ERR_ARG;
  FcDevice* dev = m->dev;
  cudaSetDevice(dev->ordinal);
  if (seq_len == 0 || seq_len > m->ctx) return fc_fail(dev, FC_ERR_SHAPE, "sequence length %u must be in 1..=%u", seq_len, m->ctx);
  if (n_seqs == 0) return FC_OK;
  const size_t rows = (size_t)n_seqs * seq_len;
  FC_TRY(arena_reserve_wide(m, chunk_bytes(m, rows, FC_TENSOR_F16), rows, mode));
  int32_t* positions = (int32_t*)arena_take(m, rows * 4);
  // positions 0..seq_len-1 per sequence (score_prep with a virtual extra token would drop the
  // last row; here every row is kept)
  {
    void* pin;
    FC_TRY(fc_pinned(dev, rows * 4, &pin));
    for (size_t i = 0; i < rows; i++) ((int32_t*)pin)[i] = (int32_t)(i % seq_len);
    FC_CUDA(dev, cudaMemcpyAsync(positions, pin, rows * 4, cudaMemcpyHostToDevice, dev->stream));
    FC_CUDA(dev, cudaStreamSynchronize(dev->stream));
  }
  if (mode == FC_EXACT_F32) return model_trunk_f32(m, ids_dev, positions, n_seqs, seq_len, (float*)hidden_dev);
  if (mode == FC_TENSOR_F16) return model_trunk_tc(m, ids_dev, positions, n_seqs, seq_len, (__half*)hidden_dev);
  return fc_fail(dev, FC_ERR_ARG, "unknown arithmetic mode %d", mode);
}

FC_API int fc_model_head_partial_dev(FcModel* m, const void* hidden_dev, const int32_t* targets_dev, uint32_t rows,
                                     int mode, float* partial_dev) {
  if (!m || !hidden_dev || !targets_dev || !partial_dev) return FC_ERR_ARG;
  FcDevice* dev = m->dev;
  cudaSetDevice(dev->ordinal);
  if (rows == 0) return FC_OK;
  if (mode == FC_TENSOR_F16) {
    FC_TRY(arena_reserve_wide(m, model_tc_head_bytes(m, rows), rows, mode));
    return model_head_partial_tc(m, (const __half*)hidden_dev, targets_dev, rows, partial_dev);
  }
  if (mode != FC_EXACT_F32) return fc_fail(dev, FC_ERR_ARG, "unknown arithmetic mode %d", mode);
  // chunk the rows so the materialised logits stay under 2 GiB
  const size_t vs = m->v1 - m->v0;
  size_t per = rows;
  while (per > 1 && per * vs * 4 > pass_cap(m, mode)) per = (per + 1) / 2;
  FC_TRY(arena_reserve_wide(m, al(per * vs * 4) + 4096, per, mode));
  float* logits_ws = (float*)arena_take(m, per * vs * 4);
  for (size_t r0 = 0; r0 < rows; r0 += per) {
    const uint32_t nr = (uint32_t)(rows - r0 < per ? rows - r0 : per);
    FC_TRY(head_partial_f32(m, (const float*)hidden_dev + r0 * m->dim, targets_dev + r0, nr, logits_ws,
                            partial_dev + r0 * 4));
  }
  return FC_OK;
}

FC_API int fc_score_combine_dev(FcDevice* dev, const float* partials_dev, uint32_t n_shards, const int32_t* targets_dev,
                                uint32_t n_seqs, uint32_t rows_per_seq, float* logprob_dev, uint8_t* greedy_dev,
                                double* nll_sum_dev) {
  if (!dev || !partials_dev || !targets_dev) return FC_ERR_ARG;
  cudaSetDevice(dev->ordinal);
  if (n_shards == 0) return fc_fail(dev, FC_ERR_ARG, "n_shards must be positive");
  if (nll_sum_dev && !logprob_dev) return fc_fail(dev, FC_ERR_ARG, "nll sums need the logprob buffer");
  const uint32_t rows = n_seqs * rows_per_seq;
  FC_TRY(k_score_combine(dev, partials_dev, n_shards, rows, targets_dev, logprob_dev, greedy_dev));
  if (nll_sum_dev) FC_TRY(k_nll_sums(dev, logprob_dev, n_seqs, rows_per_seq, nll_sum_dev));
  return FC_OK;
}

// Sequences of unequal length on the tensor cores: their rows packed one after another without padding, as many whole
// sequences per pass as the workspace bound allows, and one attention launch per layer over a list of query blocks.
// Results stay on the device until all passes are enqueued: one wait per call. (Groups of similar length, each padded
// and run as a pass of its own with its copies and waits, kept the tensor pipe idle: a server's batch is a few hundred
// rows per group. 23 sequences of 250..1000 ids on the GPT-2-124M shape: 13.3 ms so, 5.7 now.)
int model_score_packed(FcModel* m, const int32_t* ids, const uint32_t* offsets, uint32_t n_seqs, float* logprob_out, uint8_t* greedy_out) {
  FcDevice* dev = m->dev;
  const size_t cap = pass_cap(m, FC_TENSOR_F16);
  const size_t total = (size_t)offsets[n_seqs] - n_seqs; // rows: every position but each sequence's last
  // whole sequences per pass, in the caller's order
  std::vector<uint32_t> first(1, 0);
  size_t rows_max = 0;
  for (uint32_t s = 0; s < n_seqs;) {
    size_t rows = 0;
    uint32_t e = s;
    while (e < n_seqs) {
      const size_t t = offsets[e + 1] - offsets[e] - 1;
      if (rows && chunk_bytes(m, rows + t, FC_TENSOR_F16) > cap) break;
      rows += t;
      e++;
    }
    rows_max = rows > rows_max ? rows : rows_max;
    first.push_back(e);
    s = e;
  }
  const size_t b_in = al(total * 4);
  FC_TRY(arena_reserve_wide(m, chunk_bytes(m, rows_max, FC_TENSOR_F16) + 3 * b_in + al(total * 4) + al(total) + al(total * 16) + 8192, rows_max,
                            FC_TENSOR_F16));
  // everything the passes read, built once and sent in one copy: ids, targets, positions, block lists
  const size_t n_blocks_all = [&] {
    size_t b = 0;
    for (uint32_t s = 0; s < n_seqs; s++) b += (offsets[s + 1] - offsets[s] - 1 + 255) / 256;
    return b;
  }();
  const size_t in_bytes = 3 * b_in + al(n_blocks_all * 16);
  void* pin;
  FC_TRY(fc_pinned(dev, in_bytes + al(total * 4) + al(total), &pin));
  int32_t* h_ids = (int32_t*)pin;
  int32_t* h_tgt = (int32_t*)((char*)pin + b_in);
  int32_t* h_pos = (int32_t*)((char*)pin + 2 * b_in);
  uint4* h_blk = (uint4*)((char*)pin + 3 * b_in);
  for (uint32_t s = 0; s < n_seqs; s++) {
    const size_t t = offsets[s + 1] - offsets[s] - 1, at = (size_t)offsets[s] - s;
    std::copy(ids + offsets[s], ids + offsets[s] + t, h_ids + at);
    std::copy(ids + offsets[s] + 1, ids + offsets[s] + 1 + t, h_tgt + at);
    for (size_t i = 0; i < t; i++) h_pos[at + i] = (int32_t)i;
  }
  std::vector<size_t> blk_at(1, 0);
  {
    size_t b = 0;
    for (size_t c = 0; c + 1 < first.size(); c++) {
      const size_t b0 = b, row0 = (size_t)offsets[first[c]] - first[c];
      for (uint32_t s = first[c]; s < first[c + 1]; s++) {
        const uint32_t t = offsets[s + 1] - offsets[s] - 1;
        for (uint32_t q = 0; q < (t + 255) / 256; q++) h_blk[b++] = make_uint4((uint32_t)((size_t)offsets[s] - s - row0), t, q, 0);
      }
      std::stable_sort(h_blk + b0, h_blk + b, [](const uint4& x, const uint4& y) { return x.z > y.z; });
      blk_at.push_back(b);
    }
  }
  char* d_in = (char*)arena_take(m, in_bytes);
  float* d_lp = (float*)arena_take(m, total * 4);
  uint8_t* d_gr = (uint8_t*)arena_take(m, total);
  float* partial = (float*)arena_take(m, rows_max * 16);
  __half* hidden = (__half*)arena_take(m, rows_max * m->dim * 2);
  FC_CUDA(dev, cudaMemcpyAsync(d_in, pin, in_bytes, cudaMemcpyHostToDevice, dev->stream));
  const size_t mark = m->arena.off;
  for (size_t c = 0; c + 1 < first.size(); c++) {
    m->arena.off = mark;
    const size_t row0 = (size_t)offsets[first[c]] - first[c], row1 = (size_t)offsets[first[c + 1]] - first[c + 1];
    const uint32_t rows = (uint32_t)(row1 - row0);
    const int32_t* c_ids = (const int32_t*)d_in + row0;
    const int32_t* c_tgt = (const int32_t*)(d_in + b_in) + row0;
    const int32_t* c_pos = (const int32_t*)(d_in + 2 * b_in) + row0;
    const uint4* c_blk = (const uint4*)(d_in + 3 * b_in) + blk_at[c];
    FC_TRY(model_trunk_tc(m, c_ids, c_pos, 1, rows, hidden, -1, c_blk, (uint32_t)(blk_at[c + 1] - blk_at[c])));
    FC_TRY(model_head_partial_tc(m, hidden, c_tgt, rows, partial));
    FC_TRY(k_score_combine(dev, partial, 1, rows, c_tgt, d_lp + row0, d_gr + row0));
  }
  FC_TRY(tc_check_errors(dev));
  char* h_out = (char*)pin + in_bytes;
  FC_CUDA(dev, cudaMemcpyAsync(h_out, d_lp, total * 4, cudaMemcpyDeviceToHost, dev->stream));
  FC_CUDA(dev, cudaMemcpyAsync(h_out + al(total * 4), d_gr, total, cudaMemcpyDeviceToHost, dev->stream));
  FC_CUDA(dev, cudaStreamSynchronize(dev->stream));
  memcpy(logprob_out, h_out, total * 4);
  memcpy(greedy_out, h_out + al(total * 4), total);
  return FC_OK;
}
