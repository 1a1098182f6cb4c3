// The fourth kernel body of gemm_tc.cu (included there, inside its anonymous namespace): the product of many rows on
// CTA pairs, from fp16 weights that a preparation kernel decoded once for the launch (weights_f16_kernel).
//
//   D[a, b] = A[a, :] . B[b, :]       256 A rows x 256 B rows per pair and tile (tcgen05.mma.cta_group::2)
//
// Every epilogue but the head's has the weight rows as A (a thread holds one output column for 32 rows of x at a time,
// as in gemm_ts_main.cuh); the head's log-sum-exp has the activation rows as A (a thread folds its row's logits).
//
// Why beside qgemm_ts_kernel, which decodes the packed weights inside the product: there every 128 x 192 tile decodes
// its weights again, and with thousands of rows the producers' integer work and their hand-over, not the tensor pipe,
// set the pace. One decoding pass costs about 3 bytes of L2 / HBM traffic per weight whatever the rows; after it the
// main loop is TMA and MMAs only. The pair shares each tile's operands: a CTA fetches its own 128 rows of A and half of
// B's 256, 32 KB per 64 k for 128 x 256 x 64 multiply-adds - half of what two single CTAs would read, and it is the L2
// that would bound those. With few rows the decoding pass costs more than it saves: rule and
// figures at tp_takes.
//
//   warp 0        TMA: this CTA's A and B boxes of a K step; bytes are counted on the LEADER's barrier (even CTA)
//   warp 1        tensor-memory owner; in the leader one thread issues the MMAs of both CTAs
//   warps 4-11    epilogue: warp w owns lane quadrant w % 4 and B rows [128 (w - 4) / 4, + 128) of the tile
//
// Barriers: full[s] (leader: the bytes of both CTAs), empty[s] and acc_full[b] (MMA commit, multicast to both CTAs),
// acc_empty[b] (leader: 16 epilogue warps). Two accumulator buffers of 256 columns: the epilogue of a tile runs under
// the next tile's main loop. Every wait is bounded and polls the CTA's abort word.

// Packed rows -> fp16(d q), one rounding: the bits the other kernels' dequantisers produce. Bound by memory: per weight two
// bytes out and a half or one in. Rows, scales and result lie one behind the other, so the matrix is one run of eights
// (n k / 8 of them); a thread takes F16_ITEMS eights, 256 apart - all its loads first, every store instruction of a warp 512
// consecutive bytes. (One half-block per thread and row: as many blocks of one load each, 72 us for the 65 M weights of
// 32000 x 2048 Q4_0.)
constexpr int F16_ITEMS = 8;
template <int KIND>
__global__ void __launch_bounds__(256) weights_f16_kernel(QMat w, uint32_t eights, __half* __restrict__ out) {
  const uint32_t base = blockIdx.x * (256 * F16_ITEMS) + threadIdx.x;
  uint2 q[F16_ITEMS];
  uint32_t dd[F16_ITEMS];
#pragma unroll
  for (int i = 0; i < F16_ITEMS; i++) {
    const uint32_t e = min(base + i * 256, eights - 1);
    if (KIND == FC_Q8_0)
      q[i] = *reinterpret_cast<const uint2*>(w.qs + (size_t)e * 8);
    else
      q[i].x = *reinterpret_cast<const uint32_t*>(w.qs + (size_t)e * 4);
    dd[i] = (uint32_t)__half_as_ushort(w.sc[e / 4]);
  }
#pragma unroll
  for (int i = 0; i < F16_ITEMS; i++) {
    const uint32_t d = dd[i] * 0x00010001u;
    uint4 o;
    if (KIND == FC_Q8_0) {
      const uint32_t u = q[i].x ^ 0x80808080u, v = q[i].y ^ 0x80808080u;
      o.x = f16x2_mul(f16x2_sub(__byte_perm(u, 0x64646464u, 0x5140), 0x64806480u), d);
      o.y = f16x2_mul(f16x2_sub(__byte_perm(u, 0x64646464u, 0x5342), 0x64806480u), d);
      o.z = f16x2_mul(f16x2_sub(__byte_perm(v, 0x64646464u, 0x5140), 0x64806480u), d);
      o.w = f16x2_mul(f16x2_sub(__byte_perm(v, 0x64646464u, 0x5342), 0x64806480u), d);
    } else {
      const uint32_t v = q[i].x, v8 = v >> 8;
      o.x = f16x2_mul(f16x2_sub((v & 0x000f000fu) | 0x64006400u, 0x64086408u), d);
      o.y = f16x2_mul(f16x2_sub((v & 0x00f000f0u) | 0x54005400u, 0x54805480u), d);
      o.z = f16x2_mul(f16x2_sub((v8 & 0x000f000fu) | 0x64006400u, 0x64086408u), d);
      o.w = f16x2_mul(f16x2_sub((v8 & 0x00f000f0u) | 0x54005400u, 0x54805480u), d);
    }
    const uint32_t e = base + i * 256;
    if (e < eights) reinterpret_cast<uint4*>(out)[e] = o;
  }
}

template <int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(TP_THREADS, 1)
    qgemm_tp_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                    const __grid_constant__ CUtensorMap tmap_o, const TcArgs a) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (tc::smem_u32(smem_raw) + 1023u) & ~1023u; // (the 128B swizzle is a function of the address)
  uint8_t* smem = smem_raw + (base - tc::smem_u32(smem_raw));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + TP_STAGES * TP_STAGE_BYTES);
  uint64_t* empty = full + TP_STAGES;
  uint64_t* acc_full = empty + TP_STAGES;
  uint64_t* acc_empty = acc_full + 2;
  uint64_t* done = acc_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile uint32_t* abort_word = tmem_slot + 1;

  constexpr bool X_IS_A = EPI == EPI_LSE;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = blockIdx.x & 1u; // (clusters are two consecutive blocks)
  const uint32_t k_iters = a.k / TC_BK;
  const uint32_t tiles_n = (a.n + 255) / 256, tiles_x = (a.m + 255) / 256;
  const uint32_t total = tiles_n * tiles_x;
  auto place = [&](uint32_t tile, uint32_t& n0, uint32_t& x0) { n0 = (tile % tiles_n) * 256, x0 = (tile / tiles_n) * 256; };

  if (threadIdx.x == 0) {
    for (int s = 0; s < TP_STAGES; s++) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; b++) {
      tc::mbar_init(&acc_full[b], 1);
      tc::mbar_init(&acc_empty[b], 16);
    }
    tc::mbar_init(done, 1);
    *abort_word = 0;
    tc::fence_barrier_init();
    tc::prefetch_tmap(&tmap_a);
    tc::prefetch_tmap(&tmap_b);
    if (a.out_tma) tc::prefetch_tmap(&tmap_o);
  }
  if (warp == 1) {
    tc::tmem_alloc_pair(tmem_slot, TMEM_COLS);
    tc::tmem_relinquish_pair();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::cluster_sync(); // both CTAs' barriers are initialised and both tensor memories allocated
  tc::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ---- TMA ----
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (uint32_t tile = blockIdx.x >> 1; tile < total && ok; tile += gridDim.x >> 1) {
        uint32_t n0, x0;
        place(tile, n0, x0);
        const int32_t ay = (int32_t)((X_IS_A ? x0 : n0) + rank * 128), by = (int32_t)((X_IS_A ? n0 : x0) + rank * 128);
        for (uint32_t kk = 0; kk < k_iters; kk++, it++) {
          const uint32_t s = it % TP_STAGES, ph = (it / TP_STAGES) & 1;
          if (!wait_or_abort(&empty[s], ph ^ 1, abort_word)) {
            atomicExch(a.err_flag, ERR_WAIT_EMPTY);
            ok = false;
            break;
          }
          uint8_t* st = smem + s * TP_STAGE_BYTES;
          const uint32_t bar = tc::leader_addr(&full[s]);
          if (rank == 0) tc::mbar_arrive_expect_tx(&full[s], 2 * TP_STAGE_BYTES);
          tc::tma_load_2d_pair(st, &tmap_a, bar, (int32_t)(kk * TC_BK), ay);
          tc::tma_load_2d_pair(st + TP_STAGE_BYTES / 2, &tmap_b, bar, (int32_t)(kk * TC_BK), by);
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer: one thread of the leader, for both CTAs ----
    if (rank == 0 && tc::elect_one()) {
      constexpr uint32_t idesc = tc::idesc_f16_f32(256, 256);
      constexpr uint32_t desc_hi = (1024u >> 4) | (1u << 14) | (2u << 29); // stride 1024 B, version 1, 128B swizzle
      uint32_t it = 0, tcnt = 0;
      bool ok = true;
      for (uint32_t tile = blockIdx.x >> 1; tile < total && ok; tile += gridDim.x >> 1, tcnt++) {
        const uint32_t buf = tcnt & 1;
        if (!wait_or_abort(&acc_empty[buf], ((tcnt >> 1) & 1) ^ 1, abort_word)) { // both epilogues have drained this buffer
          atomicExch(a.err_flag, ERR_WAIT_ACC);
          break;
        }
        tc::tc_fence_after();
        const uint32_t d = tmem_base + buf * 256;
        for (uint32_t kk = 0; kk < k_iters; kk++, it++) {
          const uint32_t s = it % TP_STAGES;
          if (!wait_or_abort(&full[s], (it / TP_STAGES) & 1, abort_word)) {
            atomicExch(a.err_flag, ERR_WAIT_FULL);
            ok = false;
            break;
          }
          tc::tc_fence_after();
          const uint64_t da = ((uint64_t)desc_hi << 32) | ((base + s * TP_STAGE_BYTES) >> 4);
          const uint64_t db = ((uint64_t)desc_hi << 32) | ((base + s * TP_STAGE_BYTES + TP_STAGE_BYTES / 2) >> 4);
#pragma unroll
          for (uint32_t ks = 0; ks < TC_BK / 16; ks++) tc::mma_f16_pair(d, da + 2 * ks, db + 2 * ks, idesc, (kk | ks) != 0 ? 1u : 0u);
          tc::mma_commit_pair(&empty[s]);
        }
        if (ok) tc::mma_commit_pair(&acc_full[buf]);
      }
      // every MMA has finished before the tensor memory goes back (also after a wait that gave up)
      tc::mma_commit_pair(done);
    }
    __syncwarp();
    if (lane == 0) {
      volatile uint32_t never = 0;
      if (!wait_suspended(done, 0, &never)) atomicExch(a.err_flag, ERR_WAIT_ACC);
    }
    __syncwarp();
  } else if (warp >= 4) {
    // ---- epilogue ----
    const uint32_t e = (uint32_t)warp - 4, half = e >> 2, quad = (uint32_t)warp & 3u;
    uint8_t* stage = smem + TP_STG_OFF + e * (2 * STG_TILE);
    uint32_t sbuf = 0, tcnt = 0;
    for (uint32_t tile = blockIdx.x >> 1; tile < total; tile += gridDim.x >> 1, tcnt++) {
      const uint32_t buf = tcnt & 1;
      uint32_t n0, x0;
      place(tile, n0, x0);
      bool ok = wait_suspended(&acc_full[buf], (tcnt >> 1) & 1, abort_word);
      if (!ok) atomicExch(a.err_flag, ERR_WAIT_ACC);
      if (!__all_sync(0xffffffffu, ok)) break;
      tc::tc_fence_after();
      const uint32_t taddr = tmem_base + ((quad * 32u) << 16) + buf * 256 + half * 128;
      if (X_IS_A) { // this thread folds 128 logits of its row: one of the 128-column tiles that k_partial_merge takes
        const uint32_t row = x0 + rank * 128 + quad * 32 + lane, c0 = n0 + half * 128;
        LseState st;
        const int target = row < a.m ? a.targets[row] : -1;
#pragma unroll 1
        for (uint32_t c = 0; c < 4; c++) {
          uint32_t acc[32];
          tc::tmem_ld_32x32(taddr + c * 32, acc);
          tc::tmem_ld_wait();
          epilogue_lse(a, st, c0 + c * 32, target, acc);
        }
        if (row < a.m && c0 < a.n)
          *reinterpret_cast<float4*>(a.partial + ((size_t)(c0 / TC_BN + a.tile0) * a.m + row) * 4) =
              make_float4(st.mx, st.se, st.tl, (float)st.first);
      } else {
        const uint32_t ncol = n0 + rank * 128 + quad * 32, n = ncol + lane; // this thread's output column
        const bool n_ok = n < a.n;
        const float bias = (a.bias && n_ok) ? a.bias[n] : 0.0f;
#pragma unroll 1
        for (uint32_t c = 0; c < 4; c++) {
          const uint32_t x1 = x0 + half * 128 + c * 32;
          uint32_t acc[32];
          tc::tmem_ld_32x32(taddr + c * 32, acc);
          tc::tmem_ld_wait();
          if (a.out_tma) {
            uint8_t* st = stage + sbuf * STG_TILE;
            sbuf ^= 1;
            if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
            __syncwarp();
            stage_chunk<EPI>(a, st, acc, bias, lane);
            tc::fence_async_smem();
            __syncwarp();
            if (lane == 0) {
              if (ncol < a.n && x1 < a.m) store_staged<EPI>(&tmap_o, st, (int32_t)(EPI == EPI_SWIGLU ? ncol >> 1 : ncol), (int32_t)x1);
              asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
          } else if (EPI == EPI_F32) {
#pragma unroll
            for (int j = 0; j < 32; j++)
              if (n_ok && x1 + j < a.m) a.out_f32[(size_t)(x1 + j) * a.ldo + n] = __uint_as_float(acc[j]) + bias;
          }
        }
      }
      // this warp's reads of the buffer are complete: hand it back to the MMA issuer
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive_cluster(tc::leader_addr(&acc_empty[buf]));
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); // the staged tiles are out before the CTA ends
  }
  // A wait that gave up leaves copies in flight: they land within microseconds, long before this runs out.
  if (*abort_word)
    for (int i = 0; i < 1000; i++) __nanosleep(1000);
  tc::tc_fence_before();
  __syncthreads();
  __syncwarp();
  tc::cluster_sync(); // nobody leaves while the partner may still signal it or read its operands
  if (warp == 1) tc::tmem_dealloc_pair(tmem_base, TMEM_COLS);
}
