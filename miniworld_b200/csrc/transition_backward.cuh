// Backward of the pair Transition  y = x + squeeze(SiLU(expand_a(LN x)) * expand_b(LN x)),  hidden width 512.
//
// One launch per block of 128 hidden units (four launches): the weight gradients of a block (expand_a, expand_b and
// squeeze: three 128 x 128 accumulators) stay in tensor memory over all position tiles of a CTA, which leaves one
// 128-column working region; the running d x_hat is carried between the launches in HBM (fp16, in place) and the last
// launch finishes the LayerNorm backward and the residual. The first launch normalises x and scales dy and leaves both as
// fp16 tensors (and 1 / sigma) for the others. Per tile of 128 positions and block j, everything transposed like the
// prologue's backward (tensor-memory lanes = hidden units, columns = positions: a thread owns one unit and 32 positions, so
// its constants and column sums are scalars and the tiles are written in 16-byte runs):
//   dh^T = Ws_j^T dy^T -> registers    a^T = Wa_j' x_hat^T + ca -> registers    b^T = Wb_j' x_hat^T + cb
//   da = dh b silu'(a),  db = dh silu(a)  (tiles S1, S2)      h = silu(a) b  (registers, then S1)
//   d x_hat (+)= da Wa_j' + db Wb_j'   Ma_j += da x_hat   Mb_j += db x_hat   (one round)      dWs_j += dy^T h^T
// Wa' = Wa gamma, Wb' = Wb gamma (fp16), ca = Wa beta, cb = Wb beta; dy carries the power-of-two scale c of backward.cuh.
//
// 16 arithmetic warps, a warp that issues the MMAs and one that issues the copies, joined as in bwd_prologue_kernel. The
// next tile's inputs land while this one finishes: dy in S2 and x_hat in its own buffer as soon as the first gradient round
// is done. What bounds it: the chain of one tile per SM, five GEMM rounds with the working region's read between them (three
// weight matrices and four tiles fill shared memory, the accumulators three quarters of tensor memory). The form before it
// (positions on the lanes, six rounds between eleven CTA-wide barriers, LayerNorm in every launch) took 21 k cycles per tile.
#pragma once

#include "backward.cuh"

namespace trimul {

struct BwdTransitionParams {
  int num_tiles;          // ceil(positions / 128)
  long long positions;
  int block;              // hidden block j of this launch (0..3)
  const float* consts;    // [2][512]: ca, cb
  const float* grad_scale;
  const uint16_t* dx_in;  // [positions][128] fp16: c * d loss / d x_hat gathered by the earlier launches (not FIRST)
  float* rstd;            // [positions]: written by FIRST, read by LAST
  float eps;
  int residual;
  float* part_m;          // [grid][3] matrices (store_partial): Ma_j, Mb_j, dWs_j partials
  float* part_s;          // [grid][2][512]: column sums of da and db in the first 128 entries
  int* status;
};

constexpr int kTrBwdThreads = kBwdThreads + 64;
constexpr int kTrBwdSmemBytes = 7 * kBwdTile + 512 /* barriers */ + 1024;

// map_x, map_dy: FIRST the module's x and dy (bf16), else x_hat and c * dy (fp16), which FIRST stores through map_xh, map_dyc.
template <bool FIRST, bool LAST>
__global__ void __launch_bounds__(kTrBwdThreads, 1)
bwd_transition_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_dy,
                      const __grid_constant__ CUtensorMap map_wa, const __grid_constant__ CUtensorMap map_wb,
                      const __grid_constant__ CUtensorMap map_ws, const __grid_constant__ CUtensorMap map_xh,
                      const __grid_constant__ CUtensorMap map_dyc, const __grid_constant__ CUtensorMap map_out,
                      const BwdTransitionParams p) {
  // named barriers: inputs converted (FIRST), dh read, a read, da / db written, column sums taken, h written and d x_hat read,
  // output written
  constexpr int kBarN = 2, kBarR1 = 3, kBarR2 = 4, kBarA = 5, kBarS = 8, kBarH = 6, kBarC = 7;
  constexpr int kOne = kBwdThreads + 32, kTwo = kBwdThreads + 64;  // with one or both issuing warps
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t wa_s = smem_base, wb_s = wa_s + kBwdTile, ws_s = wb_s + kBwdTile, x_s = ws_s + kBwdTile;
  const uint32_t ring_s = x_s + kBwdTile;  // three buffers in the roles dy, S1, S2, which rotate from tile to tile
  const uint32_t bar_base = smem_base + 7 * kBwdTile;
  const uint32_t w_full = bar_base, x_full = bar_base + 8, y_full = bar_base + 16, dh_done = bar_base + 24;
  const uint32_t a_done = bar_base + 32, b_done = bar_base + 40, ra_done = bar_base + 48, h_done = bar_base + 56;
  const uint32_t out_free = bar_base + 64;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + 7 * kBwdTile + 72);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (uint32_t b = w_full; b <= out_free; b += 8) mbar_init(b, 1);
    *abort_flag = 0;
    fence_mbar_init();
    prefetch_tmap(&map_x);
    prefetch_tmap(&map_dy);
    prefetch_tmap(&map_out);
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (warp != kBwdThreads / 32 + 1) {
    grid_dependency_wait();
    grid_dependents_launch();
  }

  // role 0 = dy, 1 = S1 (da, then h, then the output), 2 = S2 (db): the next tile's dy comes into S2, its S1 is this tile's
  // dy buffer and its S2 this tile's S1, whose output has been stored by then
  auto ring = [&](int it_i, int r) { return ring_s + static_cast<uint32_t>((r + 2 * it_i) % 3) * kBwdTile; };
  // (thread_wait: a thread that gives up sets the abort word and carries on; every later wait of the CTA returns within
  // one poll, so that all warps walk through the same barriers to the end)
  if (warp == kBwdThreads / 32) {
    // ------------------------------------------------------------ MMAs
    if (elect_one()) thread_wait(w_full, 0, abort_flag, p.status, kDevTimeoutMma);
    __syncwarp();
    constexpr uint32_t idesc_kk = umma_idesc(128, 128, false, false, kFmtF16, kFmtF16);
    constexpr uint32_t idesc_mk = umma_idesc(128, 128, true, false, kFmtF16, kFmtF16);
    constexpr uint32_t idesc_km = umma_idesc(128, 128, false, true, kFmtF16, kFmtF16);
    constexpr uint32_t idesc_mm = umma_idesc(128, 128, true, true, kFmtF16, kFmtF16);
    auto kmaj = [](uint32_t tile, int ks) {
      return umma_desc_kmajor(tile + (ks >> 2) * 16384) + static_cast<uint64_t>((ks & 3) * 2);
    };
    auto mnmaj = [](uint32_t tile, int ks) { return umma_desc_mnmajor(tile + ks * 2048, 16384); };
    int it = 0;
    for (int tile = blockIdx.x; tile < p.num_tiles; tile += gridDim.x, ++it) {
      const uint32_t y_s = ring(it, 0), s1_s = ring(it, 1), s2_s = ring(it, 2);
      const uint32_t accum = it != 0 ? 1u : 0u;
      if constexpr (FIRST) named_bar_sync(kBarN, kTwo);
      if (elect_one()) {
        // dh^T: A = Ws_j [c][hid] read MN-major, B = dy [pos][c]
        if constexpr (!FIRST) thread_wait(y_full, it & 1, abort_flag, p.status, kDevTimeoutMma);
        tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) umma_bf16(tmem_base, mnmaj(ws_s, ks), kmaj(y_s, ks), idesc_mk, ks != 0 ? 1u : 0u);
        umma_commit(dh_done);
      }
      __syncwarp();
      named_bar_sync(kBarR1, kOne);
      if (elect_one()) {
        if constexpr (!FIRST) thread_wait(x_full, it & 1, abort_flag, p.status, kDevTimeoutMma);
        tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) umma_bf16(tmem_base, kmaj(wa_s, ks), kmaj(x_s, ks), idesc_kk, ks != 0 ? 1u : 0u);
        umma_commit(a_done);
      }
      __syncwarp();
      named_bar_sync(kBarR2, kOne);
      if (elect_one()) {
        tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) umma_bf16(tmem_base, kmaj(wb_s, ks), kmaj(x_s, ks), idesc_kk, ks != 0 ? 1u : 0u);
        umma_commit(b_done);
      }
      __syncwarp();
      named_bar_sync(kBarA, kOne);
      if (elect_one()) {
        // d x_hat (columns 0-127, lanes = positions), Ma (128-255), Mb (256-383; lanes = hidden units)
        tc_fence_after();
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int ks = 0; ks < 8; ++ks)
            umma_bf16(tmem_base, mnmaj(m == 0 ? s1_s : s2_s, ks), mnmaj(m == 0 ? wa_s : wb_s, ks), idesc_mm, (m | ks) != 0 ? 1u : 0u);
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int ks = 0; ks < 8; ++ks)
            umma_bf16(tmem_base + 128 + m * 128, kmaj(m == 0 ? s1_s : s2_s, ks), mnmaj(x_s, ks), idesc_km,
                      (ks != 0 ? 1u : 0u) | accum);
        umma_commit(ra_done);
      }
      __syncwarp();
      named_bar_sync(kBarH, kOne);
      if (elect_one()) {
        // dWs (384-511, lanes = channels c, columns = hidden units): A = dy read MN-major, B = h [hid][pos]
        tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          umma_bf16(tmem_base + 384, mnmaj(y_s, ks), kmaj(s1_s, ks), idesc_mk, (ks != 0 ? 1u : 0u) | accum);
        umma_commit(h_done);
      }
      __syncwarp();
    }
  } else if (warp == kBwdThreads / 32 + 1) {
    // ------------------------------------------------------------ copies
    auto issue_y = [&](int tile_i, int it_i) {
      mbar_arrive_expect_tx(y_full, kBwdTile);
#pragma unroll
      for (int kh = 0; kh < 2; ++kh) tma_load_2d(ring(it_i, 0) + kh * 16384, &map_dy, y_full, kh * 64, tile_i * 128);
    };
    auto issue_x = [&](int tile_i) {
      mbar_arrive_expect_tx(x_full, kBwdTile);
#pragma unroll
      for (int kh = 0; kh < 2; ++kh) tma_load_2d(x_s + kh * 16384, &map_x, x_full, kh * 64, tile_i * 128);
    };
    auto issue_w = [&]() {
      mbar_arrive_expect_tx(w_full, 3 * kBwdTile);
#pragma unroll
      for (int kh = 0; kh < 2; ++kh) {
        tma_load_2d(ws_s + kh * 16384, &map_ws, w_full, p.block * 128 + kh * 64, 0);  // Ws columns of block j, [128 c][128 hid]
        tma_load_2d(wa_s + kh * 16384, &map_wa, w_full, kh * 64, p.block * 128);      // Wa' rows of block j, [128 hid][128 k]
        tma_load_2d(wb_s + kh * 16384, &map_wb, w_full, kh * 64, p.block * 128);
      }
    };
    // What is older than the launch before this one lands while that one ends: the weights but for the first block, which
    // follows their packing; the inputs of the first block (arguments) and of the third and fourth (the first block's).
    // Forward and backward of a replayed graph: N = 48 86.6 -> 82.7 us, N = 384 366.8 -> 361.0.
    const bool inputs_early = FIRST || p.block >= 2;
    if (lane == 0) {
      if constexpr (!FIRST) issue_w();
      if (inputs_early) issue_y(blockIdx.x, 0), issue_x(blockIdx.x);
    }
    __syncwarp();
    grid_dependency_wait();
    grid_dependents_launch();
    if (lane == 0) {
      if constexpr (FIRST) issue_w();
      if (!inputs_early) issue_y(blockIdx.x, 0), issue_x(blockIdx.x);
    }
    __syncwarp();
    int it = 0;
    for (int tile = blockIdx.x; tile < p.num_tiles; tile += gridDim.x, ++it) {
      const int next = tile + static_cast<int>(gridDim.x);
      const bool has_next = next < p.num_tiles;
      if constexpr (FIRST) {
        named_bar_sync(kBarN, kTwo);
        if (lane == 0) {
#pragma unroll
          for (int kh = 0; kh < 2; ++kh) {
            tma_store_2d(&map_xh, x_s + kh * 16384, kh * 64, tile * 128);
            tma_store_2d(&map_dyc, ring(it, 0) + kh * 16384, kh * 64, tile * 128);
          }
          bulk_commit();
        }
        __syncwarp();
      }
      named_bar_sync(kBarS, kOne);  // the column sums have been read off S2
      if (lane == 0 && has_next) {
        thread_wait(ra_done, it & 1, abort_flag, p.status, kDevTimeoutProducer);
        issue_y(next, it + 1);  // into S2
        if constexpr (FIRST) bulk_wait_read<0>();
        if constexpr (!LAST) issue_x(next);
      }
      __syncwarp();
      named_bar_sync(kBarC, kOne);
      if (lane == 0) {
#pragma unroll
        for (int kh = 0; kh < 2; ++kh) tma_store_2d(&map_out, ring(it, 1) + kh * 16384, kh * 64, tile * 128);
        bulk_commit();
        if constexpr (LAST) {
          if (has_next) issue_x(next);  // (the x_hat buffer was the exchange of partial sums until here)
        }
        bulk_wait_read<0>();
        mbar_arrive(out_free);
      }
      __syncwarp();
    }
    if (lane == 0) {
      // Every copy has been waited for by its readers unless the CTA is giving up; then those in flight must land before
      // it exits (the last copies of every kind were the last tile's).
      if (*abort_flag != 0) {
        const uint32_t last = static_cast<uint32_t>((it - 1) & 1);
        const long long t0 = clock64();
        while (!mbar_try_wait(w_full, 0) || !mbar_try_wait(x_full, last) || !mbar_try_wait(y_full, last)) {
          if (clock64() - t0 > kWaitLimitCycles) {
            atomicCAS(p.status, 0, kDevTimeoutDrain);
            break;
          }
        }
      }
      bulk_wait<0>();
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ arithmetic
    const int q = warp & 3, part = warp >> 2;
    const int pos = q * 32 + lane;  // this thread's hidden unit (first part of a tile) or position (second part)
    const uint32_t lane_sel = static_cast<uint32_t>(q * 32) << 16;
    const float gc = p.grad_scale[0], gc_inv = p.grad_scale[1];
    const float ca = p.consts[p.block * 128 + pos], cb = p.consts[512 + p.block * 128 + pos];
    // column sums of da and db as the GEMMs see them (fp16), a chain per group of four positions
    float acc_a[8], acc_b[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) acc_a[c] = 0.f, acc_b[c] = 0.f;
    const float2 ca2 = make_float2(ca, ca), cb2 = make_float2(cb, cb), half2 = make_float2(0.5f, 0.5f);
    const float2 one = make_float2(1.f, 1.f), minus1 = make_float2(-1.f, -1.f);
    auto pair_of = [](uint32_t lo, uint32_t hi) { return make_float2(__uint_as_float(lo), __uint_as_float(hi)); };
    int it = 0;
    for (int tile = blockIdx.x; tile < p.num_tiles; tile += gridDim.x, ++it) {
      const uint32_t y_s = ring(it, 0), s1_s = ring(it, 1), s2_s = ring(it, 2);
      const long long gp = static_cast<long long>(tile) * 128 + pos;
      const bool inside = gp < p.positions;
      float rstd_in = 0.f;
      if constexpr (FIRST) {
        // ---- dy * c and x_hat as fp16 in place
        thread_wait(y_full, it & 1, abort_flag, p.status, kDevTimeoutStats);
#pragma unroll
        for (int ch = 0; ch < kBwdChunks; ++ch) {
          const uint32_t addr = y_s + tile_chunk(pos, part * kBwdChunks + ch);
          const uint4 v = ld_chunk(addr);
          const uint32_t w[4] = {v.x, v.y, v.z, v.w};
          uint32_t o[4];
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const float2 d = bf16x2_to_float2(w[t]);
            o[t] = pack_f16x2_sat(make_float2(d.x * gc, d.y * gc));
          }
          st_chunk(addr, o[0], o[1], o[2], o[3]);
        }
        thread_wait(x_full, it & 1, abort_flag, p.status, kDevTimeoutStats);
        // (the exchange of the statistics uses S1, the previous tile's dy buffer, once its store has read it)
        if (it != 0) thread_wait(out_free, (it - 1) & 1, abort_flag, p.status, kDevTimeoutStats);
        rstd_in = normalise_tile(x_s, s1_s, pos, part, p.eps);
        if (part == 0 && inside) p.rstd[gp] = rstd_in;
        fence_proxy_async_smem();
        __syncwarp();
        named_bar_arrive(kBarN, kTwo);
      } else if constexpr (LAST) {
        if (inside) rstd_in = __ldg(p.rstd + gp);
        // (this thread reads dy and x_hat later; their barriers are waited for here, before they can enter another phase)
        thread_wait(y_full, it & 1, abort_flag, p.status, kDevTimeoutStats);
      }
      // ---- dh, a into registers (this thread's hidden unit, 32 positions)
      uint32_t dh[32], av[32];
      thread_wait(dh_done, it & 1, abort_flag, p.status, kDevTimeoutEpilogue);
      __syncwarp();
      tc_fence_after();
      tmem_ld32(tmem_base + lane_sel + part * 32, dh);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      named_bar_arrive(kBarR1, kOne);
      if constexpr (LAST) thread_wait(x_full, it & 1, abort_flag, p.status, kDevTimeoutStats);
      thread_wait(a_done, it & 1, abort_flag, p.status, kDevTimeoutEpilogue);
      __syncwarp();
      tc_fence_after();
      tmem_ld32(tmem_base + lane_sel + part * 32, av);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      named_bar_arrive(kBarR2, kOne);
      // S2 held the previous tile's output
      if (it != 0) thread_wait(out_free, (it - 1) & 1, abort_flag, p.status, kDevTimeoutStats);
      thread_wait(b_done, it & 1, abort_flag, p.status, kDevTimeoutEpilogue);
      __syncwarp();
      tc_fence_after();
      // ---- da -> S1, db -> S2 ([hidden unit][position]), h packed in registers
      // (packed fp32 pairs: the pass is bound by its instruction count)
      uint32_t h_p[16];
      uint32_t v[2][4];
      tmem_ld4(tmem_base + lane_sel + part * 32, v[0]);
#pragma unroll
      for (int k4 = 0; k4 < 4; ++k4) {
        uint32_t da_p[4], db_p[4];
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          tmem_ld_wait();
          if (k4 * 2 + hf < 7) tmem_ld4(tmem_base + lane_sel + part * 32 + (k4 * 2 + hf + 1) * 4, v[hf ^ 1]);
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int t = hf * 2 + u, i = k4 * 8 + t * 2;
            const float2 b2 = __fadd2_rn(pair_of(v[hf][u * 2], v[hf][u * 2 + 1]), cb2);
            const float2 a2 = __fadd2_rn(pair_of(av[i], av[i + 1]), ca2);
            const float2 d2 = pair_of(dh[i], dh[i + 1]);
            const float2 ah = __fmul2_rn(a2, half2);
            const float2 sg = __ffma2_rn(make_float2(tanh_approx(ah.x), tanh_approx(ah.y)), half2, half2);
            const float2 silu = __fmul2_rn(a2, sg);
            // silu' = sg (1 + a (1 - sg))
            const float2 dsilu = __fmul2_rn(sg, __ffma2_rn(a2, __ffma2_rn(sg, minus1, one), one));
            const float2 da = __fmul2_rn(__fmul2_rn(d2, b2), dsilu);
            const float2 db = __fmul2_rn(d2, silu);
            da_p[t] = pack_f16x2_sat(da);
            db_p[t] = pack_f16x2_sat(db);
            h_p[k4 * 4 + t] = pack_f16x2_sat(__fmul2_rn(silu, b2));
          }
        }
        const uint32_t off = tile_chunk(pos, part * 4 + k4);
        st_chunk(s1_s + off, da_p[0], da_p[1], da_p[2], da_p[3]);
        st_chunk(s2_s + off, db_p[0], db_p[1], db_p[2], db_p[3]);
      }
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      named_bar_arrive(kBarA, kOne);
      // the earlier launches' running d x_hat for this thread's position: requested now, used after the GEMM round
      uint4 dx_prev[kBwdChunks];
#pragma unroll
      for (int ch = 0; ch < kBwdChunks; ++ch) dx_prev[ch] = make_uint4(0u, 0u, 0u, 0u);
      if constexpr (!FIRST) {
        if (inside) ld_gpu_chunks(reinterpret_cast<const uint4*>(p.dx_in + gp * 128 + part * kBwdCh), true, dx_prev);
      }
      // (under the GEMM round) the column sums, from the tiles this thread has written
#pragma unroll
      for (int k4 = 0; k4 < 4; ++k4) {
        auto add = [](float& s, uint32_t lo, uint32_t hi) {
          const float2 x = f16x2_to_float2(lo), y = f16x2_to_float2(hi);
          s += x.x, s += x.y, s += y.x, s += y.y;
        };
        const uint4 a = ld_chunk(s1_s + tile_chunk(pos, part * 4 + k4)), b = ld_chunk(s2_s + tile_chunk(pos, part * 4 + k4));
        add(acc_a[2 * k4], a.x, a.y), add(acc_a[2 * k4 + 1], a.z, a.w);
        add(acc_b[2 * k4], b.x, b.y), add(acc_b[2 * k4 + 1], b.z, b.w);
      }
      __syncwarp();
      named_bar_arrive(kBarS, kOne);
      thread_wait(ra_done, it & 1, abort_flag, p.status, kDevTimeoutEpilogue);
      __syncwarp();
      tc_fence_after();
      // ---- h -> S1; d x_hat of this thread's position out of tensor memory
#pragma unroll
      for (int k4 = 0; k4 < 4; ++k4)
        st_chunk(s1_s + tile_chunk(pos, part * 4 + k4), h_p[k4 * 4], h_p[k4 * 4 + 1], h_p[k4 * 4 + 2], h_p[k4 * 4 + 3]);
      uint32_t vt[kBwdChunks][8];
#pragma unroll
      for (int ch = 0; ch < kBwdChunks; ++ch) tmem_ld8(tmem_base + lane_sel + part * kBwdCh + ch * 8, vt[ch]);
      tmem_ld_wait();
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      named_bar_arrive(kBarH, kOne);
      // ---- the running d x_hat; LAST: LayerNorm backward + residual -> dx (bf16). The output goes into S1 after dWs.
      uint32_t o[kBwdChunks][4];
      if constexpr (!LAST) {
#pragma unroll
        for (int ch = 0; ch < kBwdChunks; ++ch) {
          const uint32_t iw[4] = {dx_prev[ch].x, dx_prev[ch].y, dx_prev[ch].z, dx_prev[ch].w};
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const float2 a = f16x2_to_float2(iw[t]);
            o[ch][t] = pack_f16x2_sat(
                make_float2(__uint_as_float(vt[ch][2 * t]) + a.x, __uint_as_float(vt[ch][2 * t + 1]) + a.y));
          }
        }
      } else {
        float tot[kBwdCh];
        uint4 xh[kBwdChunks];
        float s1 = 0.f, s2 = 0.f;
#pragma unroll
        for (int ch = 0; ch < kBwdChunks; ++ch) {
          xh[ch] = ld_chunk(x_s + tile_chunk(pos, part * kBwdChunks + ch));
          const uint32_t iw[4] = {dx_prev[ch].x, dx_prev[ch].y, dx_prev[ch].z, dx_prev[ch].w};
          const uint32_t xw[4] = {xh[ch].x, xh[ch].y, xh[ch].z, xh[ch].w};
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const float2 a = f16x2_to_float2(iw[t]);
            const float2 x = f16x2_to_float2(xw[t]);
            const float t0 = __uint_as_float(vt[ch][2 * t]) + a.x, t1 = __uint_as_float(vt[ch][2 * t + 1]) + a.y;
            tot[ch * 8 + 2 * t] = t0;
            tot[ch * 8 + 2 * t + 1] = t1;
            s1 += t0 + t1;
            s2 = fmaf(t0, x.x, fmaf(t1, x.y, s2));
          }
        }
        // the partial sums go where this thread's x_hat was (the GEMMs that read it are complete)
        asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(x_s + tile_chunk(pos, part * kBwdChunks)), "f"(s1), "f"(s2) : "memory");
        named_bar_sync(1, kBwdThreads);
        float m1 = 0.f, m2 = 0.f;
#pragma unroll
        for (int k = 0; k < kBwdParts; ++k) {
          float a, b;
          asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(a), "=f"(b) : "r"(x_s + tile_chunk(pos, k * kBwdChunks)));
          m1 += a, m2 += b;
        }
        m1 *= 1.0f / 128.0f, m2 *= 1.0f / 128.0f;
        const float rs = rstd_in * gc_inv;
        const float res = p.residual ? gc_inv : 0.f;  // the dy tile holds dy * c
#pragma unroll
        for (int ch = 0; ch < kBwdChunks; ++ch) {
          const uint4 dyv = ld_chunk(y_s + tile_chunk(pos, part * kBwdChunks + ch));
          const uint32_t xw[4] = {xh[ch].x, xh[ch].y, xh[ch].z, xh[ch].w};
          const uint32_t dw[4] = {dyv.x, dyv.y, dyv.z, dyv.w};
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const float2 x = f16x2_to_float2(xw[t]);
            const float2 r = f16x2_to_float2(dw[t]);
            o[ch][t] = pack_bf16x2(fmaf(rs, tot[ch * 8 + 2 * t] - m1 - x.x * m2, r.x * res),
                                   fmaf(rs, tot[ch * 8 + 2 * t + 1] - m1 - x.y * m2, r.y * res));
          }
        }
      }
      thread_wait(h_done, it & 1, abort_flag, p.status, kDevTimeoutEpilogue);
      __syncwarp();
#pragma unroll
      for (int ch = 0; ch < kBwdChunks; ++ch)
        st_chunk(s1_s + tile_chunk(pos, part * kBwdChunks + ch), o[ch][0], o[ch][1], o[ch][2], o[ch][3]);
      fence_proxy_async_smem();
      __syncwarp();
      named_bar_arrive(kBarC, kOne);
    }
    // ---- per-CTA partials of the weight gradients (every GEMM has been waited for) and of the column sums
    tc_fence_after();
    float* pm = p.part_m + static_cast<size_t>(blockIdx.x) * 3 * 128 * 128;
#pragma unroll
    for (int m = 0; m < 3; ++m) {
#pragma unroll
      for (int ch = 0; ch < kBwdChunks; ++ch) {
        uint32_t v[8];
        tmem_ld8(tmem_base + lane_sel + 128 + m * 128 + part * kBwdCh + ch * 8, v);
        tmem_ld_wait();
        store_partial(pm + m * 128 * 128, pos, part * kBwdChunks + ch, v);
      }
    }
    // the 32 groups of four positions of a hidden unit, in order (through the weights' region, which no GEMM reads any more)
    float* sc = reinterpret_cast<float*>(smem);  // [32 groups][2][128]
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      sc[((part * 8 + c) * 2 + 0) * 128 + pos] = acc_a[c];
      sc[((part * 8 + c) * 2 + 1) * 128 + pos] = acc_b[c];
    }
    named_bar_sync(1, kBwdThreads);
    if (threadIdx.x < 256) {
      float sum = 0.f;
      for (int g = 0; g < 32; ++g) sum += sc[g * 256 + threadIdx.x];
      p.part_s[static_cast<size_t>(blockIdx.x) * 2 * 512 + (threadIdx.x >> 7) * 512 + (threadIdx.x & 127)] = sum;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// ---------------------------------------------------------------------------------------------- small kernels
// Packed weights of the Transition's backward: Wa' = fp16(Wa gamma) [512][128], Wb' likewise, Ws fp16 [128][512],
// then ca = Wa beta [512], cb = Wb beta [512] (fp32). One warp per row of Wa / Wb; Ws converted elementwise.
constexpr size_t kTrBwdWa = 0, kTrBwdWb = 512 * 128 * 2, kTrBwdWs = 2 * 512 * 128 * 2, kTrBwdConst = 3 * 512 * 128 * 2;
constexpr size_t kTrBwdPackedBytes = kTrBwdConst + 2 * 512 * 4;  // 397312, a multiple of 1024
struct TrBwdPackArgs {
  const void* w_a;
  const void* w_b;
  const void* w_s;
  const float* ln_w;
  const float* ln_b;
  int f32_weights;
};
__device__ __forceinline__ float tr_load_w(const void* w, size_t i, int f32) {
  return f32 ? static_cast<const float*>(w)[i]
             : __uint_as_float(static_cast<uint32_t>(static_cast<const uint16_t*>(w)[i]) << 16);
}
// gw: 0 .. 1535: rows of Wa (0-511), Wb (512-1023), then Ws rows by 4
__device__ __forceinline__ void tr_bwd_pack_row(const TrBwdPackArgs& a, uint8_t* packed, int gw) {
  const int lane = threadIdx.x & 31;
  if (gw < 1024) {
    const int m = gw >> 9, row = gw & 511;
    const void* w = m == 0 ? a.w_a : a.w_b;
    float d = 0.f;
    uint16_t o[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int k = lane * 4 + t;
      const float v = tr_load_w(w, static_cast<size_t>(row) * 128 + k, a.f32_weights);
      o[t] = __half_as_ushort(__float2half_rn(fminf(fmaxf(v * a.ln_w[k], -65504.f), 65504.f)));
      d = fmaf(v, a.ln_b[k], d);
    }
    uint2 ov;
    ov.x = static_cast<uint32_t>(o[0]) | (static_cast<uint32_t>(o[1]) << 16);
    ov.y = static_cast<uint32_t>(o[2]) | (static_cast<uint32_t>(o[3]) << 16);
    reinterpret_cast<uint2*>(packed + (m == 0 ? kTrBwdWa : kTrBwdWb))[row * 32 + lane] = ov;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) d += __shfl_xor_sync(0xFFFFFFFFu, d, off);
    if (lane == 0) reinterpret_cast<float*>(packed + kTrBwdConst)[m * 512 + row] = d;
  } else {
    // Ws [128][512]: warp gw - 1024 (0 .. 511) converts 128 consecutive elements
    const size_t base = static_cast<size_t>(gw - 1024) * 128;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const size_t i = base + lane * 4 + t;
      const float v = tr_load_w(a.w_s, i, a.f32_weights);
      reinterpret_cast<uint16_t*>(packed + kTrBwdWs)[i] = __half_as_ushort(__float2half_rn(fminf(fmaxf(v, -65504.f), 65504.f)));
    }
  }
}

// One launch before the backward kernels: the first kTrBwdPackBlocks blocks pack the weights (eight rows each), the rest
// find max |dy| and the scale.
constexpr int kTrBwdPackBlocks = 1536 / 8;
struct TrBwdSetupArgs {
  TrBwdPackArgs w;
  uint8_t* packed;
  const uint4* dy;
  size_t n_chunks;
  unsigned int* words;
  float* scale;
};
__global__ void __launch_bounds__(256) tr_bwd_setup_kernel(const __grid_constant__ TrBwdSetupArgs a) {
  grid_dependents_launch();
  if (blockIdx.x < kTrBwdPackBlocks) {
    tr_bwd_pack_row(a.w, a.packed, blockIdx.x * 8 + (threadIdx.x >> 5));
    return;
  }
  amax_and_scale(a.dy, a.n_chunks, blockIdx.x - kTrBwdPackBlocks, gridDim.x - kTrBwdPackBlocks, a.words, a.scale);
}

// Parameter gradients of the Transition from the per-CTA partials of the four launches j:
//   part_m [4][n_parts][3] matrices (Ma_j, Mb_j: [hidden][k]; dWs_j: [c][hidden]), part_s [4][n_parts][2][512]
//   (column sums in the first 128 entries)
//   dWa[j*128+r][k] = (Ma_j[r][k] gamma[k] + sa_j[r] beta[k]) / c, dWb likewise, dWs[c][j*128+h] = dWs_j[c][h] / c
//   dgamma[k] = sum_j sum_r (Wa Ma + Wb Mb) / c,  dbeta[k] = sum_j sum_r (Wa sa + Wb sb) / c
// Grid (384, 4 blocks j): 256 blocks (group of four columns, 16 rows) of Ma and Mb, whose LayerNorm terms are one chain over
// both, and 128 blocks (group of four columns, 32 rows) of dWs; as bwd_finalize_kernel. The terms [4][8][2][128] are added by
// tr_bwd_final_ln_kernel. (A reduction per launch and a gradient kernel on 4 x 8 blocks were 4 x 5.9 + 22.4 us.)
struct TrBwdFinalArgs {
  TrBwdPackArgs w;
  const float* part_m;
  const float* part_s;
  int n_parts;
  const float* scale;
  float* d_wa;     // [512][128]
  float* d_wb;     // [512][128]
  float* d_ws;     // [128][512]
  float* ln_rows;  // [4][8][2][128]
  float* d_ln[2];  // dgamma, dbeta [128]
};
__global__ void __launch_bounds__(512) tr_bwd_final_kernel(const __grid_constant__ TrBwdFinalArgs a) {
  grid_dependency_wait();
  grid_dependents_launch();
  const bool squeeze = blockIdx.x >= 256;
  const int lane = threadIdx.x & 31, j = blockIdx.y;
  const int group = squeeze ? (blockIdx.x - 256) >> 2 : blockIdx.x >> 3, k0 = group * 4;
  const int rb = blockIdx.x & 7;  // 16 rows of Ma (lanes 0-15) and Mb (lanes 16-31)
  const int m = squeeze ? 2 : lane >> 4, r = squeeze ? (blockIdx.x & 3) * 32 + lane : rb * 16 + (lane & 15);
  const float* parts = a.part_m + (static_cast<size_t>(j) * a.n_parts * 3 + m) * 128 * 128 + (group * 128 + r) * 4;
  const float* sums = squeeze ? nullptr : a.part_s + (static_cast<size_t>(j) * a.n_parts * 2 + m) * 512 + r;
  float4 m4;
  float s1;
  sum_partials_of_rows(parts, 3 * 128 * 128, sums, 2 * 512, a.n_parts, m4, s1);
  if (threadIdx.x >= 32) return;
  const float cinv = a.scale[1];
  const float sv = s1 * cinv, mv[4] = {m4.x * cinv, m4.y * cinv, m4.z * cinv, m4.w * cinv};
  if (squeeze) {
    float* dst = a.d_ws + static_cast<size_t>(r) * 512 + j * 128 + k0;
#pragma unroll
    for (int t = 0; t < 4; ++t) dst[t] = mv[t];
    return;
  }
  const size_t wi = static_cast<size_t>(j * 128 + r) * 128 + k0;
  float* dst = (m == 0 ? a.d_wa : a.d_wb) + wi;
  __shared__ LnRow rows[32];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    dst[t] = fmaf(mv[t], a.w.ln_w[k0 + t], sv * a.w.ln_b[k0 + t]);
    rows[lane].w[t] = tr_load_w(m == 0 ? a.w.w_a : a.w.w_b, wi + t, a.w.f32_weights);
    rows[lane].mv[t] = mv[t];
  }
  rows[lane].sv = sv;
  __syncwarp();
  if (lane < 4) {
    float ag = 0.f, ab = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const LnRow &x = rows[i], &y = rows[16 + i];
      ag = fmaf(x.w[lane], x.mv[lane], fmaf(y.w[lane], y.mv[lane], ag));
      ab = fmaf(x.w[lane], x.sv, fmaf(y.w[lane], y.sv, ab));
    }
    float* terms = a.ln_rows + (j * 8 + rb) * 256 + k0 + lane;
    terms[0] = ag, terms[128] = ab;
  }
}
__global__ void __launch_bounds__(256) tr_bwd_final_ln_kernel(const TrBwdFinalArgs a) {
  grid_dependency_wait();
  grid_dependents_launch();
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < 32; ++i) s += __ldcg(a.ln_rows + i * 256 + threadIdx.x);
  a.d_ln[threadIdx.x >> 7][threadIdx.x & 127] = s;
}

}  // namespace trimul
