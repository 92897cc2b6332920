// Fused prologue: input LayerNorm + left/right gated projections + sigmoid gate + pair mask.
//
//   x_hat = LayerNorm_in(z)  (fp32 statistics, affine applied, rounded once to fp16 for the tensor cores:
//                             |x_hat| <= sqrt(127) |gamma| + |beta| fits easily and keeps three more
//                             mantissa bits than bf16; the packed weights are fp16 too)
//   left  = sigmoid(x_hat Wlg^T + blg) * (x_hat Wl^T + bl) * valid(i,k)      (biases optional)
//   right = likewise with Wrg, Wr
//
// Packed weights are fp16(0.5 * W) and d = 0.5 * bias, so that
// sigmoid(g) * p = (tanh(g/2) + 1) * (p/2) costs one MUFU op and one FMA per output.
//
// Persistent CTA pairs (tcgen05 cta_group::2), one pair per two SMs, walk tiles of 128 consecutive columns j
// of one pair row (b, i). The GEMMs are issued as D^T[h, pos] = W[h, c] * x_hat^T[c, pos], so TMEM lanes are
// channels and columns are positions: each epilogue thread owns one channel and writes runs of consecutive
// positions, which is exactly the row-plane layout [B, rows, H, N] of the outputs (written as fp16; masked
// cells are exactly zero).
//
// The two CTAs of a pair split the OUTPUTS: CTA 0 produces `left`, CTA 1 `right`, each holding only its own two matrices.
// These stay in TENSOR MEMORY as the A operand of every MMA (128 columns), so the tensor cores read nothing but the
// normalised tile from shared memory, which eight input stages and four staging buffers share. A tile is processed as two
// halves of 64 positions, because the other 384 columns hold three accumulator buffers of a half (value and gate, 64 columns
// each) but not two of a whole tile. Every MMA spans both CTAs (M = 256: rows 0-127 CTA 0's matrix, rows 128-255 CTA 1's;
// N = 64 positions, of which each CTA loads and normalises 32). So per half tile each CTA
//   * loads and LayerNorms 32 positions,
//   * receives proj / gate accumulators of ITS output for all 64 positions in its own TMEM (the MMAs of the next halves
//     overlap the epilogue of this one),
//   * gates, masks and stores 128 channels x 64 positions of its output.
// Only mbarrier signals cross between the CTAs (statistics-done and accumulator-free arrive on the leader's
// barriers; the leader's MMA commits release both CTAs' barriers); no tile is broadcast. A single-CTA version
// of this kernel (all four matrices resident, two input stages) measured 3 % slower at N = 768.
//
// What bounds it: per SM the tensor pipe and the MUFU (tanh) are busy for half of the time each, 60 % of the issue slots and
// 0.75 of the copy rate of HBM are used; the stages of the pipeline take turns at these. With the matrices in shared memory
// (128-position tiles, two accumulator buffers, five input stages) the MMAs' operand reads held up the other roles: leaving
// out most MMAs gained 18 us of 95. Now 94.8 -> 91.4 us at N = 768, 28.3 -> 27.4 at N = 384, 84.3 -> 81.2 for 8 x 256 in
// short runs (whole forwards 1 %; at N = 768 in sustained calls, which run at the power limit, no change). The 64-column
// MMAs pay only because their issuer runs on an elected lane (113 us otherwise).
//
// Outputs leave through a swizzled shared-memory staging tile and TMA stores (full 128-byte rows);
// direct per-thread 16-byte stores to 128 different channel rows ran the store path at a third of this.
//
// Warp roles (864 threads per CTA):
//   warp 0        TMA producer (input tiles)
//   warp 1        MMA issuer (leader CTA) / TMEM owner
//   warps 2-9     LayerNorm: 8 threads per position (16 channels each, their gamma / beta in registers), two
//                 passes of 32 positions computed as independent chains; normalises the tile in place.
//   warps 10-25   epilogue: four groups of four warps take half tiles in turn (one thread per channel x 64 positions:
//                 TMEM -> tanh gate -> mask -> staging -> TMA store); at the start they bring the weights to TMEM
//   warp 26       validity bitmap of the tile
#pragma once

#include "pack.cuh"
#include "ptx.cuh"

namespace trimul {

struct PrologueParams {
  int batch;           // B
  int rows;            // pair rows per sample handled by this call
  int n;               // tokens N (columns per row)
  int row_offset;      // global index of local row 0 (token-mask lookup)
  int tiles_per_row;   // ceil(N / 128)
  int num_tiles;       // B * rows * tiles_per_row
  const uint8_t* token_mask;  // [B, N] non-zero = valid, or null
  const uint8_t* pair_mask;   // [B, rows, N] non-zero = valid, or null
  // Where this kernel's matrices come from. raw = 0: `w`, the packed block of an earlier launch. raw = 1: the parameters
  // themselves (block `raw_block` of the kernel's PackLaunch), which with z, the masks and the LayerNorm parameters below are
  // older than the kernel before this one; then this launch also packs what the epilogue reads (matrices 4 and 5 of block 0,
  // matrix 4 of block 1; `pack_blocks` of them) and, if it packs anything, clears the status words of the call. The kernel with
  // LEAVES, for launches that pack, fills the rest of block 0.
  int raw, raw_block, pack_blocks;
  const uint4* w;             // [4][128][C] fp16 packed matrices: left, left gate, right, right gate
  const float* d1;            // [4][128] additive constants (0.5 * bias): left, left gate, right, right gate
  const float* ln_w;          // [128] LayerNorm gamma
  const float* ln_b;          // [128] LayerNorm beta
  float eps;
  int* status;
};

// Where the outputs go. Each output has a list of destination tensor maps; a finished tile [128 channels][128
// positions] of local row r is stored to every destination d of its list at row r + row_shift, taking the
// channels d * smem_step / 128 ... of the staging tile (smem_step = 0: every destination gets all 128 channels).
//   one GPU:            one destination per output, the [B*rows, 128, N] buffers, row_shift 0
//   rows over GPUs:     `right` additionally to the peers' gathered copies [N, 128, N] (row_shift = first local row)
//   channels over GPUs: destination d = the GPU that contracts channel group d; it receives the 128/P channels of
//                       its group for this GPU's rows, in its [N, 128/P, N] buffer (smem_step = 128/P channel rows)
// Peer destinations are plain (non-multicast) TMA stores over NVLink; they replace a separate collective pass.
constexpr int kMaxDst = 8;
struct OutputMaps {
  CUtensorMap left[kMaxDst];
  CUtensorMap right[kMaxDst];
  int n_left, n_right;
  int step_left, step_right;    // bytes between the destinations' channel slices in a 16 KiB half staging tile
  int shift_left, shift_right;  // added to the row coordinate
  // One GPU: the same two outputs with a box of 32 channel rows, so that every epilogue warp stores the 32 rows it
  // wrote by itself and the warps of a group never wait for one another (warp_store != 0).
  CUtensorMap left_warp, right_warp;
  int warp_store;
};

constexpr int kProThreads = 864;
constexpr int kProStages = 8;
constexpr int kProRing = kProStages + 4;  // mask ring entries: the input may run so many tiles ahead of an epilogue group
constexpr int kProRingBytes = 272;        // 64 pair-mask words + 4 ballots
constexpr int kProStageOutBytes = 4 * 16384;  // per epilogue group a staging buffer of [128 channels][64 positions]
constexpr int kProBarBytes = 320;
constexpr int kProAccs = 3;       // accumulator buffers (of a 64-position half tile: value and gate, 64 columns each)
constexpr int kProGroups = 4;     // epilogue groups
constexpr int kProAccBase = 128;  // tensor-memory column of the first one, behind the two weight matrices
// C = d_pair, the channels of the input tensor (128, or 64 for the narrow pair stacks); the outputs always have 128
// channels. The shared-memory budget is that of C = 128 for both.
constexpr int kProSmemBytes = kProStages * 16384 + kProStageOutBytes + kProRing * kProRingBytes + kProBarBytes + 1024;

template <bool HAS_BIAS, int C = 128, bool LEAVES = false>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kProThreads, 1)
prologue_kernel(const __grid_constant__ CUtensorMap map_z, const __grid_constant__ OutputMaps out,
                const __grid_constant__ PackLaunch params, const PrologueParams p) {
  static_assert(C == 128 || C == 64, "d_pair is 128 or 64");
  constexpr int S = kProStages;
  constexpr int kHalves = C / 64;              // 64-channel (128-byte) halves of an input row
  constexpr int kProZBytes = 64 * C * 2;       // 64 positions x C channels, 16-bit
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t z_base = smem_base;
  const uint32_t stage_out_base = z_base + S * kProZBytes;
  const uint32_t ring_base = stage_out_base + kProStageOutBytes;
  const uint32_t bar_base = ring_base + kProRing * kProRingBytes;
  uint32_t* ring_ptr = reinterpret_cast<uint32_t*>(smem + S * kProZBytes + kProStageOutBytes);
  // barriers: w_full (leader), z_full[S] (own), xn_ready[S] (leader), z_empty[S] (both), acc_full[4] (both, one per
  // epilogue group, which so sees every phase of its barrier), acc_empty[3] (leader)
  const uint32_t w_full = bar_base;
  auto z_full = [&](int s) { return bar_base + 8u * (1 + s); };
  auto xn_ready = [&](int s) { return bar_base + 8u * (1 + S + s); };
  auto z_empty = [&](int s) { return bar_base + 8u * (1 + 2 * S + s); };
  auto acc_full = [&](int g) { return bar_base + 8u * (1 + 3 * S + g); };
  auto acc_empty = [&](int a) { return bar_base + 8u * (1 + 3 * S + kProGroups + a); };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + S * kProZBytes + kProStageOutBytes +
                                                    kProRing * kProRingBytes + 8 * (1 + 3 * S + kProGroups + kProAccs));
  static_assert(8 * (1 + 3 * S + kProGroups + kProAccs) + 8 <= kProBarBytes, "barriers");
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();  // 0: leader, produces `left`; 1: produces `right`
  const int pair = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    mbar_init(w_full, 32);  // the sixteen epilogue warps of each CTA
    for (int s = 0; s < S; ++s) {
      mbar_init(z_full(s), 1);
      mbar_init(xn_ready(s), 18);  // eight LayerNorm warps and the mask warp of each CTA
      mbar_init(z_empty(s), 1);
    }
    for (int g = 0; g < kProGroups; ++g) mbar_init(acc_full(g), 1);
    for (int a = 0; a < kProAccs; ++a) mbar_init(acc_empty(a), 8);  // the four warps of an epilogue group in each CTA
    *abort_flag = 0;
    fence_mbar_init();
    prefetch_tmap(&map_z);
    prefetch_tmap(&out.left[0]);
    prefetch_tmap(&out.right[0]);
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(tmem_slot), 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // barriers of both CTAs are initialised before any signal crosses
  tc_fence_after();
  // A call's first launch may follow any kernel. With the call's arguments as the inputs of a later one only the warps that
  // store wait for the kernel before it, behind their share of the weights.
  if (!p.raw || p.pack_blocks > 0) {
    grid_dependency_wait();
    grid_dependents_launch();
  }
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs)
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0;
      int issued = 0;
      for (int tile = pair; tile < p.num_tiles; tile += num_pairs) {
        if (!mbar_wait(z_empty(s), ph ^ 1u, abort_flag, p.status, kDevTimeoutProducer)) break;
        const int row = tile / p.tiles_per_row;
        // this CTA's 64 positions: of each 64-position half of the tile the 32 that are its rows of the B operand
        const int j0 = (tile - row * p.tiles_per_row) * 128 + static_cast<int>(rank) * 32;
        mbar_arrive_expect_tx(z_full(s), kProZBytes);
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int kh = 0; kh < kHalves; ++kh)
            tma_load_3d(z_base + s * kProZBytes + kh * 8192 + u * 4096, &map_z, z_full(s), kh * 64, j0 + u * 64, row);
        ++issued;
        if (++s == S) {
          s = 0;
          ph ^= 1u;
        }
      }
      // Drain every copy this thread started before the CTA may exit.
      const int pending = issued < S ? issued : S;
      for (int q = 0; q < pending; ++q) {
        if (s == 0) {
          s = S;
          ph ^= 1u;
        }
        --s;
        const long long t0 = clock64();
        while (!mbar_try_wait(z_full(s), ph)) {
          if (clock64() - t0 > kWaitLimitCycles) {
            atomicCAS(p.status, 0, kDevTimeoutDrain);
            break;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (leader CTA only)
    if (rank != 0 && p.pack_blocks > 0) {
      // in the other CTA this warp packs what the epilogue reads
      if (pair == 0 && lane < 16) p.status[lane] = 0;
#pragma unroll 4
      for (int r = pair; r < (p.pack_blocks > 1 ? 384 : 256); r += num_pairs)
        pack_matrix_row(params.block[r >> 8], params.packed[r >> 8], 512 + (r & 255));
    }
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc = umma_idesc(256, 64, false, false, kFmtF16, kFmtF16);
      bool ok = mbar_wait(w_full, 0, abort_flag, p.status, kDevTimeoutMma);
      int s = 0;
      uint32_t ph = 0;
      int a = 0;  // accumulator buffer of the next half tile
      uint32_t aph = 1u;
      int g = 0;  // its epilogue group: 0, 2 before its tile's two halves
      for (int tile = pair; ok && tile < p.num_tiles; tile += num_pairs, g ^= 2) {
        if (!mbar_wait(xn_ready(s), ph, abort_flag, p.status, kDevTimeoutMma)) break;
        const uint64_t db0 = umma_desc_kmajor(z_base + s * kProZBytes);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          ok = mbar_wait(acc_empty(a), aph, abort_flag, p.status, kDevTimeoutMma);
          if (!ok) break;
          tc_fence_after();
#pragma unroll
          for (int m = 0; m < 2; ++m) {
            const uint32_t d_tmem = tmem_base + kProAccBase + a * 128 + m * 64;
            const uint32_t wm = tmem_base + m * (C / 2);
#pragma unroll
            for (int ks = 0; ks < C / 16; ++ks) {
              const uint64_t db = db0 + static_cast<uint64_t>((ks >> 2) * 512 + u * 256 + (ks & 3) * 2);
              umma_pair_ta(d_tmem, wm + ks * 8, db, idesc, ks != 0 ? 1u : 0u);
            }
          }
          umma_commit_pair(acc_full(g + u));
          if (++a == kProAccs) {
            a = 0;
            aph ^= 1u;
          }
        }
        if (!ok) break;
        umma_commit_pair(z_empty(s));
        if (++s == S) {
          s = 0;
          ph ^= 1u;
        }
      }
    }
  } else if (warp < 10) {
#include "prologue_stats.inc"
  } else if (warp < 26) {
#include "prologue_epilogue.inc"
  } else {
#include "prologue_mask.inc"
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // neither CTA leaves while the other may still signal its barriers or read its operands
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

}  // namespace trimul
