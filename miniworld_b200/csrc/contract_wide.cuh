// Triangle contraction with CTA pairs and output tiles of up to 256 x 512.
//
// Same math, layouts and signals as contract_pair.cuh. A tile `bn` (at most 512) columns wide takes 128 + bn / 2 operand rows
// per CTA and k block instead of 256 for every 256 columns (17 % fewer bytes from L2 at 384, 25 % at 512; a third fewer than
// two to four tiles of 128 columns). Widths are multiples of 128, and the last tile of a row is only as wide as the columns
// that are left, so that a row of 640 or 896 columns is not cut into 128-column tiles to avoid padding. The accumulator
// fills tensor memory, so there is one: two parts, columns 0-255 and the rest, which the epilogue warps hand back as soon as
// they have them in registers; the four stages that load meanwhile cover that gap (two accumulators for tiles of 256 columns
// measured the same). What bounds it: DRAM and L2 up to N = 1024, the tensor pipe at the power limit from there on.
// Contraction alone (before, 256- or 128-column pair tiles or 128 x 256 ones of one CTA -> these): N = 640 88 -> 82 us,
// 896 217 -> 180, 1152 423 -> 336, 1408 740 -> 579, 1920 1775 -> 1490, 2048 incoming 1570 -> 1508 (outgoing it is slower there, see contract_plan).
#pragma once

#include "contract_pair.cuh"

namespace trimul {

constexpr int kWideStages = 4;
constexpr int kWideMaxN = 512;
constexpr int kWideStageBytes = kBM * kBK * 2 + (kWideMaxN / 2) * kBK * 2;
constexpr int kWideContractThreads = 320;  // producer, MMA issuer, eight epilogue warps
constexpr int kWideContractSmem = kWideStages * kWideStageBytes + 8 * 4096 /* a staging buffer per warp */ + 256 + 1024;

template <int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kWideContractThreads, 1)
contract_wide_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                     const __grid_constant__ CUtensorMap map_t, const ContractParams p) {
  constexpr int S = kWideStages;
  constexpr bool A_MN = MODE == kContractIncoming;  // A operand MN-major (its k index is the tensor's row)
  constexpr bool B_MN = MODE != kContractOutgoing;  // B operand MN-major

  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t staging_base = smem_base + kWideStages * kWideStageBytes;
  const uint32_t bar_base = staging_base + 8 * 4096;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (S + s); };
  auto tfull_bar = [&](int j) { return bar_base + 8u * (2 * S + j); };
  auto tempty_bar = [&](int j) { return bar_base + 8u * (2 * S + 2 + j); };
  uint8_t* smem_aligned = smem_raw + (smem_base - smem_u32(smem_raw));
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_aligned + kWideStages * kWideStageBytes + 8 * 4096 + 8 * (2 * S + 4));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();  // 0 = leader (issues the MMAs)
  const int pair = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int j = 0; j < 2; ++j) {
      mbar_init(tfull_bar(j), 1);
      mbar_init(tempty_bar(j), 16);  // eight epilogue warps in each of the two CTAs
    }
    *abort_flag = 0;
    fence_mbar_init();
    prefetch_tmap(&map_a);
    prefetch_tmap(&map_b);
    prefetch_tmap(&map_t);
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(tmem_slot), 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // barriers of both CTAs are initialised before any signal crosses
  tc_fence_after();
  grid_dependency_wait();
  grid_dependents_launch();
  const uint32_t tmem_base = *tmem_slot;

  const int tiles_per_plane = p.m_tiles * p.n_tiles;
  const int num_tiles = p.planes * tiles_per_plane;
  struct Tile {
    int m0, n0, hh, bb;  // this CTA's first row, the tile's first column, plane
    int w0, w1;          // columns of the two parts (multiples of 128 or 0)
  };
  auto place = [&](int tile) {
    const int plane = tile / tiles_per_plane;
    const int r = tile - plane * tiles_per_plane;
    const int mt = r / p.n_tiles;
    Tile t;
    t.bb = plane / p.H;
    t.hh = plane - t.bb * p.H;
    t.m0 = mt * 256 + static_cast<int>(rank) * kBM;
    t.n0 = (r - mt * p.n_tiles) * p.bn;
    const int left = (p.n_cols - t.n0 + 127) / 128 * 128;
    const int w = left < p.bn ? left : p.bn;
    t.w0 = w < 256 ? w : 256;
    t.w1 = w - t.w0;
    return t;
  };

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs)
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0;
      int issued = 0;
      bool ok = true;
      for (int tile = pair; ok && tile < num_tiles; tile += num_pairs) {
        const Tile t = place(tile);
        const uint32_t bytes = 2u * (kBM * kBK * 2 + (t.w0 + t.w1) / 2 * kBK * 2);  // of both CTAs
        for (int kb = 0; kb < p.num_kb; ++kb) {
          if (!mbar_wait(empty_bar(s), ph ^ 1u, abort_flag, p.status, kDevTimeoutProducer)) {
            ok = false;
            break;
          }
          if (rank == 0) mbar_arrive_expect_tx(full_bar(s), bytes);
          const uint32_t lead_full = map_to_cta(full_bar(s), 0);
          const uint32_t sa = smem_base + s * kWideStageBytes;
          const uint32_t sb = sa + kBM * kBK * 2;
          const int k0 = kb * kBK;
          if constexpr (!A_MN) {
            tma_load_4d_pair(sa, &map_a, lead_full, k0, t.m0, t.hh, t.bb);
          } else {
#pragma unroll
            for (int hf = 0; hf < kBM / 64; ++hf)
              tma_load_4d_pair(sa + hf * 8192, &map_a, lead_full, p.a_col_off + t.m0 + 64 * hf, k0, t.hh, t.bb);
          }
          // this CTA's half of each part of B, in boxes of 64 of its columns
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const int w = j == 0 ? t.w0 : t.w1;
            const int n = t.n0 + j * 256 + static_cast<int>(rank) * (w / 2);
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
              if (hf * 128 >= w) break;
              if constexpr (!B_MN)
                tma_load_4d_pair(sb + j * 16384 + hf * 8192, &map_b, lead_full, k0, n + 64 * hf, t.hh, t.bb);
              else
                tma_load_4d_pair(sb + j * 16384 + hf * 8192, &map_b, lead_full, n + 64 * hf, k0, t.hh, t.bb);
            }
          }
          ++issued;
          if (++s == S) {
            s = 0;
            ph ^= 1u;
          }
        }
      }
      // Drain (leader: its `full` barriers count the bytes of both CTAs; the closing cluster barrier keeps the
      // other CTA alive until then).
      if (rank == 0) {
        const int pending = issued < S ? issued : S;
        for (int q = 0; q < pending; ++q) {
          if (s == 0) {
            s = S;
            ph ^= 1u;
          }
          --s;
          const long long t0 = clock64();
          while (!mbar_try_wait(full_bar(s), ph)) {
            if (clock64() - t0 > kWaitLimitCycles) {
              atomicCAS(p.status, 0, kDevTimeoutDrain);
              break;
            }
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (leader CTA only)
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc_0 = umma_idesc(256, 0, A_MN, B_MN, kFmtF16, kFmtF16);
      constexpr uint32_t kstep_a = A_MN ? (2048 >> 4) : (32 >> 4);
      constexpr uint32_t kstep_b = B_MN ? (2048 >> 4) : (32 >> 4);
      int s = 0;
      uint32_t ph = 0;
      uint32_t free_ph[2] = {1u, 1u};  // parities of the next hand-back of either part
      bool ok = true;
      for (int tile = pair; ok && tile < num_tiles; tile += num_pairs) {
        const Tile t = place(tile);
        for (int kb = 0; ok && kb < p.num_kb; ++kb) {
          ok = mbar_wait(full_bar(s), ph, abort_flag, p.status, kDevTimeoutMma);
          if (!ok) break;
          tc_fence_after();
          const uint32_t sa = smem_base + s * kWideStageBytes;
          const uint32_t sb = sa + kBM * kBK * 2;
          const uint64_t da = A_MN ? umma_desc_mnmajor(sa, 8192) : umma_desc_kmajor(sa);
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const int w = j == 0 ? t.w0 : t.w1;
            if (w == 0) continue;
            if (kb == 0) {  // the part's last tile has left tensor memory
              ok = mbar_wait(tempty_bar(j), free_ph[j], abort_flag, p.status, kDevTimeoutMma);
              if (!ok) break;
              free_ph[j] ^= 1u;
              tc_fence_after();
            }
            const uint64_t db = B_MN ? umma_desc_mnmajor(sb + j * 16384, 8192) : umma_desc_kmajor(sb + j * 16384);
            const uint32_t idesc = idesc_0 | static_cast<uint32_t>(w >> 3) << 17;
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k)
              umma_pair(tmem_base + j * 256, da + static_cast<uint64_t>(k * kstep_a), db + static_cast<uint64_t>(k * kstep_b),
                        idesc, (kb | k) != 0 ? 1u : 0u);
            if (kb == p.num_kb - 1) umma_commit_pair(tfull_bar(j));
          }
          if (!ok) break;
          umma_commit_pair(empty_bar(s));
          if (++s == S) {
            s = 0;
            ph ^= 1u;
          }
        }
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue warps (2..9), both CTAs
    // Two warps per TMEM lane quarter share a part's columns in groups of 64 and take every group of theirs out of tensor
    // memory before they convert and store the first; each stores its own 32 rows.
    const int q = warp & 3;
    const int hs = (warp - 2) >> 2;
    const uint32_t buf = staging_base + (warp - 2) * 4096u;
    const uint32_t t_acc = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    uint32_t full_ph[2] = {0u, 0u};
    bool ok = true;
    for (int tile = pair; ok && tile < num_tiles; tile += num_pairs) {
      const Tile t = place(tile);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int w = j == 0 ? t.w0 : t.w1;
        if (w == 0) continue;
        ok = mbar_wait_warp(tfull_bar(j), full_ph[j], abort_flag, p.status, kDevTimeoutEpilogue);
        if (!ok) break;
        full_ph[j] ^= 1u;
        tc_fence_after();
        uint32_t v[4][32];
        tmem_ld32(t_acc + j * 256 + hs * 64, v[0]);
        tmem_ld32(t_acc + j * 256 + hs * 64 + 32, v[1]);
        if (w == 256) {
          tmem_ld32(t_acc + j * 256 + 128 + hs * 64, v[2]);
          tmem_ld32(t_acc + j * 256 + 128 + hs * 64 + 32, v[3]);
        }
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_leader(tempty_bar(j), rank);
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          const int col0 = t.n0 + j * 256 + g * 128 + hs * 64;
          if (g * 128 >= w || col0 >= p.n_cols || t.m0 + q * 32 >= p.m_rows) break;
          if (lane == 0) bulk_wait_read<0>();  // this warp's previous store has read its buffer
          __syncwarp();
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const uint32_t(&x)[32] = v[2 * g + (c >> 2)];
            const int e = (c & 3) * 8;
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(buf + lane * 128 + ((c ^ (lane & 7)) << 4)),
                         "r"(pack_tri(x[e], x[e + 1])), "r"(pack_tri(x[e + 2], x[e + 3])), "r"(pack_tri(x[e + 4], x[e + 5])),
                         "r"(pack_tri(x[e + 6], x[e + 7]))
                         : "memory");
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_4d(&map_t, buf, col0, t.m0 + q * 32, t.hh, t.bb);
            bulk_commit();
          }
        }
      }
    }
    if (lane == 0) bulk_wait<0>();
    __syncwarp();
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
