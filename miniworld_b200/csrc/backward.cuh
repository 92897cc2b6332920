// Backward of the triangle update around the contraction: the epilogue's gradients (output LayerNorm, output
// projection, output gate) and the prologue's gradients (input LayerNorm, the four gated projections, the mask).
//
// Both kernels walk tiles of 128 consecutive columns j of one pair row, one CTA per SM: 16 arithmetic warps (four threads per
// position or channel, its TMEM lane, each covering a quarter of the other dimension), a warp that issues the MMAs and one
// that issues the TMA copies. Per tile:
//   1. the inputs arrive; the epilogue's backward normalises t and z in place (fp16) and leaves x_hat and 1 / sigma for the
//      prologue's backward,
//   2. the forward GEMMs are recomputed on the tensor cores (weights with the LayerNorm gamma folded in, fp16),
//   3. the threads turn the upstream gradient into the gradients of the GEMM outputs (fp16 tiles in shared memory),
//   4. the tensor cores compute, from those tiles, the gradients with respect to the normalised inputs (the same weight
//      tiles read MN-major) and accumulate the weight gradients M = dOut^T x_hat over all tiles of the CTA in TMEM,
//   5. the threads finish (LayerNorm backward) and the results leave through TMA stores.
// The four tile buffers of a CTA rotate their roles from tile to tile: the next tile's inputs are copied into the
// buffers the gradient GEMMs have finished with while the tile completes, and a store is only waited for when its
// buffer is needed again. Column sums of the dOut tiles (the bias-like terms) are accumulated per thread in
// registers. At the end every CTA writes its partial M and column sums; one pass over the partials of all launches forms
// the parameter gradients. Both kernels are templates on the input width C (128, or 64 for the narrow pair stacks); the
// epilogue's backward also has a two-launch form for an output LayerNorm over 256 channels (the bidirectional module).
//
// Gradients travel in fp16 tiles, so the upstream gradient is multiplied by a power of two c (read from device
// memory, chosen from max |dy| by `amax_and_scale`); every output of these kernels carries that
// factor, and the final kernels divide it out in fp32.
#pragma once

#include "ptx.cuh"

namespace trimul {

// threads per position, each covering 128 / kBwdParts channels. Not a knob: 16 warps (four per TMEM lane quarter, eight for each
// of t and z), 32 positions per thread and 32 groups of four rows are written into the kernels.
constexpr int kBwdParts = 4;
constexpr int kBwdThreads = 128 * kBwdParts;
constexpr int kBwdCh = 128 / kBwdParts;          // channels per thread of a 128-channel tile
constexpr int kBwdChunks = kBwdCh / 8;           // 16-byte chunks (8 channels) per thread
constexpr int kBwdTile = 32768;  // one [128][128] 16-bit tile
constexpr int kBwdXchg = kBwdParts * 128 * 8;  // float2 [kBwdParts][128]

// [128 rows][128 elements] 16-bit tiles are stored as two halves of 64 elements, each [128 rows][128 bytes] with the 128-byte
// TMA swizzle:
// offset of the 16-byte chunk holding elements 8*ch .. 8*ch+7 (ch = 0..15) of row r
__device__ __forceinline__ uint32_t tile_chunk(int r, int ch) {
  return static_cast<uint32_t>((ch >> 3) * 16384 + r * 128 + (((ch & 7) ^ (r & 7)) << 4));
}

// offset of element e of row r
__device__ __forceinline__ uint32_t tile_off(int r, int e) {
  return static_cast<uint32_t>((e >> 6) * 16384 + r * 128 + ((((e & 63) >> 3) ^ (r & 7)) << 4) + (e & 7) * 2);
}

__device__ __forceinline__ uint32_t ld_word(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ void st_word(uint32_t addr, uint32_t v) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
__device__ __forceinline__ uint32_t ld_half(uint32_t addr) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint4 ld_chunk(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ void st_chunk(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// 32 bytes per thread in one request (address 32-byte aligned): a warp whose lanes read different 128-byte lines pays
// per line and request, so half as many requests as with 16-byte loads
__device__ __forceinline__ void ldg_32B(const void* p, uint4& a, uint4& b) {
  asm volatile("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
               : "l"(p));
}
// `chunks` 16-byte pieces (an even count) from p: 32-byte requests if the address allows, else 16-byte ones
template <int CHUNKS>
__device__ __forceinline__ void ldg_chunks(const uint4* p, bool wide, uint4 (&out)[CHUNKS]) {
  static_assert(CHUNKS % 2 == 0, "pairs of 16-byte chunks");
  if (wide) {
#pragma unroll
    for (int c = 0; c < CHUNKS; c += 2) ldg_32B(p + c, out[c], out[c + 1]);
  } else {
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) out[c] = __ldg(p + c);
  }
}
__device__ __forceinline__ float sigmoid_fast(float x) { return fmaf(tanh_approx(0.5f * x), 0.5f, 0.5f); }

// (see mbar_wait_thread: a thread that gives up sets the abort word and carries on)
__device__ __forceinline__ bool thread_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status, int code) {
  return mbar_wait_thread(bar, parity, abort_flag, status, code);
}
// LayerNorm statistics of a position from the kBwdParts threads that hold a part of its channels each. The order of the additions
// is part of the results (they are repeatable bit for bit): shifted sums over a part's channels in order, then the parts.
// Mean and sum of squared deviations of 8 * CHUNKS bf16 channels.
template <int CHUNKS>
__device__ __forceinline__ float2 partial_statistics(const uint4 (&v)[CHUNKS]) {
  float pv = 0.f, s1 = 0.f, s2 = 0.f;
#pragma unroll
  for (int ch = 0; ch < CHUNKS; ++ch) {
    const uint32_t w[4] = {v[ch].x, v[ch].y, v[ch].z, v[ch].w};
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const float2 x = bf16x2_to_float2(w[t]);
      if (ch == 0 && t == 0) pv = x.x;
      const float d0 = x.x - pv, d1 = x.y - pv;
      s1 += d0 + d1;
      s2 = fmaf(d0, d0, fmaf(d1, d1, s2));
    }
  }
  constexpr float kInv = 1.0f / (8 * CHUNKS);
  return make_float2(pv + s1 * kInv, fmaxf(s2 - s1 * s1 * kInv, 0.f));
}
// Mean and 1 / sigma of position `pos` from the equal-sized partials (CH channels each) in `xchg` (float2 [kBwdParts][128]):
// mean of means, M2 = sum M2_k + n_k sum (mean_k - mean)^2.
template <int CH>
__device__ __forceinline__ float2 merge_partials(uint32_t xchg, int pos, float eps) {
  float mk[kBwdParts], qk[kBwdParts];
  float mean = 0.f, m2 = 0.f;
#pragma unroll
  for (int k = 0; k < kBwdParts; ++k) {
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(mk[k]), "=f"(qk[k]) : "r"(xchg + (k * 128 + pos) * 8));
    mean += mk[k];
    m2 += qk[k];
  }
  mean *= 1.0f / kBwdParts;
#pragma unroll
  for (int k = 0; k < kBwdParts; ++k) m2 = fmaf(static_cast<float>(CH) * (mk[k] - mean), mk[k] - mean, m2);
  return make_float2(mean, rsqrtf(m2 * (1.0f / (CH * kBwdParts)) + eps));
}
// Normalise the 128 channels of every position of a [pos][c] tile in place (bf16 in, fp16 out), the thread covering
// 128 / kBwdParts of them. Returns rstd of the thread's position. `xchg` holds float2 [kBwdParts][128]; the caller must not
// use it again without a barrier among the arithmetic threads.
__device__ __forceinline__ float normalise_tile(uint32_t tile, uint32_t xchg, int pos, int part, float eps) {
  uint4 v[kBwdChunks];
#pragma unroll
  for (int ch = 0; ch < kBwdChunks; ++ch) v[ch] = ld_chunk(tile + tile_chunk(pos, part * kBwdChunks + ch));
  const float2 m = partial_statistics<kBwdChunks>(v);
  asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(xchg + (part * 128 + pos) * 8), "f"(m.x), "f"(m.y) : "memory");
  named_bar_sync(1, kBwdThreads);
  const float2 st = merge_partials<kBwdCh>(xchg, pos, eps);
  const float rstd = st.y, nmr = -st.x * st.y;
#pragma unroll
  for (int ch = 0; ch < kBwdChunks; ++ch) {
    const uint32_t w[4] = {v[ch].x, v[ch].y, v[ch].z, v[ch].w};
    uint32_t o[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const float2 x = bf16x2_to_float2(w[t]);
      o[t] = pack_f16x2_sat(make_float2(fmaf(x.x, rstd, nmr), fmaf(x.y, rstd, nmr)));
    }
    st_chunk(tile + tile_chunk(pos, part * kBwdChunks + ch), o[0], o[1], o[2], o[3]);
  }
  return rstd;
}

// Sum of the float2 partials the kBwdParts threads of a position left in `xchg` (fixed order).
__device__ __forceinline__ void sum_partials(uint32_t xchg, int pos, float& a, float& b) {
  a = 0.f, b = 0.f;
#pragma unroll
  for (int k = 0; k < kBwdParts; ++k) {
    float x, y;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(x), "=f"(y) : "r"(xchg + (k * 128 + pos) * 8));
    a += x, b += y;
  }
}

// Eight columns (8 * chunk ..) of row `row` of a CTA's partial weight gradient. The matrix lies in memory as [32 groups of
// four columns][128 rows] float4, so that a warp, whose lanes hold consecutive rows, stores 512 contiguous bytes (row by
// row its 32 lanes would hit 32 different lines with every store: 12 us per launch for the two matrices of 148 CTAs).
__device__ __forceinline__ void store_partial(float* m, int row, int chunk, const uint32_t (&v)[8]) {
  float4* dst = reinterpret_cast<float4*>(m) + chunk * 2 * 128 + row;
  dst[0] = make_float4(__uint_as_float(v[0]), __uint_as_float(v[1]), __uint_as_float(v[2]), __uint_as_float(v[3]));
  dst[128] = make_float4(__uint_as_float(v[4]), __uint_as_float(v[5]), __uint_as_float(v[6]), __uint_as_float(v[7]));
}

struct BwdEpilogueParams {
  int tiles_per_row;   // ceil(N / 128)
  int num_tiles;       // B * N * tiles_per_row
  int n;               // N
  int ld;              // columns per row of ext_stats and ln_part (N rounded up to a multiple of 8)
  const float* consts;      // [2][128]: d_out = W_out beta_out + bias_out, d_gate = W_gate beta_in + bias_gate
  const float* grad_scale;  // [2]: c, 1 / c
  const uint16_t* drop_scale;  // [B][N][128] bf16 or null
  float eps_in;
  float eps_out;       // scaled by 2^-8: tri is stored times 2^-4
  float* part_m;       // [grid][2] matrices as store_partial lays them out: per-CTA partial sums of dproj^T t_hat and dgate^T x_hat
  float* part_s;       // [grid][2][128]: per-CTA column sums of dproj and dgate
  // the two-launch form for an output LayerNorm over 256 channels (MODE 1: first 128 channels, MODE 2: the others)
  const float2* ext_stats;  // [B*N][ld]: mean and rstd of the stored t over all 256 channels
  float2* ln_part;          // [B*N][ld]: MODE 1 writes its sums of d t_hat and d t_hat * t_hat; MODE 2 adds its own and
                            // writes back the two means over 256 channels
  float* rstd;              // [B*N][ld], not MODE 1: 1 / standard deviation of the input LayerNorm (x_hat leaves through map_xh)
  int* status;
};

// Epilogue backward. Inputs: tri [B*N][128][N] fp16 (times 2^-4), z and dy [B*N][N][128] bf16. Outputs:
//   dtri [B*N][128][N] fp16 = c * d loss / d t,  dxg [B*N][N][128] fp16 = c * (d loss / d x_hat through the output gate)
// and the per-CTA partials. Shared memory: W_out' , W_gate' (fp16, gamma folded), then four tiles: t, z, dy, dgate.
//
// MODE 0: the whole operator (128 contracted channels). MODE 1 / 2: the bidirectional module, whose output LayerNorm
// and projection span 256 channels held in two tensors; two launches with the statistics given (`ext_stats`):
//   MODE 1 (first tensor):  proj part = t_hat_1 Wo_1'^T + d_1 -> through map_dx (fp16); dproj; d t_hat_1 = dproj Wo_1'
//                           written raw through map_dt; its two LayerNorm-backward sums -> ln_part; Mo_1.
//   MODE 2 (second tensor): proj = part + t_hat_2 Wo_2'^T + d_2; dproj, dgate; d t_hat_2, dxg, Mo_2, Mg; the
//                           LayerNorm backward of its own 128 channels with the sums over all 256 (means -> ln_part);
//                           `bwd_ln_finish_kernel` then finishes the first tensor's gradient.
//
// 16 arithmetic warps, a warp that issues the MMAs and one that issues the copies (joined as in bwd_prologue_kernel). Per tile
//   arithmetic: eight warps normalise t in place, eight z -> N -> wait P / G -> dproj, dgate tiles -> A -> column sums -> S
//               -> wait d t_hat: the sums of the LayerNorm backward, d t, d x_hat -> wait weight gradients -> output tiles -> C
//   MMAs:       N: P, G;  A: d t_hat and d x_hat, then Mo and Mg
//   copies:     N: x_hat out, next tile into L2; weight gradients done: next t, z; C: output stores, then next dy
// t is stored [channel][position] while its statistics and sums run over the channels of a position: a thread normalises two
// neighbouring positions (4-byte accesses, a whole channel row per warp), and after the LayerNorm backward neighbouring lanes
// swap halves so that the gradient leaves in 4-byte accesses, too. What bounds it: the chain of one tile per SM; two weight
// matrices and four tiles, all live during the gradient GEMMs, leave no room for a second tile. (The statistics by shuffles, d
// t_hat transposed and the two sums taken from dproj save 5 us of a step of 360 at N = 384, but round otherwise: results differ
// by 3.5e-4, at the same distance from float64.)
constexpr int kBwdEpiThreads = kBwdThreads + 64;
constexpr int kBwdEpiXchg = 3 * kBwdXchg + 2048;  // three exchanges of partial sums, 1 / sigma, constants
constexpr int kBwdEpiSmemBytes = 6 * kBwdTile + kBwdEpiXchg + 512 /* barriers */ + 1024;
template <int MODE, int C = 128>
__global__ void __launch_bounds__(kBwdEpiThreads, 1)
bwd_epilogue_kernel(const __grid_constant__ CUtensorMap map_t, const __grid_constant__ CUtensorMap map_z,
                    const __grid_constant__ CUtensorMap map_dy, const __grid_constant__ CUtensorMap map_wo,
                    const __grid_constant__ CUtensorMap map_wg, const __grid_constant__ CUtensorMap map_dt,
                    const __grid_constant__ CUtensorMap map_dx, const __grid_constant__ CUtensorMap map_xh,
                    const __grid_constant__ CUtensorMap map_pp, const BwdEpilogueParams p) {
  // C = d_pair: the channels of z, dy, dproj, dgate and the rows of both weight matrices (128, or 64 for the narrow pair
  // stacks; MODE 0 only). The contracted width (channels of t) is 128 in both cases.
  static_assert(C == 128 || (C == 64 && MODE == 0), "d_pair is 128, or 64 with one output tensor");
  constexpr int kZCh = C / kBwdParts;   // z-side channels per thread
  constexpr int kZChunks = kZCh / 8;
  constexpr int kZHalves = C / 64;      // 64-channel halves of a [pos][C] tile
  constexpr uint32_t kWHalf = C * 128;  // bytes of one 64-wide k half of a weight matrix with C rows
  constexpr int kBarN = 2, kBarA = 3, kBarS = 4, kBarC = 5, kOne = kBwdThreads + 32, kTwo = kBwdThreads + 64;
  constexpr int kBarT = 6, kBarZ = 7, kBarQ = 8;  // (kBarQ .. kBarQ + 3: the threads of 32 positions)
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t wo_s = smem_base, wg_s = smem_base + kBwdTile;
  const uint32_t tiles_s = smem_base + 2 * kBwdTile;  // four tile buffers whose roles rotate from tile to tile
  // float2 [kBwdParts][128] each: partial statistics of t and of z, partial sums of the LayerNorm backward
  const uint32_t xchg = smem_base + 6 * kBwdTile, xchg_z = xchg + kBwdXchg, xchg_s = xchg_z + kBwdXchg;
  const uint32_t rstd_s = xchg_s + kBwdXchg;      // float [128]: 1 / sigma of the output LayerNorm
  float* const_ptr = reinterpret_cast<float*>(smem + 6 * kBwdTile + 3 * kBwdXchg + 512);  // d_out, d_gate [2][128]
  const uint32_t bar_base = smem_base + 6 * kBwdTile + kBwdEpiXchg;
  const uint32_t w_full = bar_base, t_full = bar_base + 8, z_full = bar_base + 16, dy_full = bar_base + 24;
  const uint32_t pp_full = bar_base + 32, fwd_done = bar_base + 40, d_done = bar_base + 48, grad_done = bar_base + 56;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + 6 * kBwdTile + kBwdEpiXchg + 64);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (uint32_t b = w_full; b <= grad_done; b += 8) mbar_init(b, 1);
    *abort_flag = 0;
    fence_mbar_init();
    prefetch_tmap(&map_t);
    prefetch_tmap(&map_z);
    prefetch_tmap(&map_dy);
    prefetch_tmap(&map_dt);
    prefetch_tmap(&map_dx);
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (threadIdx.x == kBwdThreads + 32) {
    // The first tile of the copying thread: the arguments of the call and the forward's tensors are older than the launch
    // before this one (a call begins with one that does not overlap the caller's) and land while that one ends. Forward and
    // backward of a replayed graph, with the early copies of bwd_prologue_kernel: N = 48 72.2 -> 70.7 us, 256 175.5 -> 173.0,
    // 384 316.8 -> 313.0; bidirectional 142.0 -> 139.5 (48), 369.4 -> 360.8 (256).
    const int row = blockIdx.x / p.tiles_per_row, j0 = (blockIdx.x - row * p.tiles_per_row) * 128;
    mbar_arrive_expect_tx(t_full, kBwdTile);
    mbar_arrive_expect_tx(z_full, kZHalves * 16384);
    mbar_arrive_expect_tx(dy_full, kZHalves * 16384);
#pragma unroll
    for (int kh = 0; kh < 2; ++kh) tma_load_3d(tiles_s + kh * 16384, &map_t, t_full, j0 + kh * 64, 0, row);
#pragma unroll
    for (int kh = 0; kh < kZHalves; ++kh) {
      tma_load_3d(tiles_s + kBwdTile + kh * 16384, &map_z, z_full, kh * 64, j0, row);
      tma_load_3d(tiles_s + 2 * kBwdTile + kh * 16384, &map_dy, dy_full, kh * 64, j0, row);
    }
  }
  grid_dependency_wait();
  grid_dependents_launch();
  if (threadIdx.x < 256) const_ptr[threadIdx.x] = p.consts[threadIdx.x];
  __syncthreads();

  // Buffer roles of tile `it`: t, z, dy, dgate = buffers (0, 1, 2, 3) for even it and (2, 3, 0, 1) for odd it. The outputs of
  // a tile are written over its t and z buffers and stored from there; its dy and dgate buffers are free once the gradient
  // GEMMs are done, and receive the next tile's t and z while this tile finishes. The next tile's dy (MODE 2: and the first
  // launch's part of the projection, where dgate will be) goes into this tile's t (z) buffer once the store has read it.
  auto t_buf = [&](int it_i) { return tiles_s + static_cast<uint32_t>((it_i & 1) * 2) * kBwdTile; };
  auto y_buf = [&](int it_i) { return tiles_s + static_cast<uint32_t>(((it_i & 1) ^ 1) * 2) * kBwdTile; };
  // (thread_wait: a thread that gives up sets the abort word and carries on; every later wait of the CTA returns within
  // one poll, so that all warps walk through the same barriers to the end)
  if (warp == kBwdThreads / 32) {
    // ------------------------------------------------------------ MMAs
    if (elect_one()) thread_wait(w_full, 0, abort_flag, p.status, kDevTimeoutMma);
    __syncwarp();
    int it = 0;
    for (int tile = blockIdx.x; tile < p.num_tiles; tile += gridDim.x, ++it) {
      const uint32_t t_s = t_buf(it), z_s = t_s + kBwdTile, dy_s = y_buf(it), dg_s = dy_s + kBwdTile;
      named_bar_sync(kBarN, kTwo);
      if (elect_one()) {
        // P = t_hat Wo'^T (columns 0-127), G = x_hat Wg'^T (columns 128-255); lanes = positions
        tc_fence_after();
        constexpr uint32_t idesc_p = umma_idesc(128, C, true, false, kFmtF16, kFmtF16);
        constexpr uint32_t idesc_g = umma_idesc(128, C, false, false, kFmtF16, kFmtF16);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          umma_bf16(tmem_base, umma_desc_mnmajor(t_s + ks * 2048, 16384),
                    umma_desc_kmajor(wo_s + (ks >> 2) * kWHalf) + static_cast<uint64_t>((ks & 3) * 2), idesc_p, ks != 0 ? 1u : 0u);
#pragma unroll
        for (int ks = 0; ks < C / 16; ++ks) {
          const uint64_t kb = static_cast<uint64_t>((ks & 3) * 2);
          umma_bf16(tmem_base + 128, umma_desc_kmajor(z_s + (ks >> 2) * 16384) + kb,
                    umma_desc_kmajor(wg_s + (ks >> 2) * kWHalf) + kb, idesc_g, ks != 0 ? 1u : 0u);
        }
        umma_commit(fwd_done);
      }
      __syncwarp();
      named_bar_sync(kBarA, kTwo);
      if (elect_one()) {
        // d t_hat = dproj Wo' (0-127), d x_hat = dgate Wg' (128-255; lanes = positions); Mo += dproj^T t_hat (256-383), Mg +=
        // dgate^T x_hat (384-511)
        tc_fence_after();
        constexpr uint32_t idesc_d = umma_idesc(128, 128, false, true, kFmtF16, kFmtF16);
        constexpr uint32_t idesc_dx = umma_idesc(128, C, false, true, kFmtF16, kFmtF16);
        constexpr uint32_t idesc_mo = umma_idesc(128, 128, true, false, kFmtF16, kFmtF16);
        constexpr uint32_t idesc_mg = umma_idesc(128, C, true, true, kFmtF16, kFmtF16);
        const uint32_t accum = it != 0 ? 1u : 0u;
#pragma unroll
        for (int ks = 0; ks < C / 16; ++ks) {  // K = the C channels of dproj; Wo' [C][128] read MN-major (its k halves are N blocks)
          const uint64_t kb = static_cast<uint64_t>((ks & 3) * 2);
          umma_bf16(tmem_base, umma_desc_kmajor(dy_s + (ks >> 2) * 16384) + kb, umma_desc_mnmajor(wo_s + ks * 2048, kWHalf),
                    idesc_d, ks != 0 ? 1u : 0u);
        }
        if constexpr (MODE != 1) {
#pragma unroll
          for (int ks = 0; ks < C / 16; ++ks) {
            const uint64_t kb = static_cast<uint64_t>((ks & 3) * 2);
            umma_bf16(tmem_base + 128, umma_desc_kmajor(dg_s + (ks >> 2) * 16384) + kb,
                      umma_desc_mnmajor(wg_s + ks * 2048, kWHalf), idesc_dx, ks != 0 ? 1u : 0u);
          }
        }
        umma_commit(d_done);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
          const uint64_t kb = static_cast<uint64_t>((ks & 3) * 2);
          umma_bf16(tmem_base + 256, umma_desc_mnmajor(dy_s + ks * 2048, 16384),
                    umma_desc_kmajor(t_s + (ks >> 2) * 16384) + kb, idesc_mo, (ks != 0 ? 1u : 0u) | accum);
        }
        if constexpr (MODE != 1) {
#pragma unroll
          for (int ks = 0; ks < 8; ++ks)
            umma_bf16(tmem_base + 384, umma_desc_mnmajor(dg_s + ks * 2048, 16384), umma_desc_mnmajor(z_s + ks * 2048, 16384),
                      idesc_mg, (ks != 0 ? 1u : 0u) | accum);
        }
        umma_commit(grad_done);
      }
      __syncwarp();
    }
  } else if (warp == kBwdThreads / 32 + 1) {
    // ------------------------------------------------------------ copies
    auto place = [&](int tile_i, int& row_i, int& j_i) {
      row_i = tile_i / p.tiles_per_row;
      j_i = (tile_i - row_i * p.tiles_per_row) * 128;
    };
    auto issue_tz = [&](int tile_i, int it_i) {
      int row_i, j_i;
      place(tile_i, row_i, j_i);
      const uint32_t t_i = t_buf(it_i), z_i = t_i + kBwdTile;
      mbar_arrive_expect_tx(t_full, kBwdTile);
#pragma unroll
      for (int kh = 0; kh < 2; ++kh) tma_load_3d(t_i + kh * 16384, &map_t, t_full, j_i + kh * 64, 0, row_i);
      mbar_arrive_expect_tx(z_full, kZHalves * 16384);
#pragma unroll
      for (int kh = 0; kh < kZHalves; ++kh) tma_load_3d(z_i + kh * 16384, &map_z, z_full, kh * 64, j_i, row_i);
    };
    auto issue_dy = [&](int tile_i, int it_i, bool there = false) {
      int row_i, j_i;
      place(tile_i, row_i, j_i);
      const uint32_t y_i = y_buf(it_i);
      if (!there) {
        mbar_arrive_expect_tx(dy_full, kZHalves * 16384);
#pragma unroll
        for (int kh = 0; kh < kZHalves; ++kh) tma_load_3d(y_i + kh * 16384, &map_dy, dy_full, kh * 64, j_i, row_i);
      }
      if constexpr (MODE == 2) {
        mbar_arrive_expect_tx(pp_full, kBwdTile);
#pragma unroll
        for (int kh = 0; kh < 2; ++kh) tma_load_3d(y_i + kBwdTile + kh * 16384, &map_pp, pp_full, kh * 64, j_i, row_i);
      }
    };
    if (lane == 0) {
      // Wo' [C, 128] as two k halves, Wg' [C, C] as C / 64 k halves
      mbar_arrive_expect_tx(w_full, (2 + kZHalves) * kWHalf);
#pragma unroll
      for (int kh = 0; kh < 2; ++kh) tma_load_2d(wo_s + kh * kWHalf, &map_wo, w_full, kh * 64, 0);
#pragma unroll
      for (int kh = 0; kh < kZHalves; ++kh) tma_load_2d(wg_s + kh * kWHalf, &map_wg, w_full, kh * 64, 0);
      issue_dy(blockIdx.x, 0, true);
    }
    __syncwarp();
    int it = 0;
    for (int tile = blockIdx.x; tile < p.num_tiles; tile += gridDim.x, ++it) {
      const int next = tile + static_cast<int>(gridDim.x);
      const bool has_next = next < p.num_tiles;
      int row, j0;
      place(tile, row, j0);
      const uint32_t t_s = t_buf(it), z_s = t_s + kBwdTile;
      named_bar_sync(kBarN, kTwo);
      if (lane == 0) {
        if constexpr (MODE != 1) {  // x_hat for the prologue's backward
#pragma unroll
          for (int kh = 0; kh < kZHalves; ++kh) tma_store_3d(&map_xh, z_s + kh * 16384, kh * 64, j0, row);
          bulk_commit();
        }
        if (has_next) {
          int row_n, j_n;
          place(next, row_n, j_n);
#pragma unroll
          for (int kh = 0; kh < 2; ++kh)
            if (j_n + kh * 64 < p.n) tma_prefetch_3d(&map_t, j_n + kh * 64, 0, row_n);
#pragma unroll
          for (int kh = 0; kh < kZHalves; ++kh) tma_prefetch_3d(&map_z, kh * 64, j_n, row_n);
        }
        if constexpr (MODE != 1) bulk_wait_read<0>();  // (the z buffer is written again after barrier A)
      }
      __syncwarp();
      named_bar_sync(kBarA, kTwo);
      named_bar_sync(kBarS, kOne);  // the column sums have been read off the dproj and dgate tiles
      if (lane == 0 && has_next) {
        thread_wait(grad_done, it & 1, abort_flag, p.status, kDevTimeoutProducer);
        issue_tz(next, it + 1);  // into this tile's dy and dgate buffers
      }
      __syncwarp();
      named_bar_sync(kBarC, kOne);
      if (lane == 0) {
#pragma unroll
        for (int kh = 0; kh < 2; ++kh)
          if (j0 + kh * 64 < p.n) tma_store_3d(&map_dt, t_s + kh * 16384, j0 + kh * 64, 0, row);
#pragma unroll
        for (int kh = 0; kh < kZHalves; ++kh) tma_store_3d(&map_dx, z_s + kh * 16384, kh * 64, j0, row);
        bulk_commit();
        bulk_wait_read<0>();
        if (has_next) issue_dy(next, it + 1);  // into this tile's t (and z) buffer
      }
      __syncwarp();
    }
    if (lane == 0) {
      // Every copy has been waited for by its readers unless the CTA is giving up; then those in flight must land before
      // it exits (the last copies of every kind were the last tile's).
      if (*abort_flag != 0) {
        const uint32_t last = static_cast<uint32_t>((it - 1) & 1);
        const long long t0 = clock64();
        while (!mbar_try_wait(w_full, 0) || !mbar_try_wait(t_full, last) || !mbar_try_wait(z_full, last) ||
               !mbar_try_wait(dy_full, last) || (MODE == 2 && !mbar_try_wait(pp_full, last))) {
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
    const int pos = q * 32 + lane;
    const uint32_t lane_sel = static_cast<uint32_t>(q * 32) << 16;
    const float gc = p.grad_scale[0];
    auto pair_of = [](uint32_t lo, uint32_t hi) { return make_float2(__uint_as_float(lo), __uint_as_float(hi)); };
    // Column sums of dproj and dgate (the bias / beta terms of the weight gradients): gathered from the fp16 tiles while
    // the gradient GEMMs run, this thread taking the 16-byte chunk `sum_chunk` (eight channels) of four position rows.
    const int sum_chunk = threadIdx.x & 15, sum_rows = (threadIdx.x >> 4) * 4;
    float acc_so[8], acc_sg[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) acc_so[c] = 0.f, acc_sg[c] = 0.f;
    int it = 0;
    for (int tile = blockIdx.x; tile < p.num_tiles; tile += gridDim.x, ++it) {
      const int row = tile / p.tiles_per_row;
      const int j0 = (tile - row * p.tiles_per_row) * 128;
      const int j = j0 + pos;
      const uint32_t t_s = t_buf(it), z_s = t_s + kBwdTile, dy_s = y_buf(it), dg_s = dy_s + kBwdTile;
      if (warp < 8) {
        // ---- t normalised in place: a thread takes 32 channels (`grp`) of two neighbouring positions, so that a warp reads and
        // writes a channel's 64 positions in one 128-byte access
        thread_wait(t_full, it & 1, abort_flag, p.status, kDevTimeoutStats);
        __syncwarp();
        const int p0 = (warp & 1) * 64 + 2 * lane, grp = warp >> 1;
        const uint32_t col = t_s + static_cast<uint32_t>(warp & 1) * 16384 + grp * 32 * 128 + (lane & 3) * 4;
        auto t_addr = [&](int cc) { return col + cc * 128 + (((lane >> 2) ^ (cc & 7)) << 4); };
        uint32_t x[32];
#pragma unroll
        for (int cc = 0; cc < 32; ++cc) x[cc] = ld_word(t_addr(cc));
        float2 scale, shift;  // t_hat = t scale + shift
        if constexpr (MODE == 0) {
          const float2 pv = f16x2_to_float2(x[0]), npv = make_float2(-pv.x, -pv.y);
          float2 s1 = make_float2(0.f, 0.f), s2 = make_float2(0.f, 0.f);
#pragma unroll
          for (int cc = 0; cc < 32; ++cc) {
            const float2 d = __fadd2_rn(f16x2_to_float2(x[cc]), npv);
            s1 = __fadd2_rn(s1, d);
            s2 = __ffma2_rn(d, d, s2);
          }
          constexpr float kInv = 1.0f / 32;
          asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(xchg + (grp * 128 + p0) * 8), "f"(pv.x + s1.x * kInv),
                       "f"(fmaxf(s2.x - s1.x * s1.x * kInv, 0.f)), "f"(pv.y + s1.y * kInv),
                       "f"(fmaxf(s2.y - s1.y * s1.y * kInv, 0.f)) : "memory");
          named_bar_sync(kBarT, 256);
          float2 mean_a, mean_b;
          mean_a = merge_partials<32>(xchg, p0, p.eps_out), mean_b = merge_partials<32>(xchg, p0 + 1, p.eps_out);
          scale = make_float2(mean_a.y, mean_b.y);
          shift = make_float2(-mean_a.x * mean_a.y, -mean_b.x * mean_b.y);
        } else {
          float4 st = make_float4(0.f, 0.f, 0.f, 0.f);  // (positions past the end stay zero)
          if (j0 + p0 < p.n) st = *reinterpret_cast<const float4*>(p.ext_stats + static_cast<size_t>(row) * p.ld + j0 + p0);
          if (j0 + p0 + 1 >= p.n) st.z = 0.f, st.w = 0.f;
          scale = make_float2(st.y, st.w);
          shift = make_float2(-st.x * st.y, -st.z * st.w);
        }
        if (grp == 0)
          asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(rstd_s + p0 * 4), "f"(scale.x), "f"(scale.y) : "memory");
#pragma unroll
        for (int cc = 0; cc < 32; ++cc) st_word(t_addr(cc), pack_f16x2_sat(__ffma2_rn(f16x2_to_float2(x[cc]), scale, shift)));
      } else {
        // ---- z normalised in place: a thread takes a quarter of the channels of its position, twice
        thread_wait(z_full, it & 1, abort_flag, p.status, kDevTimeoutStats);
        __syncwarp();
        const int zp = threadIdx.x & 127, first = (threadIdx.x >> 7) & 1;  // quarters `first` and `first` + 2
        uint4 v[2][kZChunks];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int grp = first + 2 * h;
#pragma unroll
          for (int ch = 0; ch < kZChunks; ++ch) v[h][ch] = ld_chunk(z_s + tile_chunk(zp, grp * kZChunks + ch));
          const float2 m = partial_statistics<kZChunks>(v[h]);
          asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(xchg_z + (grp * 128 + zp) * 8), "f"(m.x), "f"(m.y) : "memory");
        }
        named_bar_sync(kBarZ, 256);
        const float2 st = merge_partials<kZCh>(xchg_z, zp, p.eps_in);
        if constexpr (MODE != 1) {
          if (first == 0 && j0 + zp < p.n) p.rstd[static_cast<size_t>(row) * p.ld + j0 + zp] = st.y;
        }
        const float2 scale = make_float2(st.y, st.y), shift = make_float2(-st.x * st.y, -st.x * st.y);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
          for (int ch = 0; ch < kZChunks; ++ch) {
            const uint4 w = v[h][ch];
            st_chunk(z_s + tile_chunk(zp, (first + 2 * h) * kZChunks + ch),
                     pack_f16x2_sat(__ffma2_rn(bf16x2_to_float2(w.x), scale, shift)),
                     pack_f16x2_sat(__ffma2_rn(bf16x2_to_float2(w.y), scale, shift)),
                     pack_f16x2_sat(__ffma2_rn(bf16x2_to_float2(w.z), scale, shift)),
                     pack_f16x2_sat(__ffma2_rn(bf16x2_to_float2(w.w), scale, shift)));
          }
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      named_bar_arrive(kBarN, kTwo);
      // the dropout scale of this thread's position, requested before the waits
      uint4 scv[kZChunks];
#pragma unroll
      for (int ch = 0; ch < kZChunks; ++ch) scv[ch] = make_uint4(0x3F803F80u, 0x3F803F80u, 0x3F803F80u, 0x3F803F80u);  // bf16 ones
      if (p.drop_scale != nullptr && j < p.n) {
        const int b = row / p.n;
        ldg_chunks(reinterpret_cast<const uint4*>(p.drop_scale + (static_cast<size_t>(b) * p.n + j) * C + part * kZCh),
                   (reinterpret_cast<uintptr_t>(p.drop_scale) & 31u) == 0, scv);
      }
      float2 other = make_float2(0.f, 0.f);  // MODE 2: the first launch's sums of this position
      if constexpr (MODE == 2) {
        if (j < p.n) other = p.ln_part[static_cast<size_t>(row) * p.ld + j];
      }
      thread_wait(dy_full, it & 1, abort_flag, p.status, kDevTimeoutStats);
      if constexpr (MODE == 2) thread_wait(pp_full, it & 1, abort_flag, p.status, kDevTimeoutStats);
      thread_wait(fwd_done, it & 1, abort_flag, p.status, kDevTimeoutEpilogue);
      __syncwarp();
      tc_fence_after();
      // ---- dproj = c du gate, dgate = c du proj gate (1 - gate); du = dy (* dropout scale). This thread: one position,
      // kZCh channels.
      {
        const float2 half2 = make_float2(0.5f, 0.5f), gc2 = make_float2(gc, gc);
        uint32_t vp[2][8], vg[2][8];
        tmem_ld8(tmem_base + lane_sel + part * kZCh, vp[0]);
        tmem_ld8(tmem_base + lane_sel + 128 + part * kZCh, vg[0]);
#pragma unroll
        for (int ch = 0; ch < kZChunks; ++ch) {
          tmem_ld_wait();
          if (ch < kZChunks - 1) {
            tmem_ld8(tmem_base + lane_sel + part * kZCh + (ch + 1) * 8, vp[(ch + 1) & 1]);
            tmem_ld8(tmem_base + lane_sel + 128 + part * kZCh + (ch + 1) * 8, vg[(ch + 1) & 1]);
          }
          const uint32_t addr = tile_chunk(pos, part * kZChunks + ch);
          const uint4 dyv = ld_chunk(dy_s + addr);
          uint4 ppv = make_uint4(0u, 0u, 0u, 0u);
          if constexpr (MODE == 2) ppv = ld_chunk(dg_s + addr);
          const uint32_t pw[4] = {ppv.x, ppv.y, ppv.z, ppv.w};
          const uint32_t dw[4] = {dyv.x, dyv.y, dyv.z, dyv.w};
          const uint32_t sw[4] = {scv[ch].x, scv[ch].y, scv[ch].z, scv[ch].w};
          const float2* cp = reinterpret_cast<const float2*>(const_ptr + part * kZCh + ch * 8);
          uint32_t op[4], og[4];
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            float2 proj = __fadd2_rn(pair_of(vp[ch & 1][2 * t], vp[ch & 1][2 * t + 1]), cp[t]);
            if constexpr (MODE == 2) proj = __fadd2_rn(proj, f16x2_to_float2(pw[t]));
            const float2 gh = __fmul2_rn(__fadd2_rn(pair_of(vg[ch & 1][2 * t], vg[ch & 1][2 * t + 1]), cp[64 + t]), half2);
            const float2 gate = __ffma2_rn(make_float2(tanh_approx(gh.x), tanh_approx(gh.y)), half2, half2);
            const float2 du = __fmul2_rn(__fmul2_rn(bf16x2_to_float2(dw[t]), bf16x2_to_float2(sw[t])), gc2);
            const float2 dp = __fmul2_rn(du, gate);
            op[t] = pack_f16x2_sat(dp);
            // MODE 1 hands its part of proj on
            og[t] = pack_f16x2_sat(MODE == 1 ? proj
                                             : __fmul2_rn(dp, __ffma2_rn(make_float2(-proj.x, -proj.y), gate, proj)));
          }
          st_chunk(dy_s + addr, op[0], op[1], op[2], op[3]);
          // MODE 1: the part of proj leaves through the z buffer (x_hat is only needed by the G GEMM, which is done)
          st_chunk((MODE == 1 ? z_s : dg_s) + addr, og[0], og[1], og[2], og[3]);
          if constexpr (C == 64) {
            // the weight-gradient GEMMs read these tiles as 128-row operands: rows 64-127 (the second 64-channel block) are zero
            const uint32_t zaddr = tile_chunk(pos, 8 + part * kZChunks + ch);
            st_chunk(dy_s + zaddr, 0u, 0u, 0u, 0u);
            st_chunk(dg_s + zaddr, 0u, 0u, 0u, 0u);
          }
        }
      }
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      named_bar_sync(kBarA, kTwo);
      // ---- (under the gradient GEMMs) this thread's t_hat values, its position's 1 / sigma, column sums
      uint32_t th[16];  // channels part * 32 + 8 k + i and, in the upper half, + 4 (k, i = 0 .. 3)
#pragma unroll
      for (int k = 0; k < 4; ++k) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          th[k * 4 + i] = ld_half(t_s + tile_off(part * 32 + k * 8 + i, pos)) | (ld_half(t_s + tile_off(part * 32 + k * 8 + i + 4, pos)) << 16);
      }
      float rs;
      asm volatile("ld.shared.f32 %0, [%1];" : "=f"(rs) : "r"(rstd_s + pos * 4));
      rs *= 0.0625f;  // d / d t of the stored t / 16
      if (sum_chunk < C / 8) {  // column sums of the two fp16 tiles the GEMMs are reading
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const uint32_t addr = tile_chunk(sum_rows + r, sum_chunk);
          const uint4 a = ld_chunk(dy_s + addr);
          const uint32_t aw[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const float2 x = f16x2_to_float2(aw[t]);
            acc_so[2 * t] += x.x, acc_so[2 * t + 1] += x.y;
          }
          if constexpr (MODE != 1) {
            const uint4 b = ld_chunk(dg_s + addr);
            const uint32_t bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              const float2 x = f16x2_to_float2(bw[t]);
              acc_sg[2 * t] += x.x, acc_sg[2 * t + 1] += x.y;
            }
          }
        }
      }
      __syncwarp();
      named_bar_arrive(kBarS, kOne);
      // ---- LayerNorm backward of the output normalisation for this thread's position and 32 channels; d x_hat
      thread_wait(d_done, it & 1, abort_flag, p.status, kDevTimeoutEpilogue);
      __syncwarp();
      tc_fence_after();
      uint32_t dv[32];
      tmem_ld32(tmem_base + lane_sel + part * 32, dv);
      tmem_ld_wait();
      float m1 = 0.f, m2 = 0.f;
#pragma unroll
      for (int cc = 0; cc < 32; ++cc) {
        const float2 t2 = f16x2_to_float2(th[(cc >> 3) * 4 + (cc & 3)]);
        const float d = __uint_as_float(dv[cc]);
        m1 += d;
        m2 = fmaf(d, (cc & 4) ? t2.y : t2.x, m2);
      }
      asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(xchg_s + (part * 128 + pos) * 8), "f"(m1), "f"(m2) : "memory");
      named_bar_sync(kBarQ + q, 32 * kBwdParts);  // the threads of these 32 positions
      if (MODE != 1 || part == 0) sum_partials(xchg_s, pos, m1, m2);
      if constexpr (MODE == 1) {
        if (part == 0 && j < p.n) p.ln_part[static_cast<size_t>(row) * p.ld + j] = make_float2(m1, m2);
      } else if constexpr (MODE == 2) {
        m1 = (m1 + other.x) * (1.0f / 256.0f), m2 = (m2 + other.y) * (1.0f / 256.0f);
        if (part == 0 && j < p.n) p.ln_part[static_cast<size_t>(row) * p.ld + j] = make_float2(m1, m2);
      } else {
        m1 *= 1.0f / 128.0f, m2 *= 1.0f / 128.0f;
      }
      // d t = rs (d t_hat - m1 - t_hat m2). Two neighbouring lanes swap halves, the even one ending with a channel of both
      // positions and the odd one with the channel four rows on, so that a warp stores two 64-byte runs without a bank conflict
      uint32_t ot[16];
      const float2 nm1 = make_float2(-m1, -m1), nm2 = make_float2(-m2, -m2), rs2 = make_float2(rs, rs);
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        float2 d = pair_of(dv[(k >> 2) * 8 + (k & 3)], dv[(k >> 2) * 8 + (k & 3) + 4]);
        if constexpr (MODE != 1) d = __fmul2_rn(rs2, __ffma2_rn(f16x2_to_float2(th[k]), nm2, __fadd2_rn(d, nm1)));
        const uint32_t o = pack_f16x2_sat(d);  // (MODE 1: finished by bwd_ln_finish_kernel)
        const uint32_t n = __shfl_xor_sync(0xFFFFFFFFu, o, 1);
        ot[k] = (lane & 1) ? __byte_perm(n, o, 0x7632) : __byte_perm(o, n, 0x5410);
      }
      uint32_t ox[MODE != 1 ? kZChunks * 4 : 1];
      if constexpr (MODE != 1) {
#pragma unroll
        for (int ch = 0; ch < kZChunks; ++ch) {
          uint32_t x[8];
          tmem_ld8(tmem_base + lane_sel + 128 + part * kZCh + ch * 8, x);
          tmem_ld_wait();
#pragma unroll
          for (int t = 0; t < 4; ++t) ox[ch * 4 + t] = pack_f16x2_sat(pair_of(x[2 * t], x[2 * t + 1]));
        }
      }
      tc_fence_before();
      thread_wait(grad_done, it & 1, abort_flag, p.status, kDevTimeoutEpilogue);  // the GEMMs have read t_hat and x_hat
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 16; ++k)
        st_word(t_s + tile_off(part * 32 + (k >> 2) * 8 + (k & 3) + (lane & 1) * 4, pos & ~1), ot[k]);
      if constexpr (MODE != 1) {
#pragma unroll
        for (int ch = 0; ch < kZChunks; ++ch)
          st_chunk(z_s + tile_chunk(pos, part * kZChunks + ch), ox[ch * 4], ox[ch * 4 + 1], ox[ch * 4 + 2], ox[ch * 4 + 3]);
      }
      fence_proxy_async_smem();
      __syncwarp();
      named_bar_arrive(kBarC, kOne);
    }
    // ---- per-CTA partials of the weight gradients (every GEMM has been waited for) and of the column sums
    tc_fence_after();
    float* pm = p.part_m + static_cast<size_t>(blockIdx.x) * 2 * 128 * 128;
#pragma unroll
    for (int m = 0; m < 2; ++m) {
#pragma unroll
      for (int ch = 0; ch < kBwdChunks; ++ch) {
        uint32_t v[8];
        tmem_ld8(tmem_base + lane_sel + 256 + m * 128 + part * kBwdCh + ch * 8, v);
        tmem_ld_wait();
        store_partial(pm + m * 128 * 128, pos, part * kBwdChunks + ch, v);
      }
    }
    {  // the 32 row groups of a channel, fixed order (through the weights' region, which no GEMM reads any more)
      float* sc = reinterpret_cast<float*>(smem);  // [32 row groups][2][128]
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        sc[((threadIdx.x >> 4) * 2 + 0) * 128 + sum_chunk * 8 + c] = acc_so[c];
        sc[((threadIdx.x >> 4) * 2 + 1) * 128 + sum_chunk * 8 + c] = acc_sg[c];
      }
      named_bar_sync(1, kBwdThreads);
      if (threadIdx.x < 256 && (threadIdx.x & 127) < C) {
        float sum = 0.f;
        for (int g = 0; g < 32; ++g) sum += sc[g * 256 + threadIdx.x];
        p.part_s[static_cast<size_t>(blockIdx.x) * 2 * 128 + threadIdx.x] = sum;
      }
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

// Mean and rstd of the stored t over the 256 channels of two tensors [rows][128][N] (fp16): stats[row][j] = {mean,
// rsqrt(var + eps)} (eps already scaled like the stored t; `n` columns per row of statistics, channels `pitch` 16-byte pieces
// apart in t). The sums of a column are one chain over its 256 channels in
// order. A block brings eight groups of eight columns into shared memory (128 bytes per channel, all loads in flight at once);
// then one warp walks the channels, a lane two columns. (One thread per group of eight columns that loaded as it went left
// the chip idle at small N: 8192 threads at N = 256, 29 us for 34 MB.)
constexpr int kLnStatsGroups = 8;
__global__ void __launch_bounds__(256) bwd_ln_stats_kernel(const uint4* t0, const uint4* t1, int n, int pitch, long long groups, float eps,
                                                           float2* stats) {
  grid_dependency_wait();
  grid_dependents_launch();
  __shared__ uint4 tile[256][kLnStatsGroups];
  const int per_row = n / 8;
  const long long first = blockIdx.x * static_cast<long long>(kLnStatsGroups);
  {
    const int k = threadIdx.x & (kLnStatsGroups - 1), c0 = threadIdx.x / kLnStatsGroups;
    const long long g = first + k;
    if (g < groups) {
      const long long row = g / per_row;
      const long long at = row * 128 * pitch + (g - row * per_row);
      uint4 v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        v[u] = __ldg((u < 4 ? t0 : t1) + at + static_cast<long long>((c0 + 32 * u) & 127) * pitch);
#pragma unroll
      for (int u = 0; u < 8; ++u) tile[c0 + 32 * u][k] = v[u];
    }
  }
  __syncthreads();
  const long long g = first + (threadIdx.x >> 2);
  if (threadIdx.x >= 32 || g >= groups) return;
  const uint32_t* col = reinterpret_cast<const uint32_t*>(tile) + threadIdx.x;  // columns 2 * lane, 2 * lane + 1
  const float2 pv = f16x2_to_float2(col[0]), npv = make_float2(-pv.x, -pv.y);
  float2 s1 = make_float2(0.f, 0.f), s2 = make_float2(0.f, 0.f);
#pragma unroll 32
  for (int c = 0; c < 256; ++c) {
    const float2 d = __fadd2_rn(f16x2_to_float2(col[c * 32]), npv);
    s1 = __fadd2_rn(s1, d);
    s2 = __ffma2_rn(d, d, s2);
  }
  constexpr float kInv = 1.0f / 256.0f;
  const float var0 = fmaxf(s2.x - s1.x * s1.x * kInv, 0.f) * kInv, var1 = fmaxf(s2.y - s1.y * s1.y * kInv, 0.f) * kInv;
  const long long row = g / per_row;
  reinterpret_cast<float4*>(stats + row * n + (g - row * per_row) * 8)[threadIdx.x & 3] =
      make_float4(pv.x + s1.x * kInv, rsqrtf(var0 + eps), pv.y + s1.y * kInv, rsqrtf(var1 + eps));
}

// Finishes the first tensor's gradient of the 256-channel LayerNorm backward, in place over the raw d t_hat the MODE 1
// launch left in dt [rows][128][N] (fp16, times c): dt = rstd / 16 * (d t_hat - m1 - t_hat m2), t_hat recomputed from t.
// One thread per row, group of eight columns and group of 16 channels: the eight positions' statistics are read once.
constexpr int kLnFinishChannels = 16;
__global__ void __launch_bounds__(256) bwd_ln_finish_kernel(uint4* dt, const uint4* t, const float2* stats, const float2* means,
                                                            int n, int pitch, long long threads) {
  grid_dependency_wait();
  grid_dependents_launch();
  const long long g = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (g >= threads) return;
  const int per_row = n / 8;
  const long long rg = g / per_row;  // row * (128 / kLnFinishChannels) + channel group
  const int jc = static_cast<int>(g - rg * per_row);
  const long long row = rg / (128 / kLnFinishChannels);
  const int c_first = static_cast<int>(rg - row * (128 / kLnFinishChannels)) * kLnFinishChannels;
  float mean[8], k0[8], k1[8], m1[8];
  {
    const float4* sp = reinterpret_cast<const float4*>(stats + row * n + jc * 8);
    const float4* mp = reinterpret_cast<const float4*>(means + row * n + jc * 8);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float4 st = __ldg(sp + q), mm = __ldcg(mp + q);  // (the launch before this one writes the means)
      mean[2 * q] = st.x, k0[2 * q] = st.y * 0.0625f, k1[2 * q] = st.y * mm.y, m1[2 * q] = mm.x;
      mean[2 * q + 1] = st.z, k0[2 * q + 1] = st.w * 0.0625f, k1[2 * q + 1] = st.w * mm.w, m1[2 * q + 1] = mm.z;
    }
  }
  const long long base = (row * 128 + c_first) * pitch + jc;
#pragma unroll
  for (int c0 = 0; c0 < kLnFinishChannels; c0 += 4) {
    uint4 dv[4], tv[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      dv[k] = dt[base + static_cast<long long>(c0 + k) * pitch];
      tv[k] = __ldg(t + base + static_cast<long long>(c0 + k) * pitch);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t dw[4] = {dv[k].x, dv[k].y, dv[k].z, dv[k].w}, tw[4] = {tv[k].x, tv[k].y, tv[k].z, tv[k].w};
      uint32_t o[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float2 d = f16x2_to_float2(dw[q]);
        const float2 x = f16x2_to_float2(tw[q]);
        const float r0 = k0[2 * q] * (d.x - m1[2 * q] - (x.x - mean[2 * q]) * k1[2 * q]);
        const float r1 = k0[2 * q + 1] * (d.y - m1[2 * q + 1] - (x.y - mean[2 * q + 1]) * k1[2 * q + 1]);
        o[q] = pack_f16x2_sat(make_float2(r0, r1));
      }
      dt[base + static_cast<long long>(c0 + k) * pitch] = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
}

struct BwdPrologueParams {
  int tiles_per_row;
  int num_tiles;
  int n;
  int ld;                     // columns per row of rstd
  const float* consts;        // [2][128]: d_value = W beta_in + bias, d_gate likewise (this side's two matrices)
  const float* grad_scale;    // [2]: c, 1 / c
  const uint8_t* token_mask;  // [B][N] or null
  const uint8_t* pair_mask;   // [B][N][N] or null
  const void* dy;             // LAST only: non-null if the residual path's dy (map_dy) is added
  const float* rstd;          // LAST only: [B*N][ld] 1 / standard deviation of the input LayerNorm
  float* part_m;              // [grid][2] matrices (store_partial): partial dvalue^T x_hat, dgate^T x_hat
  float* part_s;              // [grid][2][128]
  int* status;
};

// Prologue backward for one side (left or right). Inputs: x_hat [B*N][N][C] fp16 and rstd (both left by the epilogue's
// backward, which normalises z anyway), dO = the contraction's gradient for this side [B*N][128][N] fp16 (times c / 16).
// It recomputes value / gate, forms dvalue = dO sig m, dgate = dO value sig (1 - sig) m, adds dvalue W_v' + dgate W_g' to
// the running d x_hat, and accumulates the two weight gradients. !LAST: the running d x_hat (fp16, times c) is written
// back through map_out. LAST: the input LayerNorm's backward and the residual finish d loss / d z (bf16, unscaled).
//
// The running d x_hat (c * d loss / d x_hat gathered so far, fp16) comes through map_dx, LAST: dy (bf16) through map_dy.
// 16 arithmetic warps (four threads per channel or position, as in the epilogue's backward), a warp that issues the MMAs and
// one that issues the copies. The arithmetic warps never wait for one another but once per tile (LAST): they arrive at
// named barriers the issuing warps wait at, and wait for MMAs and copies on mbarriers. Per tile:
//   arithmetic: wait value / gate -> dvalue, dgate tiles -> arrive A -> wait d x_hat -> out of tensor memory -> arrive B
//               -> running sum added, LAST: LayerNorm backward and residual -> output tile -> arrive C
//   MMAs:       A: d x_hat GEMMs, weight-gradient GEMMs; B: value / gate GEMMs of the NEXT tile, behind them in the pipe
//   copies:     A: next x_hat; weight gradients done: dy (LAST) and next dO; C: output store, next running sum
// Every global operand comes through TMA: read by the threads, 32 bytes per lane, the running sum alone held the load path
// for 2.8 k of the 8.8 k cycles of a tile (with dy 4-5 k).
// What bounds it: the chain value / gate GEMMs -> arithmetic -> gradient GEMMs -> read of one tile per SM; shared memory
// holds two weight matrices and five tiles and has no room for a second tile in flight.
constexpr int kBwdProThreads = kBwdThreads + 64;
constexpr int kBwdProSmemBytes = 7 * kBwdTile + 512 /* barriers */ + 1024;
template <bool LAST, int C = 128>
__global__ void __launch_bounds__(kBwdProThreads, 1)
bwd_prologue_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_do,
                    const __grid_constant__ CUtensorMap map_wv, const __grid_constant__ CUtensorMap map_wg,
                    const __grid_constant__ CUtensorMap map_dx, const __grid_constant__ CUtensorMap map_dy,
                    const __grid_constant__ CUtensorMap map_out, const BwdPrologueParams p) {
  // C = d_pair: the channels of z, d x_hat, dz and the columns of both weight matrices (128, or 64 for the narrow pair
  // stacks). The contracted width (channels of dO, rows of the weight matrices) is 128 in both cases.
  static_assert(C == 128 || C == 64, "d_pair is 128 or 64");
  constexpr int kZCh = C / kBwdParts;   // z-side channels per thread
  constexpr int kZChunks = kZCh / 8;
  constexpr int kZHalves = C / 64;      // 64-channel halves of a [pos][C] tile = k halves of a [128][C] weight matrix
  // named barriers of the arithmetic warps and the issuing warps
  constexpr int kBarA = 2, kBarB = 3, kBarC = 4, kCountA = kBwdThreads + 64, kCountB = kBwdThreads + 32;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t wv_s = smem_base, wg_s = smem_base + kBwdTile;
  const uint32_t tiles_s = smem_base + 2 * kBwdTile;  // four tile buffers whose roles rotate from tile to tile
  const uint32_t dx_s = smem_base + 6 * kBwdTile;     // the running d x_hat, later the exchange of partial sums
  const uint32_t bar_base = smem_base + 7 * kBwdTile;
  const uint32_t w_full = bar_base, x_full = bar_base + 8, do_full = bar_base + 16, dx_full = bar_base + 24;
  const uint32_t dy_full = bar_base + 32, fwd_done = bar_base + 40, dx_done = bar_base + 48, grad_done = bar_base + 56;
  const uint32_t out_free = bar_base + 64;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + 7 * kBwdTile + 72);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (uint32_t b = w_full; b <= out_free; b += 8) mbar_init(b, 1);
    *abort_flag = 0;
    fence_mbar_init();
    prefetch_tmap(&map_x);
    prefetch_tmap(&map_do);
    prefetch_tmap(&map_dx);
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
  // (the weights, x_hat and dO are older than the launch before this one, the other side's contraction or the first side's
  // pass, and land while it ends; the running d x_hat is not. Figures: bwd_epilogue_kernel)
  if (warp != kBwdThreads / 32 + 1) {
    grid_dependency_wait();
    grid_dependents_launch();
  }

  // Buffer roles (x_hat, dO, dvalue, dgate) of tile `it`, one nibble each, period 4: the next tile's x_hat and dO are
  // copied into this tile's dO buffer (free once dvalue / dgate are formed) and dgate buffer (free after the gradient
  // GEMMs); its dvalue scratch is this tile's x_hat buffer and its dgate scratch this tile's dvalue buffer, which receives
  // dy (LAST) after the gradient GEMMs and then, in place, the output, and is free once the store has read it.
  auto role = [&](int it_i, int r) {
    const uint32_t rr = static_cast<uint32_t>(0x1302012320313210ull >> (16 * (it_i & 3))) & 0xFFFFu;
    return tiles_s + ((rr >> (4 * r)) & 0xFu) * kBwdTile;
  };
  // (thread_wait: a thread that gives up sets the abort word and carries on; every later wait of the CTA returns within
  // one poll, so that all warps walk through the same barriers to the end)
  if (warp == kBwdThreads / 32) {
    // ------------------------------------------------------------ MMAs
    // value^T = Wv' x_hat^T (columns 0-127), gate^T = Wg' x_hat^T (128-255): lanes = contracted channels
    auto issue_fwd = [&](int it_i) {
      thread_wait(x_full, it_i & 1, abort_flag, p.status, kDevTimeoutMma);
      tc_fence_after();
      constexpr uint32_t idesc = umma_idesc(128, 128, false, false, kFmtF16, kFmtF16);
      const uint32_t x_s = role(it_i, 0);
#pragma unroll
      for (int m = 0; m < 2; ++m) {
#pragma unroll
        for (int ks = 0; ks < C / 16; ++ks) {
          const uint64_t kb = static_cast<uint64_t>((ks & 3) * 2);
          umma_bf16(tmem_base + m * 128, umma_desc_kmajor((m == 0 ? wv_s : wg_s) + (ks >> 2) * 16384) + kb,
                    umma_desc_kmajor(x_s + (ks >> 2) * 16384) + kb, idesc, ks != 0 ? 1u : 0u);
        }
      }
      umma_commit(fwd_done);
    };
    if (elect_one()) {
      thread_wait(w_full, 0, abort_flag, p.status, kDevTimeoutMma);
      issue_fwd(0);
    }
    __syncwarp();
    int it = 0;
    for (int tile = blockIdx.x; tile < p.num_tiles; tile += gridDim.x, ++it) {
      const uint32_t x_s = role(it, 0), dv_s = role(it, 2), dg_s = role(it, 3);
      named_bar_sync(kBarA, kCountA);  // dvalue and dgate are written, value / gate are read
      if (elect_one()) {
        // d x_hat = dvalue Wv' + dgate Wg' (columns 0-127, lanes = positions); Mv += dvalue^T x_hat (256-383), Mg +=
        // dgate^T x_hat (384-511). dvalue / dgate are [channel][position] tiles: MN-major as the A operand of the first
        // pair of GEMMs (M = positions), K-major as that of the second (M = channels, K = positions).
        tc_fence_after();
        constexpr uint32_t idesc_d = umma_idesc(128, C, true, true, kFmtF16, kFmtF16);
        constexpr uint32_t idesc_m = umma_idesc(128, C, false, true, kFmtF16, kFmtF16);
        const uint32_t accum = it != 0 ? 1u : 0u;
#pragma unroll
        for (int m = 0; m < 2; ++m) {
#pragma unroll
          for (int ks = 0; ks < 8; ++ks)
            umma_bf16(tmem_base, umma_desc_mnmajor((m == 0 ? dv_s : dg_s) + ks * 2048, 16384),
                      umma_desc_mnmajor((m == 0 ? wv_s : wg_s) + ks * 2048, 16384), idesc_d, (m | ks) != 0 ? 1u : 0u);
        }
        umma_commit(dx_done);
#pragma unroll
        for (int m = 0; m < 2; ++m) {
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) {
            const uint64_t kb = static_cast<uint64_t>((ks & 3) * 2);
            umma_bf16(tmem_base + 256 + m * 128, umma_desc_kmajor((m == 0 ? dv_s : dg_s) + (ks >> 2) * 16384) + kb,
                      umma_desc_mnmajor(x_s + ks * 2048, 16384), idesc_m, (ks != 0 ? 1u : 0u) | accum);
          }
        }
        umma_commit(grad_done);
      }
      __syncwarp();
      named_bar_sync(kBarB, kCountB);  // d x_hat has left tensor memory
      if (elect_one() && tile + static_cast<int>(gridDim.x) < p.num_tiles) issue_fwd(it + 1);
      __syncwarp();
    }
  } else if (warp == kBwdThreads / 32 + 1) {
    // ------------------------------------------------------------ copies
    auto issue_x = [&](int tile_i, int it_i) {
      const int row_i = tile_i / p.tiles_per_row;
      const int j_i = (tile_i - row_i * p.tiles_per_row) * 128;
      mbar_arrive_expect_tx(x_full, kZHalves * 16384);
#pragma unroll
      for (int kh = 0; kh < kZHalves; ++kh) tma_load_3d(role(it_i, 0) + kh * 16384, &map_x, x_full, kh * 64, j_i, row_i);
    };
    auto issue_do = [&](int tile_i, int it_i) {
      const int row_i = tile_i / p.tiles_per_row;
      const int j_i = (tile_i - row_i * p.tiles_per_row) * 128;
      mbar_arrive_expect_tx(do_full, kBwdTile);
#pragma unroll
      for (int kh = 0; kh < 2; ++kh) tma_load_3d(role(it_i, 1) + kh * 16384, &map_do, do_full, j_i + kh * 64, 0, row_i);
    };
    auto issue_dx = [&](int tile_i) {
      const int row_i = tile_i / p.tiles_per_row;
      const int j_i = (tile_i - row_i * p.tiles_per_row) * 128;
      mbar_arrive_expect_tx(dx_full, kZHalves * 16384);
#pragma unroll
      for (int kh = 0; kh < kZHalves; ++kh) tma_load_3d(dx_s + kh * 16384, &map_dx, dx_full, kh * 64, j_i, row_i);
    };
    if (lane == 0) {
      mbar_arrive_expect_tx(w_full, 2 * kZHalves * 16384);
#pragma unroll
      for (int kh = 0; kh < kZHalves; ++kh) {
        tma_load_2d(wv_s + kh * 16384, &map_wv, w_full, kh * 64, 0);
        tma_load_2d(wg_s + kh * 16384, &map_wg, w_full, kh * 64, 0);
      }
      issue_x(blockIdx.x, 0);
      issue_do(blockIdx.x, 0);
    }
    __syncwarp();
    grid_dependency_wait();
    grid_dependents_launch();
    if (lane == 0) issue_dx(blockIdx.x);
    __syncwarp();
    int it = 0;
    for (int tile = blockIdx.x; tile < p.num_tiles; tile += gridDim.x, ++it) {
      const int next = tile + static_cast<int>(gridDim.x);
      const bool has_next = next < p.num_tiles;
      const int row = tile / p.tiles_per_row;
      const int j0 = (tile - row * p.tiles_per_row) * 128;
      const uint32_t dv_s = role(it, 2);
      named_bar_sync(kBarA, kCountA);  // dO is read
      if (lane == 0) {
        if constexpr (LAST) {
          if (p.dy != nullptr) {
#pragma unroll
            for (int kh = 0; kh < kZHalves; ++kh) tma_prefetch_3d(&map_dy, kh * 64, j0, row);
          }
        }
        if (has_next) issue_x(next, it + 1);
        thread_wait(grad_done, it & 1, abort_flag, p.status, kDevTimeoutProducer);
        if constexpr (LAST) {
          if (p.dy != nullptr) {
            mbar_arrive_expect_tx(dy_full, kZHalves * 16384);
#pragma unroll
            for (int kh = 0; kh < kZHalves; ++kh) tma_load_3d(dv_s + kh * 16384, &map_dy, dy_full, kh * 64, j0, row);
          }
        }
        if (has_next) issue_do(next, it + 1);
      }
      __syncwarp();
      named_bar_sync(kBarC, kCountB);  // the output tile is written, the running sum is read
      if (lane == 0) {
#pragma unroll
        for (int kh = 0; kh < kZHalves; ++kh) tma_store_3d(&map_out, dv_s + kh * 16384, kh * 64, j0, row);
        bulk_commit();
        if (has_next) issue_dx(next);
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
        while (!mbar_try_wait(w_full, 0) || !mbar_try_wait(x_full, last) || !mbar_try_wait(do_full, last) ||
               !mbar_try_wait(dx_full, last) || (LAST && p.dy != nullptr && !mbar_try_wait(dy_full, last))) {
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
    const int pos = q * 32 + lane;
    const uint32_t lane_sel = static_cast<uint32_t>(q * 32) << 16;
    const float gc_inv = p.grad_scale[1];
    const float c_value = p.consts[pos], c_gate_half = 0.5f * p.consts[128 + pos];  // this thread's channel
    // dvalue / dgate are formed on the transposed projections (TMEM lanes = contracted channels, columns = positions): a
    // thread owns channel `pos` (its lane) and the position quarter `part`, so its constants and its column sums are
    // scalars and dO, stored [channel][position], is read in 16-byte runs of positions.
    float acc_v = 0.f, acc_g = 0.f;
    const float2 c_value2 = make_float2(c_value, c_value), c_gate_half2 = make_float2(c_gate_half, c_gate_half);
    const float2 half2 = make_float2(0.5f, 0.5f), eight2 = make_float2(8.f, 8.f);
    auto pair_of = [](uint32_t lo, uint32_t hi) { return make_float2(__uint_as_float(lo), __uint_as_float(hi)); };
    // validity of the 32 positions of this warp's quarter, one bit each. The mask bytes of the NEXT tile are requested
    // before a GEMM wait and turned into the word after it, so that their latency is off the path.
    auto mask_bytes = [&](int row_i, int j_i, uint32_t& m_i, uint32_t& m_j, uint32_t& m_p) {
      const int b = row_i / p.n;
      const int i = row_i - b * p.n;
      const int j = j_i + part * 32 + lane;
      m_i = 1u, m_j = j < p.n ? 1u : 0u, m_p = 1u;
      if (j < p.n) {
        if (p.token_mask != nullptr) {
          m_i = p.token_mask[static_cast<size_t>(b) * p.n + i];
          m_j = p.token_mask[static_cast<size_t>(b) * p.n + j];
        }
        if (p.pair_mask != nullptr) m_p = p.pair_mask[(static_cast<size_t>(b) * p.n + i) * p.n + j];
      }
    };
    // tile -> (row, column block) without a division per tile
    const int step_rows = static_cast<int>(gridDim.x) / p.tiles_per_row;
    const int step_cols = static_cast<int>(gridDim.x) - step_rows * p.tiles_per_row;
    int row = static_cast<int>(blockIdx.x) / p.tiles_per_row;
    int jt = static_cast<int>(blockIdx.x) - row * p.tiles_per_row;
    uint32_t vbits;
    {
      uint32_t m_i, m_j, m_p;
      mask_bytes(row, jt * 128, m_i, m_j, m_p);
      vbits = __ballot_sync(0xFFFFFFFFu, m_i != 0u && m_j != 0u && m_p != 0u);
    }
    int it = 0;
    for (int tile = blockIdx.x; tile < p.num_tiles; tile += gridDim.x, ++it) {
      const int j = jt * 128 + pos;
      const uint32_t x_s = role(it, 0), do_s = role(it, 1), dv_s = role(it, 2), dg_s = role(it, 3);
      float rstd_in = 0.f;
      if constexpr (LAST) {
        if (j < p.n) rstd_in = __ldg(p.rstd + static_cast<size_t>(row) * p.ld + j);
      }
      thread_wait(fwd_done, it & 1, abort_flag, p.status, kDevTimeoutEpilogue);
      __syncwarp();
      tc_fence_after();
      thread_wait(do_full, it & 1, abort_flag, p.status, kDevTimeoutStats);
      __syncwarp();
      // ---- dvalue, dgate for this thread's channel and 32 positions, stored [channel][position]
      {
        uint32_t dg_p[16];  // (the dgate buffer still holds the previous tile's output while its store reads it)
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          uint32_t vv[16], vg[16];
          tmem_ld16(tmem_base + lane_sel + part * 32 + hf * 16, vv);
          tmem_ld16(tmem_base + lane_sel + 128 + part * 32 + hf * 16, vg);
          uint4 dov[2];
#pragma unroll
          for (int k4 = 0; k4 < 2; ++k4) dov[k4] = ld_chunk(do_s + tile_chunk(pos, part * 4 + hf * 2 + k4));
          tmem_ld_wait();
#pragma unroll
          for (int k4 = 0; k4 < 2; ++k4) {
            const uint32_t dw[4] = {dov[k4].x, dov[k4].y, dov[k4].z, dov[k4].w};
            uint32_t ov[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              float2 d_o = f16x2_to_float2(dw[t]);
              const int e0 = k4 * 8 + 2 * t;
              if (vbits != 0xFFFFFFFFu) {
                d_o.x = ((vbits >> (hf * 16 + e0)) & 1u) ? d_o.x : 0.f;
                d_o.y = ((vbits >> (hf * 16 + e0 + 1)) & 1u) ? d_o.y : 0.f;
              }
              // (packed fp32 pairs: this pass is bound by its instruction count)
              const float2 val = __fadd2_rn(pair_of(vv[e0], vv[e0 + 1]), c_value2);
              const float2 gh = __ffma2_rn(pair_of(vg[e0], vg[e0 + 1]), half2, c_gate_half2);
              const float2 th = make_float2(tanh_approx(gh.x), tanh_approx(gh.y));
              const float2 sg = __ffma2_rn(th, half2, half2);
              // the contraction's outputs are stored times 2^-4: 16 sg = 8 tanh + 8
              const float2 dv = __fmul2_rn(d_o, __ffma2_rn(th, eight2, eight2));
              const float2 dg = __fmul2_rn(dv, __ffma2_rn(make_float2(-val.x, -val.y), sg, val));
              // (one chain in the order of the positions)
              acc_v += dv.x, acc_v += dv.y;
              acc_g += dg.x, acc_g += dg.y;
              ov[t] = pack_f16x2_sat(dv);
              dg_p[hf * 8 + k4 * 4 + t] = pack_f16x2_sat(dg);
            }
            st_chunk(dv_s + tile_chunk(pos, part * 4 + hf * 2 + k4), ov[0], ov[1], ov[2], ov[3]);
          }
        }
        if (it != 0) thread_wait(out_free, (it - 1) & 1, abort_flag, p.status, kDevTimeoutStats);
#pragma unroll
        for (int k4 = 0; k4 < 4; ++k4)
          st_chunk(dg_s + tile_chunk(pos, part * 4 + k4), dg_p[k4 * 4], dg_p[k4 * 4 + 1], dg_p[k4 * 4 + 2], dg_p[k4 * 4 + 3]);
      }
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      named_bar_arrive(kBarA, kCountA);
      // the next tile's mask bytes: requested now, used after the GEMM round
      const bool has_next = tile + static_cast<int>(gridDim.x) < p.num_tiles;
      row += step_rows, jt += step_cols;
      if (jt >= p.tiles_per_row) jt -= p.tiles_per_row, ++row;
      uint32_t m_i = 0u, m_j = 0u, m_p = 0u;
      if (has_next) mask_bytes(row, jt * 128, m_i, m_j, m_p);
      thread_wait(dx_done, it & 1, abort_flag, p.status, kDevTimeoutEpilogue);
      __syncwarp();
      tc_fence_after();
      uint32_t vt[kZChunks][8];
#pragma unroll
      for (int ch = 0; ch < kZChunks; ++ch) tmem_ld8(tmem_base + lane_sel + part * kZCh + ch * 8, vt[ch]);
      uint4 xh[LAST ? kZChunks : 1];
      if constexpr (LAST) {
        // x_hat is read for the last time before barrier B: the next tile's dvalue is written over it
#pragma unroll
        for (int ch = 0; ch < kZChunks; ++ch) xh[ch] = ld_chunk(x_s + tile_chunk(pos, part * kZChunks + ch));
      }
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      named_bar_arrive(kBarB, kCountB);
      vbits = __ballot_sync(0xFFFFFFFFu, m_i != 0u && m_j != 0u && m_p != 0u);
      // ---- add the running d x_hat; !LAST: write it back, LAST: LayerNorm backward + residual -> dz
      thread_wait(dx_full, it & 1, abort_flag, p.status, kDevTimeoutStats);
      __syncwarp();
      if constexpr (!LAST) {
        uint32_t o[kZChunks][4];
#pragma unroll
        for (int ch = 0; ch < kZChunks; ++ch) {
          const uint4 in = ld_chunk(dx_s + tile_chunk(pos, part * kZChunks + ch));
          const uint32_t iw[4] = {in.x, in.y, in.z, in.w};
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const float2 a = f16x2_to_float2(iw[t]);
            o[ch][t] = pack_f16x2_sat(
                make_float2(__uint_as_float(vt[ch][2 * t]) + a.x, __uint_as_float(vt[ch][2 * t + 1]) + a.y));
          }
        }
        thread_wait(grad_done, it & 1, abort_flag, p.status, kDevTimeoutEpilogue);  // the GEMMs read the dvalue buffer
#pragma unroll
        for (int ch = 0; ch < kZChunks; ++ch)
          st_chunk(dv_s + tile_chunk(pos, part * kZChunks + ch), o[ch][0], o[ch][1], o[ch][2], o[ch][3]);
      } else {
        float tot[kZCh];
        float s1 = 0.f, s2 = 0.f;
#pragma unroll
        for (int ch = 0; ch < kZChunks; ++ch) {
          const uint4 in = ld_chunk(dx_s + tile_chunk(pos, part * kZChunks + ch));
          const uint32_t iw[4] = {in.x, in.y, in.z, in.w};
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
        // the partial sums go where this thread's part of the running sum was
        asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(dx_s + tile_chunk(pos, part * kZChunks)), "f"(s1), "f"(s2) : "memory");
        named_bar_sync(1, kBwdThreads);
        float m1 = 0.f, m2 = 0.f;
#pragma unroll
        for (int k = 0; k < kBwdParts; ++k) {
          float a, b;
          asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(a), "=f"(b) : "r"(dx_s + tile_chunk(pos, k * kZChunks)));
          m1 += a, m2 += b;
        }
        m1 *= 1.0f / C, m2 *= 1.0f / C;
        const float rs = rstd_in * gc_inv;
        // dy arrives where the output goes; without it (no residual) that buffer is free once the GEMMs have read it
        if (p.dy != nullptr) thread_wait(dy_full, it & 1, abort_flag, p.status, kDevTimeoutStats);
        else thread_wait(grad_done, it & 1, abort_flag, p.status, kDevTimeoutEpilogue);
#pragma unroll
        for (int ch = 0; ch < kZChunks; ++ch) {
          const uint32_t addr = dv_s + tile_chunk(pos, part * kZChunks + ch);
          uint4 dyv = make_uint4(0u, 0u, 0u, 0u);
          if (p.dy != nullptr) dyv = ld_chunk(addr);
          const uint32_t xw[4] = {xh[ch].x, xh[ch].y, xh[ch].z, xh[ch].w};
          const uint32_t dw[4] = {dyv.x, dyv.y, dyv.z, dyv.w};
          uint32_t o[4];
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const float2 x = f16x2_to_float2(xw[t]);
            const float2 r = bf16x2_to_float2(dw[t]);
            o[t] = pack_bf16x2(fmaf(rs, tot[ch * 8 + 2 * t] - m1 - x.x * m2, r.x),
                               fmaf(rs, tot[ch * 8 + 2 * t + 1] - m1 - x.y * m2, r.y));
          }
          st_chunk(addr, o[0], o[1], o[2], o[3]);
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      named_bar_arrive(kBarC, kCountB);
    }
    // ---- per-CTA partials of the weight gradients and of the column sums
    thread_wait(grad_done, (it - 1) & 1, abort_flag, p.status, kDevTimeoutEpilogue);
    __syncwarp();
    tc_fence_after();
    float* pm = p.part_m + static_cast<size_t>(blockIdx.x) * 2 * 128 * 128;
#pragma unroll
    for (int m = 0; m < 2; ++m) {
#pragma unroll
      for (int ch = 0; ch < kBwdChunks; ++ch) {
        uint32_t v[8];
        tmem_ld8(tmem_base + lane_sel + 256 + m * 128 + part * kBwdCh + ch * 8, v);
        tmem_ld_wait();
        store_partial(pm + m * 128 * 128, pos, part * kBwdChunks + ch, v);
      }
    }
    // column sums: the four position quarters of a channel, fixed order (through the running sum's buffer, read by all)
    named_bar_sync(1, kBwdThreads);
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(dx_s + (part * 128 + pos) * 8), "f"(acc_v), "f"(acc_g) : "memory");
    named_bar_sync(1, kBwdThreads);
    if (threadIdx.x < 128) {
      float a, b;
      sum_partials(dx_s, threadIdx.x, a, b);
      float* ps = p.part_s + static_cast<size_t>(blockIdx.x) * 2 * 128;
      ps[threadIdx.x] = a;
      ps[128 + threadIdx.x] = b;
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

// ------------------------------------------------------------------------------------------------ small kernels
// Largest |dy| (bf16) over the blocks `block` of `blocks` of a launch, and from it the scale of the gradient tiles:
// scale[0] = c = the power of two that brings max |dy| into [8, 16), scale[1] = 1 / c (c = 1 for a zero gradient). `words`
// (zeroed before the launch): [0] the maximum as the bits of a non-negative float, [1] blocks that have arrived; the last
// one to arrive forms the scale, so no launch of its own is needed for it.
__device__ __forceinline__ void amax_and_scale(const uint4* dy, size_t n_chunks, int block, int blocks, unsigned int* words,
                                               float* scale) {
  // |x| of a bf16 pair compares like the unsigned integer of its bits with the sign cleared, so the maximum is taken on
  // the packed halves; eight loads per thread in flight
  constexpr int kFlight = 8;
  uint32_t mx = 0u;
  auto fold = [&](const uint4& v) {
    const uint32_t w[4] = {v.x & 0x7FFF7FFFu, v.y & 0x7FFF7FFFu, v.z & 0x7FFF7FFFu, v.w & 0x7FFF7FFFu};
#pragma unroll
    for (int t = 0; t < 4; ++t) mx = __vmaxu2(mx, w[t]);
  };
  const size_t step = static_cast<size_t>(blocks) * blockDim.x;
  for (size_t i = block * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n_chunks; i += kFlight * step) {
    uint4 v[kFlight];
#pragma unroll
    for (int u = 0; u < kFlight; ++u) v[u] = i + u * step < n_chunks ? __ldg(dy + i + u * step) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int u = 0; u < kFlight; ++u) fold(v[u]);
  }
  const uint32_t top = (mx >> 16) > (mx & 0xFFFFu) ? (mx >> 16) : (mx & 0xFFFFu);
  float m = __uint_as_float(top << 16);
  if (!(m <= 3.0e38f)) m = 0.f;  // infinities and NaN do not set the scale
  __shared__ unsigned int block_max;
  if (threadIdx.x == 0) block_max = 0u;
  __syncthreads();
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, off));
  if ((threadIdx.x & 31) == 0 && m > 0.f) atomicMax(&block_max, __float_as_uint(m));
  __syncthreads();
  // one word-sized atomic per block: they all go to one address
  if (threadIdx.x == 0) {
    if (block_max != 0u) atomicMax(words, block_max);
    __threadfence();
  }
  if (threadIdx.x == 0 && atomicAdd(words + 1, 1u) == static_cast<unsigned int>(blocks) - 1u) {
    __threadfence();
    const float amax = __uint_as_float(atomicMax(words, 0u));
    float c = 1.0f;
    if (amax > 0.f) {
      int e = 0;
      frexpf(amax, &e);           // amax = f * 2^e, f in [0.5, 1)
      e = 4 - e;                  // amax * 2^(4 - e) in [8, 16)
      e = e > 100 ? 100 : (e < -100 ? -100 : e);
      c = ldexpf(1.0f, e);
    }
    scale[0] = c;
    scale[1] = 1.0f / c;
  }
}

// Weights for the backward kernels: all six matrices (PackArgs order: left, left gate, right, right gate, out, gate)
// as dense fp16 [128][128] with the LayerNorm gamma of their input folded in, W'[r][k] = W[r][k] gamma[k], and
// d[m][r] = sum_k W[r][k] beta[k] + bias[m][r] (fp32) behind them. One warp per matrix row.
constexpr size_t kBwdPackedD = 6 * 32768;
constexpr size_t kBwdPackedBytes = kBwdPackedD + 3072;  // 199680, a multiple of 1024
__device__ __forceinline__ void bwd_pack_row(const PackArgs& a, uint8_t* packed, int gw) {  // gw: 0 .. 767
  const int lane = threadIdx.x & 31;
  const int m = gw >> 7, row = gw & 127;
  const int n_rows = m < 4 ? 128 : a.c;  // a.c = d_pair: matrices 0..3 are [128, c], 4 (out) is [c, 128], 5 (gate) [c, c]
  const int k = m == 4 ? 128 : a.c;
  if (row >= n_rows) return;
  const bool active = lane * 4 < k;
  const float* gamma = (m == 4) ? a.ln_out_w : a.ln_in_w;
  const float* beta = (m == 4) ? a.ln_out_b : a.ln_in_b;
  float w[4] = {0.f, 0.f, 0.f, 0.f};
  if (!active) {
  } else if (a.f32_weights) {
    const float4 v = reinterpret_cast<const float4*>(static_cast<const float*>(a.w[m]) + static_cast<size_t>(row) * a.ld[m])[lane];
    w[0] = v.x, w[1] = v.y, w[2] = v.z, w[3] = v.w;
  } else {
    const uint2 v = reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(a.w[m]) + static_cast<size_t>(row) * a.ld[m])[lane];
    w[0] = bf16_lo(v.x), w[1] = bf16_hi(v.x), w[2] = bf16_lo(v.y), w[3] = bf16_hi(v.y);
  }
  const float4 g = active ? reinterpret_cast<const float4*>(gamma)[lane] : make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 b = active ? reinterpret_cast<const float4*>(beta)[lane] : make_float4(0.f, 0.f, 0.f, 0.f);
  const float gg[4] = {g.x, g.y, g.z, g.w}, bb[4] = {b.x, b.y, b.z, b.w};
  float d = 0.f;
  uint16_t o[4];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    o[t] = __half_as_ushort(__float2half_rn(fminf(fmaxf(w[t] * gg[t], -65504.f), 65504.f)));
    d = fmaf(w[t], bb[t], d);
  }
  if (active) {
    uint2 ov;
    ov.x = static_cast<uint32_t>(o[0]) | (static_cast<uint32_t>(o[1]) << 16);
    ov.y = static_cast<uint32_t>(o[2]) | (static_cast<uint32_t>(o[3]) << 16);
    reinterpret_cast<uint2*>(packed + static_cast<size_t>(m) * 32768)[row * (k / 4) + lane] = ov;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) d += __shfl_xor_sync(0xFFFFFFFFu, d, off);
  if (lane == 0)
    reinterpret_cast<float*>(packed + kBwdPackedD)[m * 128 + row] = d + (a.bias[m] != nullptr ? a.bias[m][row] : 0.f);
}


// One launch before the backward kernels: blocks 0 .. 96 * halves - 1 pack the weights of the halves (eight matrix rows
// each), the rest find max |dy| and the scale.
struct BwdSetupArgs {
  PackArgs w[2];
  uint8_t* packed[2];
  int pack_blocks;  // 96 per half
  const uint4* dy;
  size_t n_chunks;
  unsigned int* words;
  float* scale;
};
__global__ void __launch_bounds__(256) bwd_setup_kernel(const __grid_constant__ BwdSetupArgs a) {
  grid_dependents_launch();
  const int block = blockIdx.x;
  if (block < a.pack_blocks) {
    const int h = block >= 96 ? 1 : 0;
    bwd_pack_row(a.w[h], a.packed[h], (block - h * 96) * 8 + (threadIdx.x >> 5));
    return;
  }
  amax_and_scale(a.dy, a.n_chunks, block - a.pack_blocks, gridDim.x - a.pack_blocks, a.words, a.scale);
}

// Parameter gradients from the per-CTA partial sums M[m] = dOut_m^T x_hat (times c) and S[m] = column sums of dOut_m
// (times c) that the launches of the epilogue's and the prologue's backward left:
//   dW_m[r][k] = (M[m][r][k] gamma[k] + S[m][r] beta[k]) / c
//   dgamma[k]  = sum_m sum_r W_m[r][k] M[m][r][k] / c,   dbeta[k] = sum_m sum_r W_m[r][k] S[m][r] / c
// over the matrices that read that LayerNorm (the output one: matrix 4; the input one: the other five).
// One set of six 128 x 128 matrices ("half"): the unidirectional module has one, the bidirectional module two, whose
// matrices are row or column blocks of the module's wider parameters, hence the leading dimensions.
// Grid (128: group of four columns and quarter of the rows, 6 matrices, halves); a block of 512 threads adds 32 rows x 4
// columns of the partials, one group of CTAs per warp, every load of a thread in flight at once, and combines the groups
// in a fixed order: the sums, the parameter gradients and this block's share of the LayerNorm sums leave in one pass over
// the partials. The earlier form (a reduction after every launch that produced partials, then a kernel for the gradients on
// 6 x 8 blocks, and one block for the LayerNorm sums) was three to six launches of 5.2 us plus 10 and 5 us.
constexpr int kFinGroups = 16;
constexpr int kFinFlight = 10;  // 16 * 10 = 160 = the largest number of CTAs
struct BwdFinalHalf {
  PackArgs w;              // raw weights (this half's blocks, with their leading dimensions) and LayerNorm parameters
  const float* part_m[6];  // per matrix: partials [n_parts][2] matrices, at this matrix of CTA 0
  const float* part_s[6];  // per matrix: [n_parts][2][128]
  float* dw[6];            // fp32 gradient blocks
  int dw_ld[6];            // their leading dimensions
  float* ln_rows;          // [6][8][2][128]: the terms of dgamma and dbeta from 16 matrix rows each
  unsigned mask;           // bit m set: matrix m is present in this half
};
struct BwdFinalArgs {
  BwdFinalHalf half[2];
  int n_parts;
  const float* scale;  // [2]
};
// Sums over the CTAs, for the block's 32 lanes: four columns of a matrix row (`m` points at the row's columns in CTA 0's
// matrix, matrices `m_stride` floats apart) and the column sum belonging to the row (`col_sum` likewise, or null). Valid in
// warp 0. The order of the additions: partial i belongs to chain i mod 16, except that the partials of an incomplete last
// sixteen are added to chain i mod 4 if it has no partial i mod 4 + 12; then the chains four apart, then the four sums.
__device__ __forceinline__ void sum_partials_of_rows(const float* m, size_t m_stride, const float* col_sum, size_t s_stride,
                                                     int n_parts, float4& mv, float& sv) {
  __shared__ float4 comb[2][kFinGroups * 32];
  __shared__ float comb_s[2][kFinGroups * 32];
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
  float4 v[kFinFlight];
  float c[kFinFlight];
#pragma unroll
  for (int u = 0; u < kFinFlight; ++u) {
    const size_t i = g + u * kFinGroups;
    const bool there = g + u * kFinGroups < n_parts;
    v[u] = there ? __ldcg(reinterpret_cast<const float4*>(m + i * m_stride)) : make_float4(0.f, 0.f, 0.f, 0.f);
    c[u] = there && col_sum != nullptr ? __ldcg(col_sum + i * s_stride) : 0.f;
  }
  // partial i = g + 16 u of an incomplete sixteen that does not stay in its chain
  const int full = n_parts & ~(kFinGroups - 1);
  const bool moved = g >= 4 && full + g < n_parts && full + (g & 3) + 12 >= n_parts;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f), tail = s;
  float t = 0.f, tail_s = 0.f;
#pragma unroll
  for (int u = 0; u < kFinFlight; ++u) {
    if (moved && u * kFinGroups == full) tail = v[u], tail_s = c[u];
    else s.x += v[u].x, s.y += v[u].y, s.z += v[u].z, s.w += v[u].w, t += c[u];
  }
  comb[0][g * 32 + lane] = s, comb[1][g * 32 + lane] = tail;
  comb_s[0][g * 32 + lane] = t, comb_s[1][g * 32 + lane] = tail_s;
  __syncthreads();
  if (g != 0) return;
  float4 q[4];
  float qs[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    float4 x[4];
    float y[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) x[k] = comb[0][(r + 4 * k) * 32 + lane], y[k] = comb_s[0][(r + 4 * k) * 32 + lane];
#pragma unroll
    for (int k = 1; k < 4; ++k) {  // (zeros where nothing moved)
      const float4 e = comb[1][(r + 4 * k) * 32 + lane];
      x[0].x += e.x, x[0].y += e.y, x[0].z += e.z, x[0].w += e.w, y[0] += comb_s[1][(r + 4 * k) * 32 + lane];
    }
    q[r].x = (x[0].x + x[1].x) + (x[2].x + x[3].x), q[r].y = (x[0].y + x[1].y) + (x[2].y + x[3].y);
    q[r].z = (x[0].z + x[1].z) + (x[2].z + x[3].z), q[r].w = (x[0].w + x[1].w) + (x[2].w + x[3].w);
    qs[r] = (y[0] + y[1]) + (y[2] + y[3]);
  }
  mv.x = (q[0].x + q[1].x) + (q[2].x + q[3].x), mv.y = (q[0].y + q[1].y) + (q[2].y + q[3].y);
  mv.z = (q[0].z + q[1].z) + (q[2].z + q[3].z), mv.w = (q[0].w + q[1].w) + (q[2].w + q[3].w);
  sv = (qs[0] + qs[1]) + (qs[2] + qs[3]);
}
// One row of the terms of dgamma and dbeta: four columns of the weights and of M / c, and S / c.
struct LnRow {
  float w[4], mv[4], sv;
};
__global__ void __launch_bounds__(512) bwd_finalize_kernel(const __grid_constant__ BwdFinalArgs args) {
  grid_dependency_wait();
  grid_dependents_launch();
  const BwdFinalHalf& a = args.half[blockIdx.z];
  const int group = blockIdx.x >> 2, q = blockIdx.x & 3, m = blockIdx.y;
  const int n_rows = m < 4 ? 128 : a.w.c, n_cols = m == 4 ? 128 : a.w.c;  // a.w.c = d_pair: 128 or 64
  if (((a.mask >> m) & 1u) == 0u || q * 32 >= n_rows || group * 4 >= n_cols) return;
  float4 m4;
  float s1;
  const int r = q * 32 + (threadIdx.x & 31), k0 = group * 4;
  sum_partials_of_rows(a.part_m[m] + (group * 128 + r) * 4, 2 * 128 * 128, a.part_s[m] + r, 2 * 128, args.n_parts, m4, s1);
  if (threadIdx.x >= 32) return;
  const float cinv = args.scale[1];
  const float sv = s1 * cinv, mv[4] = {m4.x * cinv, m4.y * cinv, m4.z * cinv, m4.w * cinv};
  const float4 gamma = *reinterpret_cast<const float4*>((m == 4 ? a.w.ln_out_w : a.w.ln_in_w) + k0);
  const float4 beta = *reinterpret_cast<const float4*>((m == 4 ? a.w.ln_out_b : a.w.ln_in_b) + k0);
  const size_t wi = static_cast<size_t>(r) * a.w.ld[m] + k0;
  float w[4];
  if (a.w.f32_weights) {
    const float4 v = *reinterpret_cast<const float4*>(static_cast<const float*>(a.w.w[m]) + wi);
    w[0] = v.x, w[1] = v.y, w[2] = v.z, w[3] = v.w;
  } else {
    const uint2 v = *reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(a.w.w[m]) + wi);
    w[0] = bf16_lo(v.x), w[1] = bf16_hi(v.x), w[2] = bf16_lo(v.y), w[3] = bf16_hi(v.y);
  }
  float* dw = a.dw[m] + static_cast<size_t>(r) * a.dw_ld[m] + k0;
  dw[0] = fmaf(mv[0], gamma.x, sv * beta.x), dw[1] = fmaf(mv[1], gamma.y, sv * beta.y);
  dw[2] = fmaf(mv[2], gamma.z, sv * beta.z), dw[3] = fmaf(mv[3], gamma.w, sv * beta.w);
  __shared__ LnRow rows[32];
  rows[threadIdx.x] = {{w[0], w[1], w[2], w[3]}, {mv[0], mv[1], mv[2], mv[3]}, sv};
  __syncwarp();
  if (threadIdx.x < 8) {  // four columns of two groups of 16 rows, in the order of the rows
    const int t = threadIdx.x & 3, half = threadIdx.x >> 2;
    float ag = 0.f, ab = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const LnRow& x = rows[half * 16 + i];
      ag = fmaf(x.w[t], x.mv[t], ag);
      ab = fmaf(x.w[t], x.sv, ab);
    }
    float* dst = a.ln_rows + (m * 8 + q * 2 + half) * 256 + k0 + t;
    dst[0] = ag, dst[128] = ab;
  }
}
// Adds the LayerNorm terms in a fixed order. Grid 1 + halves: the input LayerNorm, then the output LayerNorm's 128 channels
// of each half; thread = gamma or beta and channel.
struct BwdLnArgs {
  const float* ln_rows[2];  // per half
  unsigned mask[2];
  int halves;
  float* d_in[2];   // dgamma, dbeta of the input LayerNorm [c]
  float* d_out[2];  // of the output LayerNorm [128 * halves]: half h at + 128 h
  int c;            // d_pair
};
__global__ void __launch_bounds__(256) bwd_finalize_ln_kernel(const BwdLnArgs a) {
  grid_dependency_wait();
  grid_dependents_launch();
  const int vec = threadIdx.x >> 7, k = threadIdx.x & 127;
  const bool input = blockIdx.x == 0;
  if (input && k >= a.c) return;
  float s = 0.f;
  for (int h = input ? 0 : static_cast<int>(blockIdx.x) - 1; h < (input ? a.halves : static_cast<int>(blockIdx.x)); ++h) {
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      if ((m == 4) == input || ((a.mask[h] >> m) & 1u) == 0u) continue;
      float x[8], sm = 0.f;
#pragma unroll
      for (int rb = 0; rb < 8; ++rb) x[rb] = m < 4 || rb * 16 < a.c ? __ldcg(a.ln_rows[h] + (m * 8 + rb) * 256 + threadIdx.x) : 0.f;
#pragma unroll
      for (int rb = 0; rb < 8; ++rb) sm += x[rb];
      s += sm;
    }
  }
  (input ? a.d_in[vec] : a.d_out[vec] + 128 * (static_cast<int>(blockIdx.x) - 1))[k] = s;
}

}  // namespace trimul
