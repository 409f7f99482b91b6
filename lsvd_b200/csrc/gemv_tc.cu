// Weight-streaming W8A8 product for decode batches (1..64 tokens) on the fifth-generation tensor cores:
//   acc[tok, row] = sum_k a[tok, k] * w[row, k]      (int8 x int8 -> int32, exact), dequantised in the epilogue.
//
// A product of a decode step is an HBM stream of its weights.  Here the weights are the M operand of
// tcgen05.mma kind::i8 (128 weight rows x 16..64 tokens per instruction), so the tokens' share of the work -- fragment
// loads and MMAs once per 16 weight rows in the mma.sync forms -- costs nothing that the stream would notice: a block
// brings 128 rows x 128 bytes of K per stage into shared memory by TMA, together with the same 128 bytes of every token
// row, and one thread issues four MMAs per stage.
//   * A tile is 128 rows of one matrix, or 64 + 64 rows of a gate/up pair.  The blocks of a cluster share a tile and split
//     its K range block by block (block r of c takes the 128-byte K blocks r, r + c, ..., so that the cluster reads
//     adjacent bytes of a row at the same time); their exact int32 sums meet in distributed shared memory, token quad q in
//     block q mod c, which adds them and runs the epilogue for its tokens.
//   * With prefetch 2 the first stages' weights are requested before griddepcontrol.wait: they travel while the quantiser in front of the
//     product is still running (programmatic stream serialisation), which takes the ramp-up of the stream out of the
//     chain of short dependent kernels that a decode step is.
// Measured against the mma.sync forms in the FFN's chains (B200, graph replay): hybrid FFN 4096/11008 at 1 / 29 tokens
// 51.3 / 62.2 -> 45.3 / 55.5 us per call, 5120/13824 at 64 tokens 159 -> 88 us, mixffn 4096/14336 at 32 tokens 124 -> 79 us.
// A launch on its own (ncu, cold) is bound by its start, the sums and the epilogue: 45 MB pair 19.8 us, 45 MB down projection
// 15.3, 4 MB 7.8 at 16 tokens; 58.7 MB pair 19.0 at 32 (3.1 TB/s).  A block's start takes about 1 us, sums and epilogue 1.5 to 3.
// Every wait on an mbarrier is bounded; one that gives up, in whatever role, reports LSVD_ERR_TIMEOUT, and the block still
// attends the cluster barriers, waits for its own copies and MMAs and releases its tensor memory.
#include <algorithm>

#include "gemv.cuh"
#include "tc5.cuh"
#include "tma.cuh"

namespace lsvd {

constexpr int kTcEpiWarps = 8;           // two per quarter of the TMEM lanes
constexpr int kTcThreads = 64 + kTcEpiWarps * 32;      // TMA producer, MMA issuer, epilogue warps
constexpr int kTcMaxStages = 12;
constexpr int kTcWBytes = 128 * 128;     // the weights of a stage
constexpr int kTcSmem = 110 * 1024;      // two blocks per SM

struct TcParams {
  GemvParams g;
  int32_t dual, split, kb;               // a pair; with its own activations for the second matrix; 128-byte blocks of K
  int32_t ntok, stages;                  // tokens rounded up to a multiple of 16; stages of the ring
};

struct TcMaps {
  CUtensorMap w, w2, a, a2;
};

__device__ __forceinline__ uint32_t tc_cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void tc_cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// The token quads of one block: the cluster's shares are added and run through gemv_store's arithmetic.  A warp takes 64
// channels of four tokens, a lane two neighbouring channels; the channel scales come in registers, the token scales from
// shared memory, and the residual of the four tokens is requested before the sums.
template <int CSL, bool DUAL, bool MIX>
__device__ __forceinline__ void tc_epilogue(const GemvParams& g, const int4* part, const float* sa, const float* sb, float2 w0, float2 w1,
                                            int squads, int rank, int row0, int ew, int lane) {
  constexpr int CS = 1 << CSL;
  const int c = (DUAL ? 0 : (ew & 1) * 64) + 2 * lane, row = row0 + c;
  const bool row_ok = row < g.n;                 // n is a multiple of 16: both channels or none
  const bool vec = ((reinterpret_cast<uintptr_t>(g.out) & 3) | (g.out_row_stride & 1) | (g.out_col & 1)) == 0;
  const bool rvec = ((reinterpret_cast<uintptr_t>(g.residual) & 3) | (g.residual_row_stride & 1)) == 0;
  for (int u = ew; u < (DUAL ? squads : 2 * squads); u += kTcEpiWarps) {
    const int sq = DUAL ? u : u >> 1;
    const int tok0 = 4 * ((sq << CSL) | rank);
    if (tok0 >= g.m) break;
    __half2 res[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      res[j] = __floats2half2_rn(0.f, 0.f);
      if (g.residual != nullptr && row_ok && tok0 + j < g.m) {
        const __half* r = g.residual + (tok0 + j) * g.residual_row_stride + row;
        res[j] = rvec ? *reinterpret_cast<const __half2*>(r) : __halves2half2(r[0], r[1]);
      }
    }
    int x[2][4] = {}, y[2][4] = {};
#pragma unroll
    for (int r = 0; r < CS; ++r) {
      const int4* src = part + (r * squads + sq) * 128 + c;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int4 v = src[e];
        x[e][0] += v.x; x[e][1] += v.y; x[e][2] += v.z; x[e][3] += v.w;
        if (DUAL) {
          const int4 z = src[64 + e];
          y[e][0] += z.x; y[e][1] += z.y; y[e][2] += z.z; y[e][3] += z.w;
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int tok = tok0 + j;
      if (tok >= g.m) break;                     // the same for the whole warp
      const float ta = sa[4 * sq + j], tb = DUAL ? sb[4 * sq + j] : 0.f;
      float f[2] = {(static_cast<float>(x[0][j]) * ta) * w0.x, (static_cast<float>(x[1][j]) * ta) * w0.y};
      float av = 0.f;
      if (row_ok) {
        const int64_t at = static_cast<int64_t>(tok) * g.n + row;
        if (g.acc_out != nullptr) { g.acc_out[at] = x[0][j]; g.acc_out[at + 1] = x[1][j]; }
        if (DUAL && g.acc2_out != nullptr) { g.acc2_out[at] = y[0][j]; g.acc2_out[at + 1] = y[1][j]; }
        if (!DUAL && g.out_f32 != nullptr) { g.out_f32[at] = f[0]; g.out_f32[at + 1] = f[1]; }
        if (g.out != nullptr) {
          __half o[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            o[e] = __float2half_rn(f[e]);
            if (DUAL) {
              const float f1 = (static_cast<float>(y[e][j]) * tb) * (e ? w1.y : w1.x);
              if (MIX) {
                f[e] = f1 * (f[e] * (1.0f / (1.0f + expf(-f[e]))));
                o[e] = __float2half_rn(f[e]);
              } else {
                const __half up = __float2half_rn(f1);
                const __half sg = __float2half_rn(silu_f(__half2float(o[e])));
                o[e] = __float2half_rn(__half2float(sg) * __half2float(up));
              }
            }
            if (g.residual != nullptr) o[e] = __float2half_rn(__half2float(o[e]) + __half2float(e ? __high2half(res[j]) : __low2half(res[j])));
            av = fmaxf(av, fabsf(f[e]));
          }
          __half* dst = g.out + tok * g.out_row_stride + g.out_col + row;
          if (vec) {
            *reinterpret_cast<__half2*>(dst) = __halves2half2(o[0], o[1]);
          } else {
            dst[0] = o[0];
            dst[1] = o[1];
          }
        }
      }
      if (g.row_absmax != nullptr) {
        // absmax_split is a multiple of 16: groups of eight lanes (16 channels) belong to one word
        av = fmaxf(av, __shfl_xor_sync(0xffffffffu, av, 1));
        av = fmaxf(av, __shfl_xor_sync(0xffffffffu, av, 2));
        av = fmaxf(av, __shfl_xor_sync(0xffffffffu, av, 4));
        if ((lane & 7) == 0 && row_ok)
          atomicMax(g.row_absmax + tok * g.row_absmax_stride + (row >= g.absmax_split ? 1 : 0), __float_as_uint(av));
      }
    }
  }
}

template <int CSL>
__global__ void __launch_bounds__(kTcThreads, 2) w8a8_gemv_tc_kernel(const __grid_constant__ TcMaps maps, const __grid_constant__ TcParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  __shared__ uint64_t full_bar[kTcMaxStages], empty_bar[kTcMaxStages], acc_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile uint32_t abort_flag;
  __shared__ int issued;                   // K blocks that the producer has requested (a register live to the end: 10 % a call)
  __shared__ float sa[64], sb[64];         // token scales of this block's token slots

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int cs = 1 << CSL;
  const int rank = CSL ? static_cast<int>(tc_cluster_rank()) : 0;
  const int tile = blockIdx.x >> CSL;
  const int nb = p.split ? 2 * p.ntok : p.ntok;                    // columns of the MMA
  const int stage_bytes = kTcWBytes + nb * 128;
  const int nk = (p.kb - rank + cs - 1) >> CSL;                    // this block's K blocks: rank, rank + cs, ... (one at least)
  int4* part = reinterpret_cast<int4*>(ring + p.stages * stage_bytes);   // [source block][token quad][128]: four tokens
  const int squads = ((p.ntok >> 2) + cs - 1) >> CSL;               // token quad Q belongs to block Q mod cs
  const uint32_t tmem_cols = nb <= 32 ? 32u : (nb <= 64 ? 64u : 128u);

  grid_dependency_release();
  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&acc_bar, 1);
    abort_flag = 0;
    issued = nk;
    fence_mbar_init();
  }
  if (warp == 1) tmem_alloc(&tmem_slot, tmem_cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (CSL) tc_cluster_arrive();            // "this block is running": its shared memory may be written after the wait below
  const uint32_t tmem = tmem_slot;
  const int row0 = tile * (p.dual ? 64 : 128);

  if (warp == 0) {
    if (lane == 0) {
      const CUtensorMap* mw = &maps.w;
      const CUtensorMap* mw2 = p.dual ? &maps.w2 : mw;
      const int row1 = p.dual ? row0 : row0 + 64;
      const int pre = min(nk, p.stages);
      auto weights = [&](int i, int s) {
        uint8_t* st = ring + s * stage_bytes;
        const int x = ((i << CSL) + rank) * 128;
        mbar_arrive_expect_tx(&full_bar[s], stage_bytes);
        tma_load_2d(st, mw, x, row0, &full_bar[s]);
        tma_load_2d(st + kTcWBytes / 2, mw2, x, row1, &full_bar[s]);
      };
      auto tokens = [&](int i, int s) {
        uint8_t* st = ring + s * stage_bytes + kTcWBytes;
        const int x = ((i << CSL) + rank) * 128;
        tma_load_2d(st, &maps.a, x, 0, &full_bar[s]);
        if (p.split) tma_load_2d(st + p.ntok * 128, &maps.a2, x, 0, &full_bar[s]);
      };
      if (!p.g.prefetch) grid_dependency_wait();
      for (int i = 0; i < pre; ++i) weights(i, i);
      if (p.g.prefetch) grid_dependency_wait();
      for (int i = 0; i < pre; ++i) tokens(i, i);
      int s = 0;
      for (int i = pre; i < nk; ++i) {
        if (abort_flag || !mbar_wait_bounded(&empty_bar[s], ((i / p.stages) & 1) ^ 1)) {
          report_status(p.g.status_word, LSVD_ERR_TIMEOUT);
          abort_flag = 1;
          issued = i;
          break;
        }
        weights(i, s);
        tokens(i, s);
        if (++s == p.stages) s = 0;
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = umma_idesc_i8(128, nb);
      int s = 0;
      for (int i = 0; i < nk; ++i) {
        if (abort_flag || !mbar_wait_bounded(&full_bar[s], (i / p.stages) & 1)) {
          report_status(p.g.status_word, LSVD_ERR_TIMEOUT);
          abort_flag = 1;
          break;
        }
        tc_fence_after();
        const uint64_t wd = smem_desc_k_major_sw128(ring + s * stage_bytes);
        const uint64_t ad = smem_desc_k_major_sw128(ring + s * stage_bytes + kTcWBytes);
#pragma unroll
        for (int q = 0; q < 4; ++q) umma_i8(tmem, wd + 2 * q, ad + 2 * q, idesc, (i > 0 || q > 0) ? 1u : 0u);
        umma_commit(&empty_bar[s]);
        if (++s == p.stages) s = 0;
      }
      umma_commit(&acc_bar);
    }
  }
  __syncwarp();

  const int ew = warp - 2;
  float2 w0 = make_float2(0.f, 0.f), w1 = w0;          // channel scales of this thread's two channels
  if (warp >= 2) {
    grid_dependency_wait();                  // the epilogue reads token scales and the residual, and writes the result
    const int row = row0 + (p.dual ? 0 : (ew & 1) * 64) + 2 * lane;
    if (row < p.g.n) {
      if (p.g.w_scale != nullptr) w0 = make_float2(p.g.w_scale[row], p.g.w_scale[row + 1]);
      if (p.dual && p.g.w2_scale != nullptr) w1 = make_float2(p.g.w2_scale[row], p.g.w2_scale[row + 1]);
    }
    const int slot = threadIdx.x - 64;
    if (slot < 4 * squads) {
      const int tok = 4 * (((slot >> 2) << CSL) | rank) + (slot & 3);
      const bool on = tok < p.g.m && p.g.a_scale != nullptr;
      sa[slot] = on ? p.g.a_scale[tok * p.g.a_scale_stride] : 0.f;
      sb[slot] = (on && p.split && p.g.a2_scale != nullptr) ? p.g.a2_scale[tok * p.g.a2_scale_stride] : sa[slot];
    }
    const int quarter = warp & 3;
    const int ch = quarter * 32 + lane;      // row of the tile
    uint32_t remote[cs];
    const uint32_t mine = smem_u32(part + rank * squads * 128 + ch);
#pragma unroll
    for (int d = 0; d < cs; ++d) {
      remote[d] = mine;
      if (CSL) asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote[d]) : "r"(mine), "r"(d));
    }
    if (CSL) tc_cluster_wait();
    if (!mbar_wait_bounded(&acc_bar, 0)) {
      report_status(p.g.status_word, LSVD_ERR_TIMEOUT);
      abort_flag = 1;
    }
    tc_fence_after();
    const uint32_t taddr = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + (p.split && quarter >= 2 ? static_cast<uint32_t>(p.ntok) : 0u);
    for (int c = 16 * (ew >> 2); c < p.g.m; c += 32) {
      uint32_t v[16];
      __syncwarp();
      tmem_ld16(taddr + c, v);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (c + 4 * q < p.g.m) {
          const int sq = ((c >> 2) + q) >> CSL;          // c is a multiple of 16: the block is q mod cs, known at compile time up to 4
          const uint32_t base = CSL <= 2 ? remote[q & (cs - 1)] : ((c >> 4) & 1 ? remote[(4 + q) & (cs - 1)] : remote[q & (cs - 1)]);
          asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(base + static_cast<uint32_t>(sq) * 2048u), "r"(v[4 * q]),
                       "r"(v[4 * q + 1]), "r"(v[4 * q + 2]), "r"(v[4 * q + 3]) : "memory");
        }
      }
    }
    tc_fence_before();
  } else if (CSL) {
    tc_cluster_wait();
  }
  if (CSL) {
    tc_cluster_arrive();
    tc_cluster_wait();
  } else {
    __syncthreads();
  }
  if (warp < 2) {
    // Whoever gave up, and whenever: the barrier above has ended every role, so the flag is final.  This block's copies must
    // have landed before its shared memory goes, its MMAs have ended before their accumulators are released.
    if (lane == 0 && abort_flag) {
      if (warp == 1) mbar_wait_bounded(&acc_bar, 0);
      else for (int i = max(0, issued - p.stages); i < issued; ++i) mbar_wait_bounded(&full_bar[i % p.stages], (i / p.stages) & 1);
    }
    __syncwarp();
    if (warp == 1) {
      tc_fence_after();
      tmem_dealloc(tmem, tmem_cols);
    }
    return;
  }

  if (!p.dual) {
    tc_epilogue<CSL, false, false>(p.g, part, sa, sb, w0, w1, squads, rank, row0, ew, lane);
  } else if (p.g.epilogue == 2) {
    tc_epilogue<CSL, true, true>(p.g, part, sa, sb, w0, w1, squads, rank, row0, ew, lane);
  } else {
    tc_epilogue<CSL, true, false>(p.g, part, sa, sb, w0, w1, squads, rank, row0, ew, lane);
  }
}

// Blocks per tile: the cluster grows (to at most 8, the portable size) until the tiles fill the SMs once, as long as every
// block keeps a K block.  45 MB gate/up pair at 32 tokens, 5504 channels (86 tiles): 2 blocks per tile 16.1 us with its
// quantiser, 4 blocks 17.6; 45 MB down projection (32 tiles): 8 blocks 19.3, 4 blocks 21.
// Shared memory: two blocks per SM (110 KB each), so that the blocks of the next product of a chain find room for their
// first stages while this one drains; 76 KB measured 10 % slower on the mixffn step (fewer bytes in flight), 160 KB -- one
// block per SM -- 35 %.
int launch_gemv_tc(const GemvParams& g, bool dual, bool split, cudaStream_t st) {
  TcMaps maps;
  TcParams p{};
  p.g = g;
  p.g.prefetch = g.prefetch == 2 ? 1 : 0;          // a hint does not say that the weights are complete
  p.dual = dual ? 1 : 0;
  p.split = split ? 1 : 0;
  p.ntok = (g.m + 15) / 16 * 16;
  p.kb = (g.k + 127) / 128;
  int rc = make_map_k128(&maps.w, g.w, g.n, g.k, g.w_row_stride, 64);
  if (rc == LSVD_OK && dual) rc = make_map_k128(&maps.w2, g.w2, g.n, g.k, g.w2_row_stride, 64);
  if (rc == LSVD_OK) rc = make_map_k128(&maps.a, g.a, g.m, g.k, g.m == 1 ? g.k : g.a_row_stride, p.ntok);
  if (rc == LSVD_OK && split) rc = make_map_k128(&maps.a2, g.a2, g.m, g.k, g.m == 1 ? g.k : g.a2_row_stride, p.ntok);
  if (rc != LSVD_OK) return rc;
  const int per = dual ? 64 : 128, tiles = (g.n + per - 1) / per;
  const int sms = std::max(1, device_sm_count());
  int csl = 0;
  while (csl < 3 && tiles << csl < sms && p.kb >= 2 << csl) ++csl;
  const int stage_bytes = kTcWBytes + (split ? 2 : 1) * p.ntok * 128;
  const int part_bytes = (((p.ntok >> 2) + (1 << csl) - 1) >> csl << csl) * 2048;
  p.stages = std::max(2, std::min({kTcMaxStages, (p.kb + (1 << csl) - 1) >> csl, (kTcSmem - part_bytes - 1024) / stage_bytes}));
  const int smem = p.stages * stage_bytes + part_bytes + 1024;
  void (*kern)(TcMaps, TcParams) = csl == 0 ? w8a8_gemv_tc_kernel<0> : csl == 1 ? w8a8_gemv_tc_kernel<1>
                                   : csl == 2 ? w8a8_gemv_tc_kernel<2> : w8a8_gemv_tc_kernel<3>;
  LSVD_CUDA_TRY(ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem));
  LSVD_CUDA_TRY(launch_chained(kern, dim3(tiles << csl), dim3(kTcThreads), smem, st, 1 << csl, p.g.prefetch != 0, maps, p));
  return LSVD_OK;
}

}  // namespace lsvd
