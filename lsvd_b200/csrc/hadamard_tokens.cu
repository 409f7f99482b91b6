// (H_K kron H_nb) rotation + per-token int8 quantisation, one token per block: nb = 64 or 128, K <= 176 (the hidden vector
// 11008 = 172 x 64 and 13824 = 108 x 128 among them).
//   y[k', j] = fp16(sum_k had_K[k', k] * fp16(fwht(x[k, :])[j] / sqrt(cols))),   codes and scale of the whole row
// fake_quant/utils/hadamard_utils.py:106-113, fake_quant/utils/quant_utils.py:201-212.
//
// A token is 22 KB in and 11 KB out against K^2 nb fp16 multiply-adds (0.25 us of mma.sync per token and SM), 11 000
// butterflies and 11 000 roundings, so the kernel is built around instruction counts:
//   * the blocks are persistent and keep their rows of had_K as MMA fragments in registers (a warp holds MT 16-row tiles
//     over the whole K): had_K is read once per block, not once per token;
//   * the next token travels by cp.async while this one is transformed;
//   * a lane holds eight consecutive entries of a block: three butterfly strides in registers, the others by shuffles -- the
//     same additions in the same order as the reference's loop; the rotated blocks are stored row by row and become B
//     fragments by ldmatrix.trans (row pitch nb + 8 halves: no bank conflicts);
//   * results wait as packed fp16 pairs for the row's scale, codes are three FMA-pipe operations and an addition each
//     (ActCoder), staged in the token's own input buffer and stored 16 bytes at a time.
// MT = 2 halves the shared-memory reads of B fragments per MMA (many tokens: throughput); MT = 1 has twice the warps (a
// decode batch, at most one token per SM: latency).
#include <algorithm>

#include "common.cuh"
#include "devfn.cuh"

namespace lsvd {

__device__ __forceinline__ void ldsm_x4_trans(uint32_t (&d)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(addr) : "memory");
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

template <int KT, int NB, int MT>
__global__ void __launch_bounds__((KT + MT - 1) / MT * 32, MT == 2 ? 2 : 1) hadamard_tokens_kernel(const __grid_constant__ HadQuantParams p) {
  constexpr int NW = (KT + MT - 1) / MT, kThreads = NW * 32;
  constexpr int kPitch = NB + 8;                              // halves per row of T
  constexpr int kLanes = NB / 8;                              // lanes per block of nb entries
  constexpr int kCodePitch = NB + 16;                         // bytes per row of the staged codes
  extern __shared__ __align__(16) uint8_t smem_raw[];
  __half* T = reinterpret_cast<__half*>(smem_raw);            // [Kp][kPitch]: the rotated blocks
  uint8_t* xbuf = smem_raw + static_cast<size_t>(p.Kp) * kPitch * 2;
  const int xbytes = p.Kp * (2 * NB > kCodePitch ? 2 * NB : kCodePitch);
  __shared__ float red[2][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int K = p.K, tiles = p.Kp >> 4;
  grid_dependency_wait_release();

  auto fetch = [&](int r, int buf) {
    const uint4* src = reinterpret_cast<const uint4*>(p.x + r * p.x_row_stride);
    uint4* dst = reinterpret_cast<uint4*>(xbuf + buf * xbytes);
    for (int i = threadIdx.x; i < K * (NB / 8); i += kThreads) cp_async16(dst + i, src + i);
  };
  fetch(blockIdx.x, 0);
  asm volatile("cp.async.commit_group;" ::: "memory");

  uint4 a[MT][KT];
#pragma unroll
  for (int mi = 0; mi < MT; ++mi) {
    const int mt = warp * MT + mi;
#pragma unroll
    for (int kt = 0; kt < KT; ++kt)
      a[mi][kt] = (mt < tiles && kt < tiles) ? __ldg(p.packed + (static_cast<int64_t>(mt) * tiles + kt) * 32 + lane) : make_uint4(0u, 0u, 0u, 0u);
  }
  // rows K .. Kp of T meet zero columns of had_K in the product: they must hold numbers, not leftovers
  for (int i = threadIdx.x; i < (p.Kp - K) * kPitch; i += kThreads) T[K * kPitch + i] = __float2half_rn(0.f);

  const int sub = lane & (kLanes - 1), which = lane / kLanes;
  constexpr int kPerWarp = 32 / kLanes;                       // blocks of nb entries a warp rotates at a time
  const int g = lane >> 2, t = lane & 3;
  int buf = 0;
  for (int r = blockIdx.x; r < p.rows; r += gridDim.x, buf ^= 1) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                          // the token has landed; nobody reads the other buffer or T any more
    if (r + static_cast<int>(gridDim.x) < p.rows) {
      fetch(r + gridDim.x, buf ^ 1);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    const uint8_t* xs = xbuf + buf * xbytes;

    // ---- power-of-two part ----
    for (int k0 = warp * kPerWarp; k0 < K; k0 += NW * kPerWarp) {
      const int k = k0 + which;
      uint4 xv = make_uint4(0u, 0u, 0u, 0u);
      if (k < K) xv = *reinterpret_cast<const uint4*>(xs + k * (2 * NB) + sub * 16);
      float e[8];
      const __half2* h2 = reinterpret_cast<const __half2*>(&xv);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = __half22float2(h2[i]);
        e[2 * i] = f.x;
        e[2 * i + 1] = f.y;
      }
#pragma unroll
      for (int h = 1; h < 8; h <<= 1)
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if ((i & h) == 0) {
            const float u = e[i], v = e[i + h];
            e[i] = u + v;
            e[i + h] = u - v;
          }
#pragma unroll
      for (int h = 1; h < kLanes; h <<= 1) {                  // strides 8, 16, ...: lane bits; o - e where the bit is set
        const float sign = (sub & h) ? -1.f : 1.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) e[i] = fmaf(sign, e[i], __shfl_xor_sync(0xffffffffu, e[i], h));
      }
      if (k < K) {
        uint4 o;
        __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
        for (int i = 0; i < 4; ++i) oh[i] = __floats2half2_rn(e[2 * i] * p.rot_scale, e[2 * i + 1] * p.rot_scale);
        *reinterpret_cast<uint4*>(T + k * kPitch + sub * 8) = o;
      }
    }
    __syncthreads();

    // ---- had_K product, 32 columns at a time; a warp's rows are its own ----
    __half2 y[MT][NB / 8][2];
    __half2 top = __floats2half2_rn(0.f, 0.f);
    const uint32_t tb = smem_u32(T) + static_cast<uint32_t>(((lane & 15) * kPitch + (lane >> 4) * 8) * 2);
#pragma unroll
    for (int n0 = 0; n0 < NB; n0 += 32) {
      float d[MT][4][4];
#pragma unroll
      for (int mi = 0; mi < MT; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) d[mi][ni][0] = d[mi][ni][1] = d[mi][ni][2] = d[mi][ni][3] = 0.f;
#pragma unroll
      for (int kt = 0; kt < KT; ++kt) {
        if (kt < tiles) {
          uint32_t b[2][4];
          ldsm_x4_trans(b[0], tb + static_cast<uint32_t>((kt * 16 * kPitch + n0) * 2));
          ldsm_x4_trans(b[1], tb + static_cast<uint32_t>((kt * 16 * kPitch + n0 + 16) * 2));
#pragma unroll
          for (int mi = 0; mi < MT; ++mi)
#pragma unroll
            for (int ni = 0; ni < 4; ++ni)
              mma_f16_16x8x16(d[mi][ni], a[mi][kt].x, a[mi][kt].y, a[mi][kt].z, a[mi][kt].w, b[ni >> 1][2 * (ni & 1)], b[ni >> 1][2 * (ni & 1) + 1]);
        }
      }
#pragma unroll
      for (int mi = 0; mi < MT; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni)
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
            const __half2 v = __floats2half2_rn(d[mi][ni][2 * hf], d[mi][ni][2 * hf + 1]);   // the reference's fp16 result
            y[mi][n0 / 8 + ni][hf] = v;
            top = __hmax2(top, __habs2(v));                   // rows past K are zero
          }
    }
    float amax = warp_max(fmaxf(__low2float(top), __high2float(top)));
    if (lane == 0) red[buf][warp] = amax;
    __syncthreads();
    amax = warp_max(lane < NW ? red[buf][lane] : 0.f);
    const float s = act_scale_of(amax);
    if (threadIdx.x == 0) p.scale[r] = s;

    // ---- codes into the token's input buffer, then 16 bytes at a time to memory ----
    const ActCoder coder(s);
    uint8_t* cq = xbuf + buf * xbytes;
#pragma unroll
    for (int mi = 0; mi < MT; ++mi)
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        const int row = (warp * MT + mi) * 16 + g + 8 * hf;
        if (row < K) {
#pragma unroll
          for (int n = 0; n < NB / 8; ++n) {
            const float2 f = __half22float2(y[mi][n][hf]);
            *reinterpret_cast<uint16_t*>(cq + row * kCodePitch + n * 8 + 2 * t) = static_cast<uint16_t>(__byte_perm(coder.low(f.x), coder.low(f.y), 0x0040));
            if (p.y != nullptr) *reinterpret_cast<__half2*>(p.y + static_cast<int64_t>(r) * p.cols + row * NB + n * 8 + 2 * t) = y[mi][n][hf];
          }
        }
      }
    __syncthreads();
    int8_t* q = p.q + r * p.q_row_stride;
    if ((reinterpret_cast<uintptr_t>(q) & 15) == 0) {
      for (int i = threadIdx.x; i < K * (NB / 16); i += kThreads)
        reinterpret_cast<uint4*>(q)[i] = *reinterpret_cast<const uint4*>(cq + (i / (NB / 16)) * kCodePitch + (i % (NB / 16)) * 16);
    } else {
      for (int i = threadIdx.x; i < K * NB; i += kThreads) q[i] = static_cast<int8_t>(cq[(i / NB) * kCodePitch + i % NB]);
    }
  }
}

template <int KT, int NB>
static int launch_tokens(const HadQuantParams& p, cudaStream_t st) {
  const int sms = std::max(1, device_sm_count());
  const bool many = p.rows > sms;
  const int xbytes = p.Kp * std::max(2 * NB, NB + 16);
  const int smem = p.Kp * (NB + 8) * 2 + 2 * xbytes;
  void (*kern)(HadQuantParams) = many ? hadamard_tokens_kernel<KT, NB, 2> : hadamard_tokens_kernel<KT, NB, 1>;
  const int threads = many ? (KT + 1) / 2 * 32 : KT * 32;
  if (smem > 48 * 1024) LSVD_CUDA_TRY(ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem));
  LSVD_CUDA_TRY(launch_chained(kern, dim3(std::min(p.rows, many ? 2 * sms : sms)), dim3(threads), smem, st, 1, true, p));
  return LSVD_OK;
}

int launch_hadamard_tokens(const HadQuantParams& p, cudaStream_t st) {
  if ((p.nb != 64 && p.nb != 128) || p.Kp > 176 || !p.x_vec16) return LSVD_ERR_UNSUPPORTED;
  const int tiles = p.Kp >> 4;
  if (p.nb == 64) {
    if (tiles <= 4) return launch_tokens<4, 64>(p, st);
    if (tiles <= 7) return launch_tokens<7, 64>(p, st);
    return launch_tokens<11, 64>(p, st);
  }
  if (tiles <= 4) return launch_tokens<4, 128>(p, st);
  if (tiles <= 7) return launch_tokens<7, 128>(p, st);
  return launch_tokens<11, 128>(p, st);
}

}  // namespace lsvd
