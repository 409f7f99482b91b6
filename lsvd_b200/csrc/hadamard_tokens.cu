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
//   * a lane holds 32 consecutive entries of a block: five butterfly strides in registers, two entries per instruction from
//     the second on, the last one or two by shuffles -- the same additions in the same order as the reference's loop; the
//     rotated blocks are stored row by row and become B fragments by ldmatrix.trans (row pitch nb + 8 halves: no bank
//     conflicts; the token's input rows have the same pitch);
//   * results wait as packed fp16 pairs for the row's scale; codes are five operations per pair of entries (ActCoder),
//     staged in the token's own input buffer and stored 16 bytes at a time.
// One 16-row tile of had_K per warp: 11 warps at K = 172, two blocks per SM.  Two tiles per warp (half the shared-memory
// reads, but 12 warps per SM, eight entries per lane in the butterflies and one entry at a time in the codes) took 273 us
// for 8191 tokens of 172 x 64, issue slots 46 % busy; the block-per-token kernel before that 366 us.
#include <algorithm>

#include "common.cuh"
#include "devfn.cuh"

namespace lsvd {

__device__ __forceinline__ void ldsm_x4_trans(uint32_t (&d)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(addr) : "memory");
}

template <int KT, int NB, int PER_SM>
__global__ void __launch_bounds__(KT * 32, PER_SM) hadamard_tokens_kernel(const __grid_constant__ HadQuantParams p) {
  constexpr int kThreads = KT * 32;
  constexpr int kPitch = NB + 8;                              // halves per row of T and of the token
  constexpr int kLanes = NB / 32;                             // lanes per block of nb entries
  constexpr int kCodePitch = NB + 16;                         // bytes per row of the staged codes
  extern __shared__ __align__(16) uint8_t smem_raw[];
  __half* T = reinterpret_cast<__half*>(smem_raw);            // [Kp][kPitch]: the rotated blocks
  uint8_t* xbuf = smem_raw + static_cast<size_t>(p.Kp) * kPitch * 2;
  const int xbytes = p.Kp * kPitch * 2;
  __shared__ float red[2][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int K = p.K, tiles = p.Kp >> 4;
  grid_dependency_wait_release();

  auto fetch = [&](int r, int buf) {
    const uint4* src = reinterpret_cast<const uint4*>(p.x + r * p.x_row_stride);
    uint8_t* dst = xbuf + buf * xbytes;
    for (int i = threadIdx.x; i < K * (NB / 8); i += kThreads) cp_async16(dst + (i / (NB / 8)) * (kPitch * 2) + (i % (NB / 8)) * 16, src + i);
  };
  fetch(blockIdx.x, 0);
  asm volatile("cp.async.commit_group;" ::: "memory");

  uint4 a[KT];
#pragma unroll
  for (int kt = 0; kt < KT; ++kt)
    a[kt] = (warp < tiles && kt < tiles) ? __ldg(p.packed + (static_cast<int64_t>(warp) * tiles + kt) * 32 + lane) : make_uint4(0u, 0u, 0u, 0u);
  // rows K .. Kp of T meet zero columns of had_K in the product: they must hold numbers, not leftovers
  for (int i = threadIdx.x; i < (p.Kp - K) * kPitch; i += kThreads) T[K * kPitch + i] = __float2half_rn(0.f);

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
    for (int i0 = threadIdx.x; i0 < (K * kLanes + 31) / 32 * 32; i0 += kThreads) {      // whole warps: they shuffle
      const int k = i0 / kLanes, sub = i0 % kLanes;
      const bool on = k < K;
      float2 e[16];                                           // entries 32 sub + 2 i, + 1
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const uint4 v = on ? *reinterpret_cast<const uint4*>(xs + k * (kPitch * 2) + sub * 64 + c * 16) : make_uint4(0u, 0u, 0u, 0u);
        const __half2* h2 = reinterpret_cast<const __half2*>(&v);
#pragma unroll
        for (int i = 0; i < 4; ++i) e[4 * c + i] = __half22float2(h2[i]);
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) e[i] = make_float2(e[i].x + e[i].y, e[i].x - e[i].y);
#pragma unroll
      for (int h = 1; h < 16; h <<= 1)
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if ((i & h) == 0) {
            const float2 u = e[i], v = e[i + h];
            e[i] = add2(u, v);
            e[i + h] = fma2(v, make_float2(-1.f, -1.f), u);
          }
#pragma unroll
      for (int h = 1; h < kLanes; h <<= 1) {                  // strides 32, 64: lane bits; o - e where the bit is set
        const float sign = (sub & h) ? -1.f : 1.f;
#pragma unroll
        for (int i = 0; i < 16; ++i)
          e[i] = fma2(make_float2(sign, sign), e[i], make_float2(__shfl_xor_sync(0xffffffffu, e[i].x, h), __shfl_xor_sync(0xffffffffu, e[i].y, h)));
      }
      if (on) {
        const float2 rs = make_float2(p.rot_scale, p.rot_scale);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint4 o;
          __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
          for (int i = 0; i < 4; ++i) oh[i] = __float22half2_rn(mul2(e[4 * c + i], rs));
          *reinterpret_cast<uint4*>(T + k * kPitch + sub * 32 + c * 8) = o;
        }
      }
    }
    __syncthreads();

    // ---- had_K product, 32 columns at a time; a warp's 16 rows are its own ----
    __half2 y[NB / 8][2];
    __half2 top = __floats2half2_rn(0.f, 0.f);
    const uint32_t tb = smem_u32(T) + static_cast<uint32_t>(((lane & 15) * kPitch + (lane >> 4) * 8) * 2);
#pragma unroll
    for (int n0 = 0; n0 < NB; n0 += 32) {
      float d[4][4];
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) d[ni][0] = d[ni][1] = d[ni][2] = d[ni][3] = 0.f;
#pragma unroll
      for (int kt = 0; kt < KT; ++kt) {
        if (kt < tiles) {
          uint32_t b[2][4];
          ldsm_x4_trans(b[0], tb + static_cast<uint32_t>((kt * 16 * kPitch + n0) * 2));
          ldsm_x4_trans(b[1], tb + static_cast<uint32_t>((kt * 16 * kPitch + n0 + 16) * 2));
#pragma unroll
          for (int ni = 0; ni < 4; ++ni)
            mma_f16_16x8x16(d[ni], a[kt].x, a[kt].y, a[kt].z, a[kt].w, b[ni >> 1][2 * (ni & 1)], b[ni >> 1][2 * (ni & 1) + 1]);
        }
      }
#pragma unroll
      for (int ni = 0; ni < 4; ++ni)
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          const __half2 v = __floats2half2_rn(d[ni][2 * hf], d[ni][2 * hf + 1]);      // the reference's fp16 result
          y[n0 / 8 + ni][hf] = v;
          top = __hmax2(top, __habs2(v));                     // rows past K are zero
        }
    }
    float amax = warp_max(fmaxf(__low2float(top), __high2float(top)));
    if (lane == 0) red[buf][warp] = amax;
    __syncthreads();
    amax = warp_max(lane < KT ? red[buf][lane] : 0.f);
    const float s = act_scale_of(amax);
    if (threadIdx.x == 0) p.scale[r] = s;

    // ---- codes into the token's input buffer, then 16 bytes at a time to memory ----
    const ActCoder coder(s);
    uint8_t* cq = xbuf + buf * xbytes;
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      const int row = warp * 16 + g + 8 * hf;
      if (row < K) {
        uint16_t* dst = reinterpret_cast<uint16_t*>(cq + row * kCodePitch + 2 * t);
        if (!coder.divide) {
#pragma unroll
          for (int n = 0; n < NB / 8; ++n) dst[4 * n] = static_cast<uint16_t>(coder.pair<false>(__half22float2(y[n][hf])));
        } else {
          for (int n = 0; n < NB / 8; ++n) dst[4 * n] = static_cast<uint16_t>(coder.pair<true>(__half22float2(y[n][hf])));
        }
        if (p.y != nullptr) {
#pragma unroll
          for (int n = 0; n < NB / 8; ++n) *reinterpret_cast<__half2*>(p.y + static_cast<int64_t>(r) * p.cols + row * NB + n * 8 + 2 * t) = y[n][hf];
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

template <int KT, int NB, int PER_SM>
static int launch_tokens(const HadQuantParams& p, cudaStream_t st) {
  const int smem = 3 * p.Kp * (NB + 8) * 2;
  const int sms = std::max(1, device_sm_count());
  void (*kern)(HadQuantParams) = hadamard_tokens_kernel<KT, NB, PER_SM>;
  if (smem > 48 * 1024) LSVD_CUDA_TRY(ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem));
  LSVD_CUDA_TRY(launch_chained(kern, dim3(std::min(p.rows, PER_SM * sms)), dim3(KT * 32), smem, st, 1, ffn_chain_enabled(), p));
  return LSVD_OK;
}

// Blocks per SM.  A token per SM at most gets all the registers a block can use.  More tokens get as many blocks as shared
// memory and about 128 registers a thread admit: two of 11 warps at nb = 64 (80 registers, some spills, and still faster:
// 8191 tokens of 172 x 64 226 against 273 us), but one at 172 x 128, whose 144 KB fit once (built for two, 80 registers and
// 184 bytes of spills: 8000 tokens 555 us, so 369).  had_K of one or two tiles takes a block of as many warps, and many
// blocks: 8000 tokens of 12 x 64 took 45 us with four warps, three of them without a tile, and take 11.4; 28 x 64 52 and 20.5.
int launch_hadamard_tokens(const HadQuantParams& p, cudaStream_t st) {
  if ((p.nb != 64 && p.nb != 128) || p.Kp > 176 || !p.x_vec16) return LSVD_ERR_UNSUPPORTED;
  const int tiles = p.Kp >> 4;
  const bool many = p.rows > device_sm_count();
  if (p.nb == 64) {
    if (many && tiles == 1) return launch_tokens<1, 64, 16>(p, st);
    if (many && tiles == 2) return launch_tokens<2, 64, 8>(p, st);
    if (tiles <= 4) return many ? launch_tokens<4, 64, 2>(p, st) : launch_tokens<4, 64, 1>(p, st);
    if (tiles <= 7) return many ? launch_tokens<7, 64, 2>(p, st) : launch_tokens<7, 64, 1>(p, st);
    return many ? launch_tokens<11, 64, 2>(p, st) : launch_tokens<11, 64, 1>(p, st);
  }
  if (many && tiles == 1) return launch_tokens<1, 128, 16>(p, st);
  if (many && tiles == 2) return launch_tokens<2, 128, 8>(p, st);
  if (tiles <= 4) return many ? launch_tokens<4, 128, 2>(p, st) : launch_tokens<4, 128, 1>(p, st);
  if (tiles <= 7) return many ? launch_tokens<7, 128, 2>(p, st) : launch_tokens<7, 128, 1>(p, st);
  return launch_tokens<11, 128, 1>(p, st);
}

}  // namespace lsvd
