// BF16 tensor-core kernels of the learned denoiser: 3x3 convolutions
// (forward, gradient of the input, gradient of the weights) as implicit
// GEMMs with FP32 accumulation, and the small element-wise layers around
// them (2x2 average pool, nearest 2x upsample, channel copies for the skip
// concatenations, ReLU masks, loss, Adam).
//
// Layout: activations NHWC bf16, read and written through a channel stride
// and offset so that a concatenated buffer is just a wider tensor;
// weights [Cout][3][3][Cin] bf16 (K = tap * Cin + ci), biases fp32.
// Channel counts are multiples of 16.
//
// Two tensor-core paths.  tcgen05: rows in shared memory by TMA (zero-filled
// outside the image), one elected thread issuing operations that accumulate in
// tensor memory (k_conv_fwd_ws, k_conv_wgrad_ws; k_conv_fwd_tc streams its
// weights).  mma.sync m16n8k16 bf16 -> f32 for the shapes those do not take:
// tiles by cp.async (16-byte copies, zero-filled outside the image), fragments
// by ldmatrix (k_conv_fwd_res, k_conv_fwd, k_conv_wgrad).
#include <cooperative_groups.h>
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <climits>

#include "rx_internal.cuh"
#include "rx_runtime.h"

namespace rx {

using bf16 = __nv_bfloat16;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// 16-byte global -> shared copy; `valid` false writes zeros (no bytes read)
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(smem)), "l"(gmem),
               "r"(valid ? 16 : 0));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_u32(p)));
}
__device__ __forceinline__ void ldsm_x4_at(uint32_t (&r)[4], uint32_t saddr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(saddr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_u32(p)));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// ------------------------------------------------------------- forward conv
// y[p][co] = act(bias[co] + sum_{tap, ci} x[p + off(tap)][ci] * w[co][tap][ci])
// GEMM: M = pixels (64 per block), N = output channels (BN per block),
// K = 9 taps x Cin, BK channels per stage.  4 warps as 2 (M) x 2 (N).
template <int BN, int BK>
__global__ void __launch_bounds__(128) k_conv_fwd(rx_conv_desc d, const bf16* __restrict__ x,
                                                  const bf16* __restrict__ w, const float* __restrict__ bias,
                                                  bf16* __restrict__ y, float* __restrict__ y32, int relu) {
  constexpr int BM = 64, LDS = BK + 8;
  constexpr int KC = BK / 8;              // 16-byte chunks per row
  constexpr int A_PER = BM * KC / 128;    // A chunks per thread
  constexpr int B_CH = BN * KC;           // B chunks per stage
  constexpr int NT = BN / 16;             // n8 tiles per warp
  __shared__ __align__(16) bf16 sA[2][BM][LDS];
  __shared__ __align__(16) bf16 sB[2][BN][LDS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp & 1, wn = warp >> 1;
  const long long HW = (long long)d.H * d.W;
  const long long P = (long long)d.N * HW;
  const long long m0 = (long long)blockIdx.x * BM;
  const int n0 = blockIdx.y * BN;
  const int CB = d.Cin / BK;
  const int KT = 9 * CB;

  int a_row[A_PER], a_kc[A_PER], a_y[A_PER], a_x[A_PER];
  long long a_img[A_PER];
  bool a_ok[A_PER];
#pragma unroll
  for (int i = 0; i < A_PER; ++i) {
    int c = tid + i * 128;
    a_row[i] = c / KC;
    a_kc[i] = c % KC;
    long long pix = m0 + a_row[i];
    a_ok[i] = pix < P;
    long long n = a_ok[i] ? pix / HW : 0;
    long long r = a_ok[i] ? pix - n * HW : 0;
    a_img[i] = n * HW;
    a_y[i] = (int)(r / d.W);
    a_x[i] = (int)(r % d.W);
  }

  auto load = [&](int kt, int buf) {
    int tap = kt / CB, c0 = (kt % CB) * BK;
    int dy = tap / 3 - 1, dx = tap % 3 - 1;
#pragma unroll
    for (int i = 0; i < A_PER; ++i) {
      int yy = a_y[i] + dy, xx = a_x[i] + dx;
      bool ok = a_ok[i] && yy >= 0 && yy < d.H && xx >= 0 && xx < d.W;
      const bf16* src =
          ok ? x + (a_img[i] + (long long)yy * d.W + xx) * d.x_cstride + d.x_coff + c0 + a_kc[i] * 8 : x;
      cp_async16(&sA[buf][a_row[i]][a_kc[i] * 8], src, ok);
    }
    for (int c = tid; c < B_CH; c += 128) {
      int row = c / KC, kc = c % KC;
      int co = n0 + row;
      bool ok = co < d.Cout;
      const bf16* src = ok ? w + ((long long)co * 9 + tap) * d.Cin + c0 + kc * 8 : w;
      cp_async16(&sB[buf][row][kc * 8], src, ok);
    }
  };

  float acc[2][NT][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[i][j][k] = 0.0f;

  load(0, 0);
  cp_async_commit();
  for (int kt = 0; kt < KT; ++kt) {
    int buf = kt & 1;
    if (kt + 1 < KT) load(kt + 1, buf ^ 1);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
#pragma unroll
    for (int ks = 0; ks < BK / 16; ++ks) {
      uint32_t af[2][4];
#pragma unroll
      for (int mi = 0; mi < 2; ++mi)
        ldsm_x4(af[mi], &sA[buf][wm * 32 + mi * 16 + (lane & 15)][ks * 16 + (lane >> 4) * 8]);
#pragma unroll
      for (int nj = 0; nj < NT / 2; ++nj) {
        uint32_t bfr[4];
        ldsm_x4(bfr, &sB[buf][wn * (BN / 2) + nj * 16 + (lane & 7) + (lane >> 4) * 8][ks * 16 + ((lane >> 3) & 1) * 8]);
#pragma unroll
        for (int mi = 0; mi < 2; ++mi) {
          mma_bf16(acc[mi][2 * nj], af[mi], bfr[0], bfr[1]);
          mma_bf16(acc[mi][2 * nj + 1], af[mi], bfr[2], bfr[3]);
        }
      }
    }
    __syncthreads();
  }
  cp_async_wait<0>();

  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int mi = 0; mi < 2; ++mi)
#pragma unroll
    for (int ni = 0; ni < NT; ++ni)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        long long m = m0 + wm * 32 + mi * 16 + g + h * 8;
        int co = n0 + wn * (BN / 2) + ni * 8 + 2 * t;
        if (m >= P || co >= d.Cout) continue;
        float v0 = acc[mi][ni][2 * h], v1 = acc[mi][ni][2 * h + 1];
        if (bias) {
          v0 += bias[co];
          v1 += bias[co + 1];
        }
        if (relu) {
          v0 = fmaxf(v0, 0.0f);
          v1 = fmaxf(v1, 0.0f);
        }
        *reinterpret_cast<__nv_bfloat162*>(y + m * d.y_cstride + d.y_coff + co) = __floats2bfloat162_rn(v0, v1);
        if (y32) {
          y32[m * d.y_cstride + d.y_coff + co] = v0;
          y32[m * d.y_cstride + d.y_coff + co + 1] = v1;
        }
      }
}

// The same convolution for few input channels (KS 16-channel steps per tap)
// and many output channels -- the gradients of the layers after a concat,
// 32 -> 96 and 64 -> 192, which the tcgen05 path's groups do not cover.  The
// products of an output are added in k_conv_fwd's order (taps outer, steps
// inner), so the results are its bits.
//
// k_conv_fwd copies every tap's pixels and weights to shared memory again
// (121 and 97 us for 14.5 GFLOP each at 16x128x128).  Here a block keeps all
// nine taps' weights of its BN channels, and a tile's pixels are copied once
// with their halo (two buffers: the next tile's copies run under this tile's
// products); a tap is an offset of the ldmatrix addresses.  Tiles are
// 128 pixels of 128 >> cl rows by 1 << cl columns.  Pixel and weight rows are
// padded to an odd number of 16-byte chunks: no bank conflicts.  121 -> 65 and
// 97 -> 56 us; mma.sync keeps the tensor pipe 46-54 % busy (ncu) with the two
// warps per scheduler that the weights leave room for (its floor is 29 us).
template <int BN, int KS>
struct ResShape {
  static constexpr int CIN = 16 * KS, PX = CIN + 8, WROW = 9 * CIN + 8;  // elements
  static constexpr int W_BYTES = BN * WROW * 2;
  static int halo(int cl) { return ((128 >> cl) + 2) * ((1 << cl) + 2) * PX * 2; }
  static size_t smem(int cl) { return (size_t)W_BYTES + 2 * (size_t)halo(cl); }
};

// BIAS: there is one.  Its values sit in registers from the start, as a load
// behind the wait; 32 -> 96 channels at 16x128x128 and 64 -> 192 at 16x64x64,
// back to back: 63 and 50 us (59 and 50 without a bias; read in the epilogue
// through the untied pointer 72 and 57).
template <int BN, int KS, bool BIAS>
__global__ void __launch_bounds__(256, 1)
    k_conv_fwd_res(rx_conv_desc d, const bf16* __restrict__ x, const bf16* __restrict__ w,
                   const float* __restrict__ bias, bf16* __restrict__ y, float* __restrict__ y32, int relu, int cl,
                   int tiles_x, int tiles_y, int halo_bytes) {
  using S = ResShape<BN, KS>;
  constexpr int NT = BN / 16, KC = 2 * KS, LOADERS = 256 / KC;  // n8 tiles per warp, chunks per pixel
  extern __shared__ __align__(16) unsigned char res_smem[];
  const uint32_t sw = smem_u32(res_smem), sx = sw + S::W_BYTES;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp & 3, wn = warp >> 2;
  const int n0 = blockIdx.y * BN;
  const int HC = (1 << cl) + 2, HR = (128 >> cl) + 2;  // halo columns and rows
  const int tiles = d.N * tiles_y * tiles_x;           // fits: launch_res

  auto tile_at = [&](int t, int& n, int& y0, int& x0) {
    const int r = t / tiles_x;
    x0 = (t - r * tiles_x) << cl;
    n = r / tiles_y;
    y0 = (r - n * tiles_y) * (128 >> cl);
  };
  auto load = [&](int t, int buf) {
    int n, y0, x0;
    tile_at(t, n, y0, x0);
    const int kc = tid % KC;
    int hc = tid / KC, hr = 0;
    unsigned char* dst = res_smem + S::W_BYTES + buf * halo_bytes + kc * 16;
    const bf16* img = x + (long long)n * d.H * d.W * d.x_cstride + d.x_coff + kc * 8;
    while (true) {
      while (hc >= HC) hc -= HC, ++hr;
      if (hr >= HR) break;
      const int yy = y0 + hr - 1, xx = x0 + hc - 1;
      const bool ok = (unsigned)yy < (unsigned)d.H && (unsigned)xx < (unsigned)d.W;
      cp_async16(dst + (hr * HC + hc) * (S::PX * 2), ok ? img + ((long long)yy * d.W + xx) * d.x_cstride : x, ok);
      hc += LOADERS;
    }
  };

  chain_wait(x, w, bias);
  chain_go();
  float bias_of[NT][2] = {};  // this lane's channels
  if constexpr (BIAS) {
#pragma unroll
    for (int ni = 0; ni < NT; ++ni) {
      const int co = n0 + wn * (BN / 2) + ni * 8 + 2 * (lane & 3);
      if (co < d.Cout) bias_of[ni][0] = bias[co], bias_of[ni][1] = bias[co + 1];
    }
  }
  for (int c = tid; c < BN * 9 * KC; c += 256) {
    const int row = c / (9 * KC), k = c - row * (9 * KC);
    const bool ok = n0 + row < d.Cout;
    cp_async16(res_smem + row * (S::WROW * 2) + k * 16, ok ? w + (long long)(n0 + row) * 9 * S::CIN + k * 8 : w, ok);
  }
  int t = blockIdx.x, buf = 0;
  if (t < tiles) load(t, 0);
  cp_async_commit();

  // this lane's ldmatrix rows: two m16 tiles of pixels, BN / 32 n16 tiles of weights
  uint32_t a_at[2];
#pragma unroll
  for (int mi = 0; mi < 2; ++mi) {
    const int m = wm * 32 + mi * 16 + (lane & 15);
    a_at[mi] = ((m >> cl) * HC + (m & ((1 << cl) - 1))) * (S::PX * 2) + (lane >> 4) * 16;
  }
  const uint32_t b_at =
      sw + (wn * (BN / 2) + (lane & 7) + (lane >> 4) * 8) * (S::WROW * 2) + ((lane >> 3) & 1) * 16;

  for (; t < tiles; t += gridDim.x, buf ^= 1) {
    // one barrier a tile: this tile's copies have landed for every thread, and
    // every warp has left the other buffer, which the next tile's copies take
    cp_async_wait<0>();
    __syncthreads();
    if (t + (int)gridDim.x < tiles) load(t + gridDim.x, buf ^ 1);
    cp_async_commit();
    float acc[2][NT][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[i][j][k] = 0.0f;
    const uint32_t xb = sx + buf * halo_bytes;
    for (int ty = 0; ty < 3; ++ty) {
#pragma unroll
      for (int tx = 0; tx < 3; ++tx) {
        const uint32_t xo = xb + (ty * HC + tx) * (S::PX * 2), wo = b_at + (ty * 3 + tx) * (S::CIN * 2);
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
          uint32_t af[2][4];
#pragma unroll
          for (int mi = 0; mi < 2; ++mi) ldsm_x4_at(af[mi], xo + a_at[mi] + ks * 32);
#pragma unroll
          for (int nj = 0; nj < NT / 2; ++nj) {
            uint32_t bfr[4];
            ldsm_x4_at(bfr, wo + nj * 16 * (S::WROW * 2) + ks * 32);
#pragma unroll
            for (int mi = 0; mi < 2; ++mi) {
              mma_bf16(acc[mi][2 * nj], af[mi], bfr[0], bfr[1]);
              mma_bf16(acc[mi][2 * nj + 1], af[mi], bfr[2], bfr[3]);
            }
          }
        }
      }
    }
    int n, y0, x0;
    tile_at(t, n, y0, x0);
    const int g = lane >> 2, q = lane & 3;
#pragma unroll
    for (int mi = 0; mi < 2; ++mi)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int m = wm * 32 + mi * 16 + g + h * 8;
        const int yy = y0 + (m >> cl), xx = x0 + (m & ((1 << cl) - 1));
        if (yy >= d.H || xx >= d.W) continue;
        const long long at = (((long long)n * d.H + yy) * d.W + xx) * d.y_cstride + d.y_coff;
#pragma unroll
        for (int ni = 0; ni < NT; ++ni) {
          const int co = n0 + wn * (BN / 2) + ni * 8 + 2 * q;
          if (co >= d.Cout) continue;
          float v0 = acc[mi][ni][2 * h], v1 = acc[mi][ni][2 * h + 1];
          if constexpr (BIAS) {
            v0 += bias_of[ni][0];
            v1 += bias_of[ni][1];
          }
          if (relu) {
            v0 = fmaxf(v0, 0.0f);
            v1 = fmaxf(v1, 0.0f);
          }
          *reinterpret_cast<__nv_bfloat162*>(y + at + co) = __floats2bfloat162_rn(v0, v1);
          if (y32) {
            y32[at + co] = v0;
            y32[at + co + 1] = v1;
          }
        }
      }
  }
  cp_async_wait<0>();
}

// ------------------------------------------- forward conv on tcgen05 (UMMA)
// One CTA computes 128 consecutive pixels of one image row (the MMA's M)
// for all COUT output channels (its N), accumulating in tensor memory.
// Per chunk of 32 input channels it stages, with cp.async, a halo of 3 rows
// x 130 pixels and the 9 taps' weights in shared memory in the canonical
// K-major, no-swizzle layout (core matrices of 8 rows x 16 bytes): channel
// chunk planes [kc][row][pixel][8 channels] and [tap][kc][co][8].  A tap's
// A operand is then the same descriptor with its start moved by whole
// pixels, so the halo is loaded once for all 9 taps.  One thread issues
// 9 taps x 2 K-steps of tcgen05.mma (kind::f16, BF16 in, FP32 accumulate)
// per chunk and commits them to the chunk buffer's mbarrier; two buffers
// overlap the next chunk's copies with the current MMAs.
namespace tc {
constexpr int TILE = 128, HALO_W = TILE + 2, KCH = 4;  // 4 chunks of 8 channels = 32
constexpr int HALO_BYTES = KCH * 3 * HALO_W * 16;      // 24960
constexpr unsigned long long kSpinCycles = 4000000000ull;  // ~2 s at 1.9 GHz

__host__ __device__ constexpr int stage_bytes(int cout) { return HALO_BYTES + 9 * KCH * cout * 16; }

// K-major, no-swizzle shared-memory matrix descriptor (Blackwell version 1)
__device__ __forceinline__ uint64_t desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);
}

// instruction descriptor: FP32 accumulate, BF16 A and B, both K-major, M=128
__host__ __device__ constexpr uint32_t idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  unsigned long long t0 = clock64();
  for (;;) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
    if (clock64() - t0 > kSpinCycles) return false;
  }
}
}  // namespace tc

template <int COUT>
__global__ void __launch_bounds__(128, 1) k_conv_fwd_tc(rx_conv_desc d, const bf16* __restrict__ x,
                                                        const bf16* __restrict__ w, const float* __restrict__ bias,
                                                        bf16* __restrict__ y, float* __restrict__ y32, int relu,
                                                        int* err) {
  constexpr int SB = tc::stage_bytes(COUT);
  constexpr int TCOLS = COUT < 32 ? 32 : COUT;  // tensor-memory columns (power of two >= 32)
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) unsigned long long bars[2];
  __shared__ uint32_t tmem_base;
  __shared__ int abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int x0 = blockIdx.x * tc::TILE, yrow = blockIdx.y, n = blockIdx.z;
  const int nch = (d.Cin + 31) / 32;

  if (tid == 0) {
    abort_flag = 0;
    for (int b = 0; b < 2; ++b)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&bars[b])));
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_base)),
                 "r"(TCOLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = tmem_base;

  auto load = [&](int ch, int buf) {
    unsigned char* base = smem + buf * SB;
    const int c0 = ch * 32;
    // halo: chunk index ((r * HALO_W + px) * KCH + kc); 16 bytes each
    for (int c = tid; c < 3 * tc::HALO_W * tc::KCH; c += 128) {
      int kc = c % tc::KCH, rp = c / tc::KCH;
      int px = rp % tc::HALO_W, r = rp / tc::HALO_W;
      int yy = yrow + r - 1, xx = x0 + px - 1, ci = c0 + kc * 8;
      bool ok = yy >= 0 && yy < d.H && xx >= 0 && xx < d.W && ci < d.Cin;
      const bf16* src = ok ? x + (((long long)n * d.H + yy) * d.W + xx) * d.x_cstride + d.x_coff + ci : x;
      cp_async16(base + ((kc * 3 + r) * tc::HALO_W + px) * 16, src, ok);
    }
    // weights: chunk index ((co * 9 + tap) * KCH + kc)
    unsigned char* wb = base + tc::HALO_BYTES;
    for (int c = tid; c < COUT * 9 * tc::KCH; c += 128) {
      int kc = c % tc::KCH, ct = c / tc::KCH;
      int tap = ct % 9, co = ct / 9;
      int ci = c0 + kc * 8;
      bool ok = co < d.Cout && ci < d.Cin;
      const bf16* src = ok ? w + ((long long)co * 9 + tap) * d.Cin + ci : w;
      cp_async16(wb + ((tap * tc::KCH + kc) * COUT + co) * 16, src, ok);
    }
  };

  load(0, 0);
  cp_async_commit();
  bool ok_all = true;
  for (int ch = 0; ch < nch; ++ch) {
    const int buf = ch & 1;
    if (ch + 1 < nch) {
      const int nb = (ch + 1) & 1;
      if (ch + 1 >= 2) {
        // the MMAs of chunk ch - 1 read buffer nb: wait for their commit
        if (!tc::mbar_wait(smem_u32(&bars[nb]), (uint32_t)(((ch - 1) >> 1) & 1))) abort_flag = 1;
      }
      __syncthreads();
      if (abort_flag) {
        ok_all = false;
        break;
      }
      load(ch + 1, nb);
      cp_async_commit();
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    // copies visible to the tensor cores (async proxy) before the MMAs
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncthreads();
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const uint32_t hb = smem_u32(smem + buf * SB);
      const uint32_t wb = hb + tc::HALO_BYTES;
      constexpr uint32_t ID = tc::idesc(COUT);
#pragma unroll 1
      for (int tap = 0; tap < 9; ++tap) {
        const int dy = tap / 3, dx = tap % 3;
#pragma unroll
        for (int k2 = 0; k2 < 2; ++k2) {
          uint64_t ad = tc::desc(hb + (((2 * k2) * 3 + dy) * tc::HALO_W + dx) * 16, 3 * tc::HALO_W * 16, 128);
          uint64_t bd = tc::desc(wb + ((tap * tc::KCH + 2 * k2) * COUT) * 16, COUT * 16, 128);
          uint32_t acc = (ch > 0 || tap > 0 || k2 > 0) ? 1u : 0u;
          asm volatile(
              "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
              "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(tmem),
              "l"(ad), "l"(bd), "r"(ID), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
        }
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                       smem_u32(&bars[buf]))
                   : "memory");
    }
  }
  if (ok_all) {
    const int last = nch - 1;
    if (!tc::mbar_wait(smem_u32(&bars[last & 1]), (uint32_t)((last >> 1) & 1))) ok_all = false;
  }
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  if (ok_all) {
    // accumulator row = pixel (warp's 32 lanes), columns = output channels
    const int xx = x0 + warp * 32 + lane;
    const long long m = ((long long)n * d.H + yrow) * d.W + xx;
#pragma unroll 1
    for (int c0 = 0; c0 < COUT; c0 += 16) {
      uint32_t r[16];
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
          : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
            "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
          : "r"(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0));
      asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
      if (xx < d.W && c0 < d.Cout) {
        float v[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          v[k] = __uint_as_float(r[k]) + (bias ? bias[c0 + k] : 0.0f);
          if (relu) v[k] = fmaxf(v[k], 0.0f);
        }
        uint4 pk[2];
        uint32_t* pw = reinterpret_cast<uint32_t*>(pk);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
          pw[k] = *reinterpret_cast<uint32_t*>(&h);
        }
        uint4* dst = reinterpret_cast<uint4*>(y + m * d.y_cstride + d.y_coff + c0);
        dst[0] = pk[0];
        dst[1] = pk[1];
        if (y32) {
#pragma unroll
          for (int k = 0; k < 16; ++k) y32[m * d.y_cstride + d.y_coff + c0 + k] = v[k];
        }
      }
    }
  } else if (tid == 0) {
    atomicOr(err, ERR_BAD_NODE);
  }
  cp_async_wait<0>();
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TCOLS));
}

// --------------------------------------- forward conv, warp-specialised
// Persistent row-strip kernel for layers whose weights fit in shared memory
// beside a ring of input rows.  The weights are loaded once per CTA.  Each
// CTA owns a contiguous range of 128-pixel row tiles ordered with the row
// fastest, so consecutive tiles are vertically adjacent and share two of
// their three input rows: the input is a ring of S row slots [slot][kc]
// [pixel][8] (130 pixels, all input channels), and every input row is read
// once per strip instead of three times.  Three jobs run in separate warps
// that hand work to one another through mbarriers, so that copies, MMAs
// and epilogues of different rows overlap:
//   warp 10: producer (one elected lane).  Each input row of the strip is one
//     TMA box of 130 pixels x all channels, read as a 5-d tensor (8
//     channels, pixel, channel chunk, row, image) so that it lands in its
//     ring slot as [kc][130 px x 16 B] with zeros outside the image, and
//     completes on `full[slot]`; a slot is refilled after `empty[slot]`.
//     These 16-byte rows move at 16 B per cycle and SM (measured, from two
//     rows in flight on), a row in about 0.7 of its MMAs' time at every
//     channel count.  128 threads copying 16-byte chunks with cp.async kept
//     the MMAs waiting instead: a row could only be handed over after a
//     wait_group, one or two rows late.
//   warps 8-9: MMA issuers (one elected lane each, alternating rows).  Output
//     row y reads the slots of rows y-1, y, y+1; it accumulates into one of
//     four tensor-memory buffers, commits to `acc_full[buf]`, and commits to
//     `empty` of each slot it read (a slot is free after three commits).
//   warps 0-7: epilogue.  They load the weights, then warps 0-3 serve the
//     even rows and 4-7 the odd ones: warp w reads tensor-memory lanes
//     32 (w % 4) .. + 31 (its 32 pixels), adds the bias, applies ReLU, stores
//     bf16 (and fp32), then arrives on `acc_empty[buf]`.
// Output channels may be split into G groups of NG (blockIdx.x % G) when
// all the weights do not fit in shared memory beside the ring; the G CTAs
// of a strip run side by side and share its input rows through L2.
// Every wait is bounded: a wait that runs out (or sees another role give
// up) raises the shared abort flag, the roles stop, outstanding copies and
// MMAs are waited for (bounded), the device error flag is set.
// Bound by the MMAs' A-operand reads (40-48 cycles per M=128, K=16 MMA at
// N <= 64) in the wide layers, by the row hand-overs in the narrow ones.
// The eleven layers at 1920x1080, back to back: 880-910 us (2,157 us with one
// lane-0 issuer looping over the steps, one epilogue group and cp.async
// producers); 96 -> 32 channels 172-191 us, 600-667 TFLOP/s (472 us, 243).
// ncu: tensor pipe 13 % busy (N = 16) to 41 % (64 -> 64), DRAM 6-48 %.
namespace tc {
constexpr int PLANE = HALO_W * 16;  // one 8-channel chunk of one row
// a row slot, on the 128-byte boundary that a TMA box needs
__host__ __device__ constexpr int slot_bytes(int cin) { return ((cin / 8) * PLANE + 127) / 128 * 128; }
__host__ __device__ constexpr int weights_bytes(int cin, int cout) { return 9 * cin * cout * 2; }
constexpr int kMaxSlots = 8;
}  // namespace tc

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// single-thread bounded wait; gives up when the abort flag is raised
__device__ __forceinline__ bool mbar_wait_abortable(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (mbar_try(bar, parity)) return true;
  const unsigned long long t0 = clock64();
  for (;;) {
    if (mbar_try(bar, parity)) return true;
    if (*abort_flag) return false;
    if (clock64() - t0 > tc::kSpinCycles) {
      *abort_flag = 1;
      return false;
    }
  }
}

// whole-warp bounded wait with a warp-uniform outcome
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  const unsigned long long t0 = clock64();
  for (;;) {
    const bool ok = mbar_try(bar, parity);
    if (__all_sync(0xffffffffu, ok)) return true;
    const bool stop = *abort_flag || clock64() - t0 > tc::kSpinCycles;
    if (__any_sync(0xffffffffu, stop)) {
      *abort_flag = 1;
      return false;
    }
  }
}

// one lane of a converged warp
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(p));
  return p != 0;
}

__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}

// One M=128, N=NG, K=16 MMA on K-major, no-swizzle operands (SBO 128 B and
// descriptor version 1 in the high word); lo words as built by the caller.
template <int NG>
__device__ __forceinline__ void mma_k16(uint32_t acc_t, uint32_t a_lo, uint32_t b_lo, uint32_t acc) {
  constexpr uint64_t hi = (uint64_t)((128u >> 4) | (1u << 14)) << 32;
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(acc_t),
      "l"(hi | a_lo), "l"(hi | b_lo), "r"(tc::idesc(NG)), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
}

// The MMAs of one output row: taps in order, KS = Cin / 16 steps each; A
// moves by one pixel per tap column and two planes per step, B walks
// [tap][kc][co] in order.  The issuing thread's own instructions set the
// MMA rate unless the sequence is unrolled with compile-time offsets and
// issued by an elected lane (descriptors then live in uniform registers):
// a run-time loop over the steps on `lane == 0` took 140 (KS = 2) and 84
// (KS = 6) cycles per M=128, N=32 MMA, this takes 40 and 45; the tensor
// core's own A-operand read is about 40.
template <int NG, int KS>
__device__ __forceinline__ void issue_row(uint32_t acc_t, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t b_lo) {
  uint32_t first = 0u;  // the row's first MMA overwrites the accumulator
#pragma unroll 1
  for (int dy = 0; dy < 3; ++dy) {
    const uint32_t row = dy == 0 ? r0 : dy == 1 ? r1 : r2;
#pragma unroll
    for (int dx = 0; dx < 3; ++dx)
#pragma unroll
      for (int k = 0; k < KS; ++k)
        mma_k16<NG>(acc_t, row + (uint32_t)(dx + k * 2 * (tc::PLANE >> 4)), b_lo + (uint32_t)((dx * KS + k) * 2 * NG),
                    (dx | k) ? 1u : first);
    b_lo += 3 * KS * 2 * NG;
    first = 1u;
  }
}

// the same for other channel counts
template <int NG>
__device__ __forceinline__ void issue_row_any(int ks, uint32_t acc_t, uint32_t r0, uint32_t r1, uint32_t r2,
                                              uint32_t b_lo) {
  uint32_t acc = 0u;
#pragma unroll 1
  for (int tap = 0; tap < 9; ++tap) {
    uint32_t a_lo = (tap < 3 ? r0 : tap < 6 ? r1 : r2) + (uint32_t)(tap % 3);
#pragma unroll 1
    for (int k = 0; k < ks; ++k) {
      mma_k16<NG>(acc_t, a_lo, b_lo, acc);
      acc = 1u;
      a_lo += 2 * (tc::PLANE >> 4);
      b_lo += 2 * NG;
    }
  }
}

constexpr int kWsEpilogue = 256;   // warps 0-7: two groups of four, one per accumulator
constexpr int kWsMmaWarp = kWsEpilogue / 32;  // the first of two
constexpr int kWsThreads = kWsEpilogue + 64 + 32;
constexpr int kWsAcc = 4;          // accumulators
// resident blocks per SM the registers are kept for (shared memory allows
// more than one only for the narrow layers)
constexpr int ws_min_blocks(int ng, bool add) { return ng <= 64 && !add ? 2 : 1; }

// N consecutive 32-bit tensor-memory columns of the warp's 32 lanes
template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t (&r)[N], uint32_t addr) {
  static_assert(N == 16 || N == 32, "16 or 32 columns");
  if constexpr (N == 16)
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr));
  else
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,"
        "%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(addr));
}

// CW floats from a 32-byte aligned address (not through the read-only path:
// the kernel before wrote them)
template <int CW>
__device__ __forceinline__ void ld_global_floats(float (&v)[CW], const float* p) {
#pragma unroll
  for (int k = 0; k < CW; k += 8)
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v[k]), "=f"(v[k + 1]), "=f"(v[k + 2]), "=f"(v[k + 3]), "=f"(v[k + 4]), "=f"(v[k + 5]),
                   "=f"(v[k + 6]), "=f"(v[k + 7])
                 : "l"(p + k));
}

// 32 bytes (one sector) to a 32-byte aligned address
__device__ __forceinline__ void st_global_32B(void* p, const uint32_t* v) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]),
               "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
// acc_in (may be null): fp32 partial sums [pixel][Cout] of the other input
// channels, added before the bias (a layer split over its input channels,
// conv_fwd); y (may be null): bf16 output.
// ADD: acc_in is there; its loads take registers for one block per SM, which
// is all that fits beside a split layer's weights.
template <int NG, bool ADD>
__global__ void __launch_bounds__(kWsThreads, ws_min_blocks(NG, ADD)) k_conv_fwd_ws(const __grid_constant__ CUtensorMap xmap, rx_conv_desc d,
                                                        const bf16* __restrict__ w, const float* __restrict__ bias,
                                                        bf16* __restrict__ y, float* __restrict__ y32,
                                                        const float* __restrict__ acc_in, int relu, int S, int G,
                                                        long long per_cta, int* err) {
  constexpr int TCOLS = kWsAcc * NG;  // a power of two, 64 to 512
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long full[tc::kMaxSlots], empty[tc::kMaxSlots];
  __shared__ __align__(8) unsigned long long acc_full[kWsAcc], acc_empty[kWsAcc], w_full, mma_done;
  __shared__ uint32_t tmem_base;
  __shared__ volatile int abort_flag;
  __shared__ __align__(16) float sbias[NG];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int KC = d.Cin / 8;
  const int SB = tc::slot_bytes(d.Cin);
  unsigned char* smem = smem_raw + ((128 - (smem_u32(smem_raw) & 127)) & 127);
  unsigned char* wsm = smem;                                 // [tap][kc][co][8]
  unsigned char* rsm = smem + tc::weights_bytes(d.Cin, NG);  // S x [kc][PLANE]
  const int grp = blockIdx.x % G;
  const int xt = (d.W + tc::TILE - 1) / tc::TILE;
  const long long total = (long long)d.N * xt * d.H;  // row tiles, row fastest
  const long long u0 = (long long)(blockIdx.x / G) * per_cta;
  const long long uend = u0 + per_cta < total ? u0 + per_cta : total;

  if (tid == 0) {
    abort_flag = 0;
    for (int s = 0; s < S; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&full[s])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 3;\n" ::"r"(smem_u32(&empty[s])));
    }
    for (int b = 0; b < kWsAcc; ++b) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&acc_full[b])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;\n" ::"r"(smem_u32(&acc_empty[b])));
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(&w_full)), "r"(kWsEpilogue / 32));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 2;\n" ::"r"(smem_u32(&mma_done)));
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_base)),
                 "r"(TCOLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  // no chain_go: the next kernel's blocks, let in while this one works, took
  // more than they hid (a 1080p inference 1,255 us with it, 1,160 without,
  // 1,225 unchained)
  chain_wait(w, bias, y, y32, acc_in);
  for (int c = tid; c < NG; c += blockDim.x) sbias[c] = bias ? bias[grp * NG + c] : 0.0f;
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = tmem_base;

  if (warp > kWsMmaWarp + 1) {
    // ------------------------------------------------ producer (TMA)
    if (elect_one()) {
      const uint32_t rb = smem_u32(rsm), row_bytes = (uint32_t)(KC * tc::PLANE);
      int k = 0;  // rows issued
      bool ok = true;
      for (long long u = u0; u < uend && ok;) {
        const long long col = u / d.H;
        const int ylo = (int)(u - col * d.H);
        const int yhi = (int)((long long)ylo + (uend - u) < d.H ? (long long)ylo + (uend - u) : d.H);
        const int n = (int)(col / xt), x0 = (int)(col % xt) * tc::TILE;
        for (int r = ylo - 1; r <= yhi; ++r, ++k) {
          const int s = k % S;
          ok = mbar_wait_abortable(smem_u32(&empty[s]), (uint32_t)(((k / S) & 1) ^ 1), &abort_flag);
          if (!ok) break;
          const uint32_t bar = smem_u32(&full[s]);
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(row_bytes)
                       : "memory");
          asm volatile(
              "cp.async.bulk.tensor.5d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
              "%5, %6}], [%7];\n" ::"r"(rb + (uint32_t)(s * SB)),
              "l"(&xmap), "r"(0), "r"(x0 - 1), "r"(0), "r"(r), "r"(n), "r"(bar)
              : "memory");
        }
        u += yhi - ylo;
      }
      // no copy may be in flight when the block ends
      const unsigned long long t0 = clock64();
      for (int q = k > S ? k - S : 0; q < k; ++q)
        while (!mbar_try(smem_u32(&full[q % S]), (uint32_t)((q / S) & 1)) && clock64() - t0 < tc::kSpinCycles) {
        }
    }
    __syncwarp();
  } else if (warp >= kWsMmaWarp) {
    // ------------------------------------------------ MMA issuers
    // One elected lane of each warp walks the rows, warp 0 of the pair taking
    // the even and warp 1 the odd ones: a row's waits cost several hundred
    // cycles even when nothing has to be waited for, and the tensor core's
    // queue is too short to cover them, so the other warp's row does.
    const int mw = warp - kWsMmaWarp;
    const uint32_t rb = smem_u32(rsm), wb = smem_u32(wsm);
    // descriptor low words: (address >> 4) | (LBO >> 4) << 16, LBO = one
    // plane (A) or NG x 16 B (B)
    const uint32_t a_lo0 = (rb >> 4) | ((uint32_t)(tc::PLANE >> 4) << 16);
    const uint32_t b_lo0 = (wb >> 4) | ((uint32_t)NG << 16);
    const uint32_t slot16 = (uint32_t)SB >> 4;
    if (elect_one()) {
      auto advance = [&](int& s, uint32_t& ph) {
        if (++s == S) {
          s = 0;
          ph ^= 1u;
        }
      };
      auto wait = [&](unsigned long long* bar, uint32_t ph) {
        return mbar_wait_abortable(smem_u32(bar), ph, &abort_flag);
      };
      int s2 = 0;        // ring slot of the newest input row read so far
      uint32_t p2 = 0;   // its phase parity
      int i = 0;         // output rows so far
      bool ok = wait(&w_full, 0u);
      for (long long u = u0; u < uend && ok;) {
        const long long col = u / d.H;
        const int ylo = (int)(u - col * d.H);
        const int yhi = (int)((long long)ylo + (uend - u) < d.H ? (long long)ylo + (uend - u) : d.H);
        const int nrows = yhi - ylo;
        // rows yy - 1, yy, yy + 1 sit in slots s0, s1, s2
        int s0 = s2;
        uint32_t p0 = p2;
        int s1 = s0;
        uint32_t p1 = p0;
        advance(s1, p1);
        s2 = s1;
        p2 = p1;
        advance(s2, p2);
        for (int r = 0; r < nrows; ++r, ++i) {
          if ((i & 1) == mw) {
            const int b = i % kWsAcc;
            ok = wait(&full[s0], p0) && wait(&full[s1], p1) && wait(&full[s2], p2) &&
                 wait(&acc_empty[b], (uint32_t)(((i / kWsAcc) & 1) ^ 1));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const uint32_t acc_t = tmem + (uint32_t)(b * NG);
            const uint32_t r0 = a_lo0 + (uint32_t)s0 * slot16, r1 = a_lo0 + (uint32_t)s1 * slot16,
                           r2 = a_lo0 + (uint32_t)s2 * slot16;
            switch (KC) {
              case 2: issue_row<NG, 1>(acc_t, r0, r1, r2, b_lo0); break;
              case 4: issue_row<NG, 2>(acc_t, r0, r1, r2, b_lo0); break;
              case 8: issue_row<NG, 4>(acc_t, r0, r1, r2, b_lo0); break;
              case 12: issue_row<NG, 6>(acc_t, r0, r1, r2, b_lo0); break;
              default: issue_row_any<NG>(KC / 2, acc_t, r0, r1, r2, b_lo0); break;
            }
            tc_commit(smem_u32(&acc_full[b]));
            // an input row is free once its three output rows have read it;
            // a segment's first and last rows stand in for the missing ones
            const int n0 = r == 0 ? 3 : 1, n1 = nrows == 1 ? 3 : (r == 0 || r + 1 == nrows) ? 2 : 1,
                      n2 = r + 1 == nrows ? 3 : 1;
            for (int q = 0; q < n0; ++q) tc_commit(smem_u32(&empty[s0]));
            for (int q = 0; q < n1; ++q) tc_commit(smem_u32(&empty[s1]));
            for (int q = 0; q < n2; ++q) tc_commit(smem_u32(&empty[s2]));
          }
          s0 = s1;
          p0 = p1;
          s1 = s2;
          p1 = p2;
          advance(s2, p2);
        }
        u += nrows;  // s2: the next segment's first row follows this one's last
      }
      // every MMA issued has finished before the tensor memory is released
      tc_commit(smem_u32(&mma_done));
      const unsigned long long t0 = clock64();
      while (!mbar_try(smem_u32(&mma_done), 0u) && clock64() - t0 < tc::kSpinCycles) {
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------ epilogue (warps 0-7)
    // this group's weights first, while the producers fetch the first rows:
    // [co][tap][kc] -> [tap][kc][co][8], neighbouring threads on neighbouring
    // channels: 16-byte pieces side by side in shared memory (along kc they
    // would all meet in the same banks)
    for (int c = tid; c < NG * 9 * KC; c += kWsEpilogue) {
      const int co = c % NG, tk = c / NG;  // tk = tap * KC + kc: also the source's order
      cp_async16(wsm + c * 16, w + (long long)(grp * NG + co) * 9 * d.Cin + tk * 8, true);
    }
    cp_async_commit();
    cp_async_wait<0>();
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncwarp();
    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(&w_full)) : "memory");
    // warps 0-3 take the even output rows (accumulators 0 and 2), 4-7 the odd ones:
    // one row's tensor-memory loads, arithmetic and stores take a warp about
    // 700 cycles per 16 channels, as long as its MMAs in the narrow layers,
    // so each group gets two rows' time
    constexpr int CW = NG < 32 ? 16 : 32;  // columns per tensor-memory load
    const int eg = warp >> 2, qtr = warp & 3;  // group; tensor-memory lanes 32 qtr .. 32 qtr + 31
    const long long y_off = d.y_coff + grp * NG;
    // whole-sector stores when every 16-channel run of the view starts on one
    const bool y_sect = ((uintptr_t)y & 31) == 0 && d.y_cstride % 16 == 0 && d.y_coff % 16 == 0;
    const bool f_sect = ((uintptr_t)y32 & 31) == 0 && d.y_cstride % 8 == 0 && d.y_coff % 8 == 0;
    int i = 0;
    bool ok = true;
    for (long long u = u0; u < uend && ok;) {
      const long long col = u / d.H;
      const int ylo = (int)(u - col * d.H);
      const int yhi = (int)((long long)ylo + (uend - u) < d.H ? (long long)ylo + (uend - u) : d.H);
      const int n = (int)(col / xt), x0 = (int)(col % xt) * tc::TILE;
      const int xx = x0 + qtr * 32 + lane;
      for (int yy = ylo; yy < yhi; ++yy, ++i) {
        if ((i & 1) != eg) continue;
        const int b = i % kWsAcc;
        const uint32_t acc_t = tmem + ((uint32_t)(qtr * 32) << 16) + (uint32_t)(b * NG);
        const long long m = ((long long)n * d.H + yy) * d.W + xx;
        // the other half's sums (launch_ws_split) do not wait for this row's
        float part[CW];
        const float* part_at = acc_in + m * d.Cout + grp * NG;
        const bool add = ADD && xx < d.W;
        if (add) ld_global_floats(part, part_at);
        if (!mbar_wait_warp(smem_u32(&acc_full[b]), (uint32_t)((i / kWsAcc) & 1), &abort_flag)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll 1
        for (int c0 = 0; c0 < NG; c0 += CW) {
          uint32_t r[CW];
          if (add && c0) ld_global_floats(part, part_at + c0);
          tmem_ld(r, acc_t + (uint32_t)c0);
          asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
          if (xx < d.W) {
            float v[CW];
#pragma unroll
            for (int k = 0; k < CW; ++k) v[k] = __uint_as_float(r[k]);
            if (ADD) {
#pragma unroll
              for (int k = 0; k < CW; ++k) v[k] += part[k];
            }
#pragma unroll
            for (int k = 0; k < CW / 4; ++k) {
              const float4 bb = *reinterpret_cast<const float4*>(sbias + c0 + 4 * k);
              v[4 * k] += bb.x;
              v[4 * k + 1] += bb.y;
              v[4 * k + 2] += bb.z;
              v[4 * k + 3] += bb.w;
            }
            if (relu) {
#pragma unroll
              for (int k = 0; k < CW; ++k) v[k] = fmaxf(v[k], 0.0f);
            }
            const long long o = m * d.y_cstride + y_off + c0;
            if (y) {
              uint32_t pw[CW / 2];
#pragma unroll
              for (int k = 0; k < CW / 2; ++k) {
                __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
                pw[k] = *reinterpret_cast<uint32_t*>(&h);
              }
              if (y_sect) {
#pragma unroll
                for (int k = 0; k < CW / 16; ++k) st_global_32B(y + o + 16 * k, pw + 8 * k);
              } else {
#pragma unroll
                for (int k = 0; k < CW / 8; ++k)
                  reinterpret_cast<uint4*>(y + o)[k] = make_uint4(pw[4 * k], pw[4 * k + 1], pw[4 * k + 2],
                  pw[4 * k + 3]);
              }
            }
            if (y32) {
              if (f_sect) {
#pragma unroll
                for (int k = 0; k < CW / 8; ++k)
                  st_global_32B(y32 + o + 8 * k, reinterpret_cast<const uint32_t*>(v) + 8 * k);
              } else {
                float4* d32 = reinterpret_cast<float4*>(y32 + o);
#pragma unroll
                for (int k = 0; k < CW / 4; ++k)
                  d32[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
              }
            }
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(&acc_empty[b])) : "memory");
      }
      u += yhi - ylo;
    }
  }

  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  if (tid == 0 && abort_flag) atomicOr(err, ERR_BAD_NODE);
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TCOLS));
}

// ------------------------------------------- weight gradient on tcgen05
// dw[co][tap][ci] += sum_p dy[p][co] x[p + off(tap)][ci] as one GEMM per tap
// with the pixels as K: M = input channels (up to 128 of them), N = output
// channels, one tensor-memory accumulator per tap, all of them kept for the
// whole strip of rows a block walks.  The rows arrive by TMA in the forward
// kernel's slots [channel chunk][pixel x 16 B], which read as MN-major
// operands (8 channels contiguous, pixels 16 B apart); a tap is the same x
// slot moved by one pixel or one row, so x and dy are read once for all
// taps of a block instead of once per tap.  A block holds T taps of N output
// channels, T * N <= 512 columns: all nine taps up to N = 32, five (then
// four) at N = 64, three at N = 128; blockIdx.x % G picks its input-channel
// group, output-channel group and taps.  At the end the strips' sums meet
// in dw by fp32 atomics (32 consecutive input channels per warp).
// A width that is no multiple of 16 leaves a row's last step with pixels past
// the image, where dy is zero fill.  So is x, but for tap column 0, whose
// first such pixel reads the image's last column, and zero times an infinity
// or a NaN there would reach a sum that it does not belong to.  That step of
// that column reads 16 pixels of its own instead, loaded behind the row
// through a map that ends one column early.
//   warps 0-3: read the accumulators at the end.  warps 4-5: MMA issuers,
//   each with half of the block's taps, so that one's waits pass under the
//   other's MMAs.  warp 6: producer.  Waits are bounded as in k_conv_fwd_ws.
// Bound by the MMAs' operand reads at N <= 32 (72 MMAs of about 40 cycles
// per 128 pixels), by TMA's 16 B per cycle at N >= 64.  The eleven layers'
// weight gradients at 16 x 128^2 pixels, back to back: 1,510 us with
// k_conv_wgrad (a block per tap, each reading x and dy again), 304 us here;
// 96 -> 32 channels 390 -> 52 us.  ncu: tensor pipe 19-41 % busy, DRAM 4-19 %.
struct WgradArgs {
  int N, H, W, Cin, Cout;
  int tw, tiles;     // pixels per row tile (a multiple of 16), tiles per row
  int cm, mg;        // input channels per group, groups
  int nc, ng;        // output channels per group, groups
  int taps, tg;      // taps per group, groups
  int Sx, Sy;        // ring slots of x and dy rows
  int xslot, yslot;  // bytes
  int xcut;          // offset of the cut step's pixels in an x slot (0: no row has one)
  int tcols;         // tensor-memory columns (a power of two)
};
constexpr int kWgThreads = 224, kWgSlots = 6;

// CUT: rows may have a cut step (W not a multiple of 16).
template <bool CUT>
__global__ void __launch_bounds__(kWgThreads, 1) k_conv_wgrad_ws(const __grid_constant__ CUtensorMap xmap,
                                                                 const __grid_constant__ CUtensorMap cutmap,
                                                                 const __grid_constant__ CUtensorMap ymap, WgradArgs A,
                                                                 float* __restrict__ dw, long long per_cta, int* err) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long xfull[kWgSlots], xempty[kWgSlots], yfull[kWgSlots], yempty[kWgSlots], done;
  __shared__ uint32_t tmem_base;
  __shared__ volatile int abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t sx = (smem_u32(smem_raw) + 127) & ~127u;
  const uint32_t sy = sx + (uint32_t)(A.Sx * A.xslot);  // dy rows behind the x rows
  int g = blockIdx.x % (A.mg * A.ng * A.tg);
  const long long strip = blockIdx.x / (A.mg * A.ng * A.tg);
  const int tap0 = (g % A.tg) * A.taps, ntap = min(A.taps, 9 - tap0);
  g /= A.tg;
  const int co0 = (g % A.ng) * A.nc, ci0 = (g / A.ng) * A.cm;
  const long long total = (long long)A.N * A.tiles * A.H;  // row tiles, row fastest
  const long long u0 = strip * per_cta, uend = min(u0 + per_cta, total);

  if (tid == 0) {
    abort_flag = 0;
    for (int s = 0; s < kWgSlots; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&xfull[s])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 2;\n" ::"r"(smem_u32(&xempty[s])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&yfull[s])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 2;\n" ::"r"(smem_u32(&yempty[s])));
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 2;\n" ::"r"(smem_u32(&done)));
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_base)),
                 "r"(A.tcols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  chain_wait(dw);
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  chain_go();
  const uint32_t tmem = tmem_base;
  auto wait = [&](unsigned long long* bar, uint32_t ph) {
    return mbar_wait_abortable(smem_u32(bar), ph, &abort_flag);
  };

  if (warp == 6) {
    // ------------------------------------------------ producer
    if (elect_one()) {
      const uint32_t xbytes = (uint32_t)((A.tw + 2) * 16 * (A.cm / 8)), ybytes = (uint32_t)(A.tw * 16 * (A.nc / 8));
      auto expect = [&](uint32_t bar, uint32_t bytes) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
      };
      auto load = [&](const CUtensorMap* map, uint32_t dst, uint32_t bar, int px, int chunk, int row, int img) {
        asm volatile(
            "cp.async.bulk.tensor.5d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, "
            "%6}], [%7];\n" ::"r"(dst),
            "l"(map), "r"(0), "r"(px), "r"(chunk), "r"(row), "r"(img), "r"(bar)
            : "memory");
      };
      int kx = 0, ky = 0;  // x and dy rows issued
      bool ok = true;
      for (long long u = u0; u < uend && ok;) {
        const long long col = u / A.H;
        const int ylo = (int)(u - col * A.H), nrows = (int)min((long long)(A.H - ylo), uend - u);
        const int n = (int)(col / A.tiles), x0 = (int)(col % A.tiles) * A.tw;
        const int px = min(A.tw, A.W - x0);
        const bool cut = CUT && px % 16 != 0;  // the row's last step reaches past the image
        // first pixel of that step for tap column 0; an image of one column
        // has none to read (past its end: zeros)
        const int cut_px = A.W > 1 ? x0 - 1 + (px & ~15) : A.W;
        for (int r = -1; r <= nrows && ok; ++r) {
          const int s = kx % A.Sx;
          ok = wait(&xempty[s], (uint32_t)(((kx / A.Sx) & 1) ^ 1));
          if (!ok) break;
          const uint32_t slot = sx + (uint32_t)(s * A.xslot), bar = smem_u32(&xfull[s]);
          expect(bar, xbytes + (cut ? (uint32_t)(16 * 16 * (A.cm / 8)) : 0u));
          load(&xmap, slot, bar, x0 - 1, ci0 / 8, ylo + r, n);
          if (cut) load(&cutmap, slot + (uint32_t)A.xcut, bar, cut_px, ci0 / 8, ylo + r, n);
          ++kx;
          if (r < 1) continue;
          // dy row r - 1 goes with x rows r - 2 .. r
          const int t = ky % A.Sy;
          ok = wait(&yempty[t], (uint32_t)(((ky / A.Sy) & 1) ^ 1));
          if (!ok) break;
          expect(smem_u32(&yfull[t]), ybytes);
          load(&ymap, sy + (uint32_t)(t * A.yslot), smem_u32(&yfull[t]), x0, co0 / 8, ylo + r - 1, n);
          ++ky;
        }
        u += nrows;
      }
      // no copy may be in flight when the block ends
      const unsigned long long t0 = clock64();
      for (int q = kx > A.Sx ? kx - A.Sx : 0; q < kx; ++q)
        while (!mbar_try(smem_u32(&xfull[q % A.Sx]), (uint32_t)((q / A.Sx) & 1)) && clock64() - t0 < tc::kSpinCycles) {
        }
      for (int q = ky > A.Sy ? ky - A.Sy : 0; q < ky; ++q)
        while (!mbar_try(smem_u32(&yfull[q % A.Sy]), (uint32_t)((q / A.Sy) & 1)) && clock64() - t0 < tc::kSpinCycles) {
        }
    }
    __syncwarp();
  } else if (warp >= 4) {
    // ------------------------------------------------ MMA issuers
    if (elect_one()) {
      // M = 64 (up to 64 channels) or 128, N = nc, FP32 accumulate, BF16, both
      // operands MN-major
      const uint32_t id = tc::idesc(0) - (A.cm <= 64 ? 4u << 24 : 0u) + (1u << 15) + (1u << 16) +
                          ((uint32_t)(A.nc >> 3) << 17);
      // MN-major, no swizzle: LBO (next 8 pixels) 128 B, SBO (next 8
      // channels) one plane
      const uint64_t a_hi = (uint64_t)((uint32_t)(A.tw + 2) | (1u << 14)) << 32;
      const uint64_t b_hi = (uint64_t)((uint32_t)A.tw | (1u << 14)) << 32;
      const uint64_t cut_hi = (uint64_t)(16u | (1u << 14)) << 32;  // planes of 16 pixels
      auto mma = [&](uint32_t d, uint64_t ad, uint64_t bd, uint32_t p) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(d),
            "l"(ad), "l"(bd), "r"(id), "r"(p), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
      };
      const uint32_t a0 = (sx >> 4) | (8u << 16), b0 = (sy >> 4) | (8u << 16);
      const uint32_t xs16 = (uint32_t)A.xslot >> 4, ys16 = (uint32_t)A.yslot >> 4;
      // this warp's taps [j0, j1) of the block's
      const int j0 = warp == 4 ? 0 : (ntap + 1) / 2, j1 = warp == 4 ? (ntap + 1) / 2 : ntap;
      auto advance = [](int& slot, uint32_t& ph, int n) {
        if (++slot == n) {
          slot = 0;
          ph ^= 1u;
        }
      };
      int xs = 0, ys = 0;          // ring slots of the newest x row, of the dy row
      uint32_t xph = 0, yph = 0;   // their phase parities
      bool ok = true;
      uint32_t acc = 0u;           // the first row overwrites the accumulators
      for (long long u = u0; u < uend && ok;) {
        const long long col = u / A.H;
        const int ylo = (int)(u - col * A.H), nrows = (int)min((long long)(A.H - ylo), uend - u);
        const int x0 = (int)(col % A.tiles) * A.tw;
        const int px = min(A.tw, A.W - x0), ksteps = (px + 15) / 16;
        const bool cut = CUT && px % 16 != 0;
        // x rows yy - 1, yy, yy + 1 of output row yy
        const int sa = xs;
        ok = wait(&xfull[xs], xph);
        advance(xs, xph, A.Sx);
        const int sb = xs;
        ok = ok && wait(&xfull[xs], xph);
        advance(xs, xph, A.Sx);
        int s0 = sa, s1 = sb;
        for (int r = 0; r < nrows; ++r) {
          const int s2 = xs;
          ok = ok && wait(&xfull[s2], xph) && wait(&yfull[ys], yph);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
          const uint32_t r0 = a0 + (uint32_t)s0 * xs16, r1 = a0 + (uint32_t)s1 * xs16, r2 = a0 + (uint32_t)s2 * xs16;
          uint32_t b_lo = b0 + (uint32_t)ys * ys16;
#pragma unroll 1
          for (int j = j0; j < j1; ++j) {
            const int tap = tap0 + j;
            const int dx = tap < 3 ? tap : tap < 6 ? tap - 3 : tap - 6;
            uint32_t a_lo = (tap < 3 ? r0 : tap < 6 ? r1 : r2) + (uint32_t)dx;
            const uint32_t d = tmem + (uint32_t)(j * A.nc);
            // the last step's pixels
            const uint64_t a_last = cut && dx == 0 ? cut_hi | (a_lo + ((uint32_t)A.xcut >> 4))
                                                   : a_hi | (a_lo + 16 * (uint32_t)(ksteps - 1));
            if (ksteps == 8) {  // compile-time offsets, as in issue_row
#pragma unroll
              for (int k = 0; k < 7; ++k) mma(d, a_hi | (a_lo + 16 * k), b_hi | (b_lo + 16 * k), k ? 1u : acc);
              mma(d, a_last, b_hi | (b_lo + 16 * 7), 1u);
            } else {
#pragma unroll 1
              for (int k = 0; k < ksteps - 1; ++k)  // 16 pixels each
                mma(d, a_hi | (a_lo + 16 * k), b_hi | (b_lo + 16 * k), k ? 1u : acc);
              mma(d, a_last, b_hi | (b_lo + 16 * (ksteps - 1)), ksteps > 1 ? 1u : acc);
            }
          }
          acc = 1u;
          tc_commit(smem_u32(&yempty[ys]));
          tc_commit(smem_u32(&xempty[s0]));
          if (r + 1 == nrows) {  // the segment's last two x rows have no later reader
            tc_commit(smem_u32(&xempty[s1]));
            tc_commit(smem_u32(&xempty[s2]));
          }
          s0 = s1;
          s1 = s2;
          advance(xs, xph, A.Sx);
          advance(ys, yph, A.Sy);
        }
        u += nrows;
      }
      tc_commit(smem_u32(&done));
    }
    __syncwarp();
  }
  // every MMA issued has finished (also before the tensor memory is released)
  {
    const unsigned long long t0 = clock64();
    while (!mbar_try(smem_u32(&done), 0u)) {
      if (clock64() - t0 > tc::kSpinCycles) {
        abort_flag = 1;
        break;
      }
    }
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  if (warp < 4 && !abort_flag && u0 < uend) {
    // an M = 64 accumulator has 16 rows in each quarter of the lanes
    const int rows = A.cm <= 64 ? 16 : 32, ci = ci0 + warp * rows + lane;
    const bool mine = lane < rows && warp * rows + lane < A.cm && ci < A.Cin;
    for (int j = 0; j < ntap; ++j)
      for (int c = 0; c < A.nc; c += 16) {
        uint32_t r[16];
        tmem_ld(r, tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(j * A.nc + c));
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        if (mine) {
          float* o = dw + ((long long)(co0 + c) * 9 + tap0 + j) * A.Cin + ci;
#pragma unroll
          for (int k = 0; k < 16; ++k) atomicAdd(o + (long long)k * 9 * A.Cin, __uint_as_float(r[k]));
        }
      }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (tid == 0 && abort_flag) atomicOr(err, ERR_BAD_NODE);
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(A.tcols));
}

// ------------------------------------------------------- weight gradient
// dw[co][tap][ci] += sum_p dy[p][co] * x[p + off(tap)][ci]
// GEMM: M = output channels (64), N = input channels (64), K = pixels
// (32 per stage, `pix_per_block` per block, split-K with atomics).
__global__ void __launch_bounds__(128) k_conv_wgrad(rx_conv_desc d, const bf16* __restrict__ dy,
                                                    const bf16* __restrict__ x, float* __restrict__ dw,
                                                    int pix_per_block) {
  constexpr int BM = 64, BN = 64, BK = 32, LDA = BM + 8, LDB = BN + 8;
  __shared__ __align__(16) bf16 sA[2][BK][LDA];
  __shared__ __align__(16) bf16 sB[2][BK][LDB];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp & 1, wn = warp >> 1;
  const long long HW = (long long)d.H * d.W;
  const long long P = (long long)d.N * HW;
  const int tap = blockIdx.z;
  const int dyo = tap / 3 - 1, dxo = tap % 3 - 1;
  const int co_blocks = (d.Cout + BM - 1) / BM;
  const int co0 = (blockIdx.y % co_blocks) * BM;
  const int ci0 = (blockIdx.y / co_blocks) * BN;
  const long long p_begin = (long long)blockIdx.x * pix_per_block;
  const long long p_end = P < p_begin + pix_per_block ? P : p_begin + pix_per_block;
  const int KT = (int)((p_end - p_begin + BK - 1) / BK);

  auto load = [&](int kt, int buf) {
    long long pb = p_begin + (long long)kt * BK;
    // 32 pixels x 8 chunks of dy and of x: 256 chunks each, 2 per thread
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      int c = tid + i * 128;
      int r = c >> 3, kc = c & 7;
      long long p = pb + r;
      bool pok = p < p_end;
      int co = co0 + kc * 8;
      bool ok = pok && co < d.Cout;
      const bf16* src = ok ? dy + p * d.y_cstride + d.y_coff + co : dy;
      cp_async16(&sA[buf][r][kc * 8], src, ok);
      long long n = pok ? p / HW : 0;
      long long rem = pok ? p - n * HW : 0;
      int yy = (int)(rem / d.W) + dyo, xx = (int)(rem % d.W) + dxo;
      int ci = ci0 + kc * 8;
      bool okx = pok && ci < d.Cin && yy >= 0 && yy < d.H && xx >= 0 && xx < d.W;
      const bf16* srcx = okx ? x + (n * HW + (long long)yy * d.W + xx) * d.x_cstride + d.x_coff + ci : x;
      cp_async16(&sB[buf][r][kc * 8], srcx, okx);
    }
  };

  float acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[i][j][k] = 0.0f;

  if (KT > 0) {
    load(0, 0);
    cp_async_commit();
  }
  for (int kt = 0; kt < KT; ++kt) {
    int buf = kt & 1;
    if (kt + 1 < KT) load(kt + 1, buf ^ 1);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
#pragma unroll
    for (int ks = 0; ks < BK / 16; ++ks) {
      const int j = lane >> 3, r = lane & 7;
      uint32_t af[2][4];
#pragma unroll
      for (int mi = 0; mi < 2; ++mi)
        ldsm_x4_t(af[mi], &sA[buf][ks * 16 + r + (j >> 1) * 8][wm * 32 + mi * 16 + (j & 1) * 8]);
#pragma unroll
      for (int nj = 0; nj < 2; ++nj) {
        uint32_t bfr[4];
        ldsm_x4_t(bfr, &sB[buf][ks * 16 + r + (j & 1) * 8][wn * 32 + nj * 16 + (j >> 1) * 8]);
#pragma unroll
        for (int mi = 0; mi < 2; ++mi) {
          mma_bf16(acc[mi][2 * nj], af[mi], bfr[0], bfr[1]);
          mma_bf16(acc[mi][2 * nj + 1], af[mi], bfr[2], bfr[3]);
        }
      }
    }
    __syncthreads();
  }
  cp_async_wait<0>();
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int mi = 0; mi < 2; ++mi)
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        int co = co0 + wm * 32 + mi * 16 + g + h * 8;
        int ci = ci0 + wn * 32 + ni * 8 + 2 * t;
        if (co >= d.Cout || ci >= d.Cin) continue;
        float* dst = dw + ((long long)co * 9 + tap) * d.Cin + ci;
        atomicAdd(dst, acc[mi][ni][2 * h]);
        atomicAdd(dst + 1, acc[mi][ni][2 * h + 1]);
      }
}

// dbias[co] += sum_p dy[p][co].  Bound by reading dy once (2 B per pixel
// and channel).  A thread owns one 16-byte chunk of 8 channels and every
// `lanes`-th pixel of its block's range, so a warp reads whole pixel rows.
// The lanes meet in shared memory, the blocks of a cluster in its first
// block, both in float64, and one fp32 atomic per channel and cluster adds
// to db: eight atomics in all (an atomic per block, 592 of them, left db at
// 4.9e-7 of the float64 sum at 16 x 128^2 pixels, against 1.2e-7).
// With a thread per channel walking 4096 pixels in series (64 blocks, 32-64
// busy threads each, one 2-byte load in flight per thread) the eleven layers
// of a training step's gradients took 3,440 us.
constexpr int kBiasThreads = 1024, kBiasCluster = 8, kBiasBlocks = 64;
constexpr int kBiasWidth = 128;  // channel chunks handled side by side, at most
__global__ void __cluster_dims__(kBiasCluster, 1, 1) __launch_bounds__(kBiasThreads)
    k_bias_grad(rx_conv_desc d, const bf16* __restrict__ dy, float* __restrict__ db, int pix_per_block) {
  __shared__ float part[kBiasThreads][9];  // 8 channels, padded against bank conflicts
  __shared__ double sums[kBiasWidth * 8];
  chain_wait(dy, db);
  chain_go();
  auto cluster = cooperative_groups::this_cluster();
  const long long P = (long long)d.N * d.H * d.W;
  const long long p0 = (long long)blockIdx.x * pix_per_block;
  const long long p1 = P < p0 + pix_per_block ? P : p0 + pix_per_block;  // may be empty
  const int chunks = d.Cout / 8;
  const int width = chunks < kBiasWidth ? chunks : kBiasWidth;
  const int lanes = kBiasThreads / width;
  const int lane = threadIdx.x / width, col = threadIdx.x - lane * width;
  for (int c0 = 0; c0 < chunks; c0 += width) {
    const int ck = c0 + col;
    float s[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    if (lane < lanes && ck < chunks) {
      const bf16* src = dy + d.y_coff + ck * 8;
#pragma unroll 4
      for (long long p = p0 + lane; p < p1; p += lanes) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(src + p * d.y_cstride));
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float2 f = __bfloat1622float2(h[k]);
          s[2 * k] += f.x;
          s[2 * k + 1] += f.y;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) part[threadIdx.x][k] = s[k];
    __syncthreads();
    for (int c = threadIdx.x; c < width * 8; c += kBiasThreads) {
      double t = 0.0;
      for (int l = 0; l < lanes; ++l) t += (double)part[l * width + c / 8][c & 7];
      sums[c] = t;
    }
    cluster.sync();
    if (cluster.block_rank() == 0)
      for (int c = threadIdx.x; c < width * 8; c += kBiasThreads) {
        if (c0 + c / 8 >= chunks) continue;
        double t = 0.0;
        for (int b = 0; b < kBiasCluster; ++b) t += cluster.map_shared_rank(sums, b)[c];
        atomicAdd(db + c0 * 8 + c, (float)t);
      }
    cluster.sync();  // the sums have been read: next columns, or the end
  }
}

// ------------------------------------------------------------ element-wise
// Every element-wise kernel walks (pixel, channel) of an NHWC view
// (stride, offset) with a grid-stride loop.
#define RX_EW_LOOP(count) \
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < (count); i += (long long)gridDim.x * blockDim.x)

// w_rot[ci][tap][co] = w[co][8 - tap][ci]: the weights of the input-gradient
// convolution (a 3x3 convolution of dy with the flipped, transposed kernel).
// Eight output channels per item: lanes read eight weights each along ci and
// write one 16-byte chunk (Cout is a multiple of 16).  One weight per item,
// with 64-bit divisions and 2-byte stores, took 39 us for the ten layers of a
// training step's gradients, this 31 (a launch each).
__global__ void k_rot_weights_v8(int Cout, int Cin, const bf16* __restrict__ w, bf16* __restrict__ wr) {
  chain_wait(w, wr);
  chain_go();
  RX_EW_LOOP((long long)(Cout / 8) * 9 * Cin) {
    size_t ci, tap, co8;
    if (i <= 0xffffffffLL) {  // 32-bit divisions
      const unsigned t = (unsigned)i / (unsigned)Cin, c = t / 9u;
      ci = (unsigned)i - t * (unsigned)Cin;
      tap = t - c * 9u;
      co8 = c;
    } else {
      const long long t = i / Cin;
      ci = (size_t)(i - t * Cin);
      co8 = (size_t)(t / 9);
      tap = (size_t)t - co8 * 9;
    }
    const bf16* s = w + (co8 * 72 + (8 - tap)) * Cin + ci;
    uint4 v;
    bf16* e = reinterpret_cast<bf16*>(&v);
#pragma unroll
    for (int k = 0; k < 8; ++k) e[k] = s[(size_t)k * 9 * Cin];
    *reinterpret_cast<uint4*>(wr + (ci * 9 + tap) * Cout + co8 * 8) = v;
  }
}

// dst = src (channels [0, C) of each view); accumulate: dst += src
__global__ void k_copy_ch(long long P, int C, const bf16* __restrict__ src, int s_stride, int s_off,
                          bf16* __restrict__ dst, int d_stride, int d_off, int accumulate) {
  RX_EW_LOOP(P * C) {
    long long p = i / C;
    int c = (int)(i % C);
    float v = __bfloat162float(src[p * s_stride + s_off + c]);
    bf16* o = dst + p * d_stride + d_off + c;
    if (accumulate) v += __bfloat162float(*o);
    *o = __float2bfloat16_rn(v);
  }
}

// g = y > 0 ? g : 0  (gradient through a ReLU whose output is y)
__global__ void k_relu_mask(long long P, int C, const bf16* __restrict__ yv, int y_stride, int y_off,
                            bf16* __restrict__ g, int g_stride, int g_off) {
  RX_EW_LOOP(P * C) {
    long long p = i / C;
    int c = (int)(i % C);
    if (!(__bfloat162float(yv[p * y_stride + y_off + c]) > 0.0f)) g[p * g_stride + g_off + c] = __float2bfloat16_rn(0.0f);
  }
}

// The same on 8-channel chunks (views whose channel count, stride and offset
// are multiples of 8): the gradient is read and written only where some
// output is not positive.  Bound by memory; the ten masks of a 16x128x128
// training step's gradients 203 -> 89 us.
__global__ void k_relu_mask_v8(long long P, int C, const bf16* __restrict__ yv, int y_stride, int y_off,
                               bf16* __restrict__ g, int g_stride, int g_off) {
  chain_wait(yv, g);
  chain_go();
  const int CK = C >> 3;
  const __nv_bfloat162 zero = __floats2bfloat162_rn(0.0f, 0.0f);
  RX_EW_LOOP(P * CK) {
    long long p;
    int ck;
    if (i <= 0xffffffffLL) {
      const unsigned q = (unsigned)i / (unsigned)CK;
      p = q;
      ck = (int)((unsigned)i - q * (unsigned)CK);
    } else {
      p = i / CK;
      ck = (int)(i - p * CK);
    }
    const uint4 y = *reinterpret_cast<const uint4*>(yv + p * y_stride + y_off + ck * 8);
    const unsigned* ye = reinterpret_cast<const unsigned*>(&y);
    unsigned keep[4], all = 0xffffffffu;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      __nv_bfloat162 v;
      *reinterpret_cast<unsigned*>(&v) = ye[k];
      keep[k] = __hgt2_mask(v, zero);  // a NaN is not positive
      all &= keep[k];
    }
    if (all == 0xffffffffu) continue;
    uint4* d = reinterpret_cast<uint4*>(g + p * g_stride + g_off + ck * 8);
    uint4 v = *d;
    v.x &= keep[0], v.y &= keep[1], v.z &= keep[2], v.w &= keep[3];
    *d = v;
  }
}

// 2x2 average pool (H, W even): out (N, H/2, W/2, C)
__global__ void k_pool2(int N, int H, int W, int C, const bf16* __restrict__ x, int x_stride, int x_off,
                        bf16* __restrict__ y, int y_stride, int y_off) {
  int h2 = H / 2, w2 = W / 2;
  RX_EW_LOOP((long long)N * h2 * w2 * C) {
    int c = (int)(i % C);
    long long q = i / C;
    int xo = (int)(q % w2), yo = (int)((q / w2) % h2);
    long long n = q / ((long long)w2 * h2);
    long long b = (n * H + 2 * yo) * W + 2 * xo;
    float s = __bfloat162float(x[b * x_stride + x_off + c]) + __bfloat162float(x[(b + 1) * x_stride + x_off + c]) +
              __bfloat162float(x[(b + W) * x_stride + x_off + c]) +
              __bfloat162float(x[(b + W + 1) * x_stride + x_off + c]);
    y[q * y_stride + y_off + c] = __float2bfloat16_rn(0.25f * s);
  }
}

// The same two layers on 8-channel (16-byte) chunks, for views whose
// channel count, stride and offset are multiples of 8: one item per chunk
// of an input pixel (upsample: one load, four stores) or of an output pixel
// (pool: four loads, one store); same float32 sum order as above.
__device__ __forceinline__ void chunk_index(long long i, int CK, int W, int H, int& ck, int& x, int& y, long long& n) {
  if (i <= 0xffffffffLL) {  // 32-bit divisions, a quarter of the instructions
    const unsigned u = (unsigned)i, a = u / (unsigned)CK, b = a / (unsigned)W, c = b / (unsigned)H;
    ck = (int)(u - a * (unsigned)CK);
    x = (int)(a - b * (unsigned)W);
    y = (int)(b - c * (unsigned)H);
    n = c;
    return;
  }
  ck = (int)(i % CK);
  long long q = i / CK;
  x = (int)(q % W);
  q /= W;
  y = (int)(q % H);
  n = q / H;
}

__global__ void k_up2_v8(int N, int H, int W, int C, const bf16* __restrict__ x, int x_stride, int x_off,
                         bf16* __restrict__ y, int y_stride, int y_off) {
  chain_wait(x, y);
  chain_go();
  const int CK = C >> 3;
  RX_EW_LOOP((long long)N * H * W * CK) {
    int ck, xx, yy;
    long long n;
    chunk_index(i, CK, W, H, ck, xx, yy, n);
    const uint4 v = *reinterpret_cast<const uint4*>(x + ((n * H + yy) * W + xx) * x_stride + x_off + ck * 8);
    const long long o = (n * 2 * H + 2 * yy) * 2LL * W + 2 * xx;
    bf16* d = y + y_off + ck * 8;
    *reinterpret_cast<uint4*>(d + o * y_stride) = v;
    *reinterpret_cast<uint4*>(d + (o + 1) * y_stride) = v;
    *reinterpret_cast<uint4*>(d + (o + 2LL * W) * y_stride) = v;
    *reinterpret_cast<uint4*>(d + (o + 2LL * W + 1) * y_stride) = v;
  }
}

__global__ void k_pool2_v8(int N, int H, int W, int C, const bf16* __restrict__ x, int x_stride, int x_off,
                           bf16* __restrict__ y, int y_stride, int y_off) {
  chain_wait(x, y);
  chain_go();
  const int CK = C >> 3, h2 = H / 2, w2 = W / 2;
  RX_EW_LOOP((long long)N * h2 * w2 * CK) {
    int ck, xo, yo;
    long long n;
    chunk_index(i, CK, w2, h2, ck, xo, yo, n);
    const long long b = (n * H + 2 * yo) * W + 2 * xo;
    const bf16* s = x + x_off + ck * 8;
    uint4 q[4] = {*reinterpret_cast<const uint4*>(s + b * x_stride),
                  *reinterpret_cast<const uint4*>(s + (b + 1) * x_stride),
                  *reinterpret_cast<const uint4*>(s + (b + W) * x_stride),
                  *reinterpret_cast<const uint4*>(s + (b + W + 1) * x_stride)};
    const bf16* e[4] = {reinterpret_cast<const bf16*>(&q[0]), reinterpret_cast<const bf16*>(&q[1]),
                        reinterpret_cast<const bf16*>(&q[2]), reinterpret_cast<const bf16*>(&q[3])};
    uint4 out;
    bf16* o = reinterpret_cast<bf16*>(&out);
#pragma unroll
    for (int k = 0; k < 8; ++k)
      o[k] = __float2bfloat16_rn(0.25f * (__bfloat162float(e[0][k]) + __bfloat162float(e[1][k]) +
                                          __bfloat162float(e[2][k]) + __bfloat162float(e[3][k])));
    *reinterpret_cast<uint4*>(y + ((n * h2 + yo) * w2 + xo) * y_stride + y_off + ck * 8) = out;
  }
}

// gradient of the pool: each input pixel gets a quarter of its output's
// gradient; accumulate adds to dx
__global__ void k_pool2_bwd(int N, int H, int W, int C, const bf16* __restrict__ dy, int dy_stride, int dy_off,
                            bf16* __restrict__ dx, int dx_stride, int dx_off, int accumulate) {
  RX_EW_LOOP((long long)N * H * W * C) {
    int c = (int)(i % C);
    long long p = i / C;
    int xx = (int)(p % W), yy = (int)((p / W) % H);
    long long n = p / ((long long)W * H);
    long long q = (n * (H / 2) + yy / 2) * (W / 2) + xx / 2;
    float v = 0.25f * __bfloat162float(dy[q * dy_stride + dy_off + c]);
    bf16* o = dx + p * dx_stride + dx_off + c;
    if (accumulate) v += __bfloat162float(*o);
    *o = __float2bfloat16_rn(v);
  }
}

// The two gradients on 8-channel chunks, one item per chunk of a pooled
// (small) pixel: the pool's reads its gradient once for four input pixels,
// the upsample's sums four; float32 sums in the order of the scalar forms.
// Bound by memory; in a 16x128x128 training batch the two pools' gradients
// 86 -> 15 us, the two upsamples' 52 -> 16.
__global__ void k_pool2_bwd_v8(int N, int H, int W, int C, const bf16* __restrict__ dy, int dy_stride, int dy_off,
                               bf16* __restrict__ dx, int dx_stride, int dx_off, int accumulate) {
  chain_wait(dy, dx);
  chain_go();
  const int CK = C >> 3, h2 = H / 2, w2 = W / 2;
  RX_EW_LOOP((long long)N * h2 * w2 * CK) {
    int ck, xo, yo;
    long long n;
    chunk_index(i, CK, w2, h2, ck, xo, yo, n);
    const uint4 q = *reinterpret_cast<const uint4*>(dy + ((n * h2 + yo) * w2 + xo) * dy_stride + dy_off + ck * 8);
    const bf16* e = reinterpret_cast<const bf16*>(&q);
    const long long b = (n * H + 2 * yo) * W + 2 * xo;
    bf16* d = dx + dx_off + ck * 8;
    uint4* o[4] = {reinterpret_cast<uint4*>(d + b * dx_stride), reinterpret_cast<uint4*>(d + (b + 1) * dx_stride),
                   reinterpret_cast<uint4*>(d + (b + W) * dx_stride),
                   reinterpret_cast<uint4*>(d + (b + W + 1) * dx_stride)};
    uint4 old[4];
    if (accumulate) {
#pragma unroll
      for (int j = 0; j < 4; ++j) old[j] = *o[j];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint4 out;
      bf16* r = reinterpret_cast<bf16*>(&out);
      const bf16* oe = reinterpret_cast<const bf16*>(&old[j]);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        float v = 0.25f * __bfloat162float(e[k]);
        if (accumulate) v += __bfloat162float(oe[k]);
        r[k] = __float2bfloat16_rn(v);
      }
      *o[j] = out;
    }
  }
}

__global__ void k_up2_bwd_v8(int N, int H, int W, int C, const bf16* __restrict__ dy, int dy_stride, int dy_off,
                             bf16* __restrict__ dx, int dx_stride, int dx_off) {
  chain_wait(dy, dx);
  chain_go();
  const int CK = C >> 3;
  RX_EW_LOOP((long long)N * H * W * CK) {
    int ck, xx, yy;
    long long n;
    chunk_index(i, CK, W, H, ck, xx, yy, n);
    const long long b = (n * 2 * H + 2 * yy) * 2LL * W + 2 * xx, w2 = 2LL * W;
    const bf16* s = dy + dy_off + ck * 8;
    const uint4 q[4] = {*reinterpret_cast<const uint4*>(s + b * dy_stride),
                        *reinterpret_cast<const uint4*>(s + (b + 1) * dy_stride),
                        *reinterpret_cast<const uint4*>(s + (b + w2) * dy_stride),
                        *reinterpret_cast<const uint4*>(s + (b + w2 + 1) * dy_stride)};
    const bf16* e[4] = {reinterpret_cast<const bf16*>(&q[0]), reinterpret_cast<const bf16*>(&q[1]),
                        reinterpret_cast<const bf16*>(&q[2]), reinterpret_cast<const bf16*>(&q[3])};
    uint4 out;
    bf16* o = reinterpret_cast<bf16*>(&out);
#pragma unroll
    for (int k = 0; k < 8; ++k)
      o[k] = __float2bfloat16_rn(__bfloat162float(e[0][k]) + __bfloat162float(e[1][k]) + __bfloat162float(e[2][k]) +
                                 __bfloat162float(e[3][k]));
    *reinterpret_cast<uint4*>(dx + ((n * H + yy) * W + xx) * dx_stride + dx_off + ck * 8) = out;
  }
}

// nearest 2x upsample: out (N, 2H, 2W, C) from x (N, H, W, C)
__global__ void k_up2(int N, int H, int W, int C, const bf16* __restrict__ x, int x_stride, int x_off,
                      bf16* __restrict__ y, int y_stride, int y_off) {
  RX_EW_LOOP((long long)N * 4 * H * W * C) {
    int c = (int)(i % C);
    long long p = i / C;
    int xx = (int)(p % (2 * W)), yy = (int)((p / (2 * W)) % (2 * H));
    long long n = p / (4LL * W * H);
    long long q = (n * H + yy / 2) * W + xx / 2;
    y[p * y_stride + y_off + c] = x[q * x_stride + x_off + c];
  }
}

// gradient of the upsample: sum of the four children
__global__ void k_up2_bwd(int N, int H, int W, int C, const bf16* __restrict__ dy, int dy_stride, int dy_off,
                          bf16* __restrict__ dx, int dx_stride, int dx_off) {
  RX_EW_LOOP((long long)N * H * W * C) {
    int c = (int)(i % C);
    long long q = i / C;
    int xx = (int)(q % W), yy = (int)((q / W) % H);
    long long n = q / ((long long)W * H);
    long long b = (n * 2 * H + 2 * yy) * 2 * W + 2 * xx;
    long long w2 = 2LL * W;
    float s = __bfloat162float(dy[b * dy_stride + dy_off + c]) + __bfloat162float(dy[(b + 1) * dy_stride + dy_off + c]) +
              __bfloat162float(dy[(b + w2) * dy_stride + dy_off + c]) +
              __bfloat162float(dy[(b + w2 + 1) * dy_stride + dy_off + c]);
    dx[q * dx_stride + dx_off + c] = __float2bfloat16_rn(s);
  }
}

// Network input: 16 channels (log1p radiance, albedo, normal, depth/(1+depth),
// six zeros) from float32 (P, 3) planes; base (optional) receives the
// float32 log1p radiance the network's output is added to.
__device__ __forceinline__ void feature_pixel(const float* rad, const float* alb, const float* nrm, float dep,
                                              float* base, unsigned* o) {
  float f[10];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    f[k] = log1pf(fmaxf(rad[k], 0.0f));
    f[3 + k] = alb[k];
    f[6 + k] = nrm[k];
    base[k] = f[k];
  }
  const float dd = fmaxf(dep, 0.0f);
  f[9] = dd / (1.0f + dd);
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(f[2 * k], f[2 * k + 1]);
    o[k] = *reinterpret_cast<const unsigned*>(&v);
  }
  o[5] = o[6] = o[7] = 0;
}

__global__ void k_features(long long P, const float* __restrict__ rad, const float* __restrict__ alb,
                           const float* __restrict__ nrm, const float* __restrict__ dep, bf16* __restrict__ out,
                           float* __restrict__ base) {
  RX_EW_LOOP(P) {
    unsigned o[8];
    float l[3];
    feature_pixel(rad + 3 * i, alb + 3 * i, nrm + 3 * i, dep[i], l, o);
    if (base)
#pragma unroll
      for (int k = 0; k < 3; ++k) base[3 * i + k] = l[k];
    unsigned* d = reinterpret_cast<unsigned*>(out + 16 * i);
#pragma unroll
    for (int k = 0; k < 8; ++k) d[k] = o[k];
  }
}

// Four pixels per item (P a multiple of 4, 16-byte aligned planes): the
// three-float pixels of a plane are three 16-byte loads, a pixel's features
// two 16-byte stores.  1920x1080: 51 -> 37 us (174 MB).
__global__ void k_features_v4(long long P4, const float4* __restrict__ rad, const float4* __restrict__ alb,
                              const float4* __restrict__ nrm, const float4* __restrict__ dep, uint4* __restrict__ out,
                              float4* __restrict__ base) {
  chain_wait(rad, alb, nrm, dep, out, base);
  chain_go();
  RX_EW_LOOP(P4) {
    float4 r[3], a[3], n[3], l[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) r[k] = rad[3 * i + k], a[k] = alb[3 * i + k], n[k] = nrm[3 * i + k];
    const float4 d = dep[i];
    const float dd[4] = {d.x, d.y, d.z, d.w};
    const float *rf = reinterpret_cast<const float*>(r), *af = reinterpret_cast<const float*>(a),
                *nf = reinterpret_cast<const float*>(n);
    float* lf = reinterpret_cast<float*>(l);
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      unsigned o[8];
      feature_pixel(rf + 3 * p, af + 3 * p, nf + 3 * p, dd[p], lf + 3 * p, o);
      out[8 * i + 2 * p] = make_uint4(o[0], o[1], o[2], o[3]);
      out[8 * i + 2 * p + 1] = make_uint4(o[4], o[5], o[6], o[7]);
    }
    if (base)
#pragma unroll
      for (int k = 0; k < 3; ++k) base[3 * i + k] = l[k];
  }
}

// L1 loss in log1p space of y + base (base optional) against target t
// (P, 3): sum |y + base - t| into *loss, gradient sign(.) * scale into g
// (bf16, channel stride gs; pad channels 3..gs-1 zero)
// CHUNKS: gs is a multiple of 8 and g 16-byte aligned, so the pixel's
// channels are stored 16 bytes at a time (16x128x128, gs 16: 28 -> 18 us).
// The sum is kept in float64 up to one fp32 atomic per block of 1,024 threads,
// at most a block per SM: an atomic per warp, 8,192 on one address, left it an
// order-dependent 1.3e-6 off.
constexpr int kLossThreads = 1024;
template <bool CHUNKS>
__global__ void __launch_bounds__(kLossThreads)
    k_l1_loss(long long P, const float* __restrict__ y32, int y_stride, const float* __restrict__ base,
              const float* __restrict__ t, float scale, bf16* __restrict__ g, int gs, float* __restrict__ loss) {
  chain_wait(y32, base, t, g, loss);
  chain_go();
  double s = 0.0;
  RX_EW_LOOP(P) {
    alignas(4) bf16 v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = __float2bfloat16_rn(0.0f);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      float dlt = (y32[i * y_stride + k] + (base ? base[3 * i + k] : 0.0f)) - t[3 * i + k];
      s += (double)fabsf(dlt);
      v[k] = __float2bfloat16_rn(dlt > 0.0f ? scale : (dlt < 0.0f ? -scale : 0.0f));
    }
    if (CHUNKS) {
      uint4* d = reinterpret_cast<uint4*>(g + i * gs);
      const unsigned* w = reinterpret_cast<const unsigned*>(v);
      d[0] = make_uint4(w[0], w[1], w[2], w[3]);
      for (int k = 1; k < gs / 8; ++k) d[k] = make_uint4(0, 0, 0, 0);
    } else {
      for (int k = 0; k < 3; ++k) g[i * gs + k] = v[k];
      for (int k = 3; k < gs; ++k) g[i * gs + k] = v[7];
    }
  }
  __shared__ double warp_sum[kLossThreads / 32];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double b = 0.0;
    for (int w = 0; w < kLossThreads / 32; ++w) b += warp_sum[w];
    atomicAdd(loss, (float)b);
  }
}

// radiance = max(expm1(y + base), 0) from the head's first three channels
__global__ void k_output(long long P, const float* __restrict__ y32, int y_stride, const float* __restrict__ base,
                         float* __restrict__ out) {
  chain_wait(y32, base, out);
  chain_go();
  RX_EW_LOOP(P) {
#pragma unroll
    for (int k = 0; k < 3; ++k)
      out[3 * i + k] = fmaxf(expm1f(y32[i * y_stride + k] + (base ? base[3 * i + k] : 0.0f)), 0.0f);
  }
}

// Adam (Kingma and Ba, 2015) on float32 master weights; writes the bf16
// copy the convolutions read and clears the gradient
__global__ void k_adam(long long n, float* __restrict__ p, float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, bf16* __restrict__ p16, float lr, float b1, float b2, float eps,
                       float c1, float c2) {
  RX_EW_LOOP(n) {
    float gi = g[i];
    float mi = b1 * m[i] + (1.0f - b1) * gi;
    float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    p[i] = pi;
    if (p16) p16[i] = __float2bfloat16_rn(pi);
    g[i] = 0.0f;
  }
}

static int ew_blocks(Ctx* ctx, long long n) {
  return (int)std::max<long long>(1, std::min<long long>((n + 255) / 256, (long long)ctx->num_sms * 32));
}

static bool conv_ok(const rx_conv_desc* d) {
  return d && d->N > 0 && d->H > 0 && d->W > 0 && d->Cin > 0 && d->Cout > 0 && d->Cin % 16 == 0 &&
         d->Cout % 16 == 0 && d->x_cstride % 8 == 0 && d->x_coff % 8 == 0 && d->y_cstride % 8 == 0 &&
         d->y_coff % 8 == 0 && d->x_coff + d->Cin <= d->x_cstride && d->y_coff + d->Cout <= d->y_cstride;
}

static bool unaligned(const void* p, size_t bytes) { return (uintptr_t)p % bytes != 0; }

template <int COUT>
static int launch_tc(Ctx* ctx, const rx_conv_desc* d, const bf16* x, const bf16* w, const float* bias, bf16* y,
                     float* y32, int relu, cudaStream_t st) {
  constexpr int smem = 2 * tc::stage_bytes(COUT);
  static int attr_dev = -1;
  if (attr_dev != ctx->device) {
    CUDA_TRY(ctx, cudaFuncSetAttribute(k_conv_fwd_tc<COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    attr_dev = ctx->device;
  }
  dim3 grid((unsigned)((d->W + tc::TILE - 1) / tc::TILE), (unsigned)d->H, (unsigned)d->N);
  k_conv_fwd_tc<COUT><<<grid, 128, smem, st>>>(*d, x, w, bias, y, y32, relu, ctx->d_err);
  CUDA_TRY(ctx, cudaGetLastError());
  return RX_OK;
}

// An NHWC view (`C` channels at `v`, pixel stride `stride` elements) as the
// 5-d tensor (8 channels, W, channel chunks, H, N) whose boxes -- `px`
// pixels x `chunks` chunks of one row -- land as [chunk][pixel x 16 B], with
// zeros from pixel `cols` of a row on (W, or fewer).  False when the driver
// has no tensor maps or cannot describe the view.
static bool row_map(int N, int H, int W, int cols, int C, int stride, const bf16* v, int px_box, int chunks,
                    CUtensorMap* map) {
  using Encode = decltype(&cuTensorMapEncodeTiled);
  static const Encode encode = [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &found) != cudaSuccess) {
      cudaGetLastError();
      return (Encode)nullptr;
    }
    return found == cudaDriverEntryPointSuccess ? reinterpret_cast<Encode>(fn) : (Encode)nullptr;
  }();
  if (!encode) return false;
  const cuuint64_t px = (cuuint64_t)stride * sizeof(bf16);
  const cuuint64_t dims[5] = {8, (cuuint64_t)cols, (cuuint64_t)C / 8, (cuuint64_t)H, (cuuint64_t)N};
  const cuuint64_t strides[4] = {px, 16, px * W, px * W * H};
  const cuuint32_t box[5] = {8, (cuuint32_t)px_box, (cuuint32_t)chunks, 1, 1}, step[5] = {1, 1, 1, 1, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<bf16*>(v), dims, strides, box, step,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Dynamic shared memory of a launch with at most one block per SM: enough
// that a second block does not fit.  Blocks that come up while the kernel
// before drains would otherwise pair up on the SMs that are free first and
// leave others idle (and a pair may want all the tensor memory twice): a
// 16x256x256 batch's gradients took 4,050 instead of 3,100 us.
static int sole_block_smem(Ctx* ctx, long long blocks, int smem) {
  return blocks <= ctx->num_sms ? std::max(smem, 233472 / 2) : smem;
}

template <int NG, bool ADD>
static int launch_ws_ng(Ctx* ctx, const rx_conv_desc* d, const bf16* x, const bf16* w, const float* bias, bf16* y,
                        float* y32, const float* acc_in, int relu, int S, int smem, cudaStream_t st, int* rc) {
  const int limit = 232448 - 1024;  // opt-in shared memory per block, less the static part
  static int attr_dev = -1;
  if (attr_dev != ctx->device) {
    if (cudaFuncSetAttribute(k_conv_fwd_ws<NG, ADD>, cudaFuncAttributeMaxDynamicSharedMemorySize, limit) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    attr_dev = ctx->device;
  }
  CUtensorMap xmap;
  if (!row_map(d->N, d->H, d->W, d->W, d->Cin, d->x_cstride, x + d->x_coff, tc::HALO_W, d->Cin / 8, &xmap)) return 0;
  // resident CTAs per SM from shared memory (dynamic + static + the
  // per-block reservation), capped by the registers (ws_min_blocks) and so
  // that every resident CTA gets its tensor memory
  cudaFuncAttributes fa{};
  int smem_sm = 0, reserved = 0;
  cudaFuncGetAttributes(&fa, k_conv_fwd_ws<NG, ADD>);
  cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, ctx->device);
  cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, ctx->device);
  constexpr int tcols = kWsAcc * NG;
  int per_sm = smem_sm / (smem + (int)fa.sharedSizeBytes + reserved);
  per_sm = std::max(1, std::min(std::min(per_sm, 512 / tcols), ws_min_blocks(NG, ADD)));
  const int G = d->Cout / NG;
  const long long total = (long long)d->N * d->H * ((d->W + tc::TILE - 1) / tc::TILE);
  const long long strips_want = std::max<long long>(1, (long long)ctx->num_sms * per_sm / G);
  const long long per_cta = (total + std::min(total, strips_want) - 1) / std::min(total, strips_want);
  const long long strips = (total + per_cta - 1) / per_cta;
  launch_chained(st, true, dim3((unsigned)(strips * G)), kWsThreads, sole_block_smem(ctx, strips * G, smem),
                 k_conv_fwd_ws<NG, ADD>, xmap, *d, w, bias, y, y32, acc_in, relu, S, G, per_cta, ctx->d_err);
  cudaError_t e = cudaGetLastError();
  *rc = e == cudaSuccess ? RX_OK : (set_error(ctx, "conv_bf16_fwd: %s", cudaGetErrorString(e)), RX_ERR_CUDA);
  return 1;
}

// Warp-specialised tcgen05 kernel: the widest output-channel group (128,
// 64, 32 or 16, dividing Cout) whose weights fit in shared memory beside a
// ring of at least 4 input rows (6 where they fit).  Returns 1 if it
// launched, 0 if the shape or the pointers do not suit it.
// Output-channel group for the warp-specialised kernel at this Cin / Cout,
// and the ring's row slots; 0 when the weights do not fit.
static int ws_group(int Cin, int Cout, int* S_out, int* smem_out) {
  const int limit = 232448 - 1024;
  const int SB = tc::slot_bytes(Cin);
  int NG = 0;
  // at most two groups: every group re-reads the input rows, and a UMMA's
  // cost is mostly its A (pixel) operand read, so narrow groups do not pay
  for (int ng = 128; ng >= 16; ng >>= 1)
    if (Cout % ng == 0 && Cout / ng <= 2 && tc::weights_bytes(Cin, ng) + 4 * SB + 128 <= limit) {
      NG = ng;
      break;
    }
  if (!NG) return 0;
  *S_out = std::min(6, (limit - 128 - tc::weights_bytes(Cin, NG)) / SB);
  *smem_out = tc::weights_bytes(Cin, NG) + *S_out * SB + 128;
  return NG;
}

static int launch_ws(Ctx* ctx, const rx_conv_desc* d, const bf16* x, const bf16* w, const float* bias, bf16* y,
                     float* y32, const float* acc_in, int relu, cudaStream_t st, int* rc) {
  if (((uintptr_t)x & 15) || ((uintptr_t)w & 15) || ((uintptr_t)y & 15) || ((uintptr_t)y32 & 15) ||
      ((uintptr_t)acc_in & 15))
    return 0;
  int S = 0, smem = 0;
  const int NG = ws_group(d->Cin, d->Cout, &S, &smem);
  switch (NG) {
    case 128:
      return acc_in ? launch_ws_ng<128, true>(ctx, d, x, w, bias, y, y32, acc_in, relu, S, smem, st, rc)
                    : launch_ws_ng<128, false>(ctx, d, x, w, bias, y, y32, nullptr, relu, S, smem, st, rc);
    case 64:
      return acc_in ? launch_ws_ng<64, true>(ctx, d, x, w, bias, y, y32, acc_in, relu, S, smem, st, rc)
                    : launch_ws_ng<64, false>(ctx, d, x, w, bias, y, y32, nullptr, relu, S, smem, st, rc);
    case 32:
      return acc_in ? launch_ws_ng<32, true>(ctx, d, x, w, bias, y, y32, acc_in, relu, S, smem, st, rc)
                    : launch_ws_ng<32, false>(ctx, d, x, w, bias, y, y32, nullptr, relu, S, smem, st, rc);
    case 16:
      return acc_in ? launch_ws_ng<16, true>(ctx, d, x, w, bias, y, y32, acc_in, relu, S, smem, st, rc)
                    : launch_ws_ng<16, false>(ctx, d, x, w, bias, y, y32, nullptr, relu, S, smem, st, rc);
    default: return 0;
  }
}

// Input channels [p * cp, (p + 1) * cp) of weights [Cout][9][Cin] as
// contiguous [Cout][9][cp], for p = 0, 1 (16-byte chunks).
__global__ void k_weight_halves(int Cout, int Cin, const uint4* __restrict__ w, uint4* __restrict__ out) {
  chain_wait(w, out);
  chain_go();
  const int cp8 = Cin / 16, c8 = Cin / 8;  // chunks per half row, per row
  const long long n = (long long)Cout * 9 * c8;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long row = i / c8;
    const int k = (int)(i - row * c8), half = k / cp8;
    out[(long long)half * Cout * 9 * cp8 + row * cp8 + (k - half * cp8)] = w[i];
  }
}

// A layer whose weights do not fit beside the row ring in one launch, run
// as two launches over the halves of its input channels: the first writes
// fp32 partial sums, the second adds them before the bias and activation
// (sum over channels [0, Cin/2), then [Cin/2, Cin), then + bias).  Returns
// 1 if it launched.
static int launch_ws_split(Ctx* ctx, const rx_conv_desc* d, const bf16* x, const bf16* w, const float* bias, bf16* y,
                           float* y32, int relu, cudaStream_t st, int* rc) {
  const int cp = d->Cin / 2;
  int S = 0, smem = 0;
  if (d->Cin % 32 || !ws_group(cp, d->Cout, &S, &smem)) return 0;
  if (((uintptr_t)x & 15) || ((uintptr_t)w & 15) || ((uintptr_t)y & 15) || ((uintptr_t)y32 & 15)) return 0;
  const long long P = (long long)d->N * d->H * d->W;
  const size_t wbytes = sizeof(bf16) * (size_t)d->Cout * 9 * d->Cin;
  void* halves = nullptr;
  float* part = nullptr;
  // stream-ordered on the caller's stream, which runs the launches
  if (cudaMallocAsync(&halves, wbytes, st) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  if (cudaMallocAsync((void**)&part, sizeof(float) * (size_t)P * d->Cout, st) != cudaSuccess) {
    cudaGetLastError();
    cudaFreeAsync(halves, st);
    return 0;
  }
  const long long chunks = (long long)d->Cout * 9 * (d->Cin / 8);
  launch_chained(st, true,
                 dim3((int)std::min<long long>((chunks + 255) / 256, (long long)ctx->num_sms * 8)), 256, 0,
                 k_weight_halves, d->Cout, d->Cin, reinterpret_cast<const uint4*>(w), static_cast<uint4*>(halves));
  const bf16* w0 = static_cast<const bf16*>(halves);
  const bf16* w1 = w0 + (size_t)d->Cout * 9 * cp;
  rx_conv_desc d0 = *d, d1 = *d;
  d0.Cin = d1.Cin = cp;
  d1.x_coff = d->x_coff + cp;
  d0.y_cstride = d->Cout;  // the partial sums: [pixel][Cout]
  d0.y_coff = 0;
  const int first = launch_ws(ctx, &d0, x, w0, nullptr, nullptr, part, nullptr, 0, st, rc);
  int second = 0;
  if (first && *rc == RX_OK) second = launch_ws(ctx, &d1, x, w1, bias, y, y32, part, relu, st, rc);
  cudaFreeAsync(part, st);
  cudaFreeAsync(halves, st);
  if (!first) return 0;  // the kernel is not available: the caller falls back
  if (*rc == RX_OK && !second) {
    // same kernel and shape as the first launch, so this does not happen
    set_error(ctx, "conv_bf16_fwd: second half of a split layer did not launch");
    *rc = RX_ERR_CUDA;
  }
  return 1;
}

template <int BN, int KS>
static int launch_res_as(Ctx* ctx, const rx_conv_desc* d, const bf16* x, const bf16* w, const float* bias, bf16* y,
                         float* y32, int relu, cudaStream_t st, int* rc) {
  using S = ResShape<BN, KS>;
  // the tile shape that covers the image with the fewest tiles; wider ones
  // first (longer rows, less halo)
  int cl = 7;
  long long best = LLONG_MAX, tx = 0, ty = 0;
  for (int c = 7; c >= 3; --c) {
    const long long nx = (d->W + (1 << c) - 1) >> c, ny = (d->H + (128 >> c) - 1) / (128 >> c);
    if (nx * ny < best) best = nx * ny, cl = c, tx = nx, ty = ny;
  }
  const int limit = 232448;  // opt-in shared memory per block
  if (best * d->N > 0x3fffffffLL || S::smem(cl) > (size_t)limit) return 0;
  auto kern = bias ? k_conv_fwd_res<BN, KS, true> : k_conv_fwd_res<BN, KS, false>;
  const int smem = sole_block_smem(ctx, 0, (int)S::smem(cl));
  // the limit, not this launch's size: the attribute is the kernel's, and
  // another thread's smaller launch would take it from under this one
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, limit);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  const int ny = (d->Cout + BN - 1) / BN;
  const int nx = (int)std::max<long long>(1, std::min<long long>(best * d->N, ctx->num_sms / ny));
  launch_chained(st, true, dim3(nx, ny), 256, smem, kern, *d, x, w, bias, y, y32, relu, cl, (int)tx, (int)ty,
                 S::halo(cl));
  e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error(ctx, "conv_bf16_fwd: %s", cudaGetErrorString(e));
    *rc = RX_ERR_CUDA;
  }
  return 1;
}

// k_conv_fwd_res for 16, 32 or 64 input and more than 32 output channels, in
// blocks of 96 or 64 output channels, whichever computes fewer.  0: not for it.
static int launch_res(Ctx* ctx, const rx_conv_desc* d, const bf16* x, const bf16* w, const float* bias, bf16* y,
                      float* y32, int relu, cudaStream_t st, int* rc) {
  if (d->Cout <= 32 || d->Cout > 64 * 65535) return 0;
  const bool wide = (d->Cout + 95) / 96 * 96 <= (d->Cout + 63) / 64 * 64;
  switch (d->Cin) {
    case 16:
      return wide ? launch_res_as<96, 1>(ctx, d, x, w, bias, y, y32, relu, st, rc)
                  : launch_res_as<64, 1>(ctx, d, x, w, bias, y, y32, relu, st, rc);
    case 32:
      return wide ? launch_res_as<96, 2>(ctx, d, x, w, bias, y, y32, relu, st, rc)
                  : launch_res_as<64, 2>(ctx, d, x, w, bias, y, y32, relu, st, rc);
    case 64:
      return wide ? launch_res_as<96, 4>(ctx, d, x, w, bias, y, y32, relu, st, rc)
                  : launch_res_as<64, 4>(ctx, d, x, w, bias, y, y32, relu, st, rc);
    default: return 0;
  }
}

int conv_fwd(Ctx* ctx, const rx_conv_desc* d, const void* x, const void* w, const float* bias, void* y, float* y32,
             int relu, cudaStream_t st) {
  if (!conv_ok(d) || !x || !w || !y)
    return set_error(ctx, "conv_bf16_fwd: bad descriptor (channels multiples of 16, strides of 8)"), RX_ERR_ARG;
  // every kernel copies x and w in 16-byte pieces, the mma.sync ones store
  // pairs of channels
  if (unaligned(x, 16) || unaligned(w, 16) || unaligned(y, 4) || unaligned(bias, 4) || unaligned(y32, 4))
    return set_error(ctx, "conv_bf16_fwd: x and w must be 16-byte aligned, y, y32 and bias 4"), RX_ERR_ARG;
  if (ctx->conv_impl == 0) {
    int rc = RX_OK;
    if (launch_ws(ctx, d, static_cast<const bf16*>(x), static_cast<const bf16*>(w), bias, static_cast<bf16*>(y), y32,
                  nullptr, relu, st, &rc) ||
        launch_ws_split(ctx, d, static_cast<const bf16*>(x), static_cast<const bf16*>(w), bias,
                        static_cast<bf16*>(y), y32, relu, st, &rc))
      return rc;
  } else if (ctx->conv_impl == 2 && d->H <= 65535 && d->N <= 65535 && !unaligned(y, 16)) {
    const bf16* xb = static_cast<const bf16*>(x);
    const bf16* wb = static_cast<const bf16*>(w);
    bf16* yb = static_cast<bf16*>(y);
    switch (d->Cout) {
      case 16: return launch_tc<16>(ctx, d, xb, wb, bias, yb, y32, relu, st);
      case 32: return launch_tc<32>(ctx, d, xb, wb, bias, yb, y32, relu, st);
      case 64: return launch_tc<64>(ctx, d, xb, wb, bias, yb, y32, relu, st);
      case 128: return launch_tc<128>(ctx, d, xb, wb, bias, yb, y32, relu, st);
      default: break;
    }
  }
  {
    int rc = RX_OK;
    if (launch_res(ctx, d, static_cast<const bf16*>(x), static_cast<const bf16*>(w), bias, static_cast<bf16*>(y), y32,
                   relu, st, &rc))
      return rc;
  }
  long long P = (long long)d->N * d->H * d->W;
  dim3 grid((unsigned)((P + 63) / 64), 1);
  const bf16* xb = static_cast<const bf16*>(x);
  const bf16* wb = static_cast<const bf16*>(w);
  bf16* yb = static_cast<bf16*>(y);
  bool bk32 = d->Cin % 32 == 0;
  if (d->Cout >= 128) {
    grid.y = (unsigned)((d->Cout + 127) / 128);
    if (bk32) k_conv_fwd<128, 32><<<grid, 128, 0, st>>>(*d, xb, wb, bias, yb, y32, relu);
    else k_conv_fwd<128, 16><<<grid, 128, 0, st>>>(*d, xb, wb, bias, yb, y32, relu);
  } else if (d->Cout > 32) {
    grid.y = (unsigned)((d->Cout + 63) / 64);
    if (bk32) k_conv_fwd<64, 32><<<grid, 128, 0, st>>>(*d, xb, wb, bias, yb, y32, relu);
    else k_conv_fwd<64, 16><<<grid, 128, 0, st>>>(*d, xb, wb, bias, yb, y32, relu);
  } else {
    grid.y = (unsigned)((d->Cout + 31) / 32);
    if (bk32) k_conv_fwd<32, 32><<<grid, 128, 0, st>>>(*d, xb, wb, bias, yb, y32, relu);
    else k_conv_fwd<32, 16><<<grid, 128, 0, st>>>(*d, xb, wb, bias, yb, y32, relu);
  }
  CUDA_TRY(ctx, cudaGetLastError());
  return RX_OK;
}

int conv_bwd_data(Ctx* ctx, const rx_conv_desc* d, const void* dy, const void* w, void* w_rot, void* dx,
                  cudaStream_t st) {
  if (!conv_ok(d) || !dy || !w || !w_rot || !dx) return set_error(ctx, "conv_bf16_bwd_data: bad arguments"), RX_ERR_ARG;
  long long nw = (long long)d->Cout * 9 * d->Cin;
  if (unaligned(dy, 16) || unaligned(w_rot, 16) || unaligned(w, 2) || unaligned(dx, 4))
    return set_error(ctx, "conv_bf16_bwd_data: dy and w_rot must be 16-byte aligned, dx 4"), RX_ERR_ARG;
  launch_chained(st, true, dim3(ew_blocks(ctx, nw / 8)), 256, 0, k_rot_weights_v8, d->Cout, d->Cin,
                 static_cast<const bf16*>(w), static_cast<bf16*>(w_rot));
  CUDA_TRY(ctx, cudaGetLastError());
  // dx = conv(dy, w_rot): input channels Cout (read from the y view), output Cin (the x view)
  rx_conv_desc t = *d;
  t.Cin = d->Cout;
  t.Cout = d->Cin;
  t.x_cstride = d->y_cstride;
  t.x_coff = d->y_coff;
  t.y_cstride = d->x_cstride;
  t.y_coff = d->x_coff;
  return conv_fwd(ctx, &t, dy, w_rot, nullptr, dx, nullptr, 0, st);
}

// Pixels per partial sum of the weight gradient: enough of them to fill the
// GPU with every (tap, 64 x 64 channel block) of k_conv_wgrad.
static int wgrad_chain(Ctx* ctx, const rx_conv_desc* d) {
  const long long P = (long long)d->N * d->H * d->W;
  const int cb = ((d->Cout + 63) / 64) * ((d->Cin + 63) / 64);
  const long long want = (long long)ctx->num_sms * 4 / std::max(1, 9 * cb) + 1;
  return (int)std::max<long long>(256, ((P + want - 1) / want + 31) / 32 * 32);
}

// Weight gradient on k_conv_wgrad_ws.  Returns 1 if it launched, 0 if the
// shape does not suit it.
static int launch_wgrad_ws(Ctx* ctx, const rx_conv_desc* d, const bf16* dy, const bf16* x, float* dw, cudaStream_t st,
                           int* rc) {
  const int limit = 232448 - 1024;  // opt-in shared memory per block, less the static part
  static int attr_dev = -1;
  if (attr_dev != ctx->device) {
    for (auto kern : {k_conv_wgrad_ws<false>, k_conv_wgrad_ws<true>})
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, limit) != cudaSuccess) {
        cudaGetLastError();
        return 0;
      }
    attr_dev = ctx->device;
  }
  WgradArgs A{};
  A.N = d->N, A.H = d->H, A.W = d->W, A.Cin = d->Cin, A.Cout = d->Cout;
  // equal tiles of up to 128 pixels: every strip then sums about as many
  A.tiles = (d->W + 127) / 128;
  A.tw = ((d->W + A.tiles - 1) / A.tiles + 15) / 16 * 16;
  A.nc = 128;
  while (d->Cout % A.nc) A.nc >>= 1;  // 16 divides Cout
  A.ng = d->Cout / A.nc;
  // Pixels one accumulator sums before it meets the others in dw: the split
  // k_conv_wgrad makes.  The tensor core truncates as it accumulates, so a
  // sum's distance from the exact one grows with this length (1e-6 of it per
  // 1,300 pixels).  With k_conv_wgrad's split (7,944 pixels at 16 x 128^2) the
  // two kernels agree to a few 1e-7, both 3-7e-6 from float64.  The length is
  // for that agreement alone: one block per SM (1,772 pixels) was nearer to
  // float64 (1.3e-6; at 96 -> 32 channels it left k_conv_wgrad's result by
  // 1.7e-5) and faster (296 against 371 us, both with M = 128).
  const int chain = wgrad_chain(ctx, d);
  const long long total = (long long)d->N * d->H * A.tiles;
  const long long per_cta = std::max<long long>(1, (long long)chain * A.tiles / d->W);
  const long long strips = (total + per_cta - 1) / per_cta;
  // Blocks beyond the strips come from splitting the input channels and the
  // taps; both read rows again.  The cheapest split by the cycles of a row
  // (MMAs: about 40 each up to N = 32, N / 2 above, and 28 and 44 for N = 32
  // and 64 with M = 64, half the channels to read; TMA: 16 B per cycle), the
  // rows of a block and the rounds of blocks.  M = 64 for up to 64 channels
  // took the eleven layers of a 16x128x128 batch from 346 to 299 us.
  const int mg_min = (d->Cin + 127) / 128;
  double best = 0.0;
  for (int mg = mg_min; mg <= 4 * mg_min && (mg == mg_min || d->Cin / mg >= 16); ++mg)
    for (int tg = 1; tg <= 9; ++tg) {
      const int taps = (9 + tg - 1) / tg, cm = (d->Cin / 8 + mg - 1) / mg * 8;
      if (taps * A.nc > 512 || (tg - 1) * taps >= 9) continue;
      const int mma = A.nc > 64 ? 64 : cm <= 64 ? (A.nc <= 32 ? 28 : 44) : (A.nc <= 32 ? 40 : 48);
      const double row = std::max<double>(taps * (A.tw / 16) * mma, (double)((A.tw + 2) * cm + A.tw * A.nc) * 2 / 16);
      const long long rounds = (strips * mg * A.ng * tg + ctx->num_sms - 1) / ctx->num_sms;
      const double cost = (double)rounds * ((double)per_cta * row + 8000.0);  // 8,000: a block's start and end
      if (best == 0.0 || cost < best) best = cost, A.mg = mg, A.cm = cm, A.tg = tg, A.taps = taps;
    }
  A.tcols = 32;
  while (A.tcols < A.taps * A.nc) A.tcols <<= 1;
  const int plane = (A.tw + 2) * 16;
  A.xslot = (A.cm / 8 * plane + 127) / 128 * 128;
  if (d->W % 16) {
    A.xcut = A.xslot;
    A.xslot += A.cm / 8 * 16 * 16;
  }
  A.yslot = (A.nc / 8 * A.tw * 16 + 127) / 128 * 128;
  // M = 128 reads sixteen planes from any x slot: room behind the last one
  // (the dy slots count; rows past the group's channels are not stored)
  const int tail = std::max(16 * plane, A.xcut + 16 * 16 * 16);
  A.Sy = 3, A.Sx = kWgSlots;
  auto bytes = [&] { return std::max(A.Sx * A.xslot + A.Sy * A.yslot, (A.Sx - 1) * A.xslot + tail) + 128; };
  while (bytes() > limit && A.Sx > 4) --A.Sx;
  while (bytes() > limit && A.Sy > 2) --A.Sy;
  if (bytes() > limit) return 0;
  CUtensorMap xmap, cutmap, ymap;
  if (!row_map(d->N, d->H, d->W, d->W, d->Cin, d->x_cstride, x + d->x_coff, A.tw + 2, A.cm / 8, &xmap) ||
      !row_map(d->N, d->H, d->W, std::max(d->W - 1, 1), d->Cin, d->x_cstride, x + d->x_coff, 16, A.cm / 8, &cutmap) ||
      !row_map(d->N, d->H, d->W, d->W, d->Cout, d->y_cstride, dy + d->y_coff, A.tw, A.nc / 8, &ymap))
    return 0;
  const int G = A.mg * A.ng * A.tg;
  launch_chained(st, true, dim3((unsigned)(strips * G)), kWgThreads, sole_block_smem(ctx, strips * G, bytes()),
                 A.xcut ? k_conv_wgrad_ws<true> : k_conv_wgrad_ws<false>, xmap, cutmap, ymap, A, dw, per_cta, ctx->d_err);
  cudaError_t e = cudaGetLastError();
  *rc = e == cudaSuccess ? RX_OK : (set_error(ctx, "conv_bf16_bwd_weight: %s", cudaGetErrorString(e)), RX_ERR_CUDA);
  return 1;
}

int conv_bwd_weight(Ctx* ctx, const rx_conv_desc* d, const void* dy, const void* x, float* dw, float* db,
                    cudaStream_t st) {
  if (!conv_ok(d) || !dy || !x || !dw) return set_error(ctx, "conv_bf16_bwd_weight: bad arguments"), RX_ERR_ARG;
  if (unaligned(dy, 16) || unaligned(x, 16) || unaligned(dw, 4) || unaligned(db, 4))
    return set_error(ctx, "conv_bf16_bwd_weight: dy and x must be 16-byte aligned, dw and dbias 4"), RX_ERR_ARG;
  long long P = (long long)d->N * d->H * d->W;
  int rc = RX_OK;
  const bool ws = ctx->conv_impl == 0 && launch_wgrad_ws(ctx, d, static_cast<const bf16*>(dy),
                                                         static_cast<const bf16*>(x), dw, st, &rc);
  if (rc) return rc;
  if (!ws) {
    const int ppb = wgrad_chain(ctx, d), cb = ((d->Cout + 63) / 64) * ((d->Cin + 63) / 64);
    dim3 grid((unsigned)((P + ppb - 1) / ppb), (unsigned)cb, 9);
    k_conv_wgrad<<<grid, 128, 0, st>>>(*d, static_cast<const bf16*>(dy), static_cast<const bf16*>(x), dw, ppb);
    CUDA_TRY(ctx, cudaGetLastError());
  }
  if (db) {
    // at least eight loads per thread
    const int lanes = kBiasThreads / std::min(d->Cout / 8, kBiasWidth);
    const long long clusters = (P + 8LL * lanes * kBiasCluster - 1) / (8LL * lanes * kBiasCluster);
    const int blocks = kBiasCluster * (int)std::min<long long>(clusters, kBiasBlocks / kBiasCluster);
    const int bppb = (int)((P + blocks - 1) / blocks);
    launch_chained(st, true, dim3((unsigned)blocks), kBiasThreads, 0, k_bias_grad, *d, static_cast<const bf16*>(dy),
                   db, bppb);
    CUDA_TRY(ctx, cudaGetLastError());
  }
  return RX_OK;
}

int dn_op(Ctx* ctx, const rx_dn_op* o, cudaStream_t st) {
  if (!o) return set_error(ctx, "dn_op: NULL"), RX_ERR_ARG;
  const bf16* a = static_cast<const bf16*>(o->a);
  bf16* b = static_cast<bf16*>(o->b);
  long long P = (long long)o->N * o->H * o->W;
  // 16-byte chunks when channel count, strides, offsets and bases allow
  const bool v8 = o->C % 8 == 0 && o->a_stride % 8 == 0 && o->a_off % 8 == 0 && o->b_stride % 8 == 0 &&
                  o->b_off % 8 == 0 && ((uintptr_t)a & 15) == 0 && ((uintptr_t)b & 15) == 0;
  switch (o->kind) {
    case RX_DN_COPY:
      k_copy_ch<<<ew_blocks(ctx, P * o->C), 256, 0, st>>>(P, o->C, a, o->a_stride, o->a_off, b, o->b_stride, o->b_off,
                                                         o->flag);
      break;
    case RX_DN_RELU_MASK:
      if (v8)
        launch_chained(st, true,
                       dim3(ew_blocks(ctx, P * (o->C / 8))), 256, 0, k_relu_mask_v8, P, o->C, a, o->a_stride,
                       o->a_off, b, o->b_stride, o->b_off);
      else
        k_relu_mask<<<ew_blocks(ctx, P * o->C), 256, 0, st>>>(P, o->C, a, o->a_stride, o->a_off, b, o->b_stride,
                                                             o->b_off);
      break;
    case RX_DN_POOL:
      if (o->H % 2 || o->W % 2) return set_error(ctx, "dn_op: pool needs even H and W"), RX_ERR_ARG;
      if (v8)
        launch_chained(st, true,
                       dim3(ew_blocks(ctx, P / 4 * (o->C / 8))), 256, 0, k_pool2_v8, o->N, o->H, o->W, o->C, a,
                       o->a_stride, o->a_off, b, o->b_stride, o->b_off);
      else
        k_pool2<<<ew_blocks(ctx, P / 4 * o->C), 256, 0, st>>>(o->N, o->H, o->W, o->C, a, o->a_stride, o->a_off, b,
                                                             o->b_stride, o->b_off);
      break;
    case RX_DN_POOL_BWD:
      if (o->H % 2 || o->W % 2) return set_error(ctx, "dn_op: pool needs even H and W"), RX_ERR_ARG;
      if (v8)
        launch_chained(st, true,
                       dim3(ew_blocks(ctx, P / 4 * (o->C / 8))), 256, 0, k_pool2_bwd_v8, o->N, o->H, o->W, o->C, a,
                       o->a_stride, o->a_off, b, o->b_stride, o->b_off, o->flag);
      else
        k_pool2_bwd<<<ew_blocks(ctx, P * o->C), 256, 0, st>>>(o->N, o->H, o->W, o->C, a, o->a_stride, o->a_off, b,
                                                             o->b_stride, o->b_off, o->flag);
      break;
    case RX_DN_UP:
      if (v8)
        launch_chained(st, true,
                       dim3(ew_blocks(ctx, P * (o->C / 8))), 256, 0, k_up2_v8, o->N, o->H, o->W, o->C, a, o->a_stride,
                       o->a_off, b, o->b_stride, o->b_off);
      else
        k_up2<<<ew_blocks(ctx, 4 * P * o->C), 256, 0, st>>>(o->N, o->H, o->W, o->C, a, o->a_stride, o->a_off, b,
                                                           o->b_stride, o->b_off);
      break;
    case RX_DN_UP_BWD:
      if (v8)
        launch_chained(st, true,
                       dim3(ew_blocks(ctx, P * (o->C / 8))), 256, 0, k_up2_bwd_v8, o->N, o->H, o->W, o->C, a,
                       o->a_stride, o->a_off, b, o->b_stride, o->b_off);
      else
        k_up2_bwd<<<ew_blocks(ctx, P * o->C), 256, 0, st>>>(o->N, o->H, o->W, o->C, a, o->a_stride, o->a_off, b,
                                                           o->b_stride, o->b_off);
      break;
    default:
      return set_error(ctx, "dn_op: unknown kind %d", o->kind), RX_ERR_ARG;
  }
  CUDA_TRY(ctx, cudaGetLastError());
  return RX_OK;
}

int dn_features(Ctx* ctx, long long P, const float* rad, const float* alb, const float* nrm, const float* dep,
                void* out, float* base, cudaStream_t st) {
  if (P <= 0 || !rad || !alb || !nrm || !dep || !out) return set_error(ctx, "dn_features: bad arguments"), RX_ERR_ARG;
  const uintptr_t all = (uintptr_t)rad | (uintptr_t)alb | (uintptr_t)nrm | (uintptr_t)dep | (uintptr_t)out |
                        (uintptr_t)base;
  if (P % 4 == 0 && all % 16 == 0) {
    auto f4 = [](const float* p) { return reinterpret_cast<const float4*>(p); };
    launch_chained(st, true, dim3(ew_blocks(ctx, P / 4)), 256, 0, k_features_v4, P / 4, f4(rad), f4(alb), f4(nrm),
                   f4(dep), static_cast<uint4*>(out), reinterpret_cast<float4*>(base));
  } else {
    k_features<<<ew_blocks(ctx, P), 256, 0, st>>>(P, rad, alb, nrm, dep, static_cast<bf16*>(out), base);
  }
  CUDA_TRY(ctx, cudaGetLastError());
  return RX_OK;
}

int dn_l1_loss(Ctx* ctx, long long P, const float* y32, int y_stride, const float* base, const float* target,
               float scale, void* grad, int grad_stride, float* loss, cudaStream_t st) {
  if (P <= 0 || !y32 || !target || !grad || !loss || y_stride < 3 || grad_stride < 3)
    return set_error(ctx, "dn_l1_loss: bad arguments"), RX_ERR_ARG;
  auto kern = grad_stride % 8 == 0 && (uintptr_t)grad % 16 == 0 ? k_l1_loss<true> : k_l1_loss<false>;
  const int blocks = (int)std::min<long long>((P + kLossThreads - 1) / kLossThreads, ctx->num_sms);
  launch_chained(st, true, dim3(blocks), kLossThreads, 0, kern, P, y32, y_stride, base, target, scale,
                 static_cast<bf16*>(grad), grad_stride, loss);
  CUDA_TRY(ctx, cudaGetLastError());
  return RX_OK;
}

int dn_output(Ctx* ctx, long long P, const float* y32, int y_stride, const float* base, float* out,
              cudaStream_t st) {
  if (P <= 0 || !y32 || !out || y_stride < 3) return set_error(ctx, "dn_output: bad arguments"), RX_ERR_ARG;
  launch_chained(st, true, dim3(ew_blocks(ctx, P)), 256, 0, k_output, P, y32, y_stride, base, out);
  CUDA_TRY(ctx, cudaGetLastError());
  return RX_OK;
}

int dn_adam(Ctx* ctx, long long n, float* p, float* g, float* m, float* v, void* p16, float lr, float b1, float b2,
            float eps, int step, cudaStream_t st) {
  if (n <= 0 || !p || !g || !m || !v || step < 1) return set_error(ctx, "dn_adam: bad arguments"), RX_ERR_ARG;
  float c1 = 1.0f - powf(b1, (float)step), c2 = 1.0f - powf(b2, (float)step);
  k_adam<<<ew_blocks(ctx, n), 256, 0, st>>>(n, p, g, m, v, static_cast<bf16*>(p16), lr, b1, b2, eps, c1, c2);
  CUDA_TRY(ctx, cudaGetLastError());
  return RX_OK;
}

}  // namespace rx
