// conv.cu -- BF16 tensor-core (tcgen05, accumulators in tensor memory) 3x3
// convolutions of the learned coarse-grid correction: forward with bias and
// GELU, forward linear, backward to the input through the previous layer's
// GELU, and the weight gradient.  Images are NHWC bf16 tensors
// [batch][h][w][channels], periodic in y and x (the coarse grids they come
// from are periodic).  Weights are [c_out][9][c_in] with tap t = (dy+1)*3 +
// (dx+1): out(y, x) = sum_t W[t] x(y+dy, x+dx) (cross-correlation).
//
// Implicit GEMM.  Forward / backward-data: M = 128 output pixels x N = c_out
// channels, K = 9 taps x c_in channels.  A persistent CTA per SM walks tiles of
// 8 (small images: 4 or 2) image rows x 128 pixels; a tile's input is staged once, each tap's operand
// is a shifted descriptor into it, and producer, MMA and epilogue warps pipeline
// the tiles.  Weight gradient: D[(row, c_in)][(row, c_out)] = sum over pixels of
// x(p + tap) dz(p)^T, K = pixels; both operands are channel-major (MN-major) as
// NHWC has them, staged once per tile of 8 rows x 64 pixels, and one MMA covers
// three vertical taps of two output rows; CTAs sum with fp32 atomics.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdlib>

#include "learned/conv.h"
#include "learned/umma.cuh"

namespace pmhd {
namespace learned {

namespace {

constexpr uint32_t kWaitPolls = 1u << 22;

// GELU in the tanh form, 0.5 z (1 + tanh(y)) with y = sqrt(2/pi) (z + 0.044715
// z^3), written as z s with s = 1 / (1 + exp(-2 y)): one hardware exp2 and
// one reciprocal, and the left tail keeps its relative accuracy (s is never
// formed as a difference).  Its derivative: s + z s (1 - s) dy2/dz.
constexpr float kGeluA = 1.5957691216057308f;     // 2 sqrt(2 / pi)
constexpr float kGeluB = 0.071354816272737f;      // 2 sqrt(2 / pi) 0.044715
constexpr float kLog2e = 1.4426950408889634f;
__device__ __forceinline__ float ex2_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float gelu_sigmoid(float z) {
  const float y2 = z * (kGeluA + kGeluB * z * z);
  return rcp_approx(1.0f + ex2_approx(-y2 * kLog2e));
}
__device__ __forceinline__ float gelu(float z) { return z * gelu_sigmoid(z); }
__device__ __forceinline__ float gelu_grad(float z) {
  const float s = gelu_sigmoid(z);
  return s + z * s * (1.0f - s) * (kGeluA + 3.0f * kGeluB * z * z);
}

// Two 16-byte vectors to / from consecutive addresses: one 32-byte access (a full
// L2 sector) when the buffers allow it (`wide`: 32-byte aligned), else two.
__device__ __forceinline__ void store32(void* p, const uint4& a, const uint4& b, bool wide) {
  if (wide) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(a.x), "r"(a.y), "r"(a.z),
                 "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
                 : "memory");
  } else {
    static_cast<uint4*>(p)[0] = a;
    static_cast<uint4*>(p)[1] = b;
  }
}
__device__ __forceinline__ void load32(const void* p, uint4& a, uint4& b, bool wide) {
  if (wide) {
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
                 : "l"(p));
  } else {
    a = static_cast<const uint4*>(p)[0];
    b = static_cast<const uint4*>(p)[1];
  }
}

__device__ __forceinline__ int wrap(int v, int n) { return v < 0 ? v + n : (v >= n ? v - n : v); }

// Epilogue of 16 channels (from c0) of one output pixel p from their fp32
// accumulators; `bias` is the CTA's 16-byte-aligned shared copy (unused by
// CONV_DGELU); wide: see store32.
template <int CO, int EPI>
__device__ __forceinline__ void epilogue16(const float (&acc)[16], int c0, long long p, const float* __restrict__ bias,
                                           const __nv_bfloat16* __restrict__ zprev, void* __restrict__ out0,
                                           void* __restrict__ out1, bool wide) {
  float bb[16];
  if (EPI != CONV_DGELU) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const float4 b = reinterpret_cast<const float4*>(bias + c0)[q];
      bb[4 * q] = b.x, bb[4 * q + 1] = b.y, bb[4 * q + 2] = b.z, bb[4 * q + 3] = b.w;
    }
  }
  auto vec = [](const uint32_t* w) { return make_uint4(w[0], w[1], w[2], w[3]); };
  if (EPI == CONV_GELU) {
    uint32_t zb[8], ab[8];
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const float z0 = acc[2 * q] + bb[2 * q];
      const float z1 = acc[2 * q + 1] + bb[2 * q + 1];
      const __nv_bfloat162 z2 = __floats2bfloat162_rn(z0, z1), a2 = __floats2bfloat162_rn(gelu(z0), gelu(z1));
      zb[q] = *reinterpret_cast<const uint32_t*>(&z2);
      ab[q] = *reinterpret_cast<const uint32_t*>(&a2);
    }
    store32(static_cast<__nv_bfloat16*>(out0) + p * CO + c0, vec(zb), vec(zb + 4), wide);
    store32(static_cast<__nv_bfloat16*>(out1) + p * CO + c0, vec(ab), vec(ab + 4), wide);
  } else if (EPI == CONV_LINEAR) {
    uint32_t v[16];
#pragma unroll
    for (int q = 0; q < 16; q++) v[q] = __float_as_uint(acc[q] + bb[q]);
    float* o = static_cast<float*>(out0) + p * CO + c0;
    store32(o, vec(v), vec(v + 4), wide);
    store32(o + 8, vec(v + 8), vec(v + 12), wide);
  } else {
    uint4 za, zc;
    load32(zprev + p * CO + c0, za, zc, wide);
    const uint32_t zw[8] = {za.x, za.y, za.z, za.w, zc.x, zc.y, zc.z, zc.w};
    uint32_t db[8];
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const float2 z = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&zw[q]));
      const __nv_bfloat162 d = __floats2bfloat162_rn(acc[2 * q] * gelu_grad(z.x), acc[2 * q + 1] * gelu_grad(z.y));
      db[q] = *reinterpret_cast<const uint32_t*>(&d);
    }
    store32(static_cast<__nv_bfloat16*>(out0) + p * CO + c0, vec(db), vec(db + 4), wide);
  }
}

// B operand: for each horizontal shift dx of the input (dx + 1 = 0, 1, 2) and
// 8-channel group, the 16-byte vectors of 3 CO weights: those that take the input
// row to output rows one above (shift dy = 1), level and one below it; the
// backward pass mirrors the taps.  Thread t of nt.
template <int CG, int CO, int EPI>
__device__ __forceinline__ void stage_weights(unsigned char* sB, const __nv_bfloat16* __restrict__ wt, int t,
                                              int nt) {
  constexpr int K = 9 * CG, NG = CG / 8;
  for (int c = t; c < CO * (K / 8); c += nt) {
    const int n = c / (K / 8), g = c - n * (K / 8), tap = g / NG;
    const int sgn = EPI == CONV_DGELU ? -1 : 1, dy = sgn * (tap / 3 - 1), dx = sgn * (tap % 3 - 1);
    const uint4 v = *reinterpret_cast<const uint4*>(wt + (size_t)n * K + g * 8);
    *reinterpret_cast<uint4*>(sB + (((dx + 1) * NG + g % NG) * 3 * CO + (1 - dy) * CO + n) * 16) = v;
  }
}

// 16-byte asynchronous copy; the form with `take` zero-fills when it is false.
__device__ __forceinline__ void cp16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp16_or_zero(uint32_t dst, const void* src, bool take) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(take ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

constexpr int kRowPix = 128;               // output pixels of a row segment (M)
constexpr int kRowPitch = kRowPix + 2;     // staged pixels per input row

// A row tile: image bb, output rows y0 .., pixels x0 ..,
// of which `rows` rows and `pix` pixels lie in the image.
struct RowTile {
  long long bb;
  int y0, x0, rows, pix;
};
template <int ROWS, int PIX>
__device__ __forceinline__ RowTile row_tile(long long tile, int h, int w) {
  const int segs = (w + PIX - 1) / PIX, rblocks = (h + ROWS - 1) / ROWS;
  RowTile t;
  t.x0 = (int)(tile % segs) * PIX;
  t.y0 = (int)((tile / segs) % rblocks) * ROWS;
  t.bb = tile / ((long long)segs * rblocks);
  t.rows = h - t.y0 < ROWS ? h - t.y0 : ROWS;
  t.pix = w - t.x0 < PIX ? w - t.x0 : PIX;
  return t;
}

// Staged row r of a row tile (input row y0 - 1 + r, pixels x0 - 1 .. x0 + pix,
// periodic) by one warp: 16-byte chunks of staged pixel s at dst + s * 2 CG,
// swizzled (umma::swz).  Consecutive lanes copy consecutive 16-byte words.  ZERO:
// pixels up to PIX + 1 and rows outside the tile are zero-filled; else they are
// left alone (they feed accumulator rows that are never read).
template <int CG, int PIX, bool ZERO>
__device__ __forceinline__ void stage_halo_row(uint32_t dst, const __nv_bfloat16* __restrict__ x, const RowTile& rt,
                                               int r, int h, int w, int lane) {
  constexpr int NG = CG / 8, PER = 32 / NG;  // chunks a pixel, pixels a pass of the warp (512 bytes)
  const bool row_in = r <= rt.rows + 1;
  if (!ZERO && !row_in) return;
  const int yy = row_in ? wrap(rt.y0 - 1 + r, h) : 0;
  const __nv_bfloat16* row = x + (rt.bb * h + yy) * (long long)w * CG + lane % NG * 8;
  const int last = row_in ? rt.pix + 1 : -1;  // last staged pixel that is used
  dst = umma::swz<2 * CG>(dst + lane * 16);   // the swizzle does not see steps of 512 bytes
#pragma unroll
  for (int i = 0; i < (PIX + 2 + PER - 1) / PER; i++) {
    const int s = lane / NG + i * PER;
    const int col = wrap(rt.x0 - 1 + s, w);
    if (ZERO) {
      if (s < PIX + 2) cp16_or_zero(dst + i * 512, row + (s <= last ? (long long)col * CG : 0), s <= last);
    } else {
      if (s <= last) cp16(dst + i * 512, row + (long long)col * CG);
    }
  }
}

// The row tile's MMAs, issued by one thread.  Staged input row r, shifted by dx
// pixels (a shift of the descriptor's start address), feeds output rows r - 2,
// r - 1 and r of the tile, whose accumulators are neighbours in tensor memory
// (row o at d0 + o * CO): one MMA of N = 3 CO against the three vertical taps'
// weights, less at the tile's first and last rows.  The first MMA on an output
// row is its own (it does not accumulate).  A small MMA is bound by reading its
// 4 KB of A from shared memory whatever N is (70 cycles at N = 32 and at 64,
// measured without swizzle), so 68 MMAs of N <= 3 CO a tile of 8 rows at 32
// channels take half the time of 144 of N = CO (8 x 512^2 layer: 142 -> 131 us a
// call).
template <int CG, int CO>
__device__ __forceinline__ void issue_row_mmas(uint32_t a0, uint32_t b0, uint32_t d0, int rows) {
  constexpr uint32_t kLboB = 3u * (uint32_t)CO * 16u;
  const uint64_t a = umma::desc(a0, 16, 16 * CG, CG == 32 ? umma::kSwizzle64 : umma::kSwizzle32);
  const uint64_t b = umma::desc(b0, kLboB, 128, umma::kNoSwizzle);
  const uint32_t a_hi = umma::desc_hi(a), b_hi = umma::desc_hi(b), b_lo = umma::desc_lo(b);
  uint32_t a_lo = umma::desc_lo(a);
  // idesc of n blocks of CO columns.
  auto idesc = [](int n) { return umma::idesc_bf16(128, 0, false, false) + ((uint32_t)(n * CO >> 3) << 17); };
#pragma unroll 1
  for (int r = 0; r < rows + 2; r++, a_lo += kRowPitch * CG / 8) {
    const int lo = r < 2 ? 0 : r - 2, hi = r < rows ? r : rows - 1;  // output rows lo .. hi
    const uint32_t skip = (uint32_t)((lo - (r - 2)) * CO);            // weight blocks before row lo's
    const uint32_t d = d0 + (uint32_t)(lo * CO);
    const bool fresh = r < rows;  // row r has no accumulator yet
#pragma unroll
    for (int dx = 0; dx < 3; dx++)
#pragma unroll
      for (int kc = 0; kc < CG / 16; kc++) {
        const uint32_t al = a_lo + dx * (CG / 8) + kc * 2;
        const uint32_t bl = b_lo + (dx * (CG / 8) + kc * 2) * (kLboB / 16) + skip;
        if (dx + kc == 0 && fresh) {
          if (r > 0) umma::mma_bf16(d, al, a_hi, bl, b_hi, idesc(hi - lo), 1u);
          umma::mma_bf16(d0 + (uint32_t)(r * CO), al, a_hi, bl + (uint32_t)((hi - lo) * CO), b_hi, idesc(1), 0u);
        } else {
          umma::mma_bf16(d, al, a_hi, bl, b_hi, idesc(hi - lo + 1), 1u);
        }
      }
  }
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Bounded wait agreed by the whole warp.
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity) {
  return __all_sync(0xffffffffu, mbar_wait_bounded(bar, parity, kWaitPolls));
}

// Forward / backward-data kernel, any image size: persistent CTAs, one per SM,
// loop over row tiles.  A tile is ROWS (8, 4 or 2) image rows x 128 pixels; its
// (ROWS + 2) x 130 input pixels (periodic) are staged once as NHWC has them (umma.cuh: a swizzled K-major
// M = 128 operand whose rows are pixels), so the nine taps need no copies
// (issue_row_mmas).  Five producer warps stage tile k + 1
// while one thread issues tile k's MMAs and sixteen warps drain tile k - 1 from
// tensor memory (128 lanes x CO columns per row, the rows side by side); two
// staging and two accumulator buffers, hand-offs by mbarriers:
//   full[b]   producers -> MMA      staging buffer b holds its tile
//   empty[b]  MMA commit -> producers  the MMAs that read buffer b are done
//   tfull[b]  MMA commit -> epilogue   accumulator buffer b is complete
//   tempty[b] epilogue -> MMA          accumulator buffer b has been read
// Every wait is bounded; on expiry the CTA records the error and leaves.
// One 32 -> 32 GELU layer over 8 x 512^2 moves 403 MB (62 us at the 6.45 TB/s copy
// rate): 100 us a call, about 75 of them the kernel's, against 174 before the
// swizzled staging (full L2 sectors: 131 -> 114), the N = 3 CO MMAs, constant
// descriptor steps and sixteen epilogue warps with 32-byte stores.  What is left
// over the copy: the 16 special-function operations a clock of GELU (2.2 us of a
// tile's 4.4), the first tile's load and the last one's drain.
constexpr int kPipeEpiWarps = 16, kPipeProdWarps = 5;
constexpr int kPipeThreads = 32 * (kPipeEpiWarps + kPipeProdWarps + 1);

template <int CG, int CO, int ROWS>
struct PipeSmem {
  static constexpr uint32_t kStage = ((ROWS + 2) * kRowPitch * 2u * CG + 1023u) & ~1023u;  // one staging buffer
  static constexpr uint32_t kOffB = 2u * kStage;
  static constexpr uint32_t kBytesB = (uint32_t)CO * 9u * CG * 2u;
  static constexpr uint32_t kOffBar = (kOffB + kBytesB + 7u) & ~7u;
  static constexpr uint32_t kBytes = kOffBar + 9u * 8u + 8u;
  static constexpr uint32_t kColsBuf = umma::tmem_cols(ROWS * CO);
  static constexpr uint32_t kTmemCols = 2u * kColsBuf;
  // Shared memory requested per CTA: at least enough that no more CTAs fit
  // on an SM (228 KB) than its 512 tensor-memory columns hold.
  static constexpr uint32_t kMaxCtas = 512u / kTmemCols;
  static constexpr uint32_t kMinBytes = (228u * 1024u) / (kMaxCtas + 1u) + 1024u;
  static constexpr uint32_t kLaunchBytes = kBytes > kMinBytes ? kBytes : kMinBytes;
};

// EPI: CONV_GELU   out0 = z (bf16), out1 = gelu(z) (bf16), z = acc + bias
//      CONV_LINEAR out0 = acc + bias (fp32)
//      CONV_DGELU  out0 = acc * gelu'(zprev) (bf16); taps mirrored (the
//                  transposed convolution of the backward pass)
template <int CG, int CO, int EPI, int ROWS>
__global__ void __launch_bounds__(kPipeThreads, 1) conv3x3_pipe_kernel(const __nv_bfloat16* __restrict__ x,
                                                                       const __nv_bfloat16* __restrict__ wt,
                                                                       const float* __restrict__ bias,
                                                                       const __nv_bfloat16* __restrict__ zprev,
                                                                       long long ntiles, int h, int w,
                                                                       void* __restrict__ out0,
                                                                       void* __restrict__ out1, int wide,
                                                                       int* __restrict__ err) {
  using S = PipeSmem<CG, CO, ROWS>;
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char* sB = smem + S::kOffB;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + S::kOffBar);
  uint64_t* empty = full + 2;
  uint64_t* tfull = full + 4;
  uint64_t* tempty = full + 6;
  uint64_t* wfull = full + 8;  // epilogue warps -> MMA: weights and bias are staged
  uint32_t* tslot = reinterpret_cast<uint32_t*>(full + 9);
  __shared__ __align__(16) float sbias[CO];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (warp == 0) {
    umma::tmem_alloc(tslot, S::kTmemCols);
    umma::tmem_relinquish();
  }
  if (tid == 0) {
    for (int b = 0; b < 2; b++) {
      mbar_init(full + b, kPipeProdWarps * 32);
      mbar_init(empty + b, 1);
      mbar_init(tfull + b, 1);
      mbar_init(tempty + b, kPipeEpiWarps);
    }
    mbar_init(wfull, kPipeEpiWarps * 32);
    fence_barrier_init();
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = *tslot;
  bool ok = true;

  if (warp >= kPipeEpiWarps && warp < kPipeEpiWarps + kPipeProdWarps) {
    // Producers: stage tile k into buffer k % 2 once the MMAs of tile k - 2
    // (the buffer's previous tile) are done.
    const int pw = warp - kPipeEpiWarps;
    int k = 0;
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x, k++) {
      const int b = k & 1;
      if (k >= 2 && !warp_wait(empty + b, (uint32_t)((k >> 1) - 1) & 1u)) {
        ok = false;
        break;
      }
      const RowTile rt = row_tile<ROWS, kRowPix>(tile, h, w);
      const uint32_t dst = smem_u32(smem + b * S::kStage);
      for (int r = pw; r < ROWS + 2; r += kPipeProdWarps)
        stage_halo_row<CG, kRowPix, false>(dst + r * kRowPitch * 2 * CG, x, rt, r, h, w, lane);
      cp_wait_all();
      fence_proxy_async_smem();
      mbar_arrive(full + b);
    }
  } else if (warp == kPipeEpiWarps + kPipeProdWarps) {
    // MMA issuer: tile k from buffer k % 2 into accumulator buffer k % 2
    // once the epilogue has read that buffer's previous tile (k - 2).
    int k = 0;
    ok = warp_wait(wfull, 0);
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x, k++) {
      const int b = k & 1;
      if (!ok || !warp_wait(full + b, (uint32_t)(k >> 1) & 1u) ||
          (k >= 2 && !warp_wait(tempty + b, (uint32_t)((k >> 1) - 1) & 1u))) {
        ok = false;
        break;
      }
      umma::fence_after_sync();
      if (lane == 0) {
        issue_row_mmas<CG, CO>(smem_u32(smem + b * S::kStage), smem_u32(sB), tmem + (uint32_t)b * S::kColsBuf,
                                    row_tile<ROWS, kRowPix>(tile, h, w).rows);
        umma::commit(tfull + b);
        umma::commit(empty + b);
      }
      __syncwarp();
    }
    // The last two issued tiles' commits on empty[] have arrived before the CTA
    // leaves, also after a failed wait: no MMA runs into released tensor memory
    // (those phases are the newest of their barriers).
    for (int kk = k - 2; kk < k; kk++)
      if (kk >= 0 && !warp_wait(empty + (kk & 1), (uint32_t)(kk >> 1) & 1u)) ok = false;
  } else {
    // Epilogue warps: tile k from accumulator buffer k % 2; warp q + 4 r owns
    // lane quarter q (pixels 32 q .. 32 q + 31) of rows r, r + 4, ...  First they
    // stage the weights, while the producers load the first tile.
    if (tid < CO) sbias[tid] = EPI == CONV_DGELU ? 0.0f : bias[tid];
    stage_weights<CG, CO, EPI>(sB, wt, tid, kPipeEpiWarps * 32);
    fence_proxy_async_smem();
    mbar_arrive(wfull);
    asm volatile("bar.sync 1, %0;" ::"n"(kPipeEpiWarps * 32) : "memory");  // sbias
    const int q = warp & 3;
    int k = 0;
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x, k++) {
      const int b = k & 1;
      if (!warp_wait(tfull + b, (uint32_t)(k >> 1) & 1u)) {
        ok = false;
        break;
      }
      umma::fence_after_sync();
      const RowTile rt = row_tile<ROWS, kRowPix>(tile, h, w);
      if (q * 32 < rt.pix) {
        const bool in = q * 32 + lane < rt.pix;
#pragma unroll 1
        for (int r = warp >> 2; r < rt.rows; r += kPipeEpiWarps / 4) {
          const long long p = (rt.bb * h + rt.y0 + r) * (long long)w + rt.x0 + q * 32 + lane;
          const uint32_t t0 = tmem + (uint32_t)b * S::kColsBuf + ((uint32_t)(q * 32) << 16) + (uint32_t)(r * CO);
#pragma unroll
          for (int c = 0; c < CO; c += 16) {
            float acc[16];
            umma::ld16(t0 + c, acc);
            if (in) epilogue16<CO, EPI>(acc, c, p, sbias, zprev, out0, out1, wide != 0);
          }
        }
      }
      umma::fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty + b);
    }
  }
  if (!ok && lane == 0) *static_cast<volatile int*>(err) = PMHD_LEARNED_ERR_TIMEOUT;
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    umma::fence_after_sync();
    umma::tmem_dealloc(tmem, S::kTmemCols);
  }
}

// Weight gradient, any image size.  K = pixels, so both operands are MN-major
// with NHWC's channels along M and N, staged as NHWC has them (umma.cuh).  Staged
// rows are equidistant, so rows 2 q .. 2 q + 3 of x are four channel blocks of an
// M = 128 operand, and output rows 2 q, 2 q + 1 of dz the two of an N = 2 CO one.
// For each dx (a shift of x's start address by a pixel)
// D_dx[(row i, c_in)][(row o, c_out)] accumulates over all tiles of the CTA; the
// blocks with i - 1 - o in {-1, 0, 1} are the three vertical taps (six of eight
// blocks useful).  48 MMAs of N = 64 a tile of 8 x 64 pixels.  Six producer warps
// fill three stages; four warps sum dz for the bias gradient from the staged
// tiles (when asked to) and add the CTA's accumulators to dw at the end.
// 32 -> 32 over 8 x 512^2 reads 268 MB (42 us at the copy rate): 78 us
// against 1,110 for transposing 8 x 8 blocks of nine gathered copies into K-major
// tiles, 64 pixels at a time without overlap; 90 without swizzle (16-byte
// planes fetch every 32-byte sector twice).
constexpr int kWgRows = 8, kWgPix = 64, kWgStages = 3;
constexpr int kWgEpiWarps = 4, kWgProdWarps = 6;
constexpr int kWgThreads = 32 * (kWgEpiWarps + kWgProdWarps + 1);

template <int CO>
struct WgradSmem {
  static constexpr uint32_t kXRow = (kWgPix + 2) * 64u;  // row stride of x
  static constexpr uint32_t kBytesX = ((kWgRows + 2) * kXRow + 1023u) & ~1023u;
  static constexpr uint32_t kDRow = kWgPix * 2u * CO;    // row stride of dz
  static constexpr uint32_t kBytesD = kWgRows * kDRow;
  static constexpr uint32_t kStage = kBytesX + kBytesD;
  static constexpr uint32_t kOffBar = kWgStages * kStage;
  static constexpr uint32_t kBytes = kOffBar + (2u * kWgStages + 1u) * 8u + 8u;
  static constexpr uint32_t kTmemCols = umma::tmem_cols(3 * 2 * CO);
  static_assert(kStage % 1024 == 0, "the bias sums take a stage's base out of the swizzle");
  static_assert(2 * kBytes > 228 * 1024, "one CTA per SM (tensor memory)");
};

template <int CO>
__global__ void __launch_bounds__(kWgThreads, 1) wgrad_kernel(const __nv_bfloat16* __restrict__ x,
                                                              const __nv_bfloat16* __restrict__ dz, long long ntiles,
                                                              int h, int w, float* __restrict__ dw,
                                                              float* __restrict__ db, int* __restrict__ err) {
  using S = WgradSmem<CO>;
  constexpr int NG = CO / 8;
  extern __shared__ __align__(1024) unsigned char smem[];
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + S::kOffBar);
  uint64_t* empty = full + kWgStages;
  uint64_t* done = empty + kWgStages;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(done + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (warp == 0) {
    umma::tmem_alloc(tslot, S::kTmemCols);
    umma::tmem_relinquish();
  }
  if (tid == 0) {
    for (int b = 0; b < kWgStages; b++) {
      mbar_init(full + b, kWgProdWarps * 32);
      mbar_init(empty + b, db ? 1 + kWgEpiWarps : 1);
    }
    mbar_init(done, 1);
    fence_barrier_init();
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = *tslot;
  bool ok = true;

  if (warp >= kWgEpiWarps && warp < kWgEpiWarps + kWgProdWarps) {
    // Producers: ten input rows and eight gradient rows a tile, three a warp.
    const int pw = warp - kWgEpiWarps;
    int k = 0;
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x, k++) {
      const int b = k % kWgStages;
      if (k >= kWgStages && !warp_wait(empty + b, (uint32_t)(k / kWgStages - 1) & 1u)) {
        ok = false;
        break;
      }
      const RowTile rt = row_tile<kWgRows, kWgPix>(tile, h, w);
      const uint32_t dst = smem_u32(smem + b * S::kStage);
      for (int r = pw; r < 2 * kWgRows + 2; r += kWgProdWarps) {
        if (r < kWgRows + 2) {
          stage_halo_row<32, kWgPix, true>(dst + r * S::kXRow, x, rt, r, h, w, lane);
        } else {
          const int o = r - (kWgRows + 2);
          const bool row_in = o < rt.rows;
          const __nv_bfloat16* src =
              dz + ((rt.bb * h + rt.y0 + (row_in ? o : 0)) * (long long)w + rt.x0) * CO + lane % NG * 8;
          const uint32_t d = umma::swz<2 * CO>(dst + S::kBytesX + o * S::kDRow + lane * 16);
#pragma unroll
          for (int i = 0; i < kWgPix * NG / 32; i++) {
            const int px = lane / NG + i * (32 / NG);
            const bool take = row_in && px < rt.pix;
            cp16_or_zero(d + i * 512, src + (take ? px * CO : 0), take);
          }
        }
      }
      cp_wait_all();
      fence_proxy_async_smem();
      mbar_arrive(full + b);
    }
  } else if (warp == kWgEpiWarps + kWgProdWarps) {
    constexpr uint32_t idesc = umma::idesc_bf16(128, 2 * CO, true, true);
    int k = 0;
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x, k++) {
      const int b = k % kWgStages;
      if (!warp_wait(full + b, (uint32_t)(k / kWgStages) & 1u)) {
        ok = false;
        break;
      }
      umma::fence_after_sync();
      if (lane == 0) {
        const uint32_t a0 = smem_u32(smem + b * S::kStage);
        const uint64_t da = umma::desc(a0, S::kXRow, 512, umma::kSwizzle64);
        const uint64_t dd =
            umma::desc(a0 + S::kBytesX, S::kDRow, 16 * CO, CO == 32 ? umma::kSwizzle64 : umma::kSwizzle32);
        const uint32_t a_hi = umma::desc_hi(da), d_hi = umma::desc_hi(dd);
        uint32_t a_lo = umma::desc_lo(da), d_lo = umma::desc_lo(dd);
        const int pairs = (row_tile<kWgRows, kWgPix>(tile, h, w).rows + 1) / 2;
#pragma unroll 1
        for (int q = 0; q < pairs; q++, a_lo += 2 * S::kXRow / 16, d_lo += 2 * S::kDRow / 16)
#pragma unroll
          for (int kk = 0; kk < kWgPix; kk += 16)
#pragma unroll
            for (int dx = 0; dx < 3; dx++)
              umma::mma_bf16(tmem + dx * 2 * CO, a_lo + (kk + dx) * 4, a_hi, d_lo + kk * (CO / 8), d_hi, idesc,
                             (k | q | kk) ? 1u : 0u);
        umma::commit(empty + b);
      }
      __syncwarp();
    }
    // Every MMA has completed (also after a failed wait) before the accumulators
    // are read or released.
    if (lane == 0) umma::commit(done);
    __syncwarp();
    if (!warp_wait(done, 0)) ok = false;
  } else {
    if (db) {
      // Bias gradient: thread (px, half) sums its pixel column's NG / 2 groups.
      float s[NG / 2][8];
#pragma unroll
      for (int g = 0; g < NG / 2; g++)
#pragma unroll
        for (int c = 0; c < 8; c++) s[g][c] = 0.f;
      const int px = tid & 63, half = tid >> 6;
      int k = 0;
      for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x, k++) {
        const int b = k % kWgStages;
        if (!warp_wait(full + b, (uint32_t)(k / kWgStages) & 1u)) {
          ok = false;
          break;
        }
        const unsigned char* d = smem + b * S::kStage + S::kBytesX;
#pragma unroll
        for (int o = 0; o < kWgRows; o++)
#pragma unroll
          for (int g = 0; g < NG / 2; g++) {
            const uint4 v = *reinterpret_cast<const uint4*>(
                d + o * S::kDRow + umma::swz<2 * CO>(px * 2 * CO + (half * (NG / 2) + g) * 16));
            const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int c = 0; c < 4; c++) {
              s[g][2 * c] += __uint_as_float(u[c] << 16);
              s[g][2 * c + 1] += __uint_as_float(u[c] & 0xffff0000u);
            }
          }
        __syncwarp();
        if (lane == 0) mbar_arrive(empty + b);
      }
#pragma unroll
      for (int g = 0; g < NG / 2; g++)
#pragma unroll
        for (int c = 0; c < 8; c++) {
          float v = s[g][c];
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
          if (lane == 0 && ok) atomicAdd(db + (half * (NG / 2) + g) * 8 + c, v);
        }
    }
    // Accumulators: lane = (row i = warp, c_in = lane), columns (dx, row o, c_out).
    if (ok && !warp_wait(done, 0)) ok = false;
    umma::fence_after_sync();
    if (ok) {
#pragma unroll 1
      for (int c = 0; c < 3 * 2 * CO; c += 16) {
        float acc[16];
        umma::ld16(tmem + ((uint32_t)(warp * 32) << 16) + c, acc);
        const int dx = c / (2 * CO), o = (c / CO) & 1, co = c % CO, dy = warp - 1 - o;
        if (dy < -1 || dy > 1) continue;
        float* dst = dw + ((size_t)co * 9 + (dy + 1) * 3 + dx) * 32 + lane;
#pragma unroll
        for (int q = 0; q < 16; q++) atomicAdd(dst + (size_t)q * 9 * 32, acc[q]);
      }
    }
  }
  if (!ok && lane == 0) *static_cast<volatile int*>(err) = PMHD_LEARNED_ERR_TIMEOUT;
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    umma::fence_after_sync();
    umma::tmem_dealloc(tmem, S::kTmemCols);
  }
}

template <class K>
cudaError_t set_smem(K kernel, uint32_t bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

template <int CG, int CO, int EPI>
cudaError_t prepare_conv() {
  cudaError_t e = set_smem(conv3x3_pipe_kernel<CG, CO, EPI, 2>, PipeSmem<CG, CO, 2>::kLaunchBytes);
  if (e == cudaSuccess) e = set_smem(conv3x3_pipe_kernel<CG, CO, EPI, 4>, PipeSmem<CG, CO, 4>::kLaunchBytes);
  if (e == cudaSuccess) e = set_smem(conv3x3_pipe_kernel<CG, CO, EPI, 8>, PipeSmem<CG, CO, 8>::kLaunchBytes);
  return e;
}

int g_sms = 0;  // SM count of the device the kernels were prepared on

bool aligned32(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 31u) == 0; }

// Tiles of `rows` image rows x 128 pixels.
long long row_tiles(int batch, int h, int w, int rows) {
  return (long long)batch * ((h + rows - 1) / rows) * ((w + kRowPix - 1) / kRowPix);
}

// Persistent CTAs: one per SM, at most one per tile.  Test hook:
// PMHD_CONV_MAX_CTAS > 0 limits them, so small images still give each CTA several
// tiles (all buffers reused, barrier phases flipping).
unsigned persistent_grid(long long tiles) {
  const int sms = g_sms > 0 ? g_sms : 148;
  const char* hook_env = getenv("PMHD_CONV_MAX_CTAS");
  const long long hook = hook_env ? atoll(hook_env) : 0;
  long long grid = tiles < sms ? tiles : sms;
  if (hook > 0 && grid > hook) grid = hook;
  return (unsigned)grid;
}

template <int CG, int CO, int EPI, int ROWS>
cudaError_t launch_rows(const __nv_bfloat16* x, int batch, int h, int w, const __nv_bfloat16* wt, const float* bias,
                        const __nv_bfloat16* zprev, void* out0, void* out1, int* err, cudaStream_t s) {
  const long long tiles = row_tiles(batch, h, w, ROWS);
  const int wide = aligned32(out0) && (EPI != CONV_GELU || aligned32(out1)) && (EPI != CONV_DGELU || aligned32(zprev));
  conv3x3_pipe_kernel<CG, CO, EPI, ROWS>
      <<<persistent_grid(tiles), kPipeThreads, PipeSmem<CG, CO, ROWS>::kLaunchBytes, s>>>(x, wt, bias, zprev, tiles, h,
                                                                                         w, out0, out1, wide, err);
  return cudaGetLastError();
}

// Rows per tile: the fewest of 2, 4, 8 that leave every tile an SM of its own (a
// launch is then one tile's load, MMAs and drain in sequence: 8 x 64^2 GELU layer
// 32.5 -> 29.4 us a call with tiles of 4), else 8 (fewest halo rows).
template <int CG, int CO, int EPI>
cudaError_t launch_conv(const __nv_bfloat16* x, int batch, int h, int w, const __nv_bfloat16* wt, const float* bias,
                        const __nv_bfloat16* zprev, void* out0, void* out1, int* err, cudaStream_t s) {
  const int sms = g_sms > 0 ? g_sms : 148;
  if (row_tiles(batch, h, w, 2) <= sms)
    return launch_rows<CG, CO, EPI, 2>(x, batch, h, w, wt, bias, zprev, out0, out1, err, s);
  if (row_tiles(batch, h, w, 4) <= sms)
    return launch_rows<CG, CO, EPI, 4>(x, batch, h, w, wt, bias, zprev, out0, out1, err, s);
  return launch_rows<CG, CO, EPI, 8>(x, batch, h, w, wt, bias, zprev, out0, out1, err, s);
}

template <int CO>
cudaError_t launch_wgrad(const __nv_bfloat16* x, const __nv_bfloat16* dz, int batch, int h, int w, float* dw,
                         float* db, int* err, cudaStream_t s) {
  const long long tiles = (long long)batch * ((h + kWgRows - 1) / kWgRows) * ((w + kWgPix - 1) / kWgPix);
  wgrad_kernel<CO><<<persistent_grid(tiles), kWgThreads, WgradSmem<CO>::kBytes, s>>>(x, dz, tiles, h, w, dw, db, err);
  return cudaGetLastError();
}

}  // namespace

namespace {
std::atomic<unsigned> g_prepared{0};
}

unsigned conv_prepared() { return g_prepared.load(); }

cudaError_t conv_prepare() {
  g_prepared++;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = prepare_conv<32, 32, CONV_GELU>();
  if (e == cudaSuccess) e = prepare_conv<32, 16, CONV_LINEAR>();
  if (e == cudaSuccess) e = prepare_conv<16, 32, CONV_DGELU>();
  if (e == cudaSuccess) e = prepare_conv<32, 32, CONV_DGELU>();
  if (e == cudaSuccess) e = set_smem(wgrad_kernel<32>, WgradSmem<32>::kBytes);
  if (e == cudaSuccess) e = set_smem(wgrad_kernel<16>, WgradSmem<16>::kBytes);
  return e;
}

cudaError_t conv3x3(int mode, const __nv_bfloat16* x, int batch, int h, int w, int c_in, const __nv_bfloat16* wt,
                    const float* bias, int c_out, const __nv_bfloat16* zprev, void* out0, void* out1, int* err,
                    cudaStream_t s) {
  if (mode == CONV_GELU && c_in == 32 && c_out == 32)
    return launch_conv<32, 32, CONV_GELU>(x, batch, h, w, wt, bias, zprev, out0, out1, err, s);
  if (mode == CONV_LINEAR && c_in == 32 && c_out == 16)
    return launch_conv<32, 16, CONV_LINEAR>(x, batch, h, w, wt, bias, zprev, out0, out1, err, s);
  if (mode == CONV_DGELU && c_in == 16 && c_out == 32)
    return launch_conv<16, 32, CONV_DGELU>(x, batch, h, w, wt, bias, zprev, out0, out1, err, s);
  if (mode == CONV_DGELU && c_in == 32 && c_out == 32)
    return launch_conv<32, 32, CONV_DGELU>(x, batch, h, w, wt, bias, zprev, out0, out1, err, s);
  return cudaErrorNotSupported;
}

cudaError_t conv3x3_wgrad(const __nv_bfloat16* x, const __nv_bfloat16* dz, int batch, int h, int w, int c_in,
                          int c_out, float* dw, float* db, int* err, cudaStream_t s) {
  if (c_in == 32 && c_out == 32) return launch_wgrad<32>(x, dz, batch, h, w, dw, db, err, s);
  if (c_in == 32 && c_out == 16) return launch_wgrad<16>(x, dz, batch, h, w, dw, db, err, s);
  return cudaErrorNotSupported;
}

}  // namespace learned
}  // namespace pmhd
