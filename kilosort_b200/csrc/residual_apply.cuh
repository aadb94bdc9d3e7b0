// Subtracting spikes' waveforms amp * U_k x W from tiles of a batch: the inner
// loop of the peel's residual pass and of the reconstruction loss.
#pragma once
#include <cuda_runtime.h>

namespace {

constexpr int kXList = 64;                  // spike list entries of a warp
// Two packed FP32 operations per instruction (each half rounds as the scalar
// operation does).
__device__ __forceinline__ unsigned long long f2_pack(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void f2_unpack(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long f2_fma(unsigned long long a, unsigned long long b,
                                                     unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// c += a b in place.
__device__ __forceinline__ void f2_fma_acc(unsigned long long& c, unsigned long long a,
                                           unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long f2_mul(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// a + fl(x y), the product and the sum rounded separately.  The sum is a fused
// operation with a factor of one that the compiler cannot see (`one` of
// the callers' arguments): a packed product followed by a packed sum was
// contracted into one rounding.
__device__ __forceinline__ unsigned long long f2_add_prod(unsigned long long a,
                                                          unsigned long long x,
                                                          unsigned long long y,
                                                          unsigned long long one2) {
  return f2_fma(one2, f2_mul(x, y), a);
}

// The basis [P][nt] in shared memory with rows P .. 7 zero.  Returns whether a
// value that this thread staged is infinite or NaN.
__device__ __forceinline__ bool stage_basis(const float* W, int P, int nt, float* sW,
                                            int nthreads) {
  bool odd = false;
  for (int i = threadIdx.x; i < 8 * nt; i += nthreads) {
    const float w = i < P * nt ? W[i] : 0.f;
    odd |= !(fabsf(w) < INFINITY);
    sW[i] = w;
  }
  return odd;
}

// Per-warp scratch of the residual pass: the spike list (time, template,
// amplitude) and one spike's loadings of 16 channels.
constexpr int kXStride = 20;                // floats of a channel pair's loadings, padded
                                            // so that the stores spread over the banks
constexpr int kXU = 8 * kXStride;           // floats of one spike's loadings of 16 channels
constexpr int kXWarp = 3 * kXList + kXU;    // 4-byte words per warp
struct ResSmem {
  const float* W;  // [8][nt]: the basis, rows past P zero
  int* xl_tau;     // this warp's list, kXList entries
  int* xl_k;
  float* xl_amp;
  float* xu;       // this warp's loadings, [8 channel pairs][kXStride]: [8 components][2]
};

__device__ __forceinline__ ResSmem residual_smem(const float* W, void* scratch, int warp) {
  int* base = reinterpret_cast<int*>(scratch) + warp * kXWarp;
  ResSmem r;
  r.W = W;
  r.xl_tau = base;
  r.xl_k = base + kXList;
  r.xl_amp = reinterpret_cast<float*>(base + 2 * kXList);
  r.xu = reinterpret_cast<float*>(base + 3 * kXList);
  return r;
}

// Channels of one residual tile, and tiles per bit of a template's support
// mask: the tiles 0 .. ceil(C/16)-1 are spread over 64 bits.
constexpr int kXCh = 16;
__host__ __device__ inline int support_width(int C) { return ((C + kXCh - 1) / kXCh + 63) / 64; }

// Subtract the n listed spikes, in record order, from the tile of block blk
// and channels [cbase, cbase + 16): lanes run over the block's columns and a
// lane keeps its column's channel values in registers (x2, channel pairs).
// Per spike a lane loads its tap's PP basis components (conflict-free rows of
// W); the spike's loadings of the tile's channels come from the warp's shared
// buffer, loaded from U one spike ahead; channels are processed two at a time
// with packed FP32 operations: per element the reference's products in the
// same order, each rounded as the scalar operation.  Spikes whose template is
// exactly zero on the tile (a.sup) and whose amplitude is finite would subtract
// +0 and are passed over (callers whose spikes do not come from this basis drop
// a.sup when it is not finite: its product with a zero loading is NaN).
//
// What bounds it: issue (52 % of the slots at 29 % of the warps: about 5.5 warp
// instructions per channel row and spike) and the shared-memory round trips
// between, next to the 8CL bytes of X and Xres (185 MB, 28 us).  The
// form with lanes over channels, which applied every listed spike to an Xres
// copied from X beforehand, took 493 us + 38 us for the copy on a C=384, K=600
// batch of 60122 samples; this one takes 159 us without a copy, and the
// batched launch of 16 such batches 29.1 -> 21.6 ms.  Tiles of 32 channels
// spilled at the peel's 80 registers and pass over fewer spikes.
template <int PP, class Args>
__device__ void residual_apply(const Args& a, const ResSmem& s, int n, int c0, int cbase,
                               int bit, int lane, unsigned long long* x2) {
  const int half = a.nt / 2, nt = a.nt, P = a.P;
  const int ch = cbase + (lane & (kXCh - 1));
  const int p0 = (lane / kXCh) * (PP / 2);     // this lane loads components p0 .. p0 + PP/2 - 1
  const bool chok = ch < a.C;
  const unsigned long long one2 = f2_pack(a.one, a.one);
  for (int e0 = 0; e0 < n; e0 += 32) {
    bool hit = e0 + lane < n;
    if (hit && a.sup)
      hit = ((a.sup[s.xl_k[e0 + lane]] >> bit) & 1ull) || !(fabsf(s.xl_amp[e0 + lane]) < INFINITY);
    unsigned todo = __ballot_sync(0xffffffffu, hit);
    if (!todo) continue;
    float u[PP / 2];
    auto fetch = [&](int e) {
      const float* up = a.U + ((long long)s.xl_k[e0 + e] * P + p0) * a.C + ch;
#pragma unroll
      for (int j = 0; j < PP / 2; ++j)
        u[j] = (chok && p0 + j < P) ? __ldg(up + (long long)j * a.C) : 0.f;
    };
    fetch(__ffs(todo) - 1);
    while (todo) {
      const int e = __ffs(todo) - 1;
      todo &= todo - 1u;
      __syncwarp();                    // the previous spike's loadings are read
      {
        float* dst = s.xu + ((lane & (kXCh - 1)) >> 1) * kXStride + (lane & 1) + 2 * p0;
#pragma unroll
        for (int j = 0; j < PP / 2; ++j) dst[2 * j] = u[j];
      }
      __syncwarp();
      if (todo) fetch(__ffs(todo) - 1);
      const int t = c0 + lane - s.xl_tau[e0 + e] + half;
      const bool in = t >= 0 && t < nt;
      const float namp = -s.xl_amp[e0 + e];
      const unsigned long long amp2 = f2_pack(namp, namp);
      unsigned long long w2[PP];
#pragma unroll
      for (int p = 0; p < PP; ++p) {
        const float wv = in ? s.W[p * nt + t] : 0.f;
        w2[p] = f2_pack(wv, wv);
      }
#pragma unroll
      for (int i = 0; i < kXCh / 2; ++i) {
        const ulonglong2* u4 = reinterpret_cast<const ulonglong2*>(s.xu + i * kXStride);
        unsigned long long v = 0ull;
#pragma unroll
        for (int p = 0; p < PP; p += 2) {
          const ulonglong2 uu = u4[p >> 1];
          v = f2_fma(uu.x, w2[p], v);
          v = f2_fma(uu.y, w2[p + 1], v);
        }
        // x - fl(amp v) = x + fl(-amp v), on the columns inside the window
        if (in) x2[i] = f2_add_prod(x2[i], amp2, v, one2);
      }
    }
  }
}

}  // namespace
