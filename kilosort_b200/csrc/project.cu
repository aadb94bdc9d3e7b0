// Score projection B[k, tau] = sum_{p,c} U[k,p,c] * Y[c,p,tau],
// Y[c,p,tau] = sum_t W[p,t] X[c, tau - nt/2 + t] (zero padding),
// i.e. kilosort/template_matching.py:180-181 (conv1d then einsum).
//
// Layout in HBM (per call, carved from the caller's workspace)
//   Yt  [Lpad, Q] temporal projection, q = c*P + p contiguous ("K-major" for
//       the contraction), Lpad = roundup(L, 128), Q = roundup(roundup(C,16)*P, 64)
//       float32 (FP32 form) or two bf16 planes hi/lo (split form)
//   Uq  [Kpad, Q] templates in the same q order, zero padded; float32 or bf16 hi/lo
//   B   [K, ldb] float32 output
//
// Kernels
//   ks_prep_templates  nm[k] and Uq (both precisions)
//   ks_temporal        X -> Yt: each thread owns 8 consecutive samples of one
//                      channel and all P components, in pairs through packed
//                      multiply-adds, its samples in a register window that
//                      moves on 8 taps at a time; f32 rows turned in shared
//                      memory and written as whole sectors
//   ks_sgemm_tn        FP32 SIMT contraction with packed multiply-adds, tiles of
//                      64 to 128 rows x 128 columns or of 128 x 256, register
//                      double buffering; tile order puts the template tiles of one time
//                      tile next to each other so each Yt tile is read from HBM
//                      once
#include "ks_common.cuh"
#include "project.cuh"
#include "residual_apply.cuh"

#include <cuda_bf16.h>
#include <type_traits>

namespace ks {

// ------------------------------------------------------------------ prep
__global__ void ks_template_energy_kernel(const float* __restrict__ U, int K,
                                          int P, int C, float* __restrict__ nm) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= K) return;
  const float* u = U + (long long)warp * P * C;
  float tot = 0.f;
  for (int p = 0; p < P; ++p) {
    float s = 0.f;
    for (int c = lane; c < C; c += 32) s = __fadd_rn(s, __fmul_rn(u[p * C + c], u[p * C + c]));
    for (int o = 16; o; o >>= 1) s = __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, o));
    tot = __fadd_rn(tot, s);
  }
  if (lane == 0) nm[warp] = tot;
}

__global__ void ks_reorder_templates_kernel(const float* __restrict__ U, int K,
                                            int P, int C, int Kpad, int Q,
                                            float* __restrict__ Uf,
                                            __nv_bfloat16* __restrict__ Uhi,
                                            __nv_bfloat16* __restrict__ Ulo) {
  const long long n = (long long)Kpad * Q;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x) {
    const int k = (int)(e / Q);
    const int q = (int)(e - (long long)k * Q);
    const int c = q / P, p = q - (q / P) * P;
    float v = 0.f;
    if (k < K && c < C) v = U[((long long)k * P + p) * C + c];
    if (Uf) Uf[e] = v;
    if (Uhi) {
      const __nv_bfloat16 h = __float2bfloat16_rn(v);
      Uhi[e] = h;
      Ulo[e] = __float2bfloat16_rn(v - __bfloat162float(h));
    }
  }
}

// ------------------------------------------------------------------ temporal
constexpr int kTT = 128;   // samples per tile
constexpr int kCG = 16;    // channels per tile
constexpr int kTemporalThreads = 256;
constexpr int kPMax = 8;

// X window per channel: samples tau0 - nt/2 .. tau0 + kTT + nt + 7, padded so
// every row starts on a 16-byte boundary.
__host__ __device__ inline int temporal_xw(int nt) { return (kTT + nt + 8 + 3) & ~3; }

// Floats of a warp's turned results: half of the components of 16 channels by 16
// samples (pitch 20), or half of the samples by 16 channels.
__host__ __device__ constexpr int temporal_turn(int P) { return kCG * 20 * ((P + 1) / 2); }

// Asynchronous 4-byte global -> shared copy; src_bytes 0 fills zeros.
__device__ __forceinline__ void cp_async4(float* dst, const float* src, int src_bytes) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(src_bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_prev() {
  asm volatile("cp.async.wait_group 1;" ::: "memory");
}

// Persistent: block b takes tiles b, b + grid, ... (a tile is kTT samples x
// kCG channels).  The X window of the next tile is copied (cp.async) while the
// current one is computed.  Each thread owns 8 consecutive samples of one
// channel and all PP components; taps run in groups of 8 over a 16-sample
// register window (every operand index a compile-time constant) and each
// tap's components come from the transposed basis Wt[t][8] as two broadcast
// 16-byte loads.  acc[i][p] accumulates taps t = 0 .. nt-1 in increasing
// order, pairs of components packed.  Whole groups of taps run without a branch,
// so that the next tap's basis is loaded ahead; f32 results are turned in shared
// memory so that a store writes whole sectors.  Bound by FMA issue (235 us at
// C=384, P=6, nt=61, L=60122): 434 us there; 526 with a branch per tap, bounds
// checked per copied sample and 8-byte stores (519 with the stores alone
// so, 489 with the checks alone so).
template <int PP>
__global__ void __launch_bounds__(kTemporalThreads)
ks_temporal_kernel(const float* __restrict__ X, const float* __restrict__ W,
                   int C, int L, int nt, int Q, int tiles_t, int n_tiles,
                   float* __restrict__ Yf, __nv_bfloat16* __restrict__ Yhi,
                   __nv_bfloat16* __restrict__ Ylo, float* __restrict__ YT, long long ldyt) {
  extern __shared__ __align__(16) float sm[];
  constexpr int kS = kTT / (kTemporalThreads / kCG);   // samples per thread (8)
  const int xw = temporal_xw(nt);
  const int ntr = (nt + 7) & ~7;            // taps rounded to the group of 8
  float* sW = sm;                           // Wt[ntr][8] (zero past nt and PP)
  float* sX[2] = {sW + 8 * ntr, sW + 8 * ntr + kCG * xw};   // [kCG][xw] each
  float* sT = sX[1] + kCG * xw;             // [8 warps][kTurn]
  constexpr int kTurn = temporal_turn(PP);
  const int half = nt / 2;
  for (int i = threadIdx.x; i < 8 * ntr; i += kTemporalThreads) {
    const int t = i >> 3, p = i & 7;
    sW[i] = (p < PP && t < nt) ? W[p * nt + t] : 0.f;
  }
  auto fetch = [&](int tile, float* dst) {
    const int tau0 = (tile % tiles_t) * kTT, cg0 = (tile / tiles_t) * kCG;
    // a warp copies two channels, a lane every 32nd sample
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int w = 2 * (threadIdx.x >> 5) + h, c = cg0 + w;
      const float* src = X + (long long)(c < C ? c : 0) * L + (tau0 - half) + lane;
      float* d = dst + w * xw + lane;
      if (c < C && tau0 >= half && tau0 - half + xw <= L) {
        int u = lane;
#pragma unroll 4
        for (; u < xw; u += 32, src += 32, d += 32) cp_async4(d, src, 4);
      } else {
        for (int u = lane; u < xw; u += 32, src += 32, d += 32) {
          const int t = tau0 - half + u;
          const bool ok = c < C && t >= 0 && t < L;
          cp_async4(d, ok ? src : X, ok ? 4 : 0);
        }
      }
    }
    cp_async_commit();
  };
  const int cl = threadIdx.x & (kCG - 1);
  const int g = threadIdx.x / kCG;          // groups of kS samples
  int buf = 0;
  if (blockIdx.x < n_tiles) fetch(blockIdx.x, sX[0]);
  for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    const int next = tile + gridDim.x;
    if (next < n_tiles) fetch(next, sX[buf ^ 1]);
    else cp_async_commit();                 // keep the group count in step
    cp_async_wait_prev();                   // this tile's window has landed
    __syncthreads();
    const int tau0 = (tile % tiles_t) * kTT, cg0 = (tile / tiles_t) * kCG;
    const float4* xs4 = reinterpret_cast<const float4*>(sX[buf] + cl * xw + g * kS);
    // packed over pairs of components (the basis is zero past PP)
    constexpr int HP = (PP + 1) / 2;
    unsigned long long a2[kS][HP];
#pragma unroll
    for (int i = 0; i < kS; ++i)
#pragma unroll
      for (int p = 0; p < HP; ++p) a2[i][p] = 0ull;
    unsigned long long win[kS + 8];         // every sample twice
#pragma unroll
    for (int k = 0; k < kS / 4; ++k) {
      const float4 a = xs4[k];
      win[4 * k] = f2_pack(a.x, a.x);
      win[4 * k + 1] = f2_pack(a.y, a.y);
      win[4 * k + 2] = f2_pack(a.z, a.z);
      win[4 * k + 3] = f2_pack(a.w, a.w);
    }
    // eight taps from t0 (kTail: those below nt, a branch each)
    auto taps = [&](int t0, auto tail) {
      constexpr bool kTail = decltype(tail)::value;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const float4 a = xs4[(t0 + kS) / 4 + k];
        win[kS + 4 * k] = f2_pack(a.x, a.x);
        win[kS + 4 * k + 1] = f2_pack(a.y, a.y);
        win[kS + 4 * k + 2] = f2_pack(a.z, a.z);
        win[kS + 4 * k + 3] = f2_pack(a.w, a.w);
      }
#pragma unroll
      for (int tt = 0; tt < 8; ++tt) {
        if (!kTail || t0 + tt < nt) {
          const ulonglong2* wt = reinterpret_cast<const ulonglong2*>(sW + 8 * (t0 + tt));
          const ulonglong2 wa = wt[0], wb = HP > 2 ? wt[1] : wa;
          const unsigned long long w[4] = {wa.x, wa.y, wb.x, wb.y};
#pragma unroll
          for (int i = 0; i < kS; ++i)
#pragma unroll
            for (int p = 0; p < HP; ++p) a2[i][p] = f2_fma(w[p], win[i + tt], a2[i][p]);
        }
      }
#pragma unroll
      for (int i = 0; i < kS; ++i) win[i] = win[i + 8];
    };
    int t0 = 0;
#pragma unroll 1
    for (; t0 + 8 <= nt; t0 += 8) taps(t0, std::false_type{});
    if (t0 < nt) taps(t0, std::true_type{});
    float acc[kS][2 * HP];
#pragma unroll
    for (int i = 0; i < kS; ++i)
#pragma unroll
      for (int p = 0; p < HP; ++p) f2_unpack(a2[i][p], acc[i][2 * p], acc[i][2 * p + 1]);
    // the window is no longer read: the next fetch may overwrite this buffer
    __syncthreads();
    const long long q0 = (long long)(cg0 + cl) * PP;
    // f32 results: a warp holds 16 samples of all 16 channels, whose rows it turns
    // in shared memory so that a store writes whole sectors
    float* turn = sT + (threadIdx.x >> 5) * kTurn;
    const int lane = threadIdx.x & 31, gw = (threadIdx.x >> 5) * 2, gl = lane >> 4;
    if (YT) {
      // rows (channel, component), samples contiguous: 16 samples a row, half of
      // the components at a time
      constexpr int H = (PP + 1) / 2;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int np = h ? PP - H : H;
        __syncwarp();
#pragma unroll
        for (int p = 0; p < H; ++p)
          if (h * H + p < PP) {
            float4* d = reinterpret_cast<float4*>(turn + (p * kCG + cl) * 20 + gl * kS);
            const int pp = h * H + p < PP ? h * H + p : 0;
            d[0] = make_float4(acc[0][pp], acc[1][pp], acc[2][pp], acc[3][pp]);
            d[1] = make_float4(acc[4][pp], acc[5][pp], acc[6][pp], acc[7][pp]);
          }
        __syncwarp();
        // four lanes a row, eight rows at once
        for (int r = lane >> 2; r < np * kCG; r += 8) {
          const int c = cg0 + (r & (kCG - 1)), p = h * H + r / kCG;
          if (c < C)
            *reinterpret_cast<float4*>(YT + ((long long)c * PP + p) * ldyt + tau0 + gw * kS +
                                       4 * (lane & 3)) =
                *reinterpret_cast<const float4*>(turn + r * 20 + 4 * (lane & 3));
        }
      }
      buf ^= 1;
      continue;
    }
    if (Yf) {
      // rows (sample), channels and components contiguous: half of a thread's
      // samples at a time
      constexpr int R = kCG * PP;            // floats of a row
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        __syncwarp();
#pragma unroll
        for (int i = 0; i < kS / 2; ++i)
#pragma unroll
          for (int p = 0; p < PP; p += 2) {
            float* d = turn + (gl * (kS / 2) + i) * R + cl * PP + p;
            if (PP % 2 == 0)
              *reinterpret_cast<float2*>(d) =
                  make_float2(acc[h * kS / 2 + i][p], acc[h * kS / 2 + i][p + 1]);
            else {
              d[0] = acc[h * kS / 2 + i][p];
              if (p + 1 < PP) d[1] = acc[h * kS / 2 + i][p + 1];
            }
          }
        __syncwarp();
#pragma unroll
        for (int e = lane; e < kS * R / 4; e += 32) {
          const int r = e / (R / 4), q = e - r * (R / 4);
          const int tau = tau0 + (gw + r / (kS / 2)) * kS + h * (kS / 2) + r % (kS / 2);
          *reinterpret_cast<float4*>(Yf + (long long)tau * Q + (long long)cg0 * PP + 4 * q) =
              *reinterpret_cast<const float4*>(turn + r * R + 4 * q);
        }
      }
    }
    if (Yhi) {
#pragma unroll
      for (int i = 0; i < kS; ++i) {
        const long long o = (long long)(tau0 + g * kS + i) * Q + q0;
        // pairs of components as one 4-byte store: with PP even, o + p is even
        // for even p
#pragma unroll
        for (int p = 0; p < PP; p += 2) {
          const float v0 = acc[i][p], v1 = p + 1 < PP ? acc[i][p + 1] : 0.f;
          const __nv_bfloat162 h = __floats2bfloat162_rn(v0, v1);
          const float2 hf = __bfloat1622float2(h);
          const __nv_bfloat162 l = __floats2bfloat162_rn(v0 - hf.x, v1 - hf.y);
          if (PP % 2 == 0) {
            *reinterpret_cast<__nv_bfloat162*>(Yhi + o + p) = h;
            *reinterpret_cast<__nv_bfloat162*>(Ylo + o + p) = l;
          } else {
            Yhi[o + p] = h.x;
            Ylo[o + p] = l.x;
            if (p + 1 < PP) {
              Yhi[o + p + 1] = h.y;
              Ylo[o + p + 1] = l.y;
            }
          }
        }
      }
    }
    buf ^= 1;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

size_t temporal_smem(int nt, int P) {
  const int ntr = (nt + 7) & ~7;
  return sizeof(float) * (8 * (size_t)ntr + 2 * (size_t)kCG * temporal_xw(nt) +
                          kTemporalThreads / 32 * (size_t)temporal_turn(P));
}

// ------------------------------------------------------------------ FP32 GEMM
// Two FP32 fused operations in one instruction (each half rounds as fmaf).
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b,
                                                   unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ unsigned long long dup2(float v) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
  return r;
}

// C[m, n] = sum_q A[m, q] * Bt[n, q], every element one chain of fused
// operations over q; A is [>= tiles_m*BM, Kd], Bt is [>= tiles_n*128, Kd]
// (both zero padded), Kd % 16 == 0.  Stores m < M, n < N, row-major with
// leading dimension ldc, or (kTiled) in 32-column blocks
// C[((n/32)*M + m)*32 + n%32]; `upper` leaves out the tiles below the diagonal.
// Tiles of BM = 16 TM rows x 16 TN columns, TM x TN per thread, columns two at a
// time through packed operations.
//
// What bounds it: the FP32 pipe.  A packed operation does the work of two
// issue slots, so loads and moves no longer compete with the multiply-adds:
// 3.99 -> 3.11 ms at C=384, K=600, 60122 samples (41.6 -> 53.4 TFLOP/s), with 128
// columns per tile 3.48 ms.  Measured and dropped at 256 columns: slices of 16
// (3.60 ms), the next slice stored half way through this one (3.43), warps of 8 x
// 4 threads (3.19).
// Length of the slice of q staged at a time.
__host__ __device__ constexpr int sgemm_slice(int TN) { return TN == 8 ? 16 : 8; }

template <int TM, int TN, bool kTiled>
__global__ void __launch_bounds__(256, TN == 8 ? 2 : 1)
ks_sgemm_tn_kernel(const float* __restrict__ A, const float* __restrict__ Bt,
                   float* __restrict__ Cm, int M, int N, int Kd, long long ldc,
                   int tiles_m, bool upper) {
  constexpr int BM = 16 * TM, BN = 16 * TN, BK = sgemm_slice(TN);
  constexpr int kP = BK / 4;                           // 16-byte pieces of a row's slice
  constexpr int kALoads = (BM * kP + 255) / 256, kBLoads = BN * kP / 256;
  extern __shared__ __align__(16) float sgemm_sm[];
  float (*As)[BK][BM + 4] = reinterpret_cast<float (*)[BK][BM + 4]>(sgemm_sm);
  float (*Bs)[BK][BN + 4] = reinterpret_cast<float (*)[BK][BN + 4]>(sgemm_sm + 2 * BK * (BM + 4));
  const int tid = threadIdx.x;
  const int tm = blockIdx.x % tiles_m;
  const int tn = blockIdx.x / tiles_m;
  const long long m0 = (long long)tm * BM, n0 = (long long)tn * BN;
  if (upper && n0 + BN <= m0) return;                  // below the diagonal
  const long long last = ((N + 127LL) & ~127LL) - 1;   // the operand's last (padded) row
  const int tx = tid & 15, ty = tid >> 4;
  // a thread's pieces: row idx / kP, columns 4 (idx % kP) of the slice
  float4 ra[kALoads], rb[kBLoads];
  auto gload = [&](int k0) {
#pragma unroll
    for (int i = 0; i < kALoads; ++i) {
      const int idx = tid + i * 256;
      if (BM * kP % 256 == 0 || idx < BM * kP)
        ra[i] = *reinterpret_cast<const float4*>(A + (m0 + idx / kP) * Kd + k0 + idx % kP * 4);
    }
#pragma unroll
    for (int i = 0; i < kBLoads; ++i) {
      const int idx = tid + i * 256;
      const long long n = n0 + idx / kP;
      rb[i] = *reinterpret_cast<const float4*>(Bt + (n < last ? n : last) * Kd + k0 + idx % kP * 4);
    }
  };
  auto sstore = [&](int buf) {
#pragma unroll
    for (int i = 0; i < kALoads; ++i) {
      const int idx = tid + i * 256, kk = idx % kP * 4, r = idx / kP;
      if (BM * kP % 256 == 0 || idx < BM * kP) {
        As[buf][kk + 0][r] = ra[i].x;
        As[buf][kk + 1][r] = ra[i].y;
        As[buf][kk + 2][r] = ra[i].z;
        As[buf][kk + 3][r] = ra[i].w;
      }
    }
#pragma unroll
    for (int i = 0; i < kBLoads; ++i) {
      const int idx = tid + i * 256, kk = idx % kP * 4, r = idx / kP;
      Bs[buf][kk + 0][r] = rb[i].x;
      Bs[buf][kk + 1][r] = rb[i].y;
      Bs[buf][kk + 2][r] = rb[i].z;
      Bs[buf][kk + 3][r] = rb[i].w;
    }
  };
  // rows ty*4 .. ty*4+3 of the first 64, then TM-4 rows from 64 + ty*(TM-4) on;
  // columns 64 g + tx*4 .. +3, in pairs
  unsigned long long acc[TM][TN / 2];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;

  gload(0);
  sstore(0);
  __syncthreads();
  const int nk = Kd / BK;
  for (int kt = 0; kt < nk; ++kt) {
    const int buf = kt & 1;
    if (kt + 1 < nk) gload((kt + 1) * BK);
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float av[TM];
      {
        const float4 a0 = *reinterpret_cast<const float4*>(&As[buf][kk][ty * 4]);
        av[0] = a0.x; av[1] = a0.y; av[2] = a0.z; av[3] = a0.w;
        if (TM == 8) {
          const float4 a1 = *reinterpret_cast<const float4*>(&As[buf][kk][64 + ty * 4]);
          av[TM - 4] = a1.x; av[TM - 3] = a1.y; av[TM - 2] = a1.z; av[TM - 1] = a1.w;
        } else if (TM == 6) {
          const float2 a1 = *reinterpret_cast<const float2*>(&As[buf][kk][64 + ty * 2]);
          av[TM - 2] = a1.x; av[TM - 1] = a1.y;
        }
      }
      unsigned long long bv[TN / 2];
#pragma unroll
      for (int g = 0; g < TN / 4; ++g) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&Bs[buf][kk][64 * g + tx * 4]);
        bv[2 * g] = v.x;
        bv[2 * g + 1] = v.y;
      }
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const unsigned long long a2 = dup2(av[i]);
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = fma2(a2, bv[j], acc[i][j]);
      }
    }
    if (kt + 1 < nk) sstore(buf ^ 1);
    __syncthreads();
  }
  // the tiled layout's last block is written whole: columns past N get zeros
  const long long nw = kTiled ? (((long long)N + 31) & ~31LL) : N;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const long long m = m0 + (i < 4 ? ty * 4 + i : 64 + ty * (TM - 4) + (i - 4));
    if (m >= M) continue;
#pragma unroll
    for (int h = 0; h < TN / 4; ++h) {
      const long long n = n0 + h * 64 + tx * 4;
      float* dst = kTiled ? Cm + (((n >> 5) * M + m) << 5) + (n & 31) : Cm + m * ldc + n;
      float v[4];
#pragma unroll
      for (int e = 0; e < 4; e += 2) {
        float lo, hi;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(acc[i][h * 2 + e / 2]));
        v[e] = n + e < N ? lo : 0.f;
        v[e + 1] = n + e + 1 < N ? hi : 0.f;
      }
      if (n + 3 < nw && ((reinterpret_cast<uintptr_t>(dst) & 15) == 0)) {
        *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
        for (int e = 0; e < 4; ++e)
          if (n + e < nw) dst[e] = v[e];
      }
    }
  }
}

// Rows per tile: the height that covers M with the least work, a row of a lower
// tile counted a little dearer (its loads serve fewer rows); the operand is
// padded to 128 rows, which the tiles must not pass.
static int sgemm_rows(int64_t M) {
  const int64_t padded = round_up(M, 128);
  int best = 128;
  int64_t cost = padded * 100;
  const int rows[2] = {96, 64}, weight[2] = {104, 112};
  for (int i = 0; i < 2; ++i) {
    const int64_t r = round_up(M, rows[i]);
    if (r <= padded && r * weight[i] < cost) {
      cost = r * weight[i];
      best = rows[i];
    }
  }
  return best;
}

template <int TM, int TN>
static int launch_sgemm(const float* A, const float* Bt, float* Cm, int64_t M, int64_t N,
                        int64_t Kd, int64_t ldc, cudaStream_t stream, bool tiled,
                        bool upper) {
  const int tiles_m = (int)((M + 16 * TM - 1) / (16 * TM));
  const int tiles_n = (int)((N + 16 * TN - 1) / (16 * TN));
  const long long nblocks = (long long)tiles_m * tiles_n;
  if (nblocks > 0x7fffffffLL) return fail(KS_ERR_UNSUPPORTED, "sgemm_tn: too many tiles");
  const size_t smem = sizeof(float) * 2 * sgemm_slice(TN) * (16 * TM + 4 + 16 * TN + 4);
  const auto kernel = tiled ? ks_sgemm_tn_kernel<TM, TN, true> : ks_sgemm_tn_kernel<TM, TN, false>;
  kernel<<<(unsigned)nblocks, 256, smem, stream>>>(A, Bt, Cm, (int)M, (int)N, (int)Kd, ldc, tiles_m,
                                               upper);
  KS_CUDA(cudaGetLastError());
  return KS_OK;
}

int sgemm_tn(const float* A, const float* Bt, float* Cm, int64_t M, int64_t N,
             int64_t Kd, int64_t ldc, cudaStream_t stream, bool tiled, bool upper) {
  if (Kd % 16) return fail(KS_ERR_ARG, "sgemm_tn: Kd must be a multiple of 16");
  DeviceInfo dev;
  const int rc = device_info(&dev);
  if (rc) return rc;
  const int rows = sgemm_rows(M);
  // 256 columns by 128 rows need fewer shared-memory reads per multiply-add, one
  // block per SM; with fewer than 2.5 tiles per SM their last wave costs more than
  // that (80 x 60122 x 576: 249 us with 256 columns, 192 with 128; 3600 x 3600 x
  // 384: 197 and 219).  96 rows by 256 columns took longer for a wave than 128 rows
  // (464 and 400 us at a depth of 2304), so that height is for 128 columns only.
  const int64_t wide = ((M + 127) / 128) * ((N + 255) / 256);
  if (2 * wide >= 5 * dev.sm_count && rows != 64)
    return launch_sgemm<8, 16>(A, Bt, Cm, M, N, Kd, ldc, stream, tiled, upper);
  switch (rows) {
    case 64: return launch_sgemm<4, 8>(A, Bt, Cm, M, N, Kd, ldc, stream, tiled, upper);
    case 96: return launch_sgemm<6, 8>(A, Bt, Cm, M, N, Kd, ldc, stream, tiled, upper);
    default: return launch_sgemm<8, 8>(A, Bt, Cm, M, N, Kd, ldc, stream, tiled, upper);
  }
}

// ------------------------------------------------------------------ driver
ProjLayout proj_layout(int64_t C, int64_t L, int64_t K, int64_t P, int precision) {
  ProjLayout l;
  l.Q = round_up(round_up(C, kCG) * P, 64);
  l.Lpad = round_up(L, 128);
  l.Kpad = round_up(K, 128);
  Carve cv(nullptr);
  cv.take<int>(64);   // error word
  if (precision == KS_PROJ_FP32) {
    cv.take<float>((size_t)l.Kpad * l.Q);
    cv.take<float>((size_t)l.Lpad * l.Q);
  } else {
    cv.take<__nv_bfloat16>((size_t)l.Kpad * l.Q * 2);
    cv.take<__nv_bfloat16>((size_t)l.Lpad * l.Q * 2);
  }
  l.bytes = cv.used;
  return l;
}

int launch_template_energy(const float* U, int64_t K, int64_t P, int64_t C,
                           float* nm, cudaStream_t stream) {
  if (!U || !nm || K < 1 || P < 1 || C < 1) return fail(KS_ERR_ARG, "template_energy: bad args");
  const int threads = 256;
  const long long blocks = (K * 32 + threads - 1) / threads;
  ks_template_energy_kernel<<<(unsigned)blocks, threads, 0, stream>>>(U, (int)K, (int)P, (int)C, nm);
  KS_CUDA(cudaGetLastError());
  return KS_OK;
}

int launch_reorder_templates(const float* U, int64_t K, int64_t P, int64_t C, int64_t Kpad,
                             int64_t Q, float* Uf, __nv_bfloat16* Uhi, __nv_bfloat16* Ulo,
                             cudaStream_t stream) {
  const int blocks = (int)std::min<int64_t>(4096, (Kpad * Q + 255) / 256);
  ks_reorder_templates_kernel<<<blocks, 256, 0, stream>>>(U, (int)K, (int)P, (int)C, (int)Kpad,
                                                          (int)Q, Uf, Uhi, Ulo);
  KS_CUDA(cudaGetLastError());
  return KS_OK;
}

static int launch_temporal_simt(const float* X, const float* W, int64_t C, int64_t L,
                                int64_t P, int64_t nt, int64_t Q, int64_t Lpad, float* Yf,
                                __nv_bfloat16* Yhi, __nv_bfloat16* Ylo, float* YT,
                                int64_t ldyt, cudaStream_t stream) {
  const size_t smem = temporal_smem((int)nt, (int)P);
  const int tiles_t = (int)(Lpad / kTT);
  const long long n_tiles = (long long)tiles_t * ((C + kCG - 1) / kCG);
  if (n_tiles > 0x7fffffffLL) return fail(KS_ERR_UNSUPPORTED, "project: too many temporal tiles");
  DeviceInfo dev;
  int drc = device_info(&dev);
  if (drc) return drc;
  // persistent: as many blocks as are resident at once
  int occ = 0;
#define KS_TEMPORAL_CASE(PPV)                                                              \
  case PPV: {                                                                              \
    KS_CUDA(cudaFuncSetAttribute(ks_temporal_kernel<PPV>,                                  \
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
    KS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, ks_temporal_kernel<PPV>,   \
                                                          kTemporalThreads, smem));        \
    const unsigned grid =                                                                  \
        (unsigned)std::min<long long>(n_tiles, (long long)std::max(occ, 1) * dev.sm_count); \
    ks_temporal_kernel<PPV><<<grid, kTemporalThreads, smem, stream>>>(                     \
        X, W, (int)C, (int)L, (int)nt,                                                     \
                                                         (int)Q, tiles_t, (int)n_tiles,    \
                                                         Yf, Yhi, Ylo, YT, ldyt);          \
    break;                                                                                 \
  }
  switch (P) {
    KS_TEMPORAL_CASE(1)
    KS_TEMPORAL_CASE(2)
    KS_TEMPORAL_CASE(3)
    KS_TEMPORAL_CASE(4)
    KS_TEMPORAL_CASE(5)
    KS_TEMPORAL_CASE(6)
    KS_TEMPORAL_CASE(7)
    KS_TEMPORAL_CASE(8)
    default:
      return fail(KS_ERR_UNSUPPORTED, "project: n_pcs must be 1..8");
  }
#undef KS_TEMPORAL_CASE
  KS_CUDA(cudaGetLastError());
  return KS_OK;
}

int launch_temporal_rows(const float* X, const float* W, int64_t C, int64_t L, int64_t P,
                         int64_t nt, int64_t Lpad, float* YT, int64_t ldyt,
                         cudaStream_t stream) {
  if (Lpad % kTT || ldyt < Lpad || ldyt % 4 || (reinterpret_cast<uintptr_t>(YT) & 15))
    return fail(KS_ERR_ARG, "temporal rows: Lpad % 128, ldyt >= Lpad, 16-byte rows");
  return launch_temporal_simt(X, W, C, L, P, nt, round_up(round_up(C, kCG) * P, 64), Lpad,
                              nullptr, nullptr, nullptr, YT, ldyt, stream);
}

int launch_temporal(const float* X, const float* W, int64_t C, int64_t L,
                    int64_t P, int64_t nt, int64_t Q, int64_t Lpad, float* Yf,
                    __nv_bfloat16* Yhi, __nv_bfloat16* Ylo, int* err, cudaStream_t stream) {
  if (Yhi && Ylo && !Yf && err) {
    const int rc = launch_temporal_split_tc(X, W, C, L, P, nt, Q, Lpad, Yhi, Ylo, err, stream);
    if (rc == KS_OK) return zero_q_padding(C, P, Q, Lpad, Yf, Yhi, Ylo, stream);
    if (rc != KS_ERR_UNSUPPORTED) return rc;
  }
  const int rc = launch_temporal_simt(X, W, C, L, P, nt, Q, Lpad, Yf, Yhi, Ylo, nullptr, 0,
                                      stream);
  if (rc) return rc;
  return zero_q_padding(C, P, Q, Lpad, Yf, Yhi, Ylo, stream);
}

// q columns past the last group of 16 channels are padding: zero them.
int zero_q_padding(int64_t C, int64_t P, int64_t Q, int64_t Lpad, float* Yf, __nv_bfloat16* Yhi,
                   __nv_bfloat16* Ylo, cudaStream_t stream) {
  const int64_t qused = round_up(C, kCG) * P;
  if (qused < Q) {
    if (Yf) KS_CUDA(cudaMemset2DAsync(Yf + qused, Q * sizeof(float), 0, (Q - qused) * sizeof(float), Lpad, stream));
    if (Yhi) {
      KS_CUDA(cudaMemset2DAsync(Yhi + qused, Q * 2, 0, (Q - qused) * 2, Lpad, stream));
      KS_CUDA(cudaMemset2DAsync(Ylo + qused, Q * 2, 0, (Q - qused) * 2, Lpad, stream));
    }
  }
  return KS_OK;
}


int launch_project(const float* X, const float* U, const float* W, int64_t C,
                   int64_t L, int64_t K, int64_t P, int64_t nt, int precision,
                   float* B, int64_t ldb, bool tiled, void* ws, size_t ws_bytes,
                   int* err_out, cudaStream_t stream) {
  if (!X || !U || !W || !B) return fail(KS_ERR_ARG, "ks_project: null pointer");
  if (C < 1 || L < 1 || K < 1 || P < 1 || nt < 1 || (nt % 2) == 0)
    return fail(KS_ERR_ARG, "ks_project: need C,L,K,P >= 1 and odd nt");
  if (P > kPMax) return fail(KS_ERR_UNSUPPORTED, "ks_project: n_pcs must be <= 8");
  if (nt > 1023) return fail(KS_ERR_UNSUPPORTED, "ks_project: nt must be <= 1023");
  if (!tiled && ldb < L) return fail(KS_ERR_ARG, "ks_project: ldb < L");
  if (precision != KS_PROJ_FP32 && precision != KS_PROJ_BF16X3)
    return fail(KS_ERR_ARG, "ks_project: unknown precision");
  const ProjLayout lay = proj_layout(C, L, K, P, precision);
  if (!ws || ws_bytes < lay.bytes) return fail(KS_ERR_WORKSPACE, "ks_project: workspace too small");
  Carve cv(ws);
  int* err = cv.take<int>(64);
  KS_CUDA(cudaMemsetAsync(err, 0, sizeof(int), stream));
  const int reorder_blocks = (int)std::min<int64_t>(4096, (lay.Kpad * lay.Q + 255) / 256);
  if (precision == KS_PROJ_FP32) {
    float* Uq = cv.take<float>((size_t)lay.Kpad * lay.Q);
    float* Yt = cv.take<float>((size_t)lay.Lpad * lay.Q);
    ks_reorder_templates_kernel<<<reorder_blocks, 256, 0, stream>>>(
        U, (int)K, (int)P, (int)C, (int)lay.Kpad, (int)lay.Q, Uq, nullptr, nullptr);
    KS_CUDA(cudaGetLastError());
    int rc = launch_temporal(X, W, C, L, P, nt, lay.Q, lay.Lpad, Yt, nullptr, nullptr, nullptr, stream);
    if (rc) return rc;
    rc = sgemm_tn(Uq, Yt, B, K, L, lay.Q, ldb, stream, tiled);
    if (rc) return rc;
    if (err_out) KS_CUDA(cudaMemcpyAsync(err_out, err, sizeof(int), cudaMemcpyDeviceToDevice, stream));
    return KS_OK;
  }
  __nv_bfloat16* Uhl = cv.take<__nv_bfloat16>((size_t)lay.Kpad * lay.Q * 2);
  __nv_bfloat16* Yhl = cv.take<__nv_bfloat16>((size_t)lay.Lpad * lay.Q * 2);
  __nv_bfloat16* Uhi = Uhl;
  __nv_bfloat16* Ulo = Uhl + (size_t)lay.Kpad * lay.Q;
  __nv_bfloat16* Yhi = Yhl;
  __nv_bfloat16* Ylo = Yhl + (size_t)lay.Lpad * lay.Q;
  ks_reorder_templates_kernel<<<reorder_blocks, 256, 0, stream>>>(
      U, (int)K, (int)P, (int)C, (int)lay.Kpad, (int)lay.Q, nullptr, Uhi, Ulo);
  KS_CUDA(cudaGetLastError());
  int rc = launch_temporal(X, W, C, L, P, nt, lay.Q, lay.Lpad, nullptr, Yhi, Ylo, err, stream);
  if (rc) return rc;
  rc = gemm_bf16x3(Uhi, Ulo, Yhi, Ylo, B, K, L, lay.Q, lay.Kpad, lay.Lpad, ldb, tiled, err, stream);
  if (rc) return rc;
  if (err_out) KS_CUDA(cudaMemcpyAsync(err_out, err, sizeof(int), cudaMemcpyDeviceToDevice, stream));
  return KS_OK;
}

}  // namespace ks
