// Universal-template spike detection on the device, kilosort/spikedetect.py:133-197
// (template_match and yweighted) plus the PC features of run() (:265-266).
//
//   B[c, k, t]  = conv1d(X[c], wTEMP[k]) (padding nt/2)          FP32 temporal kernel, rows (c, k)
//   A[s, k]     = sum_j weigh[s, j, f] * B[iC[j, f], k, t]       per position f and sample t
//   As[f, t]    = max |A|,  imax[f, t] = (1 + argmax) * sign(A[argmax])   (index s*nk + k)
//   Amax[f, t]  = max over the nC2 nearest positions iC2[:, f] of As     (0 for t < nt, t >= L-nt)
//   peak        = maxpool_{+-nt0}(Amax)[f, t] == As[f, t] and As[f, t] > Th_universal
//   spikes in (f, t) order; adist[j] = B[iC[j, f], |imax|-1 mod nk, t] * sign(imax);
//   y = sum_j relu(adist_j)/sum relu(adist) * yc[iC[j, f]];
//   tF[s, j, p] = sum_u X[iC[j, f], t - nt/2 + u] * wPCA[p, u]
//
// Kernels: ks_detect_scores_tiled_kernel (a block per tile of 32 positions,
// persistent over 32-sample time tiles: the union of the positions' nearest
// channels is staged, double-buffered by cp.async, the (s, k) sums of one
// position per half warp, two samples per lane, in registers; A is never stored;
// ks_detect_scores_kernel is the form for more than 8192 channels),
// ks_detect_peaks_kernel (a block per (f, 1024-sample tile): only where the
// score exceeds the threshold and both samples beside it, the maximum over the
// neighbour rows and the +-nt0 window by a warp, left at the first larger
// value),
// count / scan / emit in (f, t) order, and one gather
// kernel per spike (adist, y) and per (spike, channel) warp (features).
#include "ks_common.cuh"
#include "project.cuh"
#include "residual_apply.cuh"

#include <algorithm>
#include <cmath>

namespace {

constexpr int kMaxNK = 8;        // universal waveforms
constexpr int kMaxNS = 8;        // template sizes
constexpr int kMaxNC = 32;       // nearest channels
constexpr int kTile = 256;       // samples per block
constexpr int kChunkWords = 32;  // peak-bit words per counting chunk (1024 samples)

__global__ void __launch_bounds__(kTile)
ks_detect_scores_kernel(const float* __restrict__ BT, long long ldb, int nk, int C,
                        const long long* __restrict__ iC, int nC,
                        const float* __restrict__ weigh, int ns, int Nfilt, int L,
                        float* __restrict__ As, signed char* __restrict__ imaxs, int* err) {
  __shared__ int sc[kMaxNC];
  __shared__ float sw[kMaxNS * kMaxNC];
  const int f = blockIdx.x;
  const int t = blockIdx.y * kTile + threadIdx.x;
  for (int j = threadIdx.x; j < nC; j += kTile) {
    long long c = iC[(long long)j * Nfilt + f];
    if (c < 0 || c >= C) {
      atomicCAS(err, 0, KS_ERR_ARG);   // reported; channel 0 stands in
      c = 0;
    }
    sc[j] = (int)c;
  }
  for (int e = threadIdx.x; e < ns * nC; e += kTile) {
    const int s = e / nC, j = e - s * nC;
    sw[e] = weigh[((long long)s * nC + j) * Nfilt + f];
  }
  __syncthreads();
  if (t >= L) return;
  float a[kMaxNS][kMaxNK];
#pragma unroll
  for (int s = 0; s < kMaxNS; ++s)
#pragma unroll
    for (int k = 0; k < kMaxNK; ++k) a[s][k] = 0.f;
  for (int j = 0; j < nC; ++j) {
    const float* b = BT + (long long)sc[j] * nk * ldb + t;
    float bk[kMaxNK];
#pragma unroll
    for (int k = 0; k < kMaxNK; ++k) bk[k] = k < nk ? __ldg(b + (long long)k * ldb) : 0.f;
#pragma unroll
    for (int s = 0; s < kMaxNS; ++s) {
      if (s < ns) {
        const float w = sw[s * nC + j];
#pragma unroll
        for (int k = 0; k < kMaxNK; ++k)
          if (k < nk) a[s][k] = fmaf(w, bk[k], a[s][k]);
      }
    }
  }
  // largest magnitude, first index in (s, k) order
  float best = -1.f, bval = 0.f;
  int bidx = 0;
#pragma unroll
  for (int s = 0; s < kMaxNS; ++s)
#pragma unroll
    for (int k = 0; k < kMaxNK; ++k)
      if (s < ns && k < nk) {
        const float m = fabsf(a[s][k]);
        if (m > best) {
          best = m;
          bval = a[s][k];
          bidx = s * nk + k;
        }
      }
  const int sg = bval > 0.f ? 1 : (bval < 0.f ? -1 : 0);
  As[(long long)f * L + t] = best;
  imaxs[(long long)f * L + t] = (signed char)((1 + bidx) * sg);
}

// The same sums for a tile of kFT consecutive positions x kTT samples: the
// block first collects the union of its positions' nearest channels (a
// bitmap over channels, compacted in channel order), stages those channels'
// convolution rows for its samples in shared memory, then each warp computes
// one position over 32 consecutive samples per round.  A tile whose union
// exceeds kMaxU channels reads its rows from global memory instead.
constexpr int kFT = 32;          // positions per block
constexpr int kTT = 32;          // samples per time tile
constexpr int kMaxU = 48;        // staged channels
constexpr int kMaxCBits = 8192;  // channels covered by the bitmap

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait1() {
  asm volatile("cp.async.wait_group 1;" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait0() {
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// The largest magnitude of the sums a[size][waveform] of one sample (half h of
// the packed pairs; -1 when all are NaN) and its signed index
// (1 + size * nk + waveform) * sign, the first index on ties: the maximum of
// each size (NaNs passed over), the first size that holds the largest, then its
// first waveform.
template <int NS, int NK>
__device__ __forceinline__ int largest_magnitude(const unsigned long long (&a)[NS][NK], bool h,
                                                 int ns, int nk, float& best) {
  auto val = [&](int q, int k) {
    float lo, hi;
    f2_unpack(a[q][k], lo, hi);
    return h ? hi : lo;
  };
  float mq[NS];
  best = -1.f;
#pragma unroll
  for (int q = 0; q < NS; ++q) {
    float m = fabsf(val(q, 0));
#pragma unroll
    for (int k = 1; k < NK; k += 2) {
      if (k + 1 < NK && k + 1 < nk)
        asm("max.f32 %0, %0, %1, %2;" : "+f"(m) : "f"(fabsf(val(q, k))), "f"(fabsf(val(q, k + 1 < NK ? k + 1 : k))));
      else if (k < nk)
        m = fmaxf(m, fabsf(val(q, k)));
    }
    mq[q] = m;
    if (q < ns) best = fmaxf(best, m);
  }
  float v[NK], x = 0.f;
  int qs = 0, ks = 0;
#pragma unroll
  for (int k = 0; k < NK; ++k) v[k] = 0.f;
#pragma unroll
  for (int q = NS - 1; q >= 0; --q) {
    const bool p = q < ns && mq[q] == best;
    qs = p ? q : qs;
#pragma unroll
    for (int k = 0; k < NK; ++k) v[k] = p ? val(q, k) : v[k];
  }
#pragma unroll
  for (int k = NK - 1; k >= 0; --k) {
    const bool p = k < nk && fabsf(v[k]) == best;
    ks = p ? k : ks;
    x = p ? v[k] : x;
  }
  const int idx = 1 + qs * nk + ks;
  return x > 0.f ? idx : (x < 0.f ? -idx : 0);
}

// Persistent over time: block (position tile, y) takes the time tiles y,
// y + gridDim.y, ...; the union of its positions' channels and their weights
// are set up once, and the channels' convolution rows of the next time tile
// are copied (cp.async, 16-byte pieces) while the current one is summed.
//
// What bounds it: the FP32 pipe and issue.  Two samples per lane through packed
// multiply-adds (the weights held twice): 2.14 ms per C=384 batch of 60122
// samples and 1532 positions; with one sample per lane 2.89 ms, with the channel
// count not known at compile time 2.45 ms.
template <int NS, int NK, int NCT>
__global__ void __launch_bounds__(256)
ks_detect_scores_tiled_kernel(const float* __restrict__ BT, long long ldb, int nk_rt, int C,
                              const long long* __restrict__ iC, int nC_rt,
                              const float* __restrict__ weigh, int ns_rt, int Nfilt, int L,
                              int n_ttiles, float* __restrict__ As,
                              signed char* __restrict__ imaxs, int* err) {
  // NS, NK: compile-time bounds of the sizes and waveforms; ns_rt, nk_rt the
  // actual counts (equal to the bounds in the specialised instantiations); NCT:
  // the nearest channels where they are known at compile time, else 0
  extern __shared__ __align__(16) float sm[];
  const int nC = NCT ? NCT : nC_rt;
  float* sB = sm;                                                // [2][kMaxU][NK][kTT]
  constexpr int kWS = (NS + 1) & ~1;                             // sizes, padded to pairs
  unsigned long long* sw = reinterpret_cast<unsigned long long*>(sB + 2 * kMaxU * NK * kTT);
                                                                 // [kFT][nC][kWS], each twice
  unsigned* bitmap = reinterpret_cast<unsigned*>(sw + kFT * kWS * nC);  // [kMaxCBits / 32]
  int* wpre = reinterpret_cast<int*>(bitmap + kMaxCBits / 32);   // [kMaxCBits / 32]
  int* ulist = wpre + kMaxCBits / 32;                            // [kMaxU]
  int* cidx = ulist + kMaxU;                                     // [kMaxNC][kFT] channel
  int* loc = cidx + kMaxNC * kFT;                                // [kMaxNC][kFT] its rows' offset
  __shared__ int nU;
  const int ns = NS == kMaxNS ? ns_rt : NS;
  const int nk = NK == kMaxNK ? nk_rt : NK;
  const int f0 = blockIdx.x * kFT;
  const int nwc = (C + 31) >> 5;
  for (int w = threadIdx.x; w < nwc; w += blockDim.x) bitmap[w] = 0u;
  __syncthreads();
  for (int e = threadIdx.x; e < nC * kFT; e += blockDim.x) {
    const int j = e / kFT, fl = e % kFT;
    const int f = f0 + fl;
    int c = 0;
    if (f < Nfilt) {
      const long long cc = iC[(long long)j * Nfilt + f];
      if (cc < 0 || cc >= C) atomicCAS(err, 0, KS_ERR_ARG);   // channel 0 stands in
      else c = (int)cc;
    }
    cidx[e] = c;
    atomicOr(bitmap + (c >> 5), 1u << (c & 31));
  }
  // weights [fl][j][q] (zero for missing sizes and positions)
  for (int e = threadIdx.x; e < kFT * nC * kWS; e += blockDim.x) {
    const int fl = e / (nC * kWS), r = e - fl * nC * kWS, j = r / kWS, q = r % kWS;
    const int f = f0 + fl;
    const float v = (f < Nfilt && q < ns) ? weigh[((long long)q * nC + j) * Nfilt + f] : 0.f;
    sw[e] = f2_pack(v, v);
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    // exclusive prefix of the bitmap words' population counts
    int run = 0;
    for (int w0 = 0; w0 < nwc; w0 += 32) {
      const int w = w0 + threadIdx.x;
      const int cnt = w < nwc ? __popc(bitmap[w]) : 0;
      int incl = cnt;
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if ((int)threadIdx.x >= o) incl += v;
      }
      if (w < nwc) wpre[w] = run + incl - cnt;
      run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (threadIdx.x == 0) nU = run;
  }
  __syncthreads();
  const bool staged = nU <= kMaxU;
  for (int e = threadIdx.x; e < nC * kFT; e += blockDim.x) {
    const int c = cidx[e];
    const int u = wpre[c >> 5] + __popc(bitmap[c >> 5] & ((1u << (c & 31)) - 1u));
    loc[e] = u * NK * kTT;
    if (staged) ulist[u] = c;
  }
  __syncthreads();
  // rows (u, k) of a time tile: kTT floats = kTT/4 16-byte pieces each
  auto fetch = [&](int tt, int buf) {
    if (staged) {
      const int n = nU * nk * (kTT / 4);
      float* dst = sB + buf * kMaxU * NK * kTT;
      for (int e = threadIdx.x; e < n; e += blockDim.x) {
        const int row = e / (kTT / 4), piece = e % (kTT / 4);
        const int u = row / nk, k = row % nk;
        cp_async16(dst + (u * NK + k) * kTT + piece * 4,
                   BT + ((long long)ulist[u] * nk + k) * ldb + (long long)tt * kTT + piece * 4);
      }
    }
    cp_async_commit();
  };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int buf = 0;
  if ((int)blockIdx.y < n_ttiles) fetch(blockIdx.y, 0);
  for (int tt = blockIdx.y; tt < n_ttiles; tt += gridDim.y) {
    const int next = tt + gridDim.y;
    if (next < n_ttiles) fetch(next, buf ^ 1);
    else cp_async_commit();
    cp_async_wait1();
    __syncthreads();
    const float* cur = sB + buf * kMaxU * NK * kTT + 2 * (lane & 15);
    // half a warp per position, two samples per lane
    const int t = tt * kTT + 2 * (lane & 15);
    for (int fl = 2 * warp + (lane >> 4); fl < kFT; fl += 16) {
      const int f = f0 + fl;
      unsigned long long a[NS][NK];
#pragma unroll
      for (int q = 0; q < NS; ++q)
#pragma unroll
        for (int k = 0; k < NK; ++k) a[q][k] = 0ull;
#pragma unroll (NCT ? NCT : 1)
      for (int j = 0; j < nC; ++j) {
        unsigned long long bk[NK];
        if (staged) {
          const float* b = cur + loc[j * kFT + fl];
#pragma unroll
          for (int k = 0; k < NK; ++k) bk[k] = *reinterpret_cast<const unsigned long long*>(b + k * kTT);
        } else {
          const float* b = BT + (long long)cidx[j * kFT + fl] * nk * ldb + t;
#pragma unroll
          for (int k = 0; k < NK; ++k)
            bk[k] = k < nk ? __ldg(reinterpret_cast<const unsigned long long*>(b + (long long)k * ldb))
                           : 0ull;
        }
        const unsigned long long* w = sw + (fl * nC + j) * kWS;
#pragma unroll
        for (int q = 0; q < NS; q += 2) {
          const ulonglong2 wq = *reinterpret_cast<const ulonglong2*>(w + q);
#pragma unroll
          for (int k = 0; k < NK; ++k) {
            f2_fma_acc(a[q][k], wq.x, bk[k]);
            if (q + 1 < NS) f2_fma_acc(a[q + 1][k], wq.y, bk[k]);
          }
        }
      }
      float best0, best1;
      const int i0 = largest_magnitude<NS, NK>(a, false, ns, nk, best0);
      const int i1 = largest_magnitude<NS, NK>(a, true, ns, nk, best1);
      if (f < Nfilt) {
        const long long o = (long long)f * L + t;
        if (t + 1 < L && (o & 1) == 0) {
          *reinterpret_cast<float2*>(As + o) = make_float2(best0, best1);
          *reinterpret_cast<char2*>(imaxs + o) = make_char2((signed char)i0, (signed char)i1);
        } else {
          if (t < L) {
            As[o] = best0;
            imaxs[o] = (signed char)i0;
          }
          if (t + 1 < L) {
            As[o + 1] = best1;
            imaxs[o + 1] = (signed char)i1;
          }
        }
      }
    }
    __syncthreads();          // the buffer is read: the next fetch may reuse it
    buf ^= 1;
  }
  cp_async_wait0();
}

size_t scores_tiled_smem(int NK, int NS, int nC) {
  return sizeof(unsigned) * (kMaxCBits / 32) * 2 + sizeof(int) * (kMaxU + 2 * kMaxNC * kFT) +
         sizeof(float) * (2 * (size_t)kFT * ((NS + 1) & ~1) * nC + 2 * (size_t)kMaxU * NK * kTT);
}

template <int NS, int NK, int NCT>
int launch_scores_tiled(const float* BT, long long ldb, int nk, int C, const long long* iC,
                        int nC, const float* weigh, int ns, int Nfilt, int L, float* As,
                        signed char* ims, int* err, cudaStream_t s) {
  const size_t smem = scores_tiled_smem(NK, NS, nC);
  KS_CUDA(cudaFuncSetAttribute(ks_detect_scores_tiled_kernel<NS, NK, NCT>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  ks::DeviceInfo dev;
  int rc = ks::device_info(&dev);
  if (rc) return rc;
  int occ = 0;
  KS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, ks_detect_scores_tiled_kernel<NS, NK, NCT>,
                                                        256, smem));
  const int ftiles = (Nfilt + kFT - 1) / kFT;
  const int n_ttiles = (L + kTT - 1) / kTT;
  // about one wave of resident blocks, each walking its share of the time tiles
  const int gy = std::max(1, std::min(n_ttiles, std::max(occ, 1) * dev.sm_count / ftiles));
  const dim3 grid((unsigned)ftiles, (unsigned)gy);
  ks_detect_scores_tiled_kernel<NS, NK, NCT><<<grid, 256, smem, s>>>(BT, ldb, nk, C, iC, nC, weigh,
                                                                ns, Nfilt, L, n_ttiles, As, ims,
                                                                err);
  KS_CUDA(cudaGetLastError());
  return KS_OK;
}

// Peak test, one block per (position f, 1024 samples).  The reference's test,
// pooled == As[f, t] && As[f, t] > th with pooled the max-pool over +-nt0 of
// the neighbour maximum (0 at the batch edges), needs the neighbour maximum
// only where As[f, t] > th and, when f is one of its own neighbours (the nearest
// position), neither sample beside it in its own row is larger.  Those
// survivors are collected, and a warp walks the rows of one at a time, its own
// row first, a lane per sample, stopping after the rows that lift the running
// maximum above As[f, t].  Where the samples beside it say nothing (nt0 = 0, or f
// not among its neighbours) every thread walks its own sample's rows, most of
// which end at the first.  Maxima are exact, so the order of the walk does not
// matter.
//
// What bounds it: reading As once (368 MB at C=384, 1532 positions, 60122
// samples) and the survivors' walks: 660 us; with every sample above the
// threshold walking the rows in its own thread 1755 us, with one row of a
// survivor in flight at a time 1290 us, with a position's tiles one after the
// other in one block 1900 us.  At nt0 = 0 and C=64 the whole detection takes 577 us
// by threads, 685 with a warp per sample above the threshold.
constexpr int kPeakTile = 1024;
constexpr int kPeakHalo = 512;   // staged beside the tile; a wider window's own row is read
                                 // from global memory
__global__ void __launch_bounds__(256)
ks_detect_peaks_kernel(const float* __restrict__ As, const long long* __restrict__ iC2,
                       int nC2, int Nfilt, int L, int nt, int nt0, float th,
                       unsigned* __restrict__ bits, int nwords) {
  extern __shared__ float sm[];
  const int halo = nt0 <= kPeakHalo ? nt0 : 0;
  float* row = sm;                                           // [kPeakTile + 2 halo]
  int* snb = reinterpret_cast<int*>(row + kPeakTile + 2 * halo);  // [nC2]
  __shared__ int list[kPeakTile];
  __shared__ unsigned sbits[kPeakTile / 32];
  __shared__ int nlist, taken, self;
  const int f = blockIdx.x;
  const int lane = threadIdx.x & 31;
  const int t0 = blockIdx.y * kPeakTile;
  if (threadIdx.x < kPeakTile / 32) sbits[threadIdx.x] = 0u;
  if (threadIdx.x == 0) nlist = taken = self = 0;
  // neighbour values exist for samples nt .. L-nt-1 only (0 elsewhere)
  const float* own = As + (long long)f * L;
  bool any = false;
  for (int i = threadIdx.x; i < kPeakTile + 2 * halo; i += 256) {
    const int t = t0 - halo + i;
    const bool in = t >= 0 && t < L;
    const float v = in ? own[t] : 0.f;
    row[i] = v;
    any |= in && i >= halo && i < halo + kPeakTile && v > th;
  }
  if (__syncthreads_or(any)) {
    for (int j = threadIdx.x; j < nC2; j += 256) {
      const long long g = iC2[(long long)j * Nfilt + f];
      const int n = (int)(g < 0 ? f : (g >= Nfilt ? f : g));
      snb[j] = n;
      if (n == f) self = 1;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kPeakTile; i += 256) {
      const int t = t0 + i;
      const float a = row[halo + i];
      bool keep = t < L && a > th;
      const int lo = max(t - nt0, nt), hi = min(t + nt0, L - nt - 1);
      if (!self || nt0 == 0) {
        // nothing to tell survivors by
        float m = 0.f;
        for (int j = 0; keep && j < nC2 && !(m > a); ++j) {
          const float* p = As + (long long)snb[j] * L;
          for (int u = lo; u <= hi; ++u) m = fmaxf(m, p[u]);
        }
        const unsigned b = __ballot_sync(0xffffffffu, keep && m == a);
        if (lane == 0) sbits[i >> 5] = b;
        continue;
      }
      if (keep && halo > 0) {
        keep = !(t - 1 >= lo && t - 1 <= hi && row[halo + i - 1] > a) &&
               !(t + 1 <= hi && t + 1 >= lo && row[halo + i + 1] > a);
      }
      const unsigned b = __ballot_sync(0xffffffffu, keep);
      if (b) {
        int o = 0;
        if (lane == 0) o = atomicAdd(&nlist, __popc(b));
        o = __shfl_sync(0xffffffffu, o, 0);
        if (keep) list[o + __popc(b & ((1u << lane) - 1u))] = i;
      }
    }
    __syncthreads();
    while (true) {
      int e = 0;
      if (lane == 0) e = atomicAdd(&taken, 1);
      e = __shfl_sync(0xffffffffu, e, 0);
      if (e >= nlist) break;
      const int i = list[e], t = t0 + i;
      const float a = row[halo + i];
      const int lo = max(t - nt0, nt), n = min(t + nt0, L - nt - 1) - lo + 1;
      float m = 0.f;                    // the lane's maximum
      bool over = false;
      if (self && halo == nt0) {        // the position's own row, staged
        const float* p = row + (lo - t0 + halo);
        for (int u = lane; u < n; u += 32) m = fmaxf(m, p[u]);
        over = __any_sync(0xffffffffu, m > a);
      }
      // four rows' windows (up to 64 samples each at a time) in flight together
      for (int j = 0; j < nC2 && !over; j += 4) {
        for (int u = lane; u - lane < n; u += 64) {
          float v[8];
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const float* p = As + (long long)snb[min(j + r, nC2 - 1)] * L + lo;
            v[2 * r] = u < n ? p[u] : 0.f;
            v[2 * r + 1] = u + 32 < n ? p[u + 32] : 0.f;
          }
#pragma unroll
          for (int r = 0; r < 8; ++r) m = fmaxf(m, v[r]);
        }
        over = __any_sync(0xffffffffu, m > a);
      }
      const bool reached = __any_sync(0xffffffffu, m == a);
      if (lane == 0 && !over && reached) atomicOr(&sbits[i >> 5], 1u << (i & 31));
    }
  }
  __syncthreads();
  const int word = (t0 >> 5) + threadIdx.x;
  if (threadIdx.x < kPeakTile / 32 && word < nwords)
    bits[(long long)f * nwords + word] = sbits[threadIdx.x];
}

__global__ void ks_detect_count_kernel(const unsigned* __restrict__ bits, int Nfilt, int nwords,
                                       int nchunks, long long* __restrict__ counts) {
  const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= (long long)Nfilt * nchunks) return;
  const int f = (int)(e / nchunks), ch = (int)(e % nchunks);
  const unsigned* b = bits + (long long)f * nwords;
  int n = 0;
  for (int w = ch * kChunkWords; w < min(nwords, (ch + 1) * kChunkWords); ++w) n += __popc(b[w]);
  counts[e] = n;
}

// Exclusive scan of n counts in place (one block), total in *total: tiles of 8
// values per thread, the next tile's loads in flight while this one is
// scanned (97 us per 90000 counts with one contiguous run per thread).
__global__ void __launch_bounds__(1024)
ks_detect_scan_kernel(long long* __restrict__ counts, long long n, long long* __restrict__ total) {
  __shared__ long long wsum[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  long long v[8];
  auto load = [&](long long i) {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = i + j < n ? counts[i + j] : 0;
  };
  long long carry = 0;
  load(8LL * threadIdx.x);
  for (long long base = 0; base < n; base += 8 * 1024) {
    const long long i = base + 8LL * threadIdx.x;
    long long e[8], run = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      e[j] = run;
      run += v[j];
    }
    load(i + 8 * 1024);
    long long incl = run;
    for (int o = 1; o < 32; o <<= 1) {
      const long long x = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += x;
    }
    __syncthreads();
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    long long w = wsum[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const long long x = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += x;
    }
    const long long prev = __shfl_sync(0xffffffffu, w, max(warp - 1, 0));
    const long long before = carry + incl - run + (warp ? prev : 0);
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (i + j < n) counts[i + j] = before + e[j];
    carry += __shfl_sync(0xffffffffu, w, 31);
  }
  if (threadIdx.x == 0) *total = carry;
}

__global__ void ks_detect_emit_kernel(const unsigned* __restrict__ bits, int Nfilt, int nwords,
                                      int nchunks, const long long* __restrict__ offsets,
                                      long long capacity, long long* __restrict__ xy) {
  const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= (long long)Nfilt * nchunks) return;
  const int f = (int)(e / nchunks), ch = (int)(e % nchunks);
  const unsigned* b = bits + (long long)f * nwords;
  long long o = offsets[e];
  for (int w = ch * kChunkWords; w < min(nwords, (ch + 1) * kChunkWords); ++w) {
    unsigned m = b[w];
    while (m) {
      const int bit = __ffs(m) - 1;
      m &= m - 1;
      if (o < capacity) {
        xy[2 * o] = f;
        xy[2 * o + 1] = (long long)w * 32 + bit;
      }
      ++o;
    }
  }
}

// Per spike: signed index, amplitude, adist over the nearest channels and
// the relu-weighted y position (float32, j in order).
__global__ void ks_detect_gather_kernel(const long long* __restrict__ xy, const long long* __restrict__ n_ptr,
                                        long long capacity, const float* __restrict__ As,
                                        const signed char* __restrict__ imaxs,
                                        const float* __restrict__ BT, long long ldb, int nk, int C,
                                        const long long* __restrict__ iC, int nC, int Nfilt,
                                        int L, const float* __restrict__ yc,
                                        long long* __restrict__ imax, float* __restrict__ amp,
                                        float* __restrict__ adist, float* __restrict__ yct) {
  const long long n = min(*n_ptr, capacity);
  const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (s >= n) return;
  const int f = (int)xy[2 * s];
  const int t = (int)xy[2 * s + 1];
  const int im = imaxs[(long long)f * L + t];
  const int sg = im > 0 ? 1 : (im < 0 ? -1 : 0);
  const int idx = abs(im) - 1;
  imax[s] = idx;
  amp[s] = As[(long long)f * L + t];
  const int k = ((idx % nk) + nk) % nk;
  float rs = 0.f;
  float r[kMaxNC];
#pragma unroll
  for (int j = 0; j < kMaxNC; ++j) {
    r[j] = 0.f;
    if (j < nC) {
      long long c = iC[(long long)j * Nfilt + f];
      if (c < 0 || c >= C) c = 0;
      const float v = BT[((long long)c * nk + k) * ldb + t] * (float)sg;
      adist[(long long)j * capacity + s] = v;
      r[j] = fmaxf(v, 0.f);
      rs = __fadd_rn(rs, r[j]);
    }
  }
  float y = 0.f;
#pragma unroll
  for (int j = 0; j < kMaxNC; ++j)
    if (j < nC) {
      long long c = iC[(long long)j * Nfilt + f];
      if (c < 0 || c >= C) c = 0;
      y = __fadd_rn(y, __fmul_rn(__fdiv_rn(r[j], rs), yc[c]));
    }
  yct[s] = y;
}

// tF[s, j, p] = sum_u X[iC[j, f], t - nt/2 + u] * wPCA[p, u]: one warp per
// (spike, channel), grid-stride over the spikes found.
__global__ void __launch_bounds__(256)
ks_detect_features_kernel(const float* __restrict__ X, int C, int L,
                          const long long* __restrict__ xy, const long long* __restrict__ n_ptr,
                          long long capacity, const long long* __restrict__ iC, int nC,
                          int Nfilt, const float* __restrict__ W, int P, int nt,
                          float* __restrict__ tF) {
  extern __shared__ float sW[];   // [P][nt]
  const long long n = min(*n_ptr, capacity);
  if ((long long)blockIdx.x * 8 >= n * nC) return;     // the whole block has no work
  for (int i = threadIdx.x; i < P * nt; i += blockDim.x) sW[i] = W[i];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (long long e = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; e < n * nC;
       e += ((long long)gridDim.x * blockDim.x) >> 5) {
    const long long s = e / nC;
    const int j = (int)(e - s * nC);
    const int f = (int)xy[2 * s];
    const int t = (int)xy[2 * s + 1];
    long long c = iC[(long long)j * Nfilt + f];
    if (c < 0 || c >= C) c = 0;
    const float* x = X + c * L + (t - nt / 2);
    float part[8];
#pragma unroll
    for (int p = 0; p < 8; ++p) part[p] = 0.f;
    for (int u = lane; u < nt; u += 32) {
      const float xv = x[u];
#pragma unroll
      for (int p = 0; p < 8; ++p)
        if (p < P) part[p] = fmaf(xv, sW[p * nt + u], part[p]);
    }
#pragma unroll
    for (int p = 0; p < 8; ++p) {
      if (p < P) {
        float v = part[p];
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) tF[(s * nC + j) * P + p] = v;
      }
    }
  }
}

__global__ void ks_detect_finish_kernel(const long long* __restrict__ total, long long capacity,
                                        const int* __restrict__ err, long long* __restrict__ info) {
  const long long n = *total;
  const int e = *err;
  info[0] = n < capacity ? n : capacity;
  info[1] = e ? e : (n > capacity ? KS_ERR_OVERFLOW : KS_OK);
  info[2] = 0;
  info[3] = n;
}

struct DetectLayout {
  int64_t Lpad, nwords, nchunks;
  size_t ctl, bt, as, im, bits, counts, bytes;
};

DetectLayout detect_layout(int64_t C, int64_t L, int64_t nk, int64_t Nfilt) {
  DetectLayout d{};
  d.Lpad = ks::round_up(L, 128);
  d.nwords = (L + 31) / 32;
  d.nchunks = (d.nwords + kChunkWords - 1) / kChunkWords;
  size_t o = 0;
  auto take = [&](size_t b) {
    const size_t at = o;
    o = ks::align256(o + b);
    return at;
  };
  d.ctl = take(256);                               // err, total
  d.bt = take(sizeof(float) * (size_t)C * nk * d.Lpad);
  d.as = take(sizeof(float) * (size_t)Nfilt * L);
  d.im = take((size_t)Nfilt * L);
  d.bits = take(sizeof(unsigned) * (size_t)Nfilt * d.nwords);
  d.counts = take(sizeof(long long) * (size_t)Nfilt * d.nchunks);
  d.bytes = o;
  return d;
}

}  // namespace

extern "C" KS_API size_t ks_detect_workspace_size(int64_t C, int64_t L, int64_t nk,
                                                  int64_t Nfilt) {
  if (C < 1 || L < 1 || nk < 1 || Nfilt < 1) return 0;
  return detect_layout(C, L, nk, Nfilt).bytes;
}

extern "C" KS_API int ks_detect(const float* X, int64_t C, int64_t L, const float* wTEMP,
                                int64_t nk, int64_t nt, const int64_t* iC, int64_t nC,
                                const int64_t* iC2, int64_t nC2, const float* weigh,
                                int64_t nsizes, int64_t Nfilt, int64_t nt0, float th,
                                const float* wPCA, int64_t P, const float* yc, int64_t capacity,
                                int64_t* xy, int64_t* imax, float* amp, float* adist, float* yct,
                                float* tF, int64_t* info, void* workspace,
                                size_t workspace_bytes, void* stream) {
  using namespace ks;
  if (!X || !wTEMP || !iC || !iC2 || !weigh || !wPCA || !yc || !info)
    return fail(KS_ERR_ARG, "ks_detect: null pointer");
  if (C < 1 || L < 1 || nk < 1 || nt < 1 || nt % 2 == 0 || nC < 1 || nC2 < 1 || nsizes < 1 ||
      Nfilt < 1 || nt0 < 0 || P < 1 || capacity < 0)
    return fail(KS_ERR_ARG, "ks_detect: bad sizes (odd nt, counts >= 1)");
  if (nk > kMaxNK || nsizes > kMaxNS || nC > kMaxNC || P > 8 || nt > 1023)
    return fail(KS_ERR_UNSUPPORTED, "ks_detect: nk, sizes <= 8, nC <= 32, P <= 8, nt <= 1023");
  if (L > 0x7fffffffLL / 2 || Nfilt > 65535 || (long long)Nfilt * L > (1LL << 40))
    return fail(KS_ERR_UNSUPPORTED, "ks_detect: batch too long or too many positions");
  if (capacity > 0 && (!xy || !imax || !amp || !adist || !yct || !tF))
    return fail(KS_ERR_ARG, "ks_detect: null output");
  const DetectLayout d = detect_layout(C, L, nk, Nfilt);
  if (!workspace || workspace_bytes < d.bytes)
    return fail(KS_ERR_WORKSPACE, "ks_detect: workspace too small");
  if (C <= kMaxCBits && !aligned16(workspace))
    return fail(KS_ERR_ARG, "ks_detect: workspace must be 16-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const long long* iCl = reinterpret_cast<const long long*>(iC);
  const long long* iC2l = reinterpret_cast<const long long*>(iC2);
  long long* xyl = reinterpret_cast<long long*>(xy);
  long long* imaxl = reinterpret_cast<long long*>(imax);
  long long* infol = reinterpret_cast<long long*>(info);
  char* base = static_cast<char*>(workspace);
  int* err = reinterpret_cast<int*>(base + d.ctl);
  long long* total = reinterpret_cast<long long*>(base + d.ctl + 8);
  float* BT = reinterpret_cast<float*>(base + d.bt);
  float* As = reinterpret_cast<float*>(base + d.as);
  signed char* ims = reinterpret_cast<signed char*>(base + d.im);
  unsigned* bits = reinterpret_cast<unsigned*>(base + d.bits);
  long long* counts = reinterpret_cast<long long*>(base + d.counts);
  KS_CUDA(cudaMemsetAsync(base + d.ctl, 0, 16, s));

  // 1. the universal waveforms convolved with the batch: rows (c, k)
  int rc = launch_temporal_rows(X, wTEMP, C, L, nk, nt, d.Lpad, BT, d.Lpad, s);
  if (rc) return rc;
  // 2. scores over sizes and waveforms
  if (C <= kMaxCBits) {
    // the reference's defaults (5 sizes, 6 waveforms, 10 channels) and their sizes
    // and waveforms with other channel counts have their own instantiations
    const auto launch = nsizes == 5 && nk == 6 ? (nC == 10 ? launch_scores_tiled<5, 6, 10>
                                                           : launch_scores_tiled<5, 6, 0>)
                                               : launch_scores_tiled<kMaxNS, kMaxNK, 0>;
    rc = launch(BT, d.Lpad, (int)nk, (int)C, iCl, (int)nC, weigh, (int)nsizes, (int)Nfilt, (int)L,
                As, ims, err, s);
    if (rc) return rc;
  } else {
    const dim3 grid((unsigned)Nfilt, (unsigned)((L + kTile - 1) / kTile));
    ks_detect_scores_kernel<<<grid, kTile, 0, s>>>(BT, d.Lpad, (int)nk, (int)C, iCl, (int)nC, weigh,
                                                   (int)nsizes, (int)Nfilt, (int)L, As, ims, err);
    KS_CUDA(cudaGetLastError());
  }
  // 3. neighbour maximum, max-pool, peaks
  {
    const size_t smem = sizeof(int) * (size_t)nC2 +
                        sizeof(float) * (size_t)(kPeakTile + 2 * (nt0 <= kPeakHalo ? nt0 : 0));
    if (sizeof(int) * (size_t)nC2 > 200 * 1024) return fail(KS_ERR_UNSUPPORTED, "ks_detect: nC2 too large");
    KS_CUDA(cudaFuncSetAttribute(ks_detect_peaks_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
    const dim3 grid((unsigned)Nfilt, (unsigned)((L + kPeakTile - 1) / kPeakTile));
    ks_detect_peaks_kernel<<<grid, 256, smem, s>>>(As, iC2l, (int)nC2, (int)Nfilt, (int)L,
                                                     (int)nt, (int)nt0, th, bits, (int)d.nwords);
    KS_CUDA(cudaGetLastError());
  }
  // 4. (f, t)-ordered compaction
  const long long ncnt = (long long)Nfilt * d.nchunks;
  const unsigned cb = (unsigned)((ncnt + 255) / 256);
  ks_detect_count_kernel<<<cb, 256, 0, s>>>(bits, (int)Nfilt, (int)d.nwords, (int)d.nchunks, counts);
  KS_CUDA(cudaGetLastError());
  ks_detect_scan_kernel<<<1, 1024, 0, s>>>(counts, ncnt, total);
  KS_CUDA(cudaGetLastError());
  if (capacity > 0) {
    ks_detect_emit_kernel<<<cb, 256, 0, s>>>(bits, (int)Nfilt, (int)d.nwords, (int)d.nchunks, counts,
                                             capacity, xyl);
    KS_CUDA(cudaGetLastError());
    // 5. per-spike outputs (grids sized for the capacity; threads past the count return)
    ks_detect_gather_kernel<<<(unsigned)((capacity + 127) / 128), 128, 0, s>>>(
        xyl, total, capacity, As, ims, BT, d.Lpad, (int)nk, (int)C, iCl, (int)nC, (int)Nfilt, (int)L,
        yc, imaxl, amp, adist, yct);
    KS_CUDA(cudaGetLastError());
    DeviceInfo dev;
    if ((rc = device_info(&dev))) return rc;
    const long long warps = capacity * nC;
    const unsigned fb = (unsigned)std::min<long long>((warps + 7) / 8, (long long)dev.sm_count * 16);
    ks_detect_features_kernel<<<fb, 256, sizeof(float) * P * nt, s>>>(
        X, (int)C, (int)L, xyl, total, capacity, iCl, (int)nC, (int)Nfilt, wPCA, (int)P, (int)nt, tF);
    KS_CUDA(cudaGetLastError());
  }
  ks_detect_finish_kernel<<<1, 1, 0, s>>>(total, capacity, err, infol);
  KS_CUDA(cudaGetLastError());
  return KS_OK;
}
