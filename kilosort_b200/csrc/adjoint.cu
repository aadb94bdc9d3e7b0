// Fixed-assignment reconstruction loss and its adjoint.
//
// Given spikes s = (tau_s, k_s) with amplitudes a_s, templates U [K,P,C] and the
// temporal basis W [P,nt], the reconstruction is
//   R[c, tau] = sum_s a_s * wave_{k_s}[c, tau - tau_s + nt/2],
//   wave_k[c, t] = sum_p U[k,p,c] * W[p,t]          (0 <= t < nt, 0 <= tau < L)
// -- the subtraction kilosort/template_matching.py:237 applies spike by spike --
// and the loss is  loss = sum_{c,tau} (X - R)^2.  With G = dloss * dLoss/dR =
// -2 * dloss * Xres (Xres = X - R):
//   d a_s      = sum_{c,t} G[c, tau_s - nt/2 + t] * wave_{k_s}[c, t]
//   d U[k,p,c] = sum_t W[p,t] * H_k[c,t]
//   d W[p,t]   = sum_k sum_c U[k,p,c] * H_k[c,t]
// where H_k[c,t] = sum_{s: k_s = k} a_s * G[c, tau_s - nt/2 + t] is the
// amplitude-weighted sum of the residual windows of template k's spikes.  The
// adjoint never stores the K x C x nt waveforms: each block recomputes the
// slice of wave_k it needs in shared memory.
//
// Determinism: every sum runs in a fixed order (spikes in index order per
// template, per-block partials reduced in block order in double precision), so
// repeated calls give identical bits.
//
// Forward kernels: count spikes per time sample, scan, bucket them by time and
// order every bucket by index, then one warp per (32-column block, 32
// channels) applies the spikes whose window meets the block in (time, index)
// order (the peel's residual_apply), writes Xres and a double partial of
// sum Xres^2.  Adjoint kernels: group spikes by template (CSR in index order),
// one block per (template, channel chunk) accumulates H in registers and the
// per-spike dot products, then fixed-order reductions.
#include "ks_common.cuh"
#include "residual_apply.cuh"

#include <algorithm>

namespace {

constexpr int kCol = 32;
constexpr int kChunkC = 32;        // channels per adjoint block (nt > 128)
constexpr int kAdjThreads = 256;
constexpr int kAdjWarps = kAdjThreads / 32;
constexpr int kAdjSpikes = 32;     // spikes whose dot products a block keeps at a time
constexpr int kDwSplits = 64;      // partial sums of dW
constexpr int kRecThreads = 256;
constexpr int kScanThreads = 1024;

struct ReconLayout {
  size_t status, cnt, off, idx, otau, ok, oamp, sup, part, cntk, offk, karr, list, dwpart, dwsum,
      dapart, bytes;
  int64_t nblk, ngrp, nchunk, nwarps;
};

// Channels of one adjoint block: a warp holds 8 elements per lane (6 at 65 to
// 96 taps) of (channel, tap), taps 32 apart.
int64_t adjoint_chunk(int64_t nt) {
  const int64_t ne = (nt + 31) / 32;
  return ne > 4 ? kChunkC : kAdjWarps * (ne == 1 ? 8 : ne == 2 ? 4 : 2);
}

ReconLayout recon_layout(int64_t C, int64_t L, int64_t K, int64_t P, int64_t nt, int64_t N) {
  ReconLayout r;
  r.nblk = (L + kCol - 1) / kCol;
  r.ngrp = (C + 31) / 32;
  r.nchunk = (C + adjoint_chunk(nt) - 1) / adjoint_chunk(nt);
  r.nwarps = r.nblk * r.ngrp;
  size_t o = 0;
  auto take = [&](size_t b) {
    const size_t at = o;
    o = ks::align256(o + b);
    return at;
  };
  r.status = take(256);
  r.cnt = take(4 * (size_t)(L + 1));
  r.off = take(4 * (size_t)(L + 1));
  r.idx = take(4 * (size_t)std::max<int64_t>(N, 1));
  r.otau = take(4 * (size_t)std::max<int64_t>(N, 1));
  r.ok = take(4 * (size_t)std::max<int64_t>(N, 1));
  r.oamp = take(4 * (size_t)std::max<int64_t>(N, 1));
  r.sup = take(8 * (size_t)K);
  r.part = take(8 * (size_t)r.nwarps);
  r.cntk = take(4 * (size_t)(K + 1));
  r.offk = take(4 * (size_t)(K + 1));
  r.karr = take(4 * (size_t)std::max<int64_t>(N, 1));
  r.list = take(4 * (size_t)std::max<int64_t>(N, 1));
  r.dwpart = take(4 * (size_t)K * r.nchunk * P * nt);
  r.dwsum = take(8 * (size_t)kDwSplits * P * nt);
  r.dapart = take(4 * (size_t)r.nchunk * std::max<int64_t>(N, 1));
  r.bytes = o + 16;              // room to align the workspace to 16 bytes
  return r;
}

// ------------------------------------------------------------------ helpers
// Exclusive scan of n ints into out[0..n] (out[n] = total), one block.  Tiles of
// kScanItems values per thread, the next tile's loads in flight while this one
// is scanned (latency-bound: 27 us per 60122 values with one contiguous run per
// thread and scalar loads).  in and out 16-byte aligned.
constexpr int kScanItems = 16;
__global__ void __launch_bounds__(kScanThreads) ks_scan_kernel(const int* __restrict__ in, int n,
                                                               int* __restrict__ out) {
  __shared__ int wsum[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int4 v[kScanItems / 4];
  auto load = [&](long long i) {
#pragma unroll
    for (int j = 0; j < kScanItems / 4; ++j) {
      const long long o = i + 4 * j;
      v[j] = make_int4(0, 0, 0, 0);
      if (o + 4 <= n) {
        v[j] = *reinterpret_cast<const int4*>(in + o);
      } else {
        if (o < n) v[j].x = in[o];
        if (o + 1 < n) v[j].y = in[o + 1];
        if (o + 2 < n) v[j].z = in[o + 2];
      }
    }
  };
  int carry = 0;
  load((long long)kScanItems * threadIdx.x);
  for (long long base = 0; base < n; base += kScanItems * kScanThreads) {
    const long long i = base + (long long)kScanItems * threadIdx.x;
    int4 e[kScanItems / 4];
    int run = 0;
#pragma unroll
    for (int j = 0; j < kScanItems / 4; ++j) {
      e[j].x = run;
      e[j].y = e[j].x + v[j].x;
      e[j].z = e[j].y + v[j].y;
      e[j].w = e[j].z + v[j].z;
      run = e[j].w + v[j].w;
    }
    load(i + kScanItems * kScanThreads);
    int incl = run;
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += x;
    }
    __syncthreads();
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    int w = wsum[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += x;
    }
    const int prev = __shfl_sync(0xffffffffu, w, max(warp - 1, 0));
    const int before = carry + incl - run + (warp ? prev : 0);
#pragma unroll
    for (int j = 0; j < kScanItems / 4; ++j) {
      const long long o = i + 4 * j;
      if (o + 4 <= n) {
        *reinterpret_cast<int4*>(out + o) =
            make_int4(before + e[j].x, before + e[j].y, before + e[j].z, before + e[j].w);
      } else {
        if (o < n) out[o] = before + e[j].x;
        if (o + 1 < n) out[o + 1] = before + e[j].y;
        if (o + 2 < n) out[o + 2] = before + e[j].z;
      }
    }
    carry += __shfl_sync(0xffffffffu, w, 31);
  }
  if (threadIdx.x == 0) out[n] = carry;
}

// Spikes per time sample; an out-of-range time or template marks the call
// invalid (the spike is skipped everywhere).  Forward: counts by time (cnt);
// adjoint: counts by template (cntk) and every spike's template, -1 for an
// invalid spike (karr).
__global__ void ks_recon_count_kernel(const long long* __restrict__ st, int N, int L, int K,
                                      int* __restrict__ cnt, int* __restrict__ cntk,
                                      int* __restrict__ karr, int* __restrict__ status) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < N; s += gridDim.x * blockDim.x) {
    const long long tau = st[2 * (long long)s], k = st[2 * (long long)s + 1];
    if (tau < 0 || tau >= L || k < 0 || k >= K) {
      atomicCAS(status, 0, KS_ERR_ARG);
      if (karr) karr[s] = -1;
      continue;
    }
    if (cnt) atomicAdd(&cnt[tau], 1);
    if (karr) {
      atomicAdd(&cntk[k], 1);
      karr[s] = (int)k;
    }
  }
}

__global__ void ks_recon_fill_kernel(const long long* __restrict__ st, int N, int L, int K,
                                     const int* __restrict__ off, int* __restrict__ fill,
                                     int* __restrict__ idx) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < N; s += gridDim.x * blockDim.x) {
    const long long tau = st[2 * (long long)s], k = st[2 * (long long)s + 1];
    if (tau < 0 || tau >= L || k < 0 || k >= K) continue;
    idx[off[tau] + atomicAdd(&fill[tau], 1)] = s;
  }
}

// The bucketed spikes in (time, index) order: an entry's place in its bucket is
// the number of smaller indices there (buckets hold a few).
__global__ void ks_recon_order_kernel(const long long* __restrict__ st,
                                      const float* __restrict__ amps, const int* __restrict__ off,
                                      const int* __restrict__ idx, int L, int* __restrict__ otau,
                                      int* __restrict__ ok, float* __restrict__ oamp) {
  const int n = off[L];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int s = idx[i];
    const int tau = (int)st[2 * (long long)s];
    const int b = off[tau], e = off[tau + 1];
    int d = b;
    for (int j = b; j < e; ++j) d += idx[j] < s ? 1 : 0;
    otau[d] = tau;
    ok[d] = (int)st[2 * (long long)s + 1];
    oamp[d] = amps[s];
  }
}

// Support mask of each template (residual_apply): a block per template.
__global__ void __launch_bounds__(256) ks_recon_support_kernel(const float* __restrict__ U, int P,
                                                               int C,
                                                               unsigned long long* __restrict__ sup) {
  __shared__ unsigned mask[2];
  if (threadIdx.x < 2) mask[threadIdx.x] = 0u;
  __syncthreads();
  const float* u = U + (long long)blockIdx.x * P * C;
  const int width = support_width(C);
  unsigned lo = 0u, hi = 0u;
#pragma unroll 4
  for (int e = threadIdx.x; e < P * C; e += 256) {
    const int bit = u[e] != 0.f ? e % C / kXCh / width : 64;
    lo |= bit < 32 ? 1u << bit : 0u;
    hi |= bit >= 32 && bit < 64 ? 1u << (bit - 32) : 0u;
  }
  lo = __reduce_or_sync(0xffffffffu, lo);
  hi = __reduce_or_sync(0xffffffffu, hi);
  if ((threadIdx.x & 31) == 0) {
    atomicOr(&mask[0], lo);
    atomicOr(&mask[1], hi);
  }
  __syncthreads();
  if (threadIdx.x == 0) sup[blockIdx.x] = (unsigned long long)mask[1] << 32 | mask[0];
}

// ------------------------------------------------------------------ forward
struct ReconArgs {
  const float* U;
  const unsigned long long* sup;
  int C, P, nt;
  float one;                     // 1 (see f2_add_prod)
};

// One warp per (32-column block, 32 channels), two tiles of 16 channels: lanes
// own columns; the spikes whose window meets the block are a run of the
// (time, index) order.  Bound by issue (half of the slots, with few warps) and the
// shared-memory round trips between: 211 us at C=384, K=600,
// 25200 spikes, where the form with lanes over channels, each lane touching its
// own row of X, took 1173 us.
template <int PP>
__global__ void __launch_bounds__(kRecThreads)
ks_recon_kernel(const float* __restrict__ X, ReconArgs a, const float* __restrict__ W,
                const int* __restrict__ off, const int* __restrict__ otau,
                const int* __restrict__ ok, const float* __restrict__ oamp, int L, int nblk,
                int ngrp, float* __restrict__ Xres, double* __restrict__ part) {
  extern __shared__ __align__(16) float sm[];
  if (__syncthreads_or(stage_basis(W, a.P, a.nt, sm, kRecThreads))) a.sup = nullptr;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long w = (long long)blockIdx.x * (kRecThreads / 32) + warp;
  if (w >= (long long)nblk * ngrp) return;
  const ResSmem s = residual_smem(sm, sm + 8 * a.nt, warp);
  const int blk = (int)(w / ngrp), cg = (int)(w % ngrp);
  const int c0 = blk * kCol, half = a.nt / 2, col = c0 + lane;
  const bool colok = col < L;
  // spike times whose window [tau - half, tau + half] meets [c0, c0 + 31]
  const int first = off[max(0, c0 - half)];
  const int total = off[min(L - 1, c0 + kCol - 1 + half) + 1] - first;
  const int width = support_width(a.C);
  double sq = 0.0;
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {
    const int cbase = cg * 32 + h * kXCh;
    if (cbase >= a.C) break;
    const float* src = X + (long long)cbase * L + col;
    float* out = Xres + (long long)cbase * L + col;
    unsigned long long x2[kXCh / 2];
#pragma unroll
    for (int i = 0; i < kXCh / 2; ++i) {
      const float lo = (colok && cbase + 2 * i < a.C) ? src[(long long)(2 * i) * L] : 0.f;
      const float hi = (colok && cbase + 2 * i + 1 < a.C) ? src[(long long)(2 * i + 1) * L] : 0.f;
      x2[i] = f2_pack(lo, hi);
    }
    for (int done = 0; done < total; done += kXList) {
      const int n = min(kXList, total - done);
      if (h == 0 || total > kXList) {
        __syncwarp();
        for (int i = lane; i < n; i += 32) {
          s.xl_tau[i] = otau[first + done + i];
          s.xl_k[i] = ok[first + done + i];
          s.xl_amp[i] = oamp[first + done + i];
        }
        __syncwarp();
      }
      residual_apply<PP>(a, s, n, c0, cbase, cbase / kXCh / width, lane, x2);
    }
#pragma unroll
    for (int i = 0; i < kXCh / 2; ++i) {
      float lo, hi;
      f2_unpack(x2[i], lo, hi);
      if (colok && cbase + 2 * i < a.C) {
        out[(long long)(2 * i) * L] = lo;
        sq += (double)lo * (double)lo;
      }
      if (colok && cbase + 2 * i + 1 < a.C) {
        out[(long long)(2 * i + 1) * L] = hi;
        sq += (double)hi * (double)hi;
      }
    }
  }
  for (int o = 16; o; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
  if (lane == 0) part[w] = sq;
}

// Fixed-order sum of the per-warp partials.
__global__ void __launch_bounds__(1024) ks_sum_double_kernel(const double* __restrict__ part,
                                                             long long n, double* __restrict__ out) {
  __shared__ double red[1024];
  double s = 0.0;
  for (long long i = threadIdx.x; i < n; i += 1024) s += part[i];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int d = 512; d; d >>= 1) {
    if (threadIdx.x < d) red[threadIdx.x] += red[threadIdx.x + d];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = red[0];
}

// ------------------------------------------------------------------ adjoint
// Spikes of each template, in index order, one block per template: every warp
// counts the template's spikes in its eighth of the list, then writes them
// behind those of the warps before it.  (With the list read 256 spikes at a
// time between block barriers, from the 16-byte records: 76 us at K=600.)
__global__ void __launch_bounds__(256) ks_group_by_template_kernel(const int* __restrict__ karr,
                                                                   int N,
                                                                   const int* __restrict__ offk,
                                                                   int* __restrict__ list) {
  __shared__ int wcount[8];
  const int k = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (offk[k + 1] == offk[k]) return;
  const long long seg = (((long long)N + 7) / 8 + 127) / 128 * 128;
  const long long s0 = warp * seg, s1 = min((long long)N, s0 + seg);
  auto load = [&](long long s) {
    int4 v = make_int4(-1, -1, -1, -1);
    if (s + 4 <= s1) {
      v = *reinterpret_cast<const int4*>(karr + s);
    } else {
      if (s < s1) v.x = karr[s];
      if (s + 1 < s1) v.y = karr[s + 1];
      if (s + 2 < s1) v.z = karr[s + 2];
    }
    return v;
  };
  int n = 0;
#pragma unroll 4
  for (long long s = s0; s < s1; s += 128) {
    const int4 v = load(s + 4 * lane);
    n += (v.x == k) + (v.y == k) + (v.z == k) + (v.w == k);
  }
  n = __reduce_add_sync(0xffffffffu, n);
  if (lane == 0) wcount[warp] = n;
  __syncthreads();
  int pos = offk[k];
  for (int i = 0; i < warp; ++i) pos += wcount[i];
  if (n == 0) return;
#pragma unroll 4
  for (long long s = s0; s < s1; s += 128) {
    const int4 v = load(s + 4 * lane);
    const unsigned below = (1u << lane) - 1u;
    const unsigned b0 = __ballot_sync(0xffffffffu, v.x == k), b1 = __ballot_sync(0xffffffffu, v.y == k);
    const unsigned b2 = __ballot_sync(0xffffffffu, v.z == k), b3 = __ballot_sync(0xffffffffu, v.w == k);
    if (!(b0 | b1 | b2 | b3)) continue;
    int o = pos + __popc(b0 & below) + __popc(b1 & below) + __popc(b2 & below) + __popc(b3 & below);
    const int s4 = (int)(s + 4 * lane);
    if (v.x == k) list[o++] = s4;
    if (v.y == k) list[o++] = s4 + 1;
    if (v.z == k) list[o++] = s4 + 2;
    if (v.w == k) list[o] = s4 + 3;
    pos += __popc(b0) + __popc(b1) + __popc(b2) + __popc(b3);
  }
}

// Block (k, chunk) of 8 * CW channels: warp w holds channels w*CW .. w*CW+CW-1,
// lane l the taps l, l + 32, ... (NE of them) of each, with its elements of
// H_k and wave_k in registers.  Spikes four at a time: their windows are loaded
// together (whole rows of taps, coalesced), H accumulates them in index order,
// and the four dot products are reduced by one exchange; 32 spikes' dot
// products are then added over the warps.
//
// What bounds it: instruction issue (70 % of the slots) around the window reads,
// C*nt residual values per spike (2.9 GB through L2 at C=384 and 25200 spikes, a
// quarter of its rate): 434 us.  With H and the waveform in shared memory, one
// spike at a time between two block barriers, it took 1246 us.
template <int NE, int CW>
__global__ void __launch_bounds__(kAdjThreads) ks_adjoint_warp_kernel(
    const float* __restrict__ Xres, const long long* __restrict__ st,
    const float* __restrict__ amps, const float* __restrict__ U, const float* __restrict__ W,
    const int* __restrict__ offk, const int* __restrict__ list, const float* __restrict__ dloss,
    int C, int L, int K, int P, int nt, int nchunk, float* __restrict__ dU,
    float* __restrict__ dwpart, float* __restrict__ dapart) {
  extern __shared__ float sm[];
  float* sW = sm;                       // [P][nt]
  float* sD = sW + P * nt;              // [kAdjWarps][P][nt] partial dW of each warp
  __shared__ int sSpike[kAdjSpikes], sTau[kAdjSpikes];
  __shared__ float sAmp[kAdjSpikes], sDot[kAdjWarps][kAdjSpikes];
  // one grid dimension: 16-channel chunks of a million channels exceed grid.y
  const int k = (int)(blockIdx.x % K), ch = (int)(blockIdx.x / K);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cw = ch * (kAdjWarps * CW) + warp * CW;     // the warp's first channel
  const int half = nt / 2;
  for (int i = threadIdx.x; i < P * nt; i += kAdjThreads) sW[i] = W[i];
  __syncthreads();
  float wave[CW][NE], H[CW][NE];
  bool ok[CW][NE];
#pragma unroll
  for (int c = 0; c < CW; ++c)
#pragma unroll
    for (int e = 0; e < NE; ++e) {
      const int t = lane + 32 * e;
      ok[c][e] = cw + c < C && t < nt;
      float v = 0.f;
      if (ok[c][e])
        for (int p = 0; p < P; ++p)
          v = fmaf(U[((long long)k * P + p) * C + cw + c], sW[p * nt + t], v);
      wave[c][e] = v;
      H[c][e] = 0.f;
    }
  const int b = offk[k], n = offk[k + 1] - b;
  for (int i0 = 0; i0 < n; i0 += kAdjSpikes) {
    const int m = min(kAdjSpikes, n - i0);
    __syncthreads();                    // the previous spikes' values are read
    if (threadIdx.x < m) {
      const int s = list[b + i0 + threadIdx.x];
      sSpike[threadIdx.x] = s;
      sTau[threadIdx.x] = (int)st[2 * (long long)s];
      sAmp[threadIdx.x] = amps[s];
    }
    __syncthreads();
    for (int j = 0; j < m; j += 4) {
      float g[4][CW][NE], dot[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int col = (j + q < m ? sTau[j + q] : L + nt) - half + lane;
        const float* x = Xres + (long long)cw * L + col;
#pragma unroll
        for (int c = 0; c < CW; ++c)
#pragma unroll
          for (int e = 0; e < NE; ++e)
            g[q][c][e] = (ok[c][e] && (unsigned)(col + 32 * e) < (unsigned)L)
                             ? __ldg(x + (long long)c * L + 32 * e) : 0.f;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        dot[q] = 0.f;
        if (j + q < m) {
          const float am = sAmp[j + q];
#pragma unroll
          for (int c = 0; c < CW; ++c)
#pragma unroll
            for (int e = 0; e < NE; ++e) {
              H[c][e] = fmaf(am, g[q][c][e], H[c][e]);
              dot[q] = fmaf(g[q][c][e], wave[c][e], dot[q]);
            }
        }
      }
      // the four sums over the lanes: lane 8 * q ends with spike j + q's
      const bool up = lane & 16, odd = lane & 8;
      const float x0 = __shfl_xor_sync(0xffffffffu, up ? dot[0] : dot[2], 16);
      const float x1 = __shfl_xor_sync(0xffffffffu, up ? dot[1] : dot[3], 16);
      const float d0 = (up ? dot[2] : dot[0]) + x0, d1 = (up ? dot[3] : dot[1]) + x1;
      float d = (odd ? d1 : d0) + __shfl_xor_sync(0xffffffffu, odd ? d0 : d1, 8);
      d += __shfl_xor_sync(0xffffffffu, d, 4);
      d += __shfl_xor_sync(0xffffffffu, d, 2);
      d += __shfl_xor_sync(0xffffffffu, d, 1);
      if ((lane & 7) == 0) sDot[warp][j + (lane >> 3)] = d;
    }
    __syncthreads();
    if (threadIdx.x < m) {
      float tot = 0.f;
      for (int w = 0; w < kAdjWarps; ++w) tot += sDot[w][threadIdx.x];
      dapart[(long long)sSpike[threadIdx.x] * nchunk + ch] = tot;
    }
  }
  const float scale = -2.f * dloss[0];
  // dU[k, p, c] = scale * sum_t W[p,t] H[c,t]; the warp's partial dW
  for (int p = 0; p < P; ++p) {
    float w[NE], dw[NE];
#pragma unroll
    for (int e = 0; e < NE; ++e) {
      const int t = lane + 32 * e;
      w[e] = t < nt ? sW[p * nt + t] : 0.f;
      dw[e] = 0.f;
    }
#pragma unroll
    for (int c = 0; c < CW; ++c) {
      if (cw + c >= C) continue;
      const float u = U[((long long)k * P + p) * C + cw + c];
      float v = 0.f;
#pragma unroll
      for (int e = 0; e < NE; ++e) {
        v = fmaf(w[e], H[c][e], v);
        dw[e] = fmaf(u, H[c][e], dw[e]);
      }
      for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) dU[((long long)k * P + p) * C + cw + c] = scale * v;
    }
#pragma unroll
    for (int e = 0; e < NE; ++e)
      if (lane + 32 * e < nt) sD[(warp * P + p) * nt + lane + 32 * e] = dw[e];
  }
  __syncthreads();
  // partial dW of this block: sum_c U[k,p,c] H[c,t] (unscaled), warps in order
  float* dst = dwpart + ((long long)k * nchunk + ch) * P * nt;
  for (int o = threadIdx.x; o < P * nt; o += kAdjThreads) {
    float v = 0.f;
    for (int w = 0; w < kAdjWarps; ++w) v += sD[w * P * nt + o];
    dst[o] = v;
  }
}

// The same for more than 128 taps (their H and waveform do not fit a warp's
// registers): H_k and wave_k over 32 channels in shared memory.
__global__ void __launch_bounds__(kAdjThreads) ks_adjoint_kernel(
    const float* __restrict__ Xres, const long long* __restrict__ st,
    const float* __restrict__ amps, const float* __restrict__ U, const float* __restrict__ W,
    const int* __restrict__ offk, const int* __restrict__ list, const float* __restrict__ dloss,
    int C, int L, int K, int P, int nt, int nchunk, float* __restrict__ dU,
    float* __restrict__ dwpart, float* __restrict__ dapart) {
  extern __shared__ float sm[];
  const int k = blockIdx.x, ch = blockIdx.y;
  const int c0 = ch * kChunkC;
  const int ncl = min(kChunkC, C - c0);
  const int ne = kChunkC * nt;
  float* sW = sm;                     // [P][nt]
  float* wave = sW + P * nt;          // [kChunkC][nt]
  float* H = wave + ne;                // [kChunkC][nt]
  float* red = H + ne;                // [kAdjThreads / 32]
  for (int i = threadIdx.x; i < P * nt; i += kAdjThreads) sW[i] = W[i];
  __syncthreads();
  for (int e = threadIdx.x; e < ne; e += kAdjThreads) {
    const int cl = e / nt, t = e - cl * nt;
    float v = 0.f;
    if (cl < ncl) {
      for (int p = 0; p < P; ++p) v = fmaf(U[((long long)k * P + p) * C + c0 + cl], sW[p * nt + t], v);
    }
    wave[e] = v;
    H[e] = 0.f;
  }
  const float scale = -2.f * dloss[0];
  const int half = nt / 2;
  const int b = offk[k], n = offk[k + 1] - b;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = 0; i < n; ++i) {
    const int s = list[b + i];
    const int tau = (int)st[2 * (long long)s];
    const float a = amps[s];
    float dot = 0.f;
    for (int e = threadIdx.x; e < ne; e += kAdjThreads) {
      const int cl = e / nt, t = e - cl * nt;
      const int col = tau - half + t;
      float g = 0.f;
      if (cl < ncl && col >= 0 && col < L) g = Xres[(long long)(c0 + cl) * L + col];
      H[e] = fmaf(a, g, H[e]);
      dot = fmaf(g, wave[e], dot);
    }
    for (int o = 16; o; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
    if (lane == 0) red[warp] = dot;
    __syncthreads();
    if (threadIdx.x == 0) {
      float tot = 0.f;
      for (int w = 0; w < kAdjThreads / 32; ++w) tot += red[w];
      dapart[(long long)s * nchunk + ch] = tot;
    }
    __syncthreads();
  }
  // H is complete (each element was written by one thread): publish it
  __syncthreads();
  // dU[k, p, c0 + cl] = scale * sum_t W[p,t] H[cl,t]
  for (int o = threadIdx.x; o < P * ncl; o += kAdjThreads) {
    const int p = o / ncl, cl = o - p * ncl;
    float v = 0.f;
    for (int t = 0; t < nt; ++t) v = fmaf(sW[p * nt + t], H[cl * nt + t], v);
    dU[((long long)k * P + p) * C + c0 + cl] = scale * v;
  }
  // partial dW of this block: sum_cl U[k,p,c0+cl] H[cl,t] (unscaled)
  float* dst = dwpart + ((long long)k * nchunk + ch) * P * nt;
  for (int o = threadIdx.x; o < P * nt; o += kAdjThreads) {
    const int p = o / nt, t = o - p * nt;
    float v = 0.f;
    for (int cl = 0; cl < ncl; ++cl) v = fmaf(U[((long long)k * P + p) * C + c0 + cl], H[cl * nt + t], v);
    dst[o] = v;
  }
}

// dW[o] = scale * sum over (template, chunk) blocks of the partials, in block
// order, accumulated in double: kDwSplits runs of blocks, then their sums.
// (One thread per output over all 7200 partials took 466 us.)
__global__ void __launch_bounds__(128) ks_adjoint_dw_part_kernel(const float* __restrict__ dwpart,
                                                                 int nblocks, int PN,
                                                                 double* __restrict__ dwsum) {
  const int o = blockIdx.x * 128 + threadIdx.x;
  if (o >= PN) return;
  const long long b0 = (long long)nblocks * blockIdx.y / kDwSplits;
  const long long b1 = (long long)nblocks * (blockIdx.y + 1) / kDwSplits;
  double s = 0.0;
#pragma unroll 8
  for (long long b = b0; b < b1; ++b) s += (double)dwpart[b * PN + o];
  dwsum[(long long)blockIdx.y * PN + o] = s;
}

__global__ void __launch_bounds__(128) ks_adjoint_dw_kernel(const double* __restrict__ dwsum, int PN,
                                                            const float* __restrict__ dloss,
                                                            float* __restrict__ dW) {
  const int o = blockIdx.x * 128 + threadIdx.x;
  if (o >= PN) return;
  double s = 0.0;
#pragma unroll 16
  for (int b = 0; b < kDwSplits; ++b) s += dwsum[(long long)b * PN + o];
  dW[o] = (float)((double)(-2.f * dloss[0]) * s);
}

// damps[s] = scale * sum over chunks of the per-chunk dot products.
__global__ void ks_adjoint_da_kernel(const float* __restrict__ dapart, const long long* __restrict__ st,
                                     int N, int L, int K, int nchunk,
                                     const float* __restrict__ dloss, float* __restrict__ damps) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < N; s += gridDim.x * blockDim.x) {
    const long long tau = st[2 * (long long)s], k = st[2 * (long long)s + 1];
    if (tau < 0 || tau >= L || k < 0 || k >= K) {
      damps[s] = 0.f;
      continue;
    }
    double v = 0.0;
    for (int ch = 0; ch < nchunk; ++ch) v += (double)dapart[(long long)s * nchunk + ch];
    damps[s] = (float)((double)(-2.f * dloss[0]) * v);
  }
}

// The workspace from its first 16-byte boundary on (vector loads of its arrays).
char* recon_base(void* workspace) {
  return reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(workspace) + 15) & ~uintptr_t(15));
}

int check_recon(int64_t C, int64_t L, int64_t K, int64_t P, int64_t nt, int64_t N) {
  if (C < 1 || L < 1 || K < 1 || P < 1 || nt < 1 || (nt % 2) == 0 || N < 0)
    return ks::fail(KS_ERR_ARG, "ks_recon: need C,L,K,P >= 1, N >= 0 and odd nt");
  if (P > 8 || nt > 1023 || L >= (1LL << 31) - 1 || N >= (1LL << 31) || C > (1 << 24))
    return ks::fail(KS_ERR_UNSUPPORTED, "ks_recon: shape beyond supported limits");
  return KS_OK;
}

}  // namespace

extern "C" KS_API size_t ks_recon_workspace_size(int64_t C, int64_t L, int64_t K, int64_t P,
                                                int64_t nt, int64_t n_spikes) {
  if (check_recon(C, L, K, P, nt, n_spikes)) return 0;
  return recon_layout(C, L, K, P, nt, n_spikes).bytes;
}

extern "C" KS_API int ks_recon_loss(const float* X, const int64_t* st, const float* amps,
                                    int64_t n_spikes, const float* U, const float* W, int64_t C,
                                    int64_t L, int64_t K, int64_t P, int64_t nt, float* Xres,
                                    double* loss, int* status, void* workspace,
                                    size_t workspace_bytes, void* stream) {
  using namespace ks;
  int rc = check_recon(C, L, K, P, nt, n_spikes);
  if (rc) return rc;
  if (!X || !U || !W || !Xres || !loss || !status || (n_spikes > 0 && (!st || !amps)))
    return fail(KS_ERR_ARG, "ks_recon_loss: null pointer");
  const ReconLayout r = recon_layout(C, L, K, P, nt, n_spikes);
  if (!workspace || workspace_bytes < r.bytes) return fail(KS_ERR_WORKSPACE, "ks_recon_loss: workspace too small");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  char* base = recon_base(workspace);
  int* cnt = reinterpret_cast<int*>(base + r.cnt);
  int* off = reinterpret_cast<int*>(base + r.off);
  int* idx = reinterpret_cast<int*>(base + r.idx);
  double* part = reinterpret_cast<double*>(base + r.part);
  const long long* stp = reinterpret_cast<const long long*>(st);
  const int N = (int)n_spikes;
  int* otau = reinterpret_cast<int*>(base + r.otau);
  int* ok = reinterpret_cast<int*>(base + r.ok);
  float* oamp = reinterpret_cast<float*>(base + r.oamp);
  ReconArgs ra;
  ra.U = U;
  ra.sup = reinterpret_cast<unsigned long long*>(base + r.sup);
  ra.C = (int)C;
  ra.P = (int)P;
  ra.nt = (int)nt;
  ra.one = 1.f;
  KS_CUDA(cudaMemsetAsync(status, 0, sizeof(int), s));
  KS_CUDA(cudaMemsetAsync(cnt, 0, 4 * (size_t)(L + 1), s));
  const int gb = (int)std::min<int64_t>(4096, std::max<int64_t>(1, (N + 255) / 256));
  if (N > 0) {
    ks_recon_count_kernel<<<gb, 256, 0, s>>>(stp, N, (int)L, (int)K, cnt, nullptr, nullptr, status);
    KS_CUDA(cudaGetLastError());
  }
  ks_scan_kernel<<<1, kScanThreads, 0, s>>>(cnt, (int)L, off);
  KS_CUDA(cudaGetLastError());
  if (N > 0) {
    KS_CUDA(cudaMemsetAsync(cnt, 0, 4 * (size_t)L, s));   // reused as fill counters
    ks_recon_fill_kernel<<<gb, 256, 0, s>>>(stp, N, (int)L, (int)K, off, cnt, idx);
    KS_CUDA(cudaGetLastError());
    ks_recon_order_kernel<<<gb, 256, 0, s>>>(stp, amps, off, idx, (int)L, otau, ok, oamp);
    KS_CUDA(cudaGetLastError());
    ks_recon_support_kernel<<<(unsigned)K, 256, 0, s>>>(
        U, (int)P, (int)C, reinterpret_cast<unsigned long long*>(base + r.sup));
    KS_CUDA(cudaGetLastError());
  }
  const unsigned grid = (unsigned)((r.nwarps + kRecThreads / 32 - 1) / (kRecThreads / 32));
  const size_t smem = sizeof(float) * (8 * (size_t)nt + (size_t)(kRecThreads / 32) * kXWarp);
  const auto kernel = P <= 6 ? ks_recon_kernel<6> : ks_recon_kernel<8>;
  kernel<<<grid, kRecThreads, smem, s>>>(X, ra, W, off, otau, ok, oamp, (int)L, (int)r.nblk,
                                         (int)r.ngrp, Xres, part);
  KS_CUDA(cudaGetLastError());
  ks_sum_double_kernel<<<1, 1024, 0, s>>>(part, r.nwarps, loss);
  KS_CUDA(cudaGetLastError());
  return KS_OK;
}

extern "C" KS_API int ks_recon_adjoint(const float* Xres, const int64_t* st, const float* amps,
                                       int64_t n_spikes, const float* U, const float* W,
                                       int64_t C, int64_t L, int64_t K, int64_t P, int64_t nt,
                                       const float* dloss, float* dU, float* dW, float* damps,
                                       int* status, void* workspace, size_t workspace_bytes,
                                       void* stream) {
  using namespace ks;
  int rc = check_recon(C, L, K, P, nt, n_spikes);
  if (rc) return rc;
  if (!Xres || !U || !W || !dloss || !dU || !dW || !status ||
      (n_spikes > 0 && (!st || !amps || !damps)))
    return fail(KS_ERR_ARG, "ks_recon_adjoint: null pointer");
  const ReconLayout r = recon_layout(C, L, K, P, nt, n_spikes);
  if (!workspace || workspace_bytes < r.bytes)
    return fail(KS_ERR_WORKSPACE, "ks_recon_adjoint: workspace too small");
  DeviceInfo dev;
  rc = device_info(&dev);
  if (rc) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  char* base = recon_base(workspace);
  int* cntk = reinterpret_cast<int*>(base + r.cntk);
  int* offk = reinterpret_cast<int*>(base + r.offk);
  int* list = reinterpret_cast<int*>(base + r.list);
  float* dwpart = reinterpret_cast<float*>(base + r.dwpart);
  float* dapart = reinterpret_cast<float*>(base + r.dapart);
  const long long* stp = reinterpret_cast<const long long*>(st);
  const int N = (int)n_spikes;
  int* karr = reinterpret_cast<int*>(base + r.karr);
  double* dwsum = reinterpret_cast<double*>(base + r.dwsum);
  KS_CUDA(cudaMemsetAsync(status, 0, sizeof(int), s));
  KS_CUDA(cudaMemsetAsync(cntk, 0, 4 * (size_t)(K + 1), s));
  const int gb = (int)std::min<int64_t>(4096, std::max<int64_t>(1, (N + 255) / 256));
  if (N > 0) {
    ks_recon_count_kernel<<<gb, 256, 0, s>>>(stp, N, (int)L, (int)K, nullptr, cntk, karr, status);
    KS_CUDA(cudaGetLastError());
  }
  ks_scan_kernel<<<1, kScanThreads, 0, s>>>(cntk, (int)K, offk);
  KS_CUDA(cudaGetLastError());
  if (N > 0) {
    ks_group_by_template_kernel<<<(unsigned)K, 256, 0, s>>>(karr, N, offk, list);
    KS_CUDA(cudaGetLastError());
  }
  const int ne = (int)((nt + 31) / 32);
  if (ne <= 4) {
    const size_t smem = sizeof(float) * (size_t)(1 + kAdjWarps) * P * nt;
    const auto kernel = ne == 1 ? ks_adjoint_warp_kernel<1, 8>
                        : ne == 2 ? ks_adjoint_warp_kernel<2, 4>
                        : ne == 3 ? ks_adjoint_warp_kernel<3, 2> : ks_adjoint_warp_kernel<4, 2>;
    KS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kernel<<<(unsigned)(K * r.nchunk), kAdjThreads, smem, s>>>(
        Xres, stp, amps, U, W, offk, list, dloss, (int)C, (int)L, (int)K, (int)P, (int)nt,
        (int)r.nchunk, dU, dwpart, dapart);
  } else {
    const size_t smem = sizeof(float) * ((size_t)P * nt + 2 * (size_t)kChunkC * nt + kAdjThreads / 32);
    if (smem > dev.smem_optin) return fail(KS_ERR_UNSUPPORTED, "ks_recon_adjoint: nt too long");
    KS_CUDA(cudaFuncSetAttribute(ks_adjoint_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const dim3 grid((unsigned)K, (unsigned)r.nchunk);
    ks_adjoint_kernel<<<grid, kAdjThreads, smem, s>>>(Xres, stp, amps, U, W, offk, list, dloss,
                                                      (int)C, (int)L, (int)K, (int)P, (int)nt,
                                                      (int)r.nchunk, dU, dwpart, dapart);
  }
  KS_CUDA(cudaGetLastError());
  const int PN = (int)(P * nt);
  const unsigned db = (unsigned)((PN + 127) / 128);
  ks_adjoint_dw_part_kernel<<<dim3(db, kDwSplits), 128, 0, s>>>(dwpart, (int)(K * r.nchunk), PN, dwsum);
  KS_CUDA(cudaGetLastError());
  ks_adjoint_dw_kernel<<<db, 128, 0, s>>>(dwsum, PN, dloss, dW);
  KS_CUDA(cudaGetLastError());
  if (N > 0) {
    ks_adjoint_da_kernel<<<gb, 256, 0, s>>>(dapart, stp, N, (int)L, (int)K, (int)r.nchunk, dloss,
                                            damps);
    KS_CUDA(cudaGetLastError());
  }
  return KS_OK;
}
