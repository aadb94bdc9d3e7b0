// Temporal projection of the split form on the tensor cores (tcgen05):
//
//   Y[tau, c*P + p] = sum_t W[p, t] * X[c, tau - nt/2 + t]     (zero padding)
//
// written as the bf16 hi/lo planes the split-BF16 contraction reads
// (kilosort/template_matching.py:180, the conv1d of the batch with wPCA).
//
// The convolution of one channel is a product with a Toeplitz operand.  With
// the window x_w[u] = X[c, tau0 - nt/2 + u], an MMA row stands for the eight
// samples tau0 + 8r + phi (phi = 0..7) and the phases go to the N dimension:
//
//   D[r, phi*P + p] = sum_k x_w[8r + k] * Wsh[phi*P + p, k],
//   Wsh[phi*P + p, k] = W[p, k - phi]  (zero outside 0 <= k - phi < nt)
//
// A[r, k] = x_w[8r + k] is the canonical non-swizzled K-major layout read
// straight from the window: rows 16 bytes (8 samples) apart inside a core
// matrix and the next 8 taps 16 bytes on (LBO); core matrices overlap in memory,
// which the tensor core does not mind.  The next 8 rows (SBO) are those of the
// next channel's window: the 128 rows of one MMA are 64 samples of 16 channels,
// so that a tile's output rows are runs of 16 channels.  A tile is 256 samples
// of 16 channels = 4 MMA row sets, N = 8P (rounded to 16), K = nt + 7 (rounded to
// 16); split-BF16 as the score contraction: x = hi + lo, Wsh = hi + lo,
// D = Ahi.Bhi + Ahi.Blo + Alo.Bhi with FP32 accumulation, then D is split again
// into the bf16 hi/lo planes of Y.
//
// Persistent, one CTA per SM, 17 warps:
//   warps 8-15 producers, four warps per shared-memory slot (every other tile): the
//              16 channel windows (f32 -> bf16 hi/lo); the slot's next loads are
//              in flight, in registers, while it is waited for
//   warp 16    one lane issues the MMAs (K/16 steps x 3 products x 4 row sets)
//              into a double-buffered TMEM accumulator and commits them to an
//              mbarrier
//   warps 0-7  epilogue, four warps per half of the phases: thread r reads its
//              row, splits it into hi/lo and stages it in shared memory as the
//              boxes of the output; one lane per warp then writes those of a phase
//              with TMA stores (no multicast) through one tensor map per phase
//              whose rows are 8 samples apart
// Bound by the output planes (4 bytes per channel, sample and component) and by
// shared-memory bandwidth (MMA operands, staging, stores): 146 us at C=384,
// P=6, L=60122 (4.4 TB/s; 97 us at the copy rate); 261 us with tiles of 1024
// samples of 4 channels, whose 48-byte rows split sectors and whose MMAs were
// issued by a producer thread.  Staging two row sets at a time, each part with
// stores of its own, hides the reads of the stores (182 -> 153 us); copying the
// staged rows out by the warps instead of TMA took 160.
// Tiles of one time range are consecutive (channel groups fastest), so the
// partial 128-byte lines at channel-group edges meet in L2.  Every mbarrier
// wait is bounded; a wait that runs out sets the error word and the CTA
// drains its MMAs, frees TMEM and returns.
#include "ks_common.cuh"
#include "project.cuh"
#include "tcgen05.cuh"

#include <algorithm>
#include <cuda_bf16.h>

namespace {

using namespace ks::tc;

constexpr int kRows = 128;                 // MMA rows (TMEM lanes)
constexpr int kChan = kRows / 8;           // channels per tile
constexpr int kSets = 4;                   // MMA row sets per tile
constexpr int kSamples = 64 * kSets;       // samples per tile
constexpr int kEpiThreads = 256;           // warps 0-7: epilogue
constexpr int kMmaWarp = kEpiThreads / 32 + 8;   // warps 8-11, 12-15: producers, 16: MMAs
constexpr int kThreads = 32 * (kMmaWarp + 1);
constexpr int kTmemCols = 512;
constexpr int kMaxK = 128;                 // taps + 7, rounded to 16
constexpr unsigned long long kLimitNs = 2000000000ull;
// sample pairs of a window per producer lane: window_len(kMaxK) / 2 / 32, rounded up
constexpr int kPairIters = (kSamples - 8 + kMaxK + 63) / 64;

template <int PP>
struct Shape {
  static constexpr int NN = (8 * PP + 15) / 16 * 16;   // MMA N
  // channels of a store box: whole sectors and few rows (a box row costs the
  // copy engine much the same whatever its length), as far as the pitch of the
  // rows keeps the lanes that stage them on different banks: 16 channels 146 us,
  // 8 channels 153 at P = 6; 4 channels 226, 8 channels 242 at P = 8
  static constexpr int kBox = PP % 4 ? 16 : 4;
  static constexpr int kBoxes = kChan / kBox;
  static constexpr int kRowBytes = 2 * kBox * PP;
  static constexpr int kBoxBytes = 16 * kRowBytes;    // 16 rows: two row sets
  // staged output: [half of the phases][half of the sets][phase][plane][box]
  // [8-sample row][kBox*PP bf16]
  static constexpr int kStageBytes = 2 * 2 * 4 * 2 * kBoxes * kBoxBytes;
};

// TMA store maps of the output planes: m[plane][phi] covers the rows
// tau = 8*y + phi of Y (base Y + phi*Q, row stride 8*Q), boxes of 16 rows x
// kBox*P columns.
struct TemporalMaps {
  CUtensorMap m[2][8];
};

__host__ __device__ constexpr int window_len(int kext) { return kSamples - 8 + kext; }

template <int PP>
struct Smem {
  int kext;
  __host__ __device__ size_t b_bytes() const { return (size_t)2 * Shape<PP>::NN * kext * 2; }
  // a window's pitch, one plane of a slot, both planes of both slots
  __host__ __device__ size_t pitch() const { return (size_t)window_len(kext) * 2; }
  __host__ __device__ size_t a_plane() const { return kChan * pitch(); }
  __host__ __device__ size_t a_bytes() const { return 4 * a_plane(); }
  __host__ __device__ size_t off_a() const { return b_bytes(); }
  __host__ __device__ size_t off_s() const { return (off_a() + a_bytes() + 127) & ~size_t(127); }
  __host__ __device__ size_t s_bytes() const { return (size_t)Shape<PP>::kStageBytes; }
  __host__ __device__ size_t off_bar() const { return (off_s() + s_bytes() + 15) & ~size_t(15); }
  __host__ __device__ size_t total() const { return off_bar() + 64 + 128; }
};

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7])
      : "r"(taddr));
}
// TMA store of a 2-D box from shared memory (no multicast), bulk-group completion.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, uint32_t src, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
          reinterpret_cast<uint64_t>(map)),
      "r"(src), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void bulk_commit() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// the source shared memory of every committed group but the last has been read
__device__ __forceinline__ void bulk_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
}
// every committed store has completed
__device__ __forceinline__ void bulk_wait_all() {
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}
__device__ __forceinline__ void tmem_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Named barrier over `count` threads that also ANDs a predicate: every
// participant gets the same answer, so a group leaves its loop together.
__device__ __forceinline__ bool group_all(bool ok, int id, int count) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "bar.red.and.pred q, %2, %3, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)ok), "r"(id), "r"(count)
      : "memory");
  return r != 0;
}
__device__ __forceinline__ void group_sync(int id, int count) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}

// N words to shared memory, as wide as the rows of P = 2N bf16 are aligned
template <int N>
__device__ __forceinline__ void store_words(unsigned char* d, const uint32_t* w) {
  if constexpr (N % 4 == 0) {
    *reinterpret_cast<uint4*>(d) = make_uint4(w[0], w[1], w[2], w[3]);
  } else if constexpr (N % 2 == 0) {
    *reinterpret_cast<uint2*>(d) = make_uint2(w[0], w[1]);
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) reinterpret_cast<uint32_t*>(d)[i] = w[i];
  }
}

__device__ __forceinline__ uint32_t bf16x2_bits(__nv_bfloat162 v) {
  return *reinterpret_cast<uint32_t*>(&v);
}

template <int PP>
__global__ void __launch_bounds__(kThreads, 1)
ks_temporal_tc_kernel(const float* __restrict__ X, const float* __restrict__ W, int C, int L,
                      int nt, int kext, int n_cg, int n_tiles,
                      const __grid_constant__ TemporalMaps maps, int* err) {
  constexpr int NN = Shape<PP>::NN;
  extern __shared__ __align__(128) unsigned char smem[];
  const Smem<PP> lay{kext};
  unsigned char* sB = smem;
  unsigned char* sA = smem + lay.off_a();
  uint32_t* sS = reinterpret_cast<uint32_t*>(smem + lay.off_s());
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + lay.off_bar());
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 8);
  const uint32_t full0 = smem_u32(bars);        // full[2]: MMAs of a buffer done
  const uint32_t tfree0 = full0 + 16;           // tfree[2]: epilogue read the accumulator
  const uint32_t afull0 = full0 + 32;           // afull[2]: the windows are staged
  const uint32_t drain = full0 + 48;
  const int warp = threadIdx.x >> 5;
  const int half = nt / 2;
  const size_t aplane = lay.a_plane();
  const size_t bplane = (size_t)NN * kext * 2;

  // shifted, split basis Wsh (hi, lo) in the K-major core-matrix layout:
  // (n, k) at ((n/8)*(kext/8) + k/8)*128 + (n%8)*16 + (k%8)*2
  for (int e = threadIdx.x; e < NN * kext; e += kThreads) {
    const int n = e / kext, k = e - n * kext;
    const int phi = n / PP, p = n - phi * PP;
    const int t = k - phi;
    const float v = (phi < 8 && t >= 0 && t < nt) ? W[p * nt + t] : 0.f;
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    const __nv_bfloat16 l = __float2bfloat16_rn(v - __bfloat162float(h));
    const size_t o = ((size_t)(n >> 3) * (kext >> 3) + (k >> 3)) * 128 + (n & 7) * 16 + (k & 7) * 2;
    *reinterpret_cast<__nv_bfloat16*>(sB + o) = h;
    *reinterpret_cast<__nv_bfloat16*>(sB + bplane + o) = l;
  }
  if (threadIdx.x == 0) {
    for (int b = 0; b < 2; ++b) {
      mbar_init(full0 + 8 * b, 1);
      mbar_init(tfree0 + 8 * b, kEpiThreads);
      mbar_init(afull0 + 8 * b, 128);
    }
    mbar_init(drain, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tmem_alloc(smem_u32(tmem_slot), kTmemCols);
  fence_proxy_async_smem();
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
  constexpr uint32_t idesc = idesc_bf16_f32(kRows, NN);
  const int nk = kext / 16;

  if (warp == kMmaWarp) {
    // ------------------------------------------------------------ MMAs
    if ((threadIdx.x & 31) == 0) {
      const uint64_t db0 = make_smem_desc(smem_u32(sB), 128, (uint32_t)(kext / 8) * 128,
                                          kSwizzleNone);
      int j = 0;
      for (int t = blockIdx.x; t < n_tiles; t += gridDim.x, ++j) {
        const int b = j & 1;
        const uint32_t use = (uint32_t)(j >> 1);
        // the windows are staged; the accumulator's previous contents have been read
        if (!mbar_wait_bounded(afull0 + 8 * b, use & 1u, err, kLimitNs)) break;
        if (use > 0 && !mbar_wait_bounded(tfree0 + 8 * b, (use - 1) & 1u, err, kLimitNs)) break;
        fence_after();
        const uint32_t d = tmem + (uint32_t)(b * 256);
        // descriptors count addresses in 16 bytes
        const uint64_t da0 = make_smem_desc(smem_u32(sA) + (uint32_t)(2 * b * aplane), 16,
                                            (uint32_t)lay.pitch(), kSwizzleNone);
        for (int kk = 0; kk < nk; ++kk) {
#pragma unroll
          for (int q = 0; q < 3; ++q) {
            const uint64_t da = da0 + 2 * kk + (q == 2 ? aplane >> 4 : 0);
            const uint64_t db = db0 + 16 * kk + (q == 1 ? bplane >> 4 : 0);
            const uint32_t acc = q > 0 || kk > 0 ? 1u : 0u;
#pragma unroll
            for (int m = 0; m < kSets; ++m) mma_f16(d + m * NN, da + 8 * m, db, idesc, acc);
          }
        }
        mma_commit(full0 + 8 * b);
      }
      // every MMA issued by this thread has completed once this commit lands
      mma_commit(drain);
      const unsigned long long t0 = ks_globaltimer();
      while (!mbar_try_wait(drain, 0u)) {
        if (ks_globaltimer() - t0 > kLimitNs) break;
      }
    }
    __syncwarp();
  } else if (warp >= kEpiThreads / 32) {
    // ------------------------------------------------------------ producer
    const int b = (warp - kEpiThreads / 32) >> 2, pw = warp & 3, lane = threadIdx.x & 31;
    const int wl = window_len(kext);
    // a warp owns four windows, a lane the sample pairs u = 2*(lane + 32*i) of
    // each; all of them are loaded before the first is converted (zero outside
    // the recording and for channels past C)
    float2 xv[4][kPairIters];
    auto load_windows = [&](int tile) {
      const int s00 = (tile / n_cg) * kSamples - half + 2 * lane;
      const int c0 = (tile % n_cg) * kChan + 4 * pw;
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const int c = c0 + g;
        const float* xr = X + (size_t)(c < C ? c : 0) * L;
#pragma unroll
        for (int i = 0; i < kPairIters; ++i) {
          const int s0 = s00 + 64 * i;
          const bool in = c < C && 2 * lane + 64 * i < wl;
          xv[g][i].x = (in && s0 >= 0 && s0 < L) ? __ldg(xr + s0) : 0.f;
          xv[g][i].y = (in && s0 + 1 >= 0 && s0 + 1 < L) ? __ldg(xr + s0 + 1) : 0.f;
        }
      }
    };
    const int step = 2 * (int)gridDim.x, first = (int)(blockIdx.x + b * gridDim.x);
    if (first < n_tiles) load_windows(first);
    uint32_t use = 0;
    for (int t = first; t < n_tiles; t += step, ++use) {
      // the slot's previous MMAs have read it
      bool ok = true;
      if (use > 0) ok = mbar_wait_bounded(full0 + 8 * b, (use - 1) & 1u, err, kLimitNs);
      if (!group_all(ok, 5 + b, 128)) break;
      unsigned char* slot = sA + 2 * b * aplane + (size_t)(4 * pw) * lay.pitch();
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        uint32_t* hi = reinterpret_cast<uint32_t*>(slot + g * lay.pitch()) + lane;
        uint32_t* lo = reinterpret_cast<uint32_t*>(slot + g * lay.pitch() + aplane) + lane;
#pragma unroll
        for (int i = 0; i < kPairIters; ++i) {
          if (2 * lane + 64 * i < wl) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(xv[g][i].x, xv[g][i].y);
            const float2 hf = __bfloat1622float2(h);
            hi[32 * i] = bf16x2_bits(h);
            lo[32 * i] = bf16x2_bits(__floats2bfloat162_rn(xv[g][i].x - hf.x, xv[g][i].y - hf.y));
          }
        }
      }
      fence_proxy_async_smem();
      mbar_arrive(afull0 + 8 * b);
      if (t + step < n_tiles) load_windows(t + step);
    }
  } else {
    // ------------------------------------------------------------ epilogue
    // Warps 4h .. 4h+3 take the half h of the phases; thread r of them holds MMA
    // row r: channel c0 + r/8, samples tau0 + 64m + 8(r%8) + phi of row set m.  It
    // reads 4P columns of two row sets at a time and writes P bf16 per sample and
    // plane to the staged row 8(m%2) + r%8 of (half of the sets, phi, plane, box);
    // one lane of each warp stores the boxes of one phase.  The two halves of the
    // phases share nothing but the accumulator, and each half of the sets is
    // staged while the other's stores are being read.
    constexpr int HV = 4 * PP;               // columns of a row set per half
    constexpr int RB = Shape<PP>::kRowBytes, BB = Shape<PP>::kBoxBytes;
    constexpr int NB = Shape<PP>::kBoxes;
    const int h = warp >> 2;
    const int r = threadIdx.x & 127;         // TMEM lane = MMA row
    const int ch = r >> 3, f0 = warp & 3;
    const bool storer = (threadIdx.x & 31) == 0;
    // (half of the sets, phi, plane, box) blocks of this half of the phases
    unsigned char* stage = reinterpret_cast<unsigned char*>(sS) + (size_t)h * 16 * NB * BB;
    const size_t mine = (size_t)(ch / Shape<PP>::kBox) * BB + (size_t)(r & 7) * RB +
                        (size_t)(ch % Shape<PP>::kBox) * 2 * PP;
    int j = 0;
    for (int t = blockIdx.x; t < n_tiles; t += gridDim.x, ++j) {
      const int b = j & 1;
      const uint32_t use = (uint32_t)(j >> 1);
      bool ok = mbar_wait_bounded(full0 + 8 * b, use & 1u, err, kLimitNs);
      const uint32_t trow = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(b * 256 + h * HV);
#pragma unroll
      for (int m0 = 0; m0 < kSets; m0 += 2) {
        // this area is free once its last stores have read it
        if (storer) bulk_wait_read();
        ok = group_all(ok, 3 + h, 128);
        if (!ok) break;
        if (m0 == 0) fence_after();
        unsigned char* area = stage + (size_t)(m0 / 2) * 8 * NB * BB;
        uint32_t v[2][HV];
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int i = 0; i < HV / 8; ++i)
            tmem_ld8(trow + (uint32_t)((m0 + m) * NN + 8 * i), &v[m][8 * i]);
        tmem_wait_ld();
        if (m0 + 2 == kSets) {
          // the accumulator may be overwritten once both halves are here
          fence_before();
          mbar_arrive(tfree0 + 8 * b);
        }
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int f = 0; f < 4; ++f) {
            uint32_t hw[PP / 2], lw[PP / 2];
#pragma unroll
            for (int i = 0; i < PP / 2; ++i) {
              const float a = __uint_as_float(v[m][f * PP + 2 * i]);
              const float c = __uint_as_float(v[m][f * PP + 2 * i + 1]);
              const __nv_bfloat162 hv = __floats2bfloat162_rn(a, c);
              const float2 hf = __bfloat1622float2(hv);
              hw[i] = bf16x2_bits(hv);
              lw[i] = bf16x2_bits(__floats2bfloat162_rn(a - hf.x, c - hf.y));
            }
            unsigned char* dh = area + mine + (size_t)(2 * f * NB) * BB + (size_t)(8 * m) * RB;
            store_words<PP / 2>(dh, hw);
            store_words<PP / 2>(dh + (size_t)NB * BB, lw);
          }
        fence_proxy_async_smem();
        group_sync(3 + h, 128);
        if (storer) {
          const int y = (t / n_cg) * (kSamples / 8) + 8 * m0, x = (t % n_cg) * kChan * PP;
          const uint32_t s0 = smem_u32(area) + (uint32_t)(2 * f0 * NB * BB);
          for (int pl = 0; pl < 2; ++pl)
#pragma unroll
            for (int bx = 0; bx < NB; ++bx)
              tma_store_2d(&maps.m[pl][4 * h + f0], s0 + (uint32_t)((pl * NB + bx) * BB),
                           x + bx * Shape<PP>::kBox * PP, y);
          bulk_commit();
        }
      }
      if (!ok) break;
    }
    // the stores in flight are complete before the CTA exits
    if (storer) bulk_wait_all();
  }
  fence_before();
  __syncthreads();
  fence_after();
  if (warp == 0) tmem_dealloc(tmem, kTmemCols);
}

template <int PP>
int launch_pp(const float* X, const float* W, int64_t C, int64_t L, int64_t nt, int64_t Q,
              int64_t Lpad, __nv_bfloat16* Yhi, __nv_bfloat16* Ylo, int* err,
              cudaStream_t stream) {
  using namespace ks;
  const int kext = (int)round_up(nt + 7, 16);
  const Smem<PP> lay{kext};
  const size_t smem = lay.total();
  DeviceInfo dev;
  int rc = device_info(&dev);
  if (rc) return rc;
  if (smem > (size_t)dev.smem_optin) return KS_ERR_UNSUPPORTED;
  const int n_cg = (int)(round_up(C, 16) / kChan);
  const long long n_tiles = ((Lpad + kSamples - 1) / kSamples) * (long long)n_cg;
  if (n_tiles > 0x7fffffffLL) return fail(KS_ERR_UNSUPPORTED, "temporal: too many tiles");
  static thread_local int attr_device = -1;
  if (attr_device != dev.device) {
    KS_CUDA(cudaFuncSetAttribute(ks_temporal_tc_kernel<PP>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)dev.smem_optin));
    attr_device = dev.device;
  }
  const int grid = (int)std::min<long long>(n_tiles, dev.sm_count);
  if (grid < 1) return KS_OK;
  static thread_local TemporalMaps maps;
  for (int pl = 0; pl < 2; ++pl)
    for (int phi = 0; phi < 8; ++phi) {
      rc = make_bf16_store_map(&maps.m[pl][phi], (pl ? Ylo : Yhi) + phi * Q, Lpad / 8, Q, 8 * Q,
                               Shape<PP>::kBox * PP, 16);
      if (rc) return rc;
    }
  ks_temporal_tc_kernel<PP><<<grid, kThreads, smem, stream>>>(X, W, (int)C, (int)L, (int)nt, kext,
                                                              n_cg, (int)n_tiles, maps, err);
  KS_CUDA(cudaGetLastError());
  return KS_OK;
}

}  // namespace

namespace ks {

int launch_temporal_split_tc(const float* X, const float* W, int64_t C, int64_t L, int64_t P,
                             int64_t nt, int64_t Q, int64_t Lpad, __nv_bfloat16* Yhi,
                             __nv_bfloat16* Ylo, int* err, cudaStream_t stream) {
  if (!err || nt + 7 > kMaxK || Lpad > 0x7fffffffLL - kSamples ||
      (reinterpret_cast<uintptr_t>(Yhi) & 15) || (reinterpret_cast<uintptr_t>(Ylo) & 15) ||
      (Q % 8) || (Lpad % 8))
    return KS_ERR_UNSUPPORTED;
  switch (P) {
    case 2: return launch_pp<2>(X, W, C, L, nt, Q, Lpad, Yhi, Ylo, err, stream);
    case 4: return launch_pp<4>(X, W, C, L, nt, Q, Lpad, Yhi, Ylo, err, stream);
    case 6: return launch_pp<6>(X, W, C, L, nt, Q, Lpad, Yhi, Ylo, err, stream);
    case 8: return launch_pp<8>(X, W, C, L, nt, Q, Lpad, Yhi, Ylo, err, stream);
    default: return KS_ERR_UNSUPPORTED;
  }
}

}  // namespace ks
