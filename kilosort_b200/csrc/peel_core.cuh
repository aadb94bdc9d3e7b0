// Device code of the greedy peel, shared by the single-batch launch
// (peel.cu) and the multi-batch launch (batched.cu).
// Greedy peel (matching pursuit) of one batch as a single persistent,
// cooperative kernel.  Semantics follow kilosort/template_matching.py:183-244.
//
// Layout in HBM
//   Bt     [nblk][K][32] f32   score matrix B[k, tau] tiled by 32-column blocks
//                              (nblk = ceil(L/32)): a block's K rows are one
//                              contiguous 128*K-byte run, so rescoring a block
//                              streams it instead of touching K scattered lines
//   ctcT   [K][K][2nt+1] f32   ctcT[k][j][l] = ctc[j][k][l]: the cross-
//                              correlations a peak of template k subtracts are
//                              one contiguous slab
//   Xres   [C][L] f32          residual, written once after the loop from X
//   cfmax [L] f32 / imax [L] i32  settled best score relu(B)^2/nm over
//                              templates, and its template, per column
//   pack   [2][L] u64          rescoring of dirty columns per iteration:
//                              (score bits << 32) | ~template under atomicMax,
//                              so the larger score and, on ties, the smaller
//                              template index win
//   per-iteration (double buffered by parity): dirty-block bitmap, touch
//   lists (peaks within +-nt of each dirty block) and a work counter
//
// Iteration it (p = it & 1, q = p ^ 1), two phases between device-wide barriers:
//   DETECT  per 256-column chunk whose +-nt neighbourhood changed in it-1:
//           settle the rescored columns (pack[q] -> cfmax/imax); pooled =
//           max of cfmax over +-nt (doubling levels of a sliding max); a column
//           is a peak iff pooled > th2 and |pooled - cfmax| < 1e-9 (kilosort
//           :206-212).  Peaks are compacted in time order; amplitude
//           B[k,tau]/nm[k] and sqrt(pooled) come from the pre-subtraction B
//           (:225-229).  Each peak registers in the touch lists of the blocks
//           within +-nt of it; the first registration sets the block's dirty bit
//           and clears its pack[p] entries.
//   UPDATE  every block computes the exclusive prefix of the chunk counts (a
//           peak's global index in the iteration) and of the dirty bitmap.
//           Records are written in (iteration, tau) order, after the updates.
//           Warps scan the dirty blocks and, past a barrier, work through the
//           units found (grouped update; with few dirty blocks a warp updates a
//           (block, group) pair as it looks at it, without the barrier), or take
//           work items (dirty block in column order, row range) from a counter
//           (ungrouped; large teams: round-robin, the last round from the
//           counter): B[j,c] -= amp*ctc[j,k,c-tau+nt] for the peaks touching column c,
//           even-indexed peaks first, then odd-indexed -- the order of the
//           reference's two interleaved groups (:235-238) -- product and
//           difference rounded separately; rescored rows fold into pack[p].
// The loop ends when no peak is found or after max_peels iterations, decided
// identically by every block from the same counts.  The residual (:237) is not
// read inside the loop, so its updates run once afterwards: per 32-column
// block the spikes whose windows cover it are gathered from the time-sorted
// records of each iteration and subtracted element by element in record order,
// the order of the reference's iterations; every element of Xres is read and
// written once instead of once per touching spike.  Every device-wide wait is
// bounded; a wait that runs out records KS_ERR_TIMEOUT and all blocks leave.
#pragma once
#include "ks_common.cuh"
#include "project.cuh"
#include "residual_apply.cuh"

namespace {

constexpr int kThreads = 256;
// Resident blocks per SM.  The single-batch launch (its phases end at
// barriers of the whole device, so fewer, faster blocks pay): 1.53 ms with 2,
// 1.63 ms with 3 for the iterations of a C=384, K=600 batch.  Teams work
// through many units per phase: 11.0 ms with 3, 11.5 with 2, 13.2 with 4 for 16
// such batches by 16 teams.
constexpr int kBlocksPerSm = 2;
constexpr int kTeamBlocksPerSm = 3;
constexpr int kWarps = kThreads / 32;
constexpr int kChunk = 256;          // detection chunk, one column per thread
constexpr int kCol = 32;             // update block, one column per lane
constexpr int kRowsPerWarp = 16;     // template rows in flight per lane (ungrouped update)
constexpr int kItemRows = 64;        // template rows per update item, large teams (at most)
constexpr int kItemRowsSmall = 640;  // the same, small teams: a whole block's rows per
                                     // item (one fold per column instead of ten)
constexpr int kStaticWarps = 1024;   // teams of at least this many warps deal items statically
constexpr int kTouch = 8;            // peaks touching one block (more: ties)
constexpr int kMaxChunks = 16384;
constexpr int kMaxIters = 4096;      // iterations whose record offsets are kept
constexpr int kMaxTemplates = 65536; // templates of one batch
constexpr int kXCap = 32;            // spikes recorded per block for the residual
constexpr int kGroup = 32;           // template rows of one group (grouped update)
constexpr long long kStaticUnits = 4; // units per warp up to which they are dealt round-robin
__host__ __device__ inline int n_groups(long long K) { return (int)((K + kGroup - 1) / kGroup); }
constexpr int kTileBytes = 4096;     // a warp's tile: a unit's ctc rows (4 KB), a scan's
                                     // metadata, a detection chunk's windows; larger tiles
                                     // leave L1 too few lines for the loads in flight (units
                                     // 6.7 ms of the 16-batch launch, 8.1 with 6 KB)
constexpr int kScanGroups = 14;      // groups whose metadata a scan stages at once
static_assert(kScanGroups * 32 * 9 <= kTileBytes && kScanGroups <= 32 &&
              kGroup * 32 * 4 <= kTileBytes, "a warp's tile is too small");

// Phase timeline for profiling builds (-DKS_PEEL_TRACE): block 0 writes
// %globaltimer stamps to info[8 + 8*it + slot]; the caller sizes info.
#ifdef KS_PEEL_TRACE
#define KS_TRACE(it, slot, value)                                        \
  do {                                                                   \
    if (a.trace && blockIdx.x == 0 && threadIdx.x == 0 && (it) < 200)    \
      a.info[8 + 8 * (it) + (slot)] = (long long)(value);                \
  } while (0)
// every block's end-of-work stamp of iterations < 8 at info[1608 + it*G + block]
#define KS_TRACE_CTA(it, value)                                                  \
  do {                                                                           \
    if (a.trace && threadIdx.x == 0 && (it) < 8)                                 \
      a.info[1608 + (it) * gridDim.x + blockIdx.x] = (long long)(value);          \
  } while (0)
#else
#define KS_TRACE(it, slot, value) \
  do {                           \
  } while (0)
#define KS_TRACE_CTA(it, value) \
  do {                          \
  } while (0)
#endif

struct Touch {
  int tau;
  int k;
  float amp;
  int slot;  // chunk * kChunk + index in chunk
};

struct PeelArgs {
  float* Bt;
  const float* X;             // the batch; Xres = X - residual updates (may be Xres)
  float* Xres;
  const float* U;
  const float* W;
  const float* ctcT;
  const float* nm;
  const unsigned long long* sup;  // [K] channel groups where a template is not all zero
                                  //     (support_width; null: taken as everywhere)
  const float2* nmi;          // {nm[j], 1/nm[j]} (1/nm NaN when nm is not a positive normal)
  int C, L, K, P, nt;
  float th2;
  float one;                  // 1 (see f2_add_prod)
  int max_peels;
  long long capacity;
  long long* st;
  float* amps;
  float* th_amps;
  long long* info;
  // scratch
  float* cfmax;
  int* imax;
  unsigned long long* pack;   // [2][L]
  int* chunk_cnt;
  int* chunk_tau;
  int* chunk_k;
  float* chunk_amp;
  float* chunk_th;
  int* tcount;                // [2][nblk]
  Touch* touch;               // [2][nblk * kTouch]
  unsigned* dbits;            // [2][nwords]
  unsigned* wctr;             // [6] work counters by iteration parity: [0,1] update
                              //     items, [2,3] grouped units written, [4,5] taken
  int* itoff;                 // [kMaxIters] first record of each iteration
  int* xcount;                // [nblk] spikes whose residual window meets the block
  int* xlist;                 // [nblk * kXCap] their record indices (unordered)
  unsigned long long* ctl;    // the team's control word (barrier count, error)
  const int* upstream_err;    // error word of the producer of Bt (may be null)
  // grouped update (null rperm: every row of a touched column is rewritten)
  const int* rperm;           // [K] template rows in group order (group g: rows
                              //     rperm[32g .. 32g+31])
  const float2* nmip;         // [K] {nm, 1/sqrt(nm)} in group order (the scale NaN for an
                              //     nm outside [2^-30, 2^30])
  const float* mg;            // [K][ng] largest |ctcT[k][j][l]| over the rows j
                              //     of group g and all lags
  unsigned long long* gbest;  // [nblk][ng][32] packed best score of each group
                              //     per column (pack_score)
  unsigned char* gexp;        // [nblk][ng][32] smallest exponent field of |B|
                              //     over each group's rows per column (noop_expo)
  int* blist;                 // [nblk][32] a dirty block's ordered touch list for
                              //     its units: n, tau[kTouch], k[kTouch], amp bits
  uint2* units;               // [nblk*ng] (block << 11 | group, columns to process)
  int ng;                     // groups, ceil(K / kGroup)
  int nchunks, nblk, nwords;
  int trace;                  // profiling builds: 1 where info has room for the timeline
  unsigned long long limit_ns;
};

// Detection by one warp per chunk: where a chunk's two window buffers and its
// template indices fit in the warp's tile (nt <= 64) and the team has fewer
// blocks than the batch has chunks.  A block finishes one chunk sooner (3 us
// against 5 us), but a team of 18 blocks took 50 us an iteration for the 235
// chunks of 60122 samples one after the other, and 14 us by warps.
__host__ __device__ inline bool warp_detection(int nt, bool grouped, int nchunks, unsigned G) {
  return grouped && (2 * (kChunk + 2 * nt) + kChunk) * 4 <= kTileBytes && (unsigned)nchunks > G;
}

constexpr int kUnitBytes = 2 * 512;  // inputs of a warp's units in flight (UnitIn)

struct Smem {
  float* W;        // [8][nt] (the fused residual's basis)
  int* prefix;     // nchunks+1   exclusive prefix of chunk peak counts
  int* wprefix;    // nwords+1    exclusive prefix of dirty-bitmap popcounts
  unsigned* dw;    // nwords      the iteration's dirty bitmap
  float* win;      // kChunk + 2*nt   column scores around the chunk (block detection)
  float* mx0;      // kChunk + 2*nt   sliding-max doubling levels (ping-pong)
  float* mx1;      // kChunk + 2*nt
  int* kidx;       // kChunk          best template of the chunk's own columns
  int* wcnt;       // kWarps+1
  int* tl_tau;     // kWarps*kTouch ordered touch list of each warp's item
  int* tl_k;       // kWarps*kTouch
  float* tl_amp;   // kWarps*kTouch
  unsigned char* eb;  // kWarps*kTouch*32  bound exponents of a warp's touching peaks
  float* stage;       // kWarps*kTileBytes (grouped update only): a warp's tile (of ctc
                      //   rows [kGroup][32], then of the updated scores)
  struct UnitIn* unit;  // kWarps*kUnitSlots (grouped update only): inputs of a warp's units
};

__device__ __forceinline__ Smem carve_smem(const PeelArgs& a, char* base, bool grouped) {
  Smem s;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char* p = base + off;
    off = (off + bytes + 15) & ~size_t(15);
    return p;
  };
  const int wn = kChunk + 2 * a.nt;
  s.W = reinterpret_cast<float*>(take(sizeof(float) * 8 * a.nt));
  s.prefix = reinterpret_cast<int*>(take(sizeof(int) * (a.nchunks + 1)));
  s.wprefix = reinterpret_cast<int*>(take(sizeof(int) * (a.nwords + 1)));
  s.dw = reinterpret_cast<unsigned*>(take(sizeof(unsigned) * a.nwords));
  s.win = reinterpret_cast<float*>(take(sizeof(float) * wn));
  s.mx0 = reinterpret_cast<float*>(take(sizeof(float) * wn));
  s.mx1 = reinterpret_cast<float*>(take(sizeof(float) * wn));
  s.kidx = reinterpret_cast<int*>(take(sizeof(int) * kChunk));
  s.wcnt = reinterpret_cast<int*>(take(sizeof(int) * (kWarps + 1)));
  s.tl_tau = reinterpret_cast<int*>(take(sizeof(int) * kWarps * kTouch));
  s.tl_k = reinterpret_cast<int*>(take(sizeof(int) * kWarps * kTouch));
  s.tl_amp = reinterpret_cast<float*>(take(sizeof(float) * kWarps * kTouch));
  s.eb = reinterpret_cast<unsigned char*>(take(kWarps * kTouch * 32));
  s.stage = grouped ? reinterpret_cast<float*>(take(kWarps * kTileBytes)) : nullptr;
  s.unit = grouped ? reinterpret_cast<UnitIn*>(take(kWarps * kUnitBytes)) : nullptr;
  return s;
}

size_t smem_bytes(int P, int nt, int nchunks, int nwords, bool grouped) {
  auto r = [](size_t b) { return (b + 15) & ~size_t(15); };
  const size_t wn = kChunk + 2 * (size_t)nt;
  (void)P;
  return r(sizeof(float) * 8 * nt) + r(sizeof(int) * (nchunks + 1)) +
         r(sizeof(int) * (nwords + 1)) + r(sizeof(unsigned) * nwords) +
         3 * r(sizeof(float) * wn) +
         r(sizeof(int) * kChunk) + r(sizeof(int) * (kWarps + 1)) +
         3 * r(sizeof(int) * kWarps * kTouch) + r(kWarps * kTouch * 32) +
         (grouped ? r(kWarps * kTileBytes) + r(kWarps * kUnitBytes) : 0);
}

__device__ __forceinline__ unsigned long long pack_score(float cf, int j) {
  return ((unsigned long long)__float_as_uint(cf) << 32) | (unsigned)(~(unsigned)j);
}
__device__ __forceinline__ float pack_value(unsigned long long v) {
  return __uint_as_float((unsigned)(v >> 32));
}
__device__ __forceinline__ int pack_index(unsigned long long v) {
  return (int)(~(unsigned)(v & 0xffffffffull));
}
// Fold row j's score relu(b)^2/nm[j] into (best, arg) -- larger score wins,
// the earlier (smaller) row on ties -- computing the IEEE quotient only where
// it can matter: sq*(1/nm) is within a relative 2^-22 of sq/nm, so a row whose
// quotient could reach best has sq*(1/nm) >= best*(1 - 2^-20).  Rows failing
// that test cannot change (best, arg).  The quotient itself is the exactly
// rounded division, as in the reference.
__device__ __forceinline__ void fold_score(float b, float2 nmi, int j, float& best, int& arg) {
  const float rl = b > 0.f ? b : 0.f;
  const float sq = __fmul_rn(rl, rl);
  const float approx = __fmul_rn(sq, nmi.y);
  const bool maybe = best < 0.f || !(approx < best * 0.99999905f) || approx != approx;
  if (maybe) {
    const float cf = __fdiv_rn(sq, nmi.x);
    if (cf > best) {
      best = cf;
      arg = j;
    }
  }
}

__device__ __forceinline__ const float* bt_row(const PeelArgs& a, int blk, int j) {
  return a.Bt + ((size_t)blk * a.K + j) * kCol;
}

// A warp's tile.
__device__ __forceinline__ float* unit_tile(const Smem& s, int warp) {
  return s.stage + (size_t)warp * (kTileBytes / 4);
}

// ---------------------------------------------------------------- DETECT
__device__ void detect_chunk(const PeelArgs& a, const Smem& s, int ch, int it) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nt = a.nt, L = a.L;
  const int p = it & 1, q = p ^ 1;
  const int a0 = ch * kChunk;
  const int a1 = min(a0 + kChunk, L);
  const int wn = kChunk + 2 * nt;
  const int* tprev = a.tcount + (size_t)q * a.nblk;
  const unsigned long long* pprev = a.pack + (size_t)q * L;
  // Column scores: rescored columns of the last iteration come from pack[q]
  // (and are settled into cfmax/imax by the chunk that owns them), the others
  // from cfmax.  The candidate loads are independent and issued together; if
  // nothing within +-nt of the chunk changed, its peak test cannot change and
  // the chunk is skipped.
  int any_fresh = 0;
  for (int i = tid; i < wn; i += kThreads) {
    const int col = a0 - nt + i;
    float v;
    if (col < 0 || col >= L) {
      v = -INFINITY;
    } else if (col < nt || col >= L - nt) {
      v = 0.f;
    } else {
      const bool fresh = it == 0 || tprev[col / kCol] > 0;
      const unsigned long long pv = pprev[col];
      const float cv = a.cfmax[col];
      const bool own = i >= nt && i < nt + kChunk && col < a1;
      const int iv = own ? a.imax[col] : 0;
      any_fresh |= fresh;
      v = fresh ? pack_value(pv) : cv;
      if (own) {
        const int kb = fresh ? pack_index(pv) : iv;
        s.kidx[i - nt] = kb;
        if (fresh) {
          a.cfmax[col] = v;
          a.imax[col] = kb;
        }
      }
    }
    s.win[i] = v;
  }
  if (!__syncthreads_or(any_fresh)) {
    if (tid == 0) a.chunk_cnt[ch] = 0;
    return;
  }
  // sliding max over 2nt+1 columns: doubling levels up to the largest power
  // of two m <= 2nt+1, then the union of two overlapping m-windows
  const int len = 2 * nt + 1;
  int m = 1;
  const float* src = s.win;
  float* dst = s.mx0;
  while (2 * m <= len) {
    for (int i = tid; i + 2 * m <= wn; i += kThreads) dst[i] = fmaxf(src[i], src[i + m]);
    __syncthreads();
    m *= 2;
    src = dst;
    dst = (dst == s.mx0) ? s.mx1 : s.mx0;
  }
  const int tau = a0 + tid;
  bool pk = false;
  float pooled = 0.f;
  if (tid < kChunk && tau < a1 && tau >= nt && tau < L - nt) {
    pooled = fmaxf(src[tid], src[tid + len - m]);
    const float best = s.win[tid + nt];
    pk = (pooled > a.th2) && (fabsf(__fsub_rn(pooled, best)) < 1e-9f);
  }
  const unsigned bal = __ballot_sync(0xffffffffu, pk);
  if (lane == 0) s.wcnt[warp] = __popc(bal);
  __syncthreads();
  if (tid == 0) {
    int acc = 0;
    for (int w = 0; w < kWarps; ++w) {
      const int c = s.wcnt[w];
      s.wcnt[w] = acc;
      acc += c;
    }
    s.wcnt[kWarps] = acc;
  }
  __syncthreads();
  if (pk) {
    const int idx = s.wcnt[warp] + __popc(bal & ((1u << lane) - 1u));
    const int k = s.kidx[tid];
    const float amp = __fdiv_rn(bt_row(a, tau / kCol, k)[tau % kCol], a.nm[k]);
    const float th = __fsqrt_rn(pooled);
    const int slot = ch * kChunk + idx;
    a.chunk_tau[slot] = tau;
    a.chunk_k[slot] = k;
    a.chunk_amp[slot] = amp;
    a.chunk_th[slot] = th;
    int* tcur = a.tcount + (size_t)p * a.nblk;
    Touch* tch = a.touch + (size_t)p * a.nblk * kTouch;
    unsigned* bits = a.dbits + (size_t)p * a.nwords;
    unsigned long long* pcur = a.pack + (size_t)p * L;
    const int b0 = (tau - nt) / kCol, b1 = (tau + nt) / kCol;
    for (int bb = b0; bb <= b1; bb += 8) {
      int pos[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) pos[i] = (bb + i <= b1) ? atomicAdd(&tcur[bb + i], 1) : -1;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int b = bb + i;
        if (pos[i] < 0) continue;
        if (pos[i] == 0) {
          atomicOr(&bits[b >> 5], 1u << (b & 31));
          const int c_hi = min(L, (b + 1) * kCol);
          for (int c = b * kCol; c < c_hi; ++c) pcur[c] = 0ull;
        }
        if (pos[i] < kTouch) tch[(size_t)b * kTouch + pos[i]] = Touch{tau, k, amp, slot};
        else ks_ctl_fail(a.ctl, KS_ERR_DEGENERATE);
      }
    }
  }
  if (tid == 0) a.chunk_cnt[ch] = s.wcnt[kWarps];
  __syncthreads();
}

// detect_chunk by one warp in its tile, so that a team's chunks proceed side by
// side instead of one per block and latency chain.  The columns whose blocks
// were rescored come from pack[q], the others from cfmax (one load each); a
// chunk without a rescored block within +-nt has no peak.
//
// What bounds it: the latency of its few dependent loads and atomics.
__device__ void detect_chunk_warp(const PeelArgs& a, float* tile, int ch, int it, int lane) {
  const int nt = a.nt, L = a.L;
  const int p = it & 1, q = p ^ 1;
  const int a0 = ch * kChunk, a1 = min(a0 + kChunk, L);
  const int wn = kChunk + 2 * nt;
  const unsigned long long* pprev = a.pack + (size_t)q * L;
  // rescored blocks among those within +-nt (at most 13: nt <= 64)
  const int bb0 = max(a0 - nt, 0) / kCol, bb1 = min(a1 - 1 + nt, L - 1) / kCol;
  unsigned fresh = 0xffffffffu;
  if (it > 0) {
    const bool f = bb0 + lane <= bb1 && a.tcount[(size_t)q * a.nblk + bb0 + lane] > 0;
    fresh = __ballot_sync(0xffffffffu, f);
    if (!fresh) {
      if (lane == 0) a.chunk_cnt[ch] = 0;
      return;
    }
  }
  float* w0 = tile;
  float* w1 = tile + wn;
  int* kidx = reinterpret_cast<int*>(tile + 2 * wn);
  __syncwarp();                         // the tile's earlier readers are done
  for (int i0 = 0; i0 < wn; i0 += 128) {
    unsigned long long pv[4];
    float cv[4];
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const int i = i0 + 32 * h + lane, col = a0 - nt + i;
      const bool in = i < wn && col >= nt && col < L - nt;
      const bool fr = in && ((fresh >> (col / kCol - bb0)) & 1u);
      pv[h] = fr ? pprev[col] : 0ull;
      cv[h] = in && !fr ? a.cfmax[col] : 0.f;
    }
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const int i = i0 + 32 * h + lane, col = a0 - nt + i;
      if (i >= wn) continue;
      const bool in = col >= nt && col < L - nt;
      const bool fr = in && ((fresh >> (col / kCol - bb0)) & 1u);
      const float v = col < 0 || col >= L ? -INFINITY : (fr ? pack_value(pv[h]) : cv[h]);
      w0[i] = v;
      if (i >= nt && i < nt + kChunk) {
        kidx[i - nt] = fr ? pack_index(pv[h]) : -1;
        if (fr) {
          a.cfmax[col] = v;
          a.imax[col] = pack_index(pv[h]);
        }
      }
    }
  }
  __syncwarp();
  const int len = 2 * nt + 1;
  // the chunk's own scores leave the window before the levels overwrite it
  float own[kChunk / 32];
#pragma unroll
  for (int h = 0; h < kChunk / 32; ++h) own[h] = w0[nt + 32 * h + lane];
  int m = 1;
  float* src = w0;
  float* dst = w1;
  while (2 * m <= len) {
    for (int i = lane; i + 2 * m <= wn; i += 32) dst[i] = fmaxf(src[i], src[i + m]);
    __syncwarp();
    m *= 2;
    float* t = src;
    src = dst;
    dst = t;
  }
  // peaks in time order: their columns to the free buffer
  int* list = reinterpret_cast<int*>(dst);
  int total = 0;
#pragma unroll
  for (int h = 0; h < kChunk / 32; ++h) {
    const int i = 32 * h + lane, tau = a0 + i;
    bool pk = false;
    if (tau < a1 && tau >= nt && tau < L - nt) {
      const float pooled = fmaxf(src[i], src[i + len - m]);
      pk = (pooled > a.th2) && (fabsf(__fsub_rn(pooled, own[h])) < 1e-9f);
    }
    const unsigned bal = __ballot_sync(0xffffffffu, pk);
    if (pk) list[total + __popc(bal & ((1u << lane) - 1u))] = i;
    total += __popc(bal);
  }
  __syncwarp();
  int* tcur = a.tcount + (size_t)p * a.nblk;
  Touch* tch = a.touch + (size_t)p * a.nblk * kTouch;
  unsigned* bits = a.dbits + (size_t)p * a.nwords;
  unsigned long long* pcur = a.pack + (size_t)p * L;
  for (int e0 = 0; e0 < total; e0 += 32) {
    const int e = e0 + lane;
    const bool have = e < total;
    int tau = 0, k = 0;
    float amp = 0.f;
    const int slot = ch * kChunk + e;
    if (have) {
      const int i = list[e];
      tau = a0 + i;
      k = kidx[i];
      if (k < 0) k = a.imax[tau];
      amp = __fdiv_rn(bt_row(a, tau / kCol, k)[tau % kCol], a.nm[k]);
      a.chunk_tau[slot] = tau;
      a.chunk_k[slot] = k;
      a.chunk_amp[slot] = amp;
      a.chunk_th[slot] = __fsqrt_rn(fmaxf(src[i], src[i + len - m]));
    }
    const int b0 = (tau - nt) / kCol, b1 = have ? (tau + nt) / kCol : b0 - 1;
    const int nb = (2 * nt) / kCol + 2;               // blocks a peak can touch
    for (int o = 0; o < nb; o += 8) {
      int pos[8];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        pos[i] = (b0 + o + i <= b1) ? atomicAdd(&tcur[b0 + o + i], 1) : -1;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int b = b0 + o + i;
        if (pos[i] == 0) atomicOr(&bits[b >> 5], 1u << (b & 31));
        if (pos[i] >= 0) {
          if (pos[i] < kTouch) tch[(size_t)b * kTouch + pos[i]] = Touch{tau, k, amp, slot};
          else ks_ctl_fail(a.ctl, KS_ERR_DEGENERATE);
        }
        // a block's first registration clears its rescoring slots
        for (unsigned f = __ballot_sync(0xffffffffu, pos[i] == 0); f; f &= f - 1u) {
          const int c = __shfl_sync(0xffffffffu, b, __ffs(f) - 1) * kCol + lane;
          if (c < L) pcur[c] = 0ull;
        }
      }
    }
  }
  if (lane == 0) a.chunk_cnt[ch] = total;
}

// Both exclusive prefixes an iteration needs, in one pass: of the chunk peak
// counts into s.prefix[0..nchunks] and of the dirty-bitmap word popcounts into
// s.wprefix[0..nwords].  All threads of the block take part.
__device__ void two_prefix(const int* cnt, int nchunks, const unsigned* bits, int nwords,
                           const Smem& s, int& total, int& ndirty) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int pc = (nchunks + kThreads - 1) / kThreads;
  const int pw = (nwords + kThreads - 1) / kThreads;
  int lc = 0, lw = 0;
  for (int i = 0; i < pc; ++i) {
    const int c = tid * pc + i;
    if (c < nchunks) lc += cnt[c];
  }
  for (int i = 0; i < pw; ++i) {
    const int w = tid * pw + i;
    if (w < nwords) lw += __popc(bits[w]);
  }
  int ic = lc, iw = lw;
  for (int o = 1; o < 32; o <<= 1) {
    const int vc = __shfl_up_sync(0xffffffffu, ic, o);
    const int vw = __shfl_up_sync(0xffffffffu, iw, o);
    if (lane >= o) { ic += vc; iw += vw; }
  }
  int* wc = s.wcnt;                 // [kWarps+1] chunk totals per warp
  int* ww = s.kidx;                 // [kWarps+1] word totals per warp (kidx is free here)
  if (lane == 31) { wc[warp] = ic; ww[warp] = iw; }
  __syncthreads();
  if (tid == 0) {
    int ac = 0, aw = 0;
    for (int w = 0; w < kWarps; ++w) {
      const int c = wc[w], x = ww[w];
      wc[w] = ac; ww[w] = aw;
      ac += c; aw += x;
    }
    wc[kWarps] = ac; ww[kWarps] = aw;
  }
  __syncthreads();
  int rc = wc[warp] + ic - lc, rw = ww[warp] + iw - lw;
  for (int i = 0; i < pc; ++i) {
    const int c = tid * pc + i;
    if (c < nchunks) { s.prefix[c] = rc; rc += cnt[c]; }
  }
  for (int i = 0; i < pw; ++i) {
    const int w = tid * pw + i;
    if (w < nwords) {
      const unsigned v = bits[w];
      s.dw[w] = v;
      s.wprefix[w] = rw;
      rw += __popc(v);
    }
  }
  if (tid == 0) { s.prefix[nchunks] = wc[kWarps]; s.wprefix[nwords] = ww[kWarps]; }
  __syncthreads();
  total = s.prefix[nchunks];
  ndirty = s.wprefix[nwords];
}

// ---------------------------------------------------------------- UPDATE
// Ordered touch list of one block in the warp's shared-memory slot: entry e
// (application order: even global index first, then odd, each ascending) has
// peak time tau[e], template k[e], amplitude amp[e].
struct TouchList {
  int n;
  const int* tau;
  const int* k;
  const float* amp;
};

// The lane's registration of block blk (lanes below kTouch) and their number.
struct TouchWord {
  Touch t;
  int n;
};
__device__ __forceinline__ TouchWord touch_word(const PeelArgs& a, int p, int blk, int lane) {
  TouchWord w{Touch{0, 0, 0.f, 0}, 0};
  if (lane < kTouch) w.t = a.touch[((size_t)p * a.nblk + blk) * kTouch + lane];
  w.n = a.tcount[(size_t)p * a.nblk + blk];
  return w;
}

__device__ __forceinline__ TouchList order_touch_warp(const Smem& s, const TouchWord& w, int lane,
                                                      int warp) {
  const int n = min(w.n, kTouch);
  int key = 0x7fffffff;
  if (lane < n) {
    const int ch = w.t.slot / kChunk;
    const int g = s.prefix[ch] + (w.t.slot - ch * kChunk);
    key = ((g & 1) << 30) | g;
  }
  int rank = 0;
  for (int j = 0; j < n; ++j) {
    const int kj = __shfl_sync(0xffffffffu, key, j);
    rank += (kj < key) ? 1 : 0;
  }
  int* tau = s.tl_tau + warp * kTouch;
  int* kk = s.tl_k + warp * kTouch;
  float* amp = s.tl_amp + warp * kTouch;
  __syncwarp();
  if (lane < n) {
    tau[rank] = w.t.tau;
    kk[rank] = w.t.k;
    amp[rank] = w.t.amp;
  }
  __syncwarp();
  return TouchList{n, tau, kk, amp};
}

__device__ __forceinline__ TouchList load_touch_warp(const PeelArgs& a, const Smem& s,
                                                     int p, int blk, int lane, int warp) {
  return order_touch_warp(s, touch_word(a, p, blk, lane), lane, warp);
}

// Columns of block blk x template rows [j_lo, j_hi): subtract the touching
// peaks, store the changed rows, fold the rescored rows into pack_out.  Most
// columns are touched by one peak; its cross-correlations are loaded with the
// rows of B (16 rows per round trip).  Later peaks of the same column (at
// most one more unless scores tie exactly) are applied in a second round, in
// the same order.  A column no peak touches keeps its rows, so its score is
// its settled one (cfmax/imax): the item holding row 0 passes that on instead
// of re-reading the rows (all columns are scored from B when init is set).
template <int kRows>
__device__ void update_warp_item(const PeelArgs& a, const TouchList& tl, int blk,
                                 int j_lo, int j_hi, unsigned long long* pack_out,
                                 int lane, bool init = false) {
  const int c = blk * kCol + lane;
  const bool colok = c < a.L;
  const int nt = a.nt, K = a.K, nlag = 2 * nt + 1;
  int e0 = -1;
  unsigned rest = 0u;                                 // further touching entries
  for (int e = 0; e < tl.n; ++e) {
    const int d = c - tl.tau[e];
    if (colok && d >= -nt && d <= nt) {
      if (e0 < 0) e0 = e;
      else rest |= 1u << e;
    }
  }
  const bool touched = e0 >= 0;
  const bool score = init || touched;
  const bool any_rest = __any_sync(0xffffffffu, rest != 0u);
  const float* cp0 = a.ctcT;
  float amp0 = 0.f;
  if (e0 >= 0) { cp0 = a.ctcT + (size_t)tl.k[e0] * K * nlag + (c - tl.tau[e0] + nt); amp0 = tl.amp[e0]; }
  float* bcol = a.Bt + (size_t)blk * K * kCol + lane;
  float best = -1.f;
  int arg = 0;
  for (int j0 = j_lo; j0 < j_hi; j0 += kRows) {
    float bv[kRows], w0[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const int j = j0 + r;
      const bool ok = score && colok && j < j_hi;
      bv[r] = ok ? bcol[(size_t)j * kCol] : 0.f;
      w0[r] = (ok && e0 >= 0) ? __ldg(cp0 + (size_t)j * nlag) : 0.f;
    }
    if (e0 >= 0) {
#pragma unroll
      for (int r = 0; r < kRows; ++r) bv[r] = __fsub_rn(bv[r], __fmul_rn(amp0, w0[r]));
    }
    if (any_rest) {
      for (int e = 0; e < tl.n; ++e) {
        if ((rest >> e) & 1u) {
          const float amp = tl.amp[e];
          const float* cp = a.ctcT + (size_t)tl.k[e] * K * nlag + (c - tl.tau[e] + nt);
#pragma unroll
          for (int r = 0; r < kRows; ++r) {
            const int j = j0 + r;
            w0[r] = (j < j_hi) ? __ldg(cp + (size_t)j * nlag) : 0.f;
          }
#pragma unroll
          for (int r = 0; r < kRows; ++r) bv[r] = __fsub_rn(bv[r], __fmul_rn(amp, w0[r]));
        }
      }
    }
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const int j = j0 + r;
      if (score && colok && j < j_hi) {
        if (touched) bcol[(size_t)j * kCol] = bv[r];
        fold_score(bv[r], __ldg(a.nmi + j), j, best, arg);
      }
    }
  }
  if (colok) {
    if (score) {
      if (best >= 0.f) atomicMax(&pack_out[c], pack_score(best, arg));
    } else if (j_lo == 0) {
      atomicMax(&pack_out[c], pack_score(a.cfmax[c], a.imax[c]));
    }
  }
}

// Exponent field of |x| as the no-op test reads a score: the biased exponent
// of a normal number; 0 for zero, subnormal, infinite and NaN values, whose
// groups then always take the exact path.
__device__ __forceinline__ int noop_expo(float x) {
  const int e = (int)((__float_as_uint(x) >> 23) & 0xffu);
  return e == 255 ? 0 : e;
}

// Exponent field of a non-negative product bound (255 for infinity or NaN,
// which never passes the test).
__device__ __forceinline__ int bound_expo(float b) {
  return (int)((__float_as_uint(b) >> 23) & 0xffu);
}

// cp.async global -> shared of 16 bytes (L2 only), and the wait for this
// thread's copies.
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// ----------------------------------------------------------- grouped update
// Grouped form of update_warp_item.  The K template rows are cut into groups
// of kGroup rows in the order rperm (templates sorted by the channel centroid
// of their energy, so one group holds templates of neighbouring sites).
// Before touching a group, a column decides from per-group metadata alone
// whether the subtractions can change any of its rows:
//   the product that a subtraction rounds, p = fl(amp * ctc[j,k,l]), has
//   |p| <= fl(|amp| * mg[k][g]) = bnd, because |ctc[j,k,l]| <= mg[k][g] (the
//   group's largest magnitude over rows and lags) and rounding is monotone;
//   if bnd's exponent field Eb satisfies Eb <= gexp - 26, where gexp is the
//   smallest exponent field of |B[j,c]| over the group's rows, then
//   |p| < 2^(Eb-126) <= 2^(gexp-152) <= ulp(B[j,c]) / 4 for every row j of
//   the group, so fl(B[j,c] - p) = B[j,c] exactly (also when B[j,c] is a power
//   of two, where the spacing below it is ulp / 2), for each of the peaks
//   touching the column in turn.
// Zero, subnormal, infinite and NaN scores give gexp = 0, and an infinite or
// NaN bound gives Eb = 255, so those always take the exact path.  A (column,
// group) pair that passes is left as it is: its rows are not read, its
// cross-correlations are not loaded and its cached best (gbest) stands.  The
// other pairs are updated exactly as update_warp_item does (same peaks, same
// order, same roundings), and their gbest and gexp are rewritten.  The
// column's best is the packed maximum over all groups (larger score, then the
// smaller template index), which equals update_warp_item's in-order fold.
//
// An iteration's update runs in two phases separated by a team barrier, so
// that the uneven work (a dirty block needs anywhere from none to all of its
// groups) is spread evenly: group_scan (one warp per dirty block) reads
// only metadata, folds the cached bests of the groups its columns leave
// alone into the column maxima and appends each group that some column must
// process to the iteration's unit list; run_units processes one such group tile.

// Per-lane view of an ordered touch list: the first entry touching this
// column (-1: none) and the mask of the others.
struct LaneEntries {
  int e0;
  unsigned rest;
};

// Inputs of a unit (a group tile that some columns of a block must process)
// in shared memory: the block's ordered touch list as the scan published it,
// the group's row indices and {nm, 1/sqrt(nm)}.  The tables are padded to whole
// groups with copies of the last template, whose rows are then read, updated
// and written with the same values more than once and fold to the same best.
struct UnitIn {
  int list[32];        // n, tau[kTouch], k[kTouch], amp bits[kTouch]
  int row[kGroup];
  float2 nm[kGroup];
};
constexpr int kUnitSlots = 2;
static_assert(sizeof(UnitIn) * kUnitSlots == kUnitBytes && sizeof(UnitIn) == 512 && 1 + 3 * kTouch <= 32, "one 16-byte piece per lane");

__device__ __forceinline__ UnitIn* unit_in(const Smem& s, int warp, int i) {
  return s.unit + warp * kUnitSlots + i % kUnitSlots;
}

// Where a unit's touch list comes from: none (initial scores), the list that the
// scan published, or the unit's slot, where the warp itself has put it (kPair).
enum UnitKind { kInit, kListed, kPair };

// Request unit u's inputs (cp.async, a 16-byte piece per lane).
template <UnitKind kKind>
__device__ __forceinline__ void unit_fetch(const PeelArgs& a, uint2 u, UnitIn* in, int lane) {
  const char* src;
  if (lane < 8) src = reinterpret_cast<const char*>(a.blist + (size_t)(u.x >> 11) * 32) + lane * 16;
  else if (lane < 16) src = reinterpret_cast<const char*>(a.rperm + (u.x & 2047u) * kGroup) + (lane - 8) * 16;
  else src = reinterpret_cast<const char*>(a.nmip + (u.x & 2047u) * kGroup) + (lane - 16) * 16;
  if (kKind == kListed || lane >= 8) cp_async16(reinterpret_cast<char*>(in) + lane * 16, src);
  cp_async_commit();
}

// min(m, |x|, |y|), NaN when any of them is; max(m, x, y), NaNs passed over.
__device__ __forceinline__ float min_abs_nan(float m, float x, float y) {
  float r;
  asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(m), "f"(fabsf(x)), "f"(fabsf(y)));
  return r;
}
// All ones where x >= y, else 0 (also for NaN).
__device__ __forceinline__ unsigned mask_ge(float x, float y) {
  unsigned r;
  asm("set.ge.u32.f32 %0, %1, %2;" : "=r"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float max3(float m, float x, float y) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(m), "f"(x), "f"(y));
  return r;
}

// The columns of a group tile a lane reads, and the one it owns: lane
// (rq, cq) = (lane / 8, lane % 8) holds rows 4i + rq and columns 4cq .. 4cq+3
// of the 32 x 32 tile, and owns column 4cq + rq.
__device__ __forceinline__ int own_column(int lane) { return 4 * (lane & 7) + (lane >> 3); }

// Stage, for the columns with `mine`, the cross-correlations of one peak (cp:
// row 0 of its slab at this lane's column) with the group's rows into a tile;
// the other columns get zeros.
__device__ __forceinline__ void stage_ctc(float* Cs, const float* cp, bool mine, const int* row,
                                          int nlag, int lane) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(Cs + lane);
  const int bytes = mine ? 4 : 0;
#pragma unroll 2
  for (int r = 0; r < kGroup; r += 4) {
    const int4 j = *reinterpret_cast<const int4*>(row + r);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d + r * 128), "l"(cp + (unsigned)(j.x * nlag)), "r"(bytes) : "memory");
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d + r * 128 + 128), "l"(cp + (unsigned)(j.y * nlag)), "r"(bytes) : "memory");
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d + r * 128 + 256), "l"(cp + (unsigned)(j.z * nlag)), "r"(bytes) : "memory");
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d + r * 128 + 384), "l"(cp + (unsigned)(j.w * nlag)), "r"(bytes) : "memory");
  }
  cp_async_commit();
}

// b += (-amp) * c over the lane's 8 x 4 elements: the product and the sum are
// rounded separately, b - fl(amp c).  A column that takes no part has
// n = -0 and c = +0: b + (-0) = b exactly.
__device__ __forceinline__ void apply_ctc(const float* Cs, unsigned long long n01,
                                          unsigned long long n23, unsigned long long one2,
                                          unsigned long long (&b)[8][2], int lane) {
  const float* c = Cs + (lane >> 3) * 32 + (lane & 7) * 4;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(c + i * 128);
    b[i][0] = f2_add_prod(b[i][0], n01, v.x, one2);
    b[i][1] = f2_add_prod(b[i][1], n23, v.y, one2);
  }
}

// The four columns' values of a per-column quantity, packed in pairs.
__device__ __forceinline__ void column_pairs(float v, int lane, unsigned long long& p01,
                                             unsigned long long& p23) {
  const int c = 4 * (lane & 7);
  const float v0 = __shfl_sync(0xffffffffu, v, c), v1 = __shfl_sync(0xffffffffu, v, c + 1);
  const float v2 = __shfl_sync(0xffffffffu, v, c + 2), v3 = __shfl_sync(0xffffffffu, v, c + 3);
  p01 = f2_pack(v0, v1);
  p23 = f2_pack(v2, v3);
}

// This lane's column's address in the slab of entry e's template.
__device__ __forceinline__ const float* entry_slab(const PeelArgs& a, const UnitIn* in, int e, int c) {
  return a.ctcT + (size_t)in->list[1 + kTouch + e] * a.K * (2 * a.nt + 1) +
         (c - in->list[1 + e] + a.nt);
}

// Start of a unit whose inputs have landed: every column in `cols` stages its
// first touching peak's cross-correlations (not waited for).  Returns the
// lane's column's entries.
__device__ __forceinline__ LaneEntries unit_begin(const PeelArgs& a, const UnitIn* in, uint2 u,
                                                  float* Cs, int lane) {
  const int c = (int)(u.x >> 11) * kCol + lane;
  LaneEntries le{-1, 0u};
  if ((u.y >> lane) & 1u) {
    const int n = in->list[0];
    for (int e = 0; e < n; ++e) {
      const int d = c - in->list[1 + e];
      if (c < a.L && d >= -a.nt && d <= a.nt) {
        if (le.e0 < 0) le.e0 = e;
        else le.rest |= 1u << e;
      }
    }
  }
  __syncwarp();
  const bool first = le.e0 >= 0;
  stage_ctc(Cs, first ? entry_slab(a, in, le.e0, c) : a.ctcT, first, in->row, 2 * a.nt + 1, lane);
  return le;
}

// The unit's 32 rows x 32 columns of B, whole rows as 16-byte pieces: a lane
// holds 8 rows x 4 columns.
__device__ __forceinline__ void unit_rows(const PeelArgs& a, const UnitIn* in, uint2 u,
                                          unsigned long long (&b)[8][2], int lane) {
  const int* row = in->row + (lane >> 3);
  const float* brow = a.Bt + (size_t)(u.x >> 11) * a.K * kCol + (lane & 7) * 4;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(brow + (unsigned)row[4 * i] * kCol);
    b[i][0] = v.x;
    b[i][1] = v.y;
  }
}

// The scores of a unit's updated rows (b, and kept in the slot's tile): the
// smallest magnitude e0, the largest t and the candidate rows of the lane's
// own column (own_column), found in two passes over the lane's 8 x 4 elements;
// unit_fold then folds the candidates.
//
// The best over the group's rows is found without a division per row.  With
// t = fl(b * fl(1/sqrt(nm))), nm in [2^-30, 2^30], t is within a relative
// 2^-23 of b/sqrt(nm), so for a largest t in [2^-45, 2^48] (its b is then in
// [2^-60, 2^63], its square and quotient normal, and no row's square infinite)
// the exactly rounded scores cf = fl(fl(b^2) / nm) of two rows are
// ordered as their t wherever those differ by more than a relative 2^-21: only
// rows with t >= (1 - 2^-20) max t can hold the best, and only their quotients
// are computed and folded (larger score, then the smaller template index).
// When no t is above 0 every row's score is +0 exactly (NaN scores count as 0,
// as relu of a failed comparison), and the smallest template index wins.  A
// largest t outside that interval, or a group with an nm outside its range
// (marked by a NaN scale), folds every row's quotient.
//
// What bounds it: latency (a launch of teams uses 37 % of the issue slots, 45 % of
// L1's rate, 21 % of L2's): the unit's loads (about 14 KB), then the phase's
// barrier.  Four columns per lane make one 16-byte access, one
// row index and one scale serve four elements, and the products, differences
// and scores run two per packed FP32 instruction; the form with one column per
// lane and a division-free fold of larger state took about three times the
// instructions (peel of a C=384, K=600 batch 2.40 -> 1.70 ms, of 16 such
// batches by 16 teams 21.6 -> 14.0 ms, with the scan and detection below).
// Measured and dropped: the next unit's rows and cross-correlations requested
// a unit ahead (registers and a second tile: 6.5-7.5 ms of units in the
// 16-batch launch against 6.2), loads past L1, cross-correlations through
// registers instead of cp.async, more or fewer warps per SM at equal tiles.
struct UnitScore {
  float e0;        // smallest |b| (NaN if any is)
  float mo;        // largest t
  unsigned rows;   // bit 8k + i: row 4i + k is a candidate
};

// b becomes t.
__device__ __forceinline__ UnitScore unit_score(const UnitIn* in, unsigned long long (&b)[8][2],
                                                int lane) {
  const int rq = lane >> 3;
  float ea[4] = {INFINITY, INFINITY, INFINITY, INFINITY};
  float m[4] = {-1.f, -1.f, -1.f, -1.f};
#pragma unroll
  for (int i = 0; i < 8; i += 2) {
    const float sa = in->nm[4 * i + rq].y, sb = in->nm[4 * i + 4 + rq].y;
    const unsigned long long s2 = f2_pack(sa, sa), s3 = f2_pack(sb, sb);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float x0, x1, y0, y1, t0, t1, u0, u1;
      f2_unpack(b[i][h], x0, x1);
      f2_unpack(b[i + 1][h], y0, y1);
      ea[2 * h] = min_abs_nan(ea[2 * h], x0, y0);
      ea[2 * h + 1] = min_abs_nan(ea[2 * h + 1], x1, y1);
      b[i][h] = f2_mul(b[i][h], s2);
      b[i + 1][h] = f2_mul(b[i + 1][h], s3);
      f2_unpack(b[i][h], t0, t1);
      f2_unpack(b[i + 1][h], u0, u1);
      m[2 * h] = max3(m[2 * h], t0, u0);
      m[2 * h + 1] = max3(m[2 * h + 1], t1, u1);
    }
  }
#pragma unroll
  for (int o = 8; o <= 16; o <<= 1)
#pragma unroll
    for (int h = 0; h < 4; ++h) m[h] = fmaxf(m[h], __shfl_xor_sync(0xffffffffu, m[h], o));
  // candidate rows: bit i of byte h stands for row 4i + rq of column 4cq + h
  unsigned cand = 0u;
  {
    float thr[4];
#pragma unroll
    for (int h = 0; h < 4; ++h) thr[h] = m[h] > 0.f ? m[h] * 0.99999905f : INFINITY;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float t0, t1;
        f2_unpack(b[i][h], t0, t1);
        cand |= mask_ge(t0, thr[2 * h]) & (1u << (8 * (2 * h) + i));
        cand |= mask_ge(t1, thr[2 * h + 1]) & (1u << (8 * (2 * h + 1) + i));
      }
    }
  }
  // hand every column to its owner: its smallest magnitude, largest t and the
  // candidate bits of the four lanes that hold its rows
  const bool up = lane & 16, odd = lane & 8;
  UnitScore r;
  float e0 = up ? ea[2] : ea[0], e1 = up ? ea[3] : ea[1];
  const float x0 = up ? ea[0] : ea[2], x1 = up ? ea[1] : ea[3];
  const float y0 = __shfl_xor_sync(0xffffffffu, x0, 16), y1 = __shfl_xor_sync(0xffffffffu, x1, 16);
  e0 = min_abs_nan(e0, y0, y0);
  e1 = min_abs_nan(e1, y1, y1);
  const float z = __shfl_xor_sync(0xffffffffu, odd ? e0 : e1, 8);
  r.e0 = min_abs_nan(odd ? e1 : e0, z, z);
  r.mo = up ? (odd ? m[3] : m[2]) : (odd ? m[1] : m[0]);
  r.rows = 0u;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const unsigned v = __shfl_sync(0xffffffffu, cand, 8 * k + (lane & 7));
    r.rows |= ((v >> (8 * rq)) & 0xffu) << (8 * k);
  }
  return r;
}

// The group's packed best of the lane's own column when it is in `cols` (its
// gbest and gexp are rewritten), 0 otherwise.
__device__ __forceinline__ unsigned long long unit_fold(const PeelArgs& a, const UnitScore& us,
                                                        const float* Cs, const UnitIn* in, uint2 u,
                                                        int lane) {
  const int oc = own_column(lane);
  const bool ond = (u.y >> oc) & 1u;
  const float scale = in->nm[lane].y;
  const bool odd_nm = __any_sync(0xffffffffu, scale != scale);
  const float mo = us.mo;
  float best = 0.f;
  int arg = __reduce_min_sync(0xffffffffu, in->row[lane]);
  const bool all = odd_nm || !(mo <= 0.f || (mo >= 2.8421709e-14f && mo <= 2.8147498e14f));
  unsigned rows = us.rows;
  if (!ond || all || !(mo > 0.f)) rows = 0u;
  if (rows) best = -1.f;
  for (; rows; rows &= rows - 1u) {   // usually one row
    const int bit = __ffs(rows) - 1;
    const int r = 4 * (bit & 7) + (bit >> 3);
    const float x = Cs[r * 32 + oc];
    const float cf = __fdiv_rn(__fmul_rn(x, x), in->nm[r].x);
    const int j = in->row[r];
    if (cf > best || (cf == best && j < arg)) {
      best = cf;
      arg = j;
    }
  }
  if (__any_sync(0xffffffffu, ond && all)) {
    if (all) {
      best = -1.f;
      arg = 0x7fffffff;
      for (int r = 0; r < kGroup; ++r) {
        const float x = Cs[r * 32 + oc];
        const float rl = x > 0.f ? x : 0.f;
        const float sq = __fmul_rn(rl, rl);
        const float nm = in->nm[r].x;
        const bool normal = nm >= 1.17549435e-38f && nm <= 3.40282347e38f;
        const float cf = (sq == 0.f && normal) ? 0.f : __fdiv_rn(sq, nm);
        const int j = in->row[r];
        if (cf > best || (cf == best && j < arg)) {
          best = cf;
          arg = j;
        }
      }
    }
  }
  unsigned long long gb = 0ull;
  if (ond) {
    gb = best >= 0.f ? pack_score(best, arg) : 0ull;
    const size_t mi = ((size_t)(u.x >> 11) * a.ng + (u.x & 2047u)) * 32 + oc;
    a.gbest[mi] = gb;
    a.gexp[mi] = (unsigned char)noop_expo(us.e0);
  }
  return gb;
}

// The units first, first + step, ... (nu of them) of the iteration's list (one
// unit with kPair), or (kInit) of all nblk * ng tiles, whose initial scores are
// folded (nothing is subtracted or written back).  Per unit: its rows and staged
// cross-correlations are waited for, the columns subtract their touching peaks
// in application order (further peaks stage theirs in the tile once it is
// read), the rows are written back and scored.  The next unit's inputs are
// fetched once this one's peaks are applied.
template <UnitKind kKind>
__device__ void run_units(const PeelArgs& a, const Smem& s, long long first, long long step,
                          int nu, uint2 rec, unsigned long long* pack_out, int lane, int warp) {
  auto record = [&](int i) {
    if (kKind == kInit) {
      const unsigned w = (unsigned)first + (unsigned)i * (unsigned)step, ng = (unsigned)a.ng;
      const int blk = (int)(w / ng), left = a.L - blk * kCol;
      return make_uint2(((unsigned)blk << 11) | (w % ng),
                        left >= kCol ? 0xffffffffu : (1u << left) - 1u);
    }
    return make_uint2(__shfl_sync(0xffffffffu, rec.x, i), __shfl_sync(0xffffffffu, rec.y, i));
  };
  if (nu <= 0) return;
  uint2 u = record(0);
  float* Cs = unit_tile(s, warp);
  __syncwarp();                       // the tile's and the slots' earlier readers are done
  unit_fetch<kKind>(a, u, unit_in(s, warp, 0), lane);
#pragma unroll 1
  for (int i = 0; i < nu; ++i) {
    const UnitIn* in = unit_in(s, warp, i);
    cp_async_wait_all();
    __syncwarp();                     // the unit's inputs have landed
    unsigned long long b[8][2];
    LaneEntries le{-1, 0u};
    if (kKind != kInit) le = unit_begin(a, in, u, Cs, lane);
    unit_rows(a, in, u, b, lane);
    uint2 un = u;
    if (i + 1 < nu) un = record(i + 1);
    if (kKind != kInit) {
      const unsigned long long one2 = f2_pack(a.one, a.one);
      unsigned long long n01, n23;
      column_pairs(le.e0 >= 0 ? -__int_as_float(in->list[1 + 2 * kTouch + le.e0]) : -0.f, lane, n01,
                   n23);
      cp_async_wait_all();
      __syncwarp();                   // every lane's staged column has landed
      apply_ctc(Cs, n01, n23, one2, b, lane);
#pragma unroll 1
      for (unsigned m = __reduce_or_sync(0xffffffffu, le.rest); m; m &= m - 1u) {
        const int e = __ffs(m) - 1;
        const bool mine = (le.rest >> e) & 1u;
        __syncwarp();                 // the tile is read
        stage_ctc(Cs, mine ? entry_slab(a, in, e, (int)(u.x >> 11) * kCol + lane) : a.ctcT, mine,
                  in->row, 2 * a.nt + 1, lane);
        column_pairs(mine ? -__int_as_float(in->list[1 + 2 * kTouch + e]) : -0.f, lane, n01, n23);
        cp_async_wait_all();
        __syncwarp();
        apply_ctc(Cs, n01, n23, one2, b, lane);
      }
    }
    if (i + 1 < nu) unit_fetch<kKind>(a, un, unit_in(s, warp, i + 1), lane);
    // write back; the tile keeps the scores for the quotients
    {
      const int rq = lane >> 3;
      float* cs = Cs + rq * 32 + (lane & 7) * 4;
      float* brow = a.Bt + (size_t)(u.x >> 11) * a.K * kCol + (lane & 7) * 4;
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const ulonglong2 v = make_ulonglong2(b[r][0], b[r][1]);
        if (kKind != kInit)
          *reinterpret_cast<ulonglong2*>(brow + (unsigned)in->row[4 * r + rq] * kCol) = v;
        *reinterpret_cast<ulonglong2*>(cs + r * 128) = v;
      }
    }
    const UnitScore us = unit_score(in, b, lane);
    __syncwarp();                     // the tile holds every lane's scores
    const unsigned long long gb = unit_fold(a, us, Cs, in, u, lane);
    if (gb) atomicMax(&pack_out[(u.x >> 11) * kCol + own_column(lane)], gb);
    u = un;
  }
}

// Block of the rank-th set bit of the dirty bitmap (s.wprefix holds the
// exclusive prefix of the word popcounts).
__device__ __forceinline__ int dirty_block(const Smem& s, int nwords, int rank) {
  int lo = 0, hi = nwords - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (s.wprefix[mid] <= rank) lo = mid; else hi = mid - 1;
  }
  const unsigned word = s.dw[lo];
  const int bit = (int)__fns(word, 0, rank - s.wprefix[lo] + 1);
  return lo * 32 + bit;
}

// Phase A over the dirty blocks w, w + step, ... below ndirty, one warp per
// block: publish the block's ordered touch list for its units, decide per
// column and group from the metadata, fold the cached bests of the groups a
// column leaves alone (and the settled score of a column no peak touches)
// into pack_out, and append the groups some column must process to the unit
// list.  The next block's touch list is read, and the place of this block's
// units in the list comes back, while the next block's metadata is on its way.
//
// What bounds it: the latency of its chain (touch list, bounds, metadata); with
// every step of it exposed, a block took 13 us at K = 600.
__device__ void group_scan(const PeelArgs& a, const Smem& s, int p, long long w, long long step,
                           int ndirty, unsigned long long* pack_out, int lane, int warp) {
  if (w >= ndirty) return;
  const int nt = a.nt, ng = a.ng;
  // the block's metadata, kScanGroups groups at a time: [gn][32] bests, then
  // [gn][32] exponents
  unsigned long long* sb = reinterpret_cast<unsigned long long*>(unit_tile(s, warp));
  unsigned char* se = reinterpret_cast<unsigned char*>(sb + kScanGroups * 32);
  auto fetch = [&](int blk, int gc, int gn) {
    const char* gb = reinterpret_cast<const char*>(a.gbest + ((size_t)blk * ng + gc) * 32);
    const char* ge = reinterpret_cast<const char*>(a.gexp + ((size_t)blk * ng + gc) * 32);
    for (int i = lane; i < gn * 16; i += 32) cp_async16(reinterpret_cast<char*>(sb) + i * 16, gb + i * 16);
    for (int i = lane; i < gn * 2; i += 32) cp_async16(reinterpret_cast<char*>(se) + i * 16, ge + i * 16);
    cp_async_commit();
  };
  unsigned char* eb = s.eb + warp * (kTouch * 32);
  unsigned* ucount = a.wctr + 2 + p;
  // units whose place in the list has been asked for: lane i holds group
  // (at & 2047) + i's columns
  unsigned base = 0u, pend = 0u, pcols = 0u, at = 0u;
  auto flush = [&]() {
    if (pend) {
      const unsigned first = __shfl_sync(0xffffffffu, base, 0);
      if ((pend >> lane) & 1u)
        a.units[first + __popc(pend & ((1u << lane) - 1u))] = make_uint2(at + lane, pcols);
      pend = 0u;
    }
  };
  int blk = dirty_block(s, a.nwords, (int)w);
  TouchWord t = touch_word(a, p, blk, lane);
  while (true) {
    const int c = blk * kCol + lane;
    const bool colok = c < a.L;
    __syncwarp();                       // the tile's earlier readers are done
    fetch(blk, 0, min(kScanGroups, ng));
    const TouchList tl = order_touch_warp(s, t, lane, warp);
    w += step;
    const int next = w < ndirty ? dirty_block(s, a.nwords, (int)w) : -1;
    if (next >= 0) t = touch_word(a, p, next, lane);
    int* bl = a.blist + (size_t)blk * 32;
    if (lane == 0) bl[0] = tl.n;
    if (lane < tl.n) {
      bl[1 + lane] = tl.tau[lane];
      bl[1 + kTouch + lane] = tl.k[lane];
      bl[1 + 2 * kTouch + lane] = __float_as_int(tl.amp[lane]);
    }
    unsigned tmask = 0u;
    for (int e = 0; e < tl.n; ++e) {
      const int d = c - tl.tau[e];
      if (colok && d >= -nt && d <= nt) tmask |= 1u << e;
    }
    const bool touched = tmask != 0u;
    unsigned long long colbest = 0ull;
    for (int gc = 0; gc < ng; gc += kScanGroups) {
      const int gn = min(kScanGroups, ng - gc);
      if (gc > 0) {
        __syncwarp();
        fetch(blk, gc, gn);
      }
      // exponent fields of the product bounds of every touching peak plus 26,
      // for the groups gc + lane
      for (int e = 0; e < tl.n; ++e) {
        int x = 255;
        if (lane < gn)
          x = min(255, 26 + bound_expo(__fmul_rn(fabsf(tl.amp[e]),
                                                 __ldg(a.mg + (size_t)tl.k[e] * ng + gc + lane))));
        eb[e * 32 + lane] = (unsigned char)x;
      }
      flush();
      cp_async_wait_all();
      __syncwarp();
      // groups that the lane's first peak can change, then those that a further
      // peak can (exponents are at most 254: a bound of 255 always passes)
      unsigned need = 0u;
      if (touched) {
        const unsigned char* b0 = eb + (__ffs(tmask) - 1) * 32;
#pragma unroll 4
        for (int i = 0; i < gn; ++i) need |= b0[i] > se[i * 32 + lane] ? 1u << i : 0u;
        for (unsigned m = tmask & (tmask - 1u); m; m &= m - 1u) {
          const unsigned char* b1 = eb + (__ffs(m) - 1) * 32;
          for (int i = 0; i < gn; ++i) need |= b1[i] > se[i * 32 + lane] ? 1u << i : 0u;
        }
        for (unsigned m = ~need & (gn == 32 ? 0xffffffffu : (1u << gn) - 1u); m; m &= m - 1u) {
          const unsigned long long gb = sb[(__ffs(m) - 1) * 32 + lane];
          colbest = gb > colbest ? gb : colbest;
        }
      }
      const unsigned proc = __reduce_or_sync(0xffffffffu, need);
      if (proc) {
        if (lane == 0) base = atomicAdd(ucount, (unsigned)__popc(proc));
        for (unsigned m = proc; m; m &= m - 1u) {
          const int i = __ffs(m) - 1;
          const unsigned b = __ballot_sync(0xffffffffu, (need >> i) & 1u);
          if (lane == i) pcols = b;
        }
        pend = proc;
        at = ((unsigned)blk << 11) | (unsigned)gc;
      }
    }
    if (colok) {
      if (touched) {
        if (colbest) atomicMax(&pack_out[c], colbest);
      } else {
        atomicMax(&pack_out[c], pack_score(a.cfmax[c], a.imax[c]));
      }
    }
    if (next < 0) break;
    blk = next;
  }
  flush();
}

// (dirty block, group) pairs per warp up to which pairs are updated as they are
// looked at: peel at C=96, K=80, L=60122 173 us with the list alone, 164 with one
// pair per warp, 154 with two or four (more pairs are better dealt as the units
// that the list leaves of them).
constexpr long long kFusedItems = 2;

// The records of nu units from `first` in steps of `step`: one per lane.
__device__ __forceinline__ uint2 unit_records(const PeelArgs& a, long long first, long long step,
                                              int nu, int lane) {
  return lane < nu ? a.units[first + lane * step] : make_uint2(0u, 0u);
}

// One (dirty block, group) pair w: what group_scan does for one group (the warp
// of group 0 also folds the untouched columns), then the unit if there is one.
__device__ __forceinline__ void scan_and_update(const PeelArgs& a, const Smem& s, int p, int w,
                                                unsigned long long* pack_out, int lane, int warp) {
  const int nt = a.nt, ng = a.ng;
  const int blk = dirty_block(s, a.nwords, w / ng), g = w % ng;
  const int c = blk * kCol + lane;
  const bool colok = c < a.L;
  const size_t at = ((size_t)blk * ng + g) * 32 + lane;
  const unsigned long long best = a.gbest[at];
  const int expo = a.gexp[at];
  const TouchList tl = order_touch_warp(s, touch_word(a, p, blk, lane), lane, warp);
  // exponent field of the lane's peak's product bound plus 26
  int x = 255;
  if (lane < tl.n)
    x = min(255, 26 + bound_expo(__fmul_rn(fabsf(tl.amp[lane]),
                                           __ldg(a.mg + (size_t)tl.k[lane] * ng + g))));
  bool touched = false, need = false;
  for (int e = 0; e < tl.n; ++e) {
    const int d = c - tl.tau[e];
    const int xe = __shfl_sync(0xffffffffu, x, e);
    if (colok && d >= -nt && d <= nt) {
      touched = true;
      need |= xe > expo;
    }
  }
  if (touched) {
    if (!need && best) atomicMax(&pack_out[c], best);
  } else if (colok && g == 0) {
    atomicMax(&pack_out[c], pack_score(a.cfmax[c], a.imax[c]));
  }
  const unsigned cols = __ballot_sync(0xffffffffu, need);
  if (!cols) return;
  // the list goes to the warp's own slot: the warps of this block's other groups
  // have theirs at the same time
  int* list = unit_in(s, warp, 0)->list;
  __syncwarp();                         // the slot's earlier readers are done
  if (lane == 0) list[0] = tl.n;
  if (lane < tl.n) {
    list[1 + lane] = tl.tau[lane];
    list[1 + kTouch + lane] = tl.k[lane];
    list[1 + 2 * kTouch + lane] = __float_as_int(tl.amp[lane]);
  }
  run_units<kPair>(a, s, 0, 1, 1, make_uint2(((unsigned)blk << 11) | (unsigned)g, cols), pack_out,
                   lane, warp);
}

// Outcome of one batch's peel, the same in every block of the team.
struct PeelOutcome {
  long long n_out;
  int iters;
  int status;
};

// The peel of one batch by a team of G co-resident blocks (this block has
// rank `rank` in it); epoch is the team barrier's count of passed barriers,
// carried across the batches a team processes.  The team first clears the
// batch's per-run state, then runs the iterations; the outcome goes to info
// (written by one thread) and is returned to every thread.  When the status
// is KS_OK every record and residual list of the batch is complete and
// visible to the team (the last pass ended at a team barrier).
// `again`: another batch follows in the same scratch.
template <int kRows, bool kGrouped>
__device__ PeelOutcome run_peel(const PeelArgs& a, const Smem& s, int rank, unsigned G,
                                unsigned& epoch, bool again) {
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  // warps are numbered across the blocks, so that fewer items than warps are
  // spread over every SM
  const long long gwarp = (long long)warp * G + rank;
  const long long nwarps = (long long)G * kWarps;
  stage_basis(a.W, a.P, a.nt, s.W, kThreads);
  // a failed producer of the score matrix fails the peel
  if (rank == 0 && tid == 0 && a.upstream_err) {
    const int ue = ks_ld_volatile(a.upstream_err);
    if (ue) ks_ctl_fail(a.ctl, ue);
  }
  // per-batch state starts empty: registration counts, dirty bitmaps, both
  // rescoring buffers (pack[1] receives the initial scores), work counters and
  // the residual lists
  {
    const long long t0 = (long long)rank * kThreads + tid, ts = (long long)G * kThreads;
    for (long long i = t0; i < 2LL * a.nblk; i += ts) a.tcount[i] = 0;
    for (long long i = t0; i < 2LL * a.nwords; i += ts) a.dbits[i] = 0u;
    for (long long i = t0; i < 2LL * a.L; i += ts) a.pack[i] = 0ull;
    for (long long i = t0; i < a.nblk; i += ts) a.xcount[i] = 0;
    if (t0 < 6) a.wctr[t0] = 0u;
  }
  if (!ks_grid_sync(a.ctl, G, epoch, a.limit_ns)) {
    const int e = ks_ctl_error(a.ctl);
    if (rank == 0 && tid == 0) {
      a.info[0] = 0;
      a.info[1] = e;
      a.info[2] = 0;
      a.info[3] = 0;
    }
    return PeelOutcome{0, 0, e ? e : KS_ERR_TIMEOUT};
  }

  // initial scores of every column, folded into pack[1]
  {
    unsigned long long* pinit = a.pack + (size_t)a.L;
    if (kGrouped) {
      // every (block, group) tile: the group metadata of every column too
      const long long n_items = (long long)a.nblk * a.ng;
      if (gwarp < n_items)
        run_units<kInit>(a, s, gwarp, nwarps, (int)((n_items - gwarp + nwarps - 1) / nwarps),
                        make_uint2(0u, 0u), pinit, lane, warp);
    } else {
      const int rg = (a.K + kItemRows - 1) / kItemRows;
      const TouchList none{0, nullptr, nullptr, nullptr};
      const long long n_items = (long long)a.nblk * rg;
      for (long long w = gwarp; w < n_items; w += nwarps) {
        const int blk = (int)(w / rg), r = (int)(w % rg);
        update_warp_item<kRows>(a, none, blk, r * kItemRows, min(a.K, (r + 1) * kItemRows),
                                pinit, lane, true);
      }
    }
  }

  long long n_out = 0;
  int it = 0;
  int status = KS_OK;
  KS_TRACE(199, 0, ks_globaltimer());
  bool ok = ks_grid_sync(a.ctl, G, epoch, a.limit_ns);
  for (; ok && it < a.max_peels; ++it) {
    const int p = it & 1, q = p ^ 1;
    KS_TRACE(it, 0, ks_globaltimer());
    if (warp_detection(a.nt, kGrouped, a.nchunks, G)) {
      for (long long ch = gwarp; ch < a.nchunks; ch += nwarps)
        detect_chunk_warp(a, unit_tile(s, warp), (int)ch, it, lane);
    } else {
      for (int ch = rank; ch < a.nchunks; ch += (int)G) detect_chunk(a, s, ch, it);
    }
    KS_TRACE(it, 1, ks_globaltimer());
    if (!ks_grid_sync(a.ctl, G, epoch, a.limit_ns)) break;
    KS_TRACE(it, 2, ks_globaltimer());

    const unsigned* bits = a.dbits + (size_t)p * a.nwords;
    int total, ndirty;
    two_prefix(a.chunk_cnt, a.nchunks, bits, a.nwords, s, total, ndirty);
    if (total == 0) break;
    if (n_out + total > a.capacity) {
      status = KS_ERR_OVERFLOW;
      if (rank == 0 && tid == 0) a.info[3] = n_out + total;
      break;
    }
    unsigned long long* pcur = a.pack + (size_t)p * a.L;
    KS_TRACE(it, 3, ks_globaltimer());
    if (kGrouped) {
      if ((long long)ndirty * a.ng <= kFusedItems * nwarps) {
        // few (dirty block, group) pairs (a small batch, or the last iterations
        // of a larger one): each pair is looked at and updated by one warp, without
        // a list and its barrier (109 -> 91 us of peel at C=32, K=24, L=4122; 1423
        // -> 1385 at C=384, K=600, L=60122)
        for (long long w = gwarp; w < (long long)ndirty * a.ng; w += nwarps)
          scan_and_update(a, s, p, (int)w, pcur, lane, warp);
      } else {
        // phase A: one warp per dirty block, dealt round-robin (metadata only,
        // about the same work per block)
        group_scan(a, s, p, gwarp, nwarps, ndirty, pcur, lane, warp);
        if (!ks_grid_sync(a.ctl, G, epoch, a.limit_ns)) break;
        // phase B: the units.  Up to kStaticUnits per warp are dealt round-robin
        // (neighbouring warps run one block's groups at the same time; a counter
        // taken one unit at a time by thousands of warps would be their queue);
        // more are taken from a counter in claims of about a quarter of a warp's
        // share (at most 32).  A warp reads its records at once and fetches each
        // unit's inputs while it runs the one before.
        KS_TRACE(it, 7, ks_globaltimer());
        const unsigned n_units = ks_ld_acquire(a.wctr + 2 + p);
        const bool dealt = (long long)n_units <= kStaticUnits * nwarps;
        const unsigned claim =
            (unsigned)min(32LL, max(1LL, (long long)n_units / (nwarps * 4)));
        if (dealt) {
          if (gwarp < n_units) {
            const int nu = (int)((n_units - gwarp + nwarps - 1) / nwarps);
            run_units<kListed>(a, s, gwarp, nwarps, nu, unit_records(a, gwarp, nwarps, nu, lane),
                               pcur, lane, warp);
          }
        } else {
          while (true) {
            unsigned first = 0;
            if (lane == 0) first = atomicAdd(&a.wctr[4 + p], claim);
            first = __shfl_sync(0xffffffffu, first, 0);
            if (first >= n_units) break;
            const int nu = (int)(min(n_units, first + claim) - first);
            run_units<kListed>(a, s, first, 1, nu, unit_records(a, first, 1, nu, lane), pcur,
                               lane, warp);
          }
        }
      }
    } else {
      // update items: (dirty block in column order, row range): the split
      // whose most loaded warp has the least work (row steps of kRows plus one
      // step's worth of per-item set-up)
      const int item_cap = nwarps >= kStaticWarps ? kItemRows : kItemRowsSmall;
      int rows = kItemRows;
      if (ndirty > 0) {
        long long best_cost = -1;
        for (int r = kRows; r <= item_cap; r += kRows) {
          const long long items = (long long)ndirty * ((a.K + r - 1) / r);
          const long long per_warp = (items + nwarps - 1) / nwarps;
          const long long cost = per_warp * (r / kRows + 1);
          if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            rows = r;
          }
        }
      }
      const int rgroups = (a.K + rows - 1) / rows;
      const long long n_items = (long long)ndirty * rgroups;
      // Items go to warps in item order, so consecutive items (neighbouring
      // blocks, which share the slabs of their peaks) run at about the same
      // time.  A small team takes every item from the counter: warps that ran
      // into slower memory take fewer of them (a static deal left the blocks
      // of a 14-block team up to 20 % of an iteration apart at the closing
      // barrier).  A large team deals all but its last round round-robin, so
      // thousands of warps do not queue on one counter.
      const long long rounds = n_items / nwarps;
      const long long n_static =
          (nwarps >= kStaticWarps && rounds > 1) ? (rounds - 1) * nwarps : 0;
      for (long long w = gwarp; w < n_static; w += nwarps) {
        const int blk = dirty_block(s, a.nwords, (int)(w / rgroups));
        const int r = (int)(w % rgroups);
        const TouchList tl = load_touch_warp(a, s, p, blk, lane, warp);
        update_warp_item<kRows>(a, tl, blk, r * rows, min(a.K, (r + 1) * rows), pcur, lane);
      }
      while (true) {
        unsigned next = 0;
        if (lane == 0) next = atomicAdd(&a.wctr[p], 1u);
        const long long w = n_static + (long long)__shfl_sync(0xffffffffu, next, 0);
        if (w >= n_items) break;
        const int blk = dirty_block(s, a.nwords, (int)(w / rgroups));
        const int r = (int)(w % rgroups);
        const TouchList tl = load_touch_warp(a, s, p, blk, lane, warp);
        update_warp_item<kRows>(a, tl, blk, r * rows, min(a.K, (r + 1) * rows), pcur, lane);
      }
    }
    // The records of this iteration's spikes and the empty lists of the next one
    // have no reader before the closing barrier, so they come after the units, on
    // the warps that were dealt the fewest: one warp per chunk (the chunks' peak
    // counts are independent loads).  Ahead of the scan they held up every
    // iteration by a chain of three loads and an atomic: 1566 -> 1519 us of peel at
    // C=384, K=600, L=60122, 125 -> 118 us at C=32, K=24, L=4122.
    for (long long ch = nwarps - 1 - gwarp; ch < a.nchunks; ch += nwarps) {
      const int c_n = a.chunk_cnt[ch];
      for (int i = lane; i < c_n; i += 32) {
        const long long slot = ch * kChunk + i;
        const long long o = n_out + s.prefix[ch] + i;
        const int tau = a.chunk_tau[slot];
        a.st[2 * o] = tau;
        a.st[2 * o + 1] = a.chunk_k[slot];
        a.amps[o] = a.chunk_amp[slot];
        a.th_amps[o] = a.chunk_th[slot];
        // blocks whose columns this spike's residual window covers
        const int xb0 = (tau - a.nt / 2) / kCol, xb1 = (tau + a.nt / 2) / kCol;
        for (int b = xb0; b <= xb1; ++b) {
          const int pos = atomicAdd(&a.xcount[b], 1);
          if (pos < kXCap) a.xlist[(size_t)b * kXCap + pos] = (int)o;
        }
      }
    }
    // registration lists, bitmap and work counter of the next iteration start empty
    for (int w = rank * kThreads + tid; w < a.nblk; w += (int)G * kThreads)
      a.tcount[(size_t)q * a.nblk + w] = 0;
    for (int w = rank * kThreads + tid; w < a.nwords; w += (int)G * kThreads)
      a.dbits[(size_t)q * a.nwords + w] = 0u;
    if (rank == 0 && tid == 0) {
      a.wctr[q] = 0u;
      a.wctr[2 + q] = 0u;
      a.wctr[4 + q] = 0u;
    }
    if (rank == 0 && tid == 0) a.itoff[it] = (int)n_out;
    KS_TRACE(it, 4, ks_globaltimer());
    __syncthreads();
    KS_TRACE_CTA(it, ks_globaltimer());
    KS_TRACE(it, 5, total);
    KS_TRACE(it, 6, ndirty);
    n_out += total;
    ok = ks_grid_sync(a.ctl, G, epoch, a.limit_ns);
  }
  // one decision on the error for the whole block
  int e = __syncthreads_or(tid == 0 && ks_ctl_error(a.ctl) != 0) ? ks_ctl_error(a.ctl) : 0;
  // The next batch's clearing and scores overwrite this scratch, and the blocks
  // that left on the peak counts (no peak, too many) have passed no barrier since
  // they read them: nobody goes on before all have.
  if (again && !e && !ks_grid_sync(a.ctl, G, epoch, a.limit_ns)) e = ks_ctl_error(a.ctl);
  if (rank == 0 && tid == 0) {
    a.info[0] = n_out;
    a.info[1] = e ? e : status;
    a.info[2] = it;
    if (status != KS_ERR_OVERFLOW) a.info[3] = n_out;
  }
  return PeelOutcome{n_out, it, e ? e : status};
}

// kGrouped: the grouped update (a.rperm, a.nmip, a.mg and the group metadata
// set); the ungrouped form needs no group metadata.
template <bool kGrouped>
__global__ void __launch_bounds__(kThreads, kGrouped ? kBlocksPerSm : kTeamBlocksPerSm) peel_kernel(PeelArgs a) {
  extern __shared__ __align__(16) char smem_raw[];
  const Smem s = carve_smem(a, smem_raw, kGrouped);
  unsigned epoch = 0;
  run_peel<kRowsPerWarp, kGrouped>(a, s, blockIdx.x, gridDim.x, epoch, false);
}

// the batched peel's residual scratch fits in the warp tiles
static_assert(4 * kXWarp <= kTileBytes, "residual scratch exceeds a tile");

// ---------------------------------------------------------------- RESIDUAL
// After the loop: Xres[c, col] -= amp_s * sum_p U[k_s,p,c] W[p, col-tau_s+nt/2]
// for every spike s whose window covers col, applied in record order
// (iteration, then time) -- per element the order in which the reference's
// iterations subtract (:237).  Each element is read and written once.
//
// Gather, into the warp's list, the spikes of record positions
// [skip, skip + kXList) among those whose window meets columns [c0, c0+32):
// lanes binary-search the time-sorted run of one iteration each.  Returns the
// total number of such spikes.
__device__ int gather_residual(const PeelArgs& a, const ResSmem& s, int n_iter,
                               long long n_out, int c0, int skip, int lane) {
  __syncwarp();   // earlier readers of the warp's list are done
  const int half = a.nt / 2;
  const long long wlo = (long long)c0 - half, whi = (long long)c0 + kCol - 1 + half;
  int* ltau = s.xl_tau;
  int* lk = s.xl_k;
  float* lamp = s.xl_amp;
  int total = 0;
  for (int i0 = 0; i0 < n_iter; i0 += 32) {
    const int i = i0 + lane;
    long long first = 0, last = 0;
    if (i < n_iter) {
      long long lo = a.itoff[i];
      const long long end = (i + 1 < n_iter) ? a.itoff[i + 1] : n_out;
      long long hi = end;
      while (lo < hi) {                       // first record with tau >= wlo
        const long long mid = (lo + hi) >> 1;
        if (a.st[2 * mid] < wlo) lo = mid + 1; else hi = mid;
      }
      first = lo;
      last = lo;
      while (last < end && a.st[2 * last] <= whi) ++last;
    }
    const int cnt = (int)(last - first);
    int incl = cnt;
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    const int base = total + incl - cnt;
    for (int e = 0; e < cnt; ++e) {
      const int pos = base + e - skip;
      if (pos >= 0 && pos < kXList) {
        const long long o = first + e;
        ltau[pos] = (int)a.st[2 * o];
        lk[pos] = (int)a.st[2 * o + 1];
        lamp[pos] = a.amps[o];
      }
    }
    total += __shfl_sync(0xffffffffu, incl, 31);
  }
  __syncwarp();
  return total;
}

// Load into the warp's list the spikes whose residual window meets block blk,
// in record order.  Returns their number; when it exceeds kXCap the per-block
// record list overflowed and the caller gathers with gather_residual instead.
__device__ int load_residual_list(const PeelArgs& a, const ResSmem& s, int blk, int lane) {
  __syncwarp();
  const int n = a.xcount[blk];
  if (n > kXCap) return n;
  const int o = lane < n ? a.xlist[(size_t)blk * kXCap + lane] : 0x7fffffff;
  int rank = 0;
  for (int j = 0; j < n; ++j) {
    const int oj = __shfl_sync(0xffffffffu, o, j);
    rank += (oj < o) ? 1 : 0;
  }
  if (lane < n) {
    s.xl_tau[rank] = (int)a.st[2 * (long long)o];
    s.xl_k[rank] = (int)a.st[2 * (long long)o + 1];
    s.xl_amp[rank] = a.amps[o];
  }
  __syncwarp();
  return n;
}

// Residual of block blk for channels [32*cg, 32*cg + 32), two tiles: X is
// read, the block's spikes are subtracted and Xres is written (Xres may be X).
template <int PP>
__device__ void residual_item(const PeelArgs& a, const ResSmem& s, int n_iter, long long n_out,
                              int blk, int cg, int lane) {
  const int c0 = blk * kCol;
  const long long col = c0 + lane;
  const bool colok = col < a.L;
  const bool copy = a.X != a.Xres;
  int total = n_out > 0 ? load_residual_list(a, s, blk, lane) : 0;
  const bool gathered = total > kXCap;
  if (gathered) total = gather_residual(a, s, n_iter, n_out, c0, 0, lane);
  if (!copy && total == 0) return;
  const int width = support_width(a.C);
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {
    const int cbase = cg * 32 + h * kXCh;
    if (cbase >= a.C) break;
    const float* src = a.X + (long long)cbase * a.L + col;
    float* out = a.Xres + (long long)cbase * a.L + col;
    unsigned long long x2[kXCh / 2];
#pragma unroll
    for (int i = 0; i < kXCh / 2; ++i) {
      const float lo = (colok && cbase + 2 * i < a.C) ? src[(long long)(2 * i) * a.L] : 0.f;
      const float hi = (colok && cbase + 2 * i + 1 < a.C) ? src[(long long)(2 * i + 1) * a.L] : 0.f;
      x2[i] = f2_pack(lo, hi);
    }
    // more spikes than the warp's list holds: gathered kXList at a time
    for (int done = 0; done < total; done += kXList) {
      if (gathered && total > kXList)
        gather_residual(a, s, n_iter, n_out, c0, done, lane);
      residual_apply<PP>(a, s, min(kXList, total - done), c0, cbase, cbase / kXCh / width, lane,
                         x2);
    }
#pragma unroll
    for (int i = 0; i < kXCh / 2; ++i) {
      float lo, hi;
      f2_unpack(x2[i], lo, hi);
      if (colok && cbase + 2 * i < a.C) out[(long long)(2 * i) * a.L] = lo;
      if (colok && cbase + 2 * i + 1 < a.C) out[(long long)(2 * i + 1) * a.L] = hi;
    }
  }
}

// The residual of every (block, channel group) w, w + step, ... below the
// batch's count.
__device__ __forceinline__ void residual_items(const PeelArgs& a, const ResSmem& s, int n_iter,
                                               long long n_out, long long w, long long step,
                                               int lane) {
  const int xg = (a.C + 31) / 32;
  const long long n_items = (long long)a.nblk * xg;
  for (; w < n_items; w += step) {
    const int blk = (int)(w / xg), cg = (int)(w % xg);
    if (a.P <= 6) residual_item<6>(a, s, n_iter, n_out, blk, cg, lane);
    else residual_item<8>(a, s, n_iter, n_out, blk, cg, lane);
  }
}

constexpr int kResThreads = 256;
constexpr int kResWarps = kResThreads / 32;

// One warp per (32-column block, 32 channels) of the residual; runs after the
// peel kernel on the same stream and reads its outcome from info (a failed
// peel leaves Xres = X).
__global__ void __launch_bounds__(kResThreads)
ks_residual_kernel(PeelArgs a) {
  extern __shared__ __align__(16) char smem_raw[];
  float* sW = reinterpret_cast<float*>(smem_raw);
  if (__syncthreads_or(stage_basis(a.W, a.P, a.nt, sW, kResThreads))) a.sup = nullptr;
  const long long n_out = (int)a.info[1] == KS_OK ? a.info[0] : 0;
  const int n_iter = (int)a.info[2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const ResSmem s = residual_smem(sW, sW + 8 * a.nt, warp);
  residual_items(a, s, n_iter, n_out, (long long)blockIdx.x * kResWarps + warp,
                 (long long)gridDim.x * kResWarps, lane);
}

size_t residual_smem_bytes(int nt) {
  return sizeof(float) * (8 * (size_t)nt + (size_t)kResWarps * kXWarp);
}

__global__ void ks_nm_pair_kernel(const float* __restrict__ nm, int K, float2* __restrict__ nmi) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < K; j += gridDim.x * blockDim.x) {
    const float v = nm[j];
    const bool normal = v >= 1.17549435e-38f && v <= 3.40282347e38f;
    nmi[j] = make_float2(v, normal ? __frcp_rn(v) : __int_as_float(0x7fc00000));
  }
}

// ------------------------------------------------------------------ relayout
__global__ void ks_tile_rows_kernel(const float* __restrict__ B, long long ldb, int K,
                                    int L, int nblk, float* __restrict__ Bt) {
  const long long n = (long long)nblk * K * kCol;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(e % kCol);
    const long long bj = e / kCol;
    const int j = (int)(bj % K);
    const int blk = (int)(bj / K);
    const int col = blk * kCol + c;
    Bt[e] = col < L ? B[(long long)j * ldb + col] : 0.f;
  }
}

__global__ void ks_untile_rows_kernel(const float* __restrict__ Bt, int K, int L,
                                      float* __restrict__ B, long long ldb) {
  const long long n = (long long)K * L;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x) {
    const int col = (int)(e % L);
    const int j = (int)(e / L);
    B[(long long)j * ldb + col] = Bt[((long long)(col / kCol) * K + j) * kCol + (col % kCol)];
  }
}

// ctcT[k][j][l] = ctc[j][k][l]: a block moves the rows of 8 k by 4 j, a warp one
// k with its 16 loads of 4 rows in flight, so that runs of eight rows are read
// and of four written.  Bound by the two passes over memory (54 us at K = 600);
// one row per block took 170 us there, now 66 (5.4 TB/s).
__global__ void __launch_bounds__(256) ks_ctc_transpose_kernel(const float* __restrict__ ctc, int K,
                                                               int nlag, float* __restrict__ ctcT) {
  const int tk = (K + 7) / 8, tj = (K + 3) / 4;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (long long t = blockIdx.x; t < (long long)tk * tj; t += gridDim.x) {
    const int k = (int)(t / tj) * 8 + warp, j0 = (int)(t % tj) * 4;
    if (k >= K) continue;
    for (int l0 = 0; l0 < nlag; l0 += 128) {
      float v[4][4];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int j = j0 + r, l = l0 + 32 * q + lane;
          v[r][q] = j < K && l < nlag ? ctc[((long long)j * K + k) * nlag + l] : 0.f;
        }
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int j = j0 + r, l = l0 + 32 * q + lane;
          if (j < K && l < nlag) ctcT[((long long)k * K + j) * nlag + l] = v[r][q];
        }
    }
  }
}

// ------------------------------------------------------------ group order
// Setup of the grouped update.  The order only decides how many (column,
// group) pairs the no-op test can leave alone; any order gives the same
// results.
//
// Per template: the energy nm = sum_{p,c} U^2 (when nm_out is given; else nm_in
// holds it), {nm, 1/nm} (NaN when nm is not a positive normal), the spatial key
// (the channel centroid sum_c c*e_c / sum_c e_c of its energy e_c =
// sum_p U[k,p,c]^2, 0 for a template without energy) and the support mask: bit
// (c/16)/support_width(C) is set where some U[k,p,c] is not zero.  One block
// of 8 warps per template, fixed summation orders: the energy a warp per
// component, lanes over channels, then the components in turn
// (ks_template_energy's order).  Latency-bound: 7 us at C=371, K=533, where
// one warp per template in three kernels took 33 us.
__global__ void __launch_bounds__(256)
ks_template_setup_kernel(const float* __restrict__ U, int K, int P, int C,
                         const float* __restrict__ nm_in, float* __restrict__ nm_out,
                         float2* __restrict__ nmi, float* __restrict__ key,
                         unsigned long long* __restrict__ sup) {
  __shared__ float sp[8];
  __shared__ double sse[8], ssc[8];
  __shared__ unsigned smask[2];
  const int k = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float* u = U + (size_t)k * P * C;
  if (threadIdx.x < 2) smask[threadIdx.x] = 0u;
  if (nm_out && warp < P) {
    float s = 0.f;
#pragma unroll 4
    for (int c = lane; c < C; c += 32) {
      const float v = u[warp * C + c];
      s = __fadd_rn(s, __fmul_rn(v, v));
    }
    for (int o = 16; o; o >>= 1) s = __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, o));
    if (lane == 0) sp[warp] = s;
  }
  const int width = support_width(C);
  double se = 0.0, sc = 0.0;
  unsigned lo = 0u, hi = 0u;
  for (int c = threadIdx.x; c < C; c += 256) {
    float e = 0.f;
    bool nz = false;
    for (int p = 0; p < P; ++p) {
      const float v = u[p * C + c];
      e = fmaf(v, v, e);
      nz |= v != 0.f;
    }
    se += e;
    sc += (double)c * e;
    if (nz) {
      const int bit = c / kXCh / width;
      if (bit < 32) lo |= 1u << bit;
      else hi |= 1u << (bit - 32);
    }
  }
  for (int o = 16; o; o >>= 1) {
    se += __shfl_xor_sync(0xffffffffu, se, o);
    sc += __shfl_xor_sync(0xffffffffu, sc, o);
  }
  lo = __reduce_or_sync(0xffffffffu, lo);
  hi = __reduce_or_sync(0xffffffffu, hi);
  __syncthreads();
  if (lane == 0) {
    sse[warp] = se;
    ssc[warp] = sc;
    atomicOr(&smask[0], lo);
    atomicOr(&smask[1], hi);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double e = 0.0, c = 0.0;
    for (int w = 0; w < 8; ++w) {
      e += sse[w];
      c += ssc[w];
    }
    key[k] = e > 0.0 ? (float)(c / e) : 0.f;
    sup[k] = (unsigned long long)smask[1] << 32 | smask[0];
    float nm = nm_out ? 0.f : nm_in[k];
    if (nm_out) {
      for (int p = 0; p < P; ++p) nm = __fadd_rn(nm, sp[p]);
      nm_out[k] = nm;
    }
    const bool normal = nm >= 1.17549435e-38f && nm <= 3.40282347e38f;
    nmi[k] = make_float2(nm, normal ? __frcp_rn(nm) : __int_as_float(0x7fc00000));
  }
}

__device__ __forceinline__ unsigned sortable_key(float f) {
  const unsigned u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// rperm[r] = the template of rank r in ascending key order (the smaller
// template index first on equal keys), and {nm, 1/sqrt(nm)} of the templates in
// that order; an nm outside [2^-30, 2^30], where the group fold's comparison of
// scores by b/sqrt(nm) could leave the normal range, gets a NaN scale.  The
// last template fills the positions past K up to whole groups.  Eight threads
// count the keys below each template's, staged through shared memory 1024 at a
// time.
__global__ void __launch_bounds__(256) ks_group_order_kernel(const float* __restrict__ key, int K,
                                                             const float2* __restrict__ nmi,
                                                             int* __restrict__ rperm,
                                                             float2* __restrict__ nmip) {
  __shared__ unsigned sk[1024];
  const int k = blockIdx.x * 32 + (threadIdx.x >> 3), part = threadIdx.x & 7;
  const unsigned mine = k < K ? sortable_key(key[k]) : 0u;
  int rank = 0;
  for (int j0 = 0; j0 < K; j0 += 1024) {
    const int n = min(1024, K - j0);
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) sk[i] = sortable_key(key[j0 + i]);
    __syncthreads();
#pragma unroll 4
    for (int i = part; i < n; i += 8) {
      const unsigned v = sk[i];
      rank += (v < mine || (v == mine && j0 + i < k)) ? 1 : 0;
    }
  }
  for (int o = 4; o; o >>= 1) rank += __shfl_xor_sync(0xffffffffu, rank, o);
  if (k >= K || part) return;
  const float nm = nmi[k].x;
  const bool ok = nm >= 9.3132257e-10f && nm <= 1.0737418e9f;
  const float2 v = make_float2(nm, ok ? __frsqrt_rn(nm) : __int_as_float(0x7fc00000));
  rperm[rank] = k;
  nmip[rank] = v;
  if (rank == K - 1)
    for (int r = K; r < n_groups(K) * kGroup; ++r) {
      rperm[r] = k;
      nmip[r] = v;
    }
}

// mg[k][g] = the largest |ctcT[k][j][l]| over the rows j of group g (rows
// rperm[32g ..]) and all lags l, by the integer maximum of the magnitude bits
// (so a NaN anywhere gives a NaN bound, which never passes the no-op test).
// One block of 256 threads per (template, group), a warp's 16 loads of its four
// rows in flight: bound by reading ctcT once (140 MB at K = 533: 29 us; 41 with
// one row of loads in flight).
__global__ void __launch_bounds__(256) ks_group_bound_kernel(const float* __restrict__ ctcT,
                                                             const int* __restrict__ rperm, int K,
                                                             int nlag, int ng,
                                                             float* __restrict__ mg) {
  __shared__ unsigned wm[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long items = (long long)K * ng;
  for (long long item = blockIdx.x; item < items; item += gridDim.x) {
    const int k = (int)(item / ng), g = (int)(item % ng);
    unsigned m = 0u;
    // the warp's four rows (the positions past K repeat the last template)
    const float* row[kGroup / 8];
#pragma unroll
    for (int r = 0; r < kGroup / 8; ++r)
      row[r] = ctcT + ((size_t)k * K + rperm[g * kGroup + warp + 8 * r]) * nlag;
    for (int l0 = 0; l0 < nlag; l0 += 128) {
#pragma unroll
      for (int r = 0; r < kGroup / 8; ++r)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int l = l0 + 32 * q + lane;
          if (l < nlag) m = max(m, __float_as_uint(row[r][l]) & 0x7fffffffu);
        }
    }
    for (int o = 16; o; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    __syncthreads();
    if (lane == 0) wm[warp] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned x = 0u;
      for (int w = 0; w < 8; ++w) x = max(x, wm[w]);
      mg[item] = __uint_as_float(x);
    }
  }
}

// Scratch of one team (reused for every batch it processes), for batches of
// up to L padded samples and K templates: [ctl 256 B: control word] [cfmax L]
// [imax L] [pack 2L] [chunk counts] [chunk buffers 4 x nchunks*kChunk]
// [tcount 2 nblk] [touch 2 nblk*kTouch] [dbits 2 nwords] [work counters 6], and
// for the grouped update [gbest nblk*ng*32 u64] [gexp nblk*ng*32 u8]
// [blist nblk*32 int] [units nblk*ng uint2] (K = 0: none).  Only the control
// word needs zeroing before a launch; the team clears the rest per batch (the
// initial scoring writes every gbest and gexp entry).
struct TeamLayout {
  size_t cfmax, imax, pack, chunk_cnt, chunk_tau, chunk_k, chunk_amp, chunk_th, tcount,
      touch, dbits, wctr, gbest, gexp, blist, units, bytes;
};

__host__ __device__ inline size_t al256(size_t x) { return (x + 255) & ~size_t(255); }

__host__ __device__ inline TeamLayout team_layout(long long L, long long K) {
  const long long nchunks = (L + kChunk - 1) / kChunk, nblk = (L + kCol - 1) / kCol;
  const long long nwords = (nblk + 31) / 32;
  const size_t meta = (size_t)nblk * n_groups(K) * 32;
  TeamLayout t;
  size_t o = 256;
  t.cfmax = o; o = al256(o + 4 * (size_t)L);
  t.imax = o; o = al256(o + 4 * (size_t)L);
  t.pack = o; o = al256(o + 16 * (size_t)L);
  t.chunk_cnt = o; o = al256(o + 4 * (size_t)nchunks);
  t.chunk_tau = o; o = al256(o + 4 * (size_t)nchunks * kChunk);
  t.chunk_k = o; o = al256(o + 4 * (size_t)nchunks * kChunk);
  t.chunk_amp = o; o = al256(o + 4 * (size_t)nchunks * kChunk);
  t.chunk_th = o; o = al256(o + 4 * (size_t)nchunks * kChunk);
  t.tcount = o; o = al256(o + 8 * (size_t)nblk);
  t.touch = o; o = al256(o + 2 * sizeof(Touch) * (size_t)nblk * kTouch);
  t.dbits = o; o = al256(o + 8 * (size_t)nwords);
  t.wctr = o; o = al256(o + 24);
  t.gbest = o; o = al256(o + 8 * meta);
  t.gexp = o; o = al256(o + meta);
  t.blist = o; o = al256(o + (K > 0 ? 128 * (size_t)nblk : 0));
  t.units = o; o = al256(o + 8 * (size_t)nblk * n_groups(K));
  t.bytes = o;
  return t;
}

// Lists a batch keeps until its residual pass: [iteration offsets kMaxIters]
// [residual counts nblk] [residual lists nblk*kXCap].
struct ListLayout {
  size_t itoff, xcount, xlist, bytes;
};

__host__ __device__ inline ListLayout list_layout(long long L) {
  const long long nblk = (L + kCol - 1) / kCol;
  ListLayout t;
  size_t o = 0;
  t.itoff = o; o = al256(o + 4 * (size_t)kMaxIters);
  t.xcount = o; o = al256(o + 4 * (size_t)nblk);
  t.xlist = o; o = al256(o + 4 * (size_t)nblk * kXCap);
  t.bytes = o;
  return t;
}

// Point the scratch fields of a at a team region and a list region; with
// grouped, also the group metadata (a.K must be set).
__host__ __device__ inline void bind_scratch(PeelArgs& a, char* team, char* lists,
                                             bool grouped) {
  const TeamLayout t = team_layout(a.L, grouped ? a.K : 0);
  const ListLayout l = list_layout(a.L);
  a.ctl = reinterpret_cast<unsigned long long*>(team);
  a.cfmax = reinterpret_cast<float*>(team + t.cfmax);
  a.imax = reinterpret_cast<int*>(team + t.imax);
  a.pack = reinterpret_cast<unsigned long long*>(team + t.pack);
  a.chunk_cnt = reinterpret_cast<int*>(team + t.chunk_cnt);
  a.chunk_tau = reinterpret_cast<int*>(team + t.chunk_tau);
  a.chunk_k = reinterpret_cast<int*>(team + t.chunk_k);
  a.chunk_amp = reinterpret_cast<float*>(team + t.chunk_amp);
  a.chunk_th = reinterpret_cast<float*>(team + t.chunk_th);
  a.tcount = reinterpret_cast<int*>(team + t.tcount);
  a.touch = reinterpret_cast<Touch*>(team + t.touch);
  a.dbits = reinterpret_cast<unsigned*>(team + t.dbits);
  a.wctr = reinterpret_cast<unsigned*>(team + t.wctr);
  a.itoff = reinterpret_cast<int*>(lists + l.itoff);
  a.xcount = reinterpret_cast<int*>(lists + l.xcount);
  a.xlist = reinterpret_cast<int*>(lists + l.xlist);
  a.gbest = grouped ? reinterpret_cast<unsigned long long*>(team + t.gbest) : nullptr;
  a.gexp = grouped ? reinterpret_cast<unsigned char*>(team + t.gexp) : nullptr;
  a.blist = grouped ? reinterpret_cast<int*>(team + t.blist) : nullptr;
  a.units = grouped ? reinterpret_cast<uint2*>(team + t.units) : nullptr;
  a.ng = grouped ? n_groups(a.K) : 0;
  a.nchunks = (int)((a.L + kChunk - 1) / kChunk);
  a.nblk = (int)((a.L + kCol - 1) / kCol);
  a.nwords = (a.nblk + 31) / 32;
}

}  // namespace
