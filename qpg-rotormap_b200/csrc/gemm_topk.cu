// gemm_topk.cu -- the read x index similarity search: a persistent tcgen05
// fp8 GEMM whose epilogue is a streaming per-row top-k, plus the merge of
// the per-split partial lists and the engine object behind the C ABI.
//
// Replaces the reference's chunk loop batch_gemm_topk!
// (RotorMap/search/engine_fp8.jl:399-437): cuBLASLt fp8 GEMM into an fp16 C
// chunk in HBM (gemm/fp8_lt.jl:128-168) followed by seg_rowtopk_merge_kernel!
// (gemm/topk_kernels.jl:213-329).  Here the score tile lives only in TMEM.
//
// Kernel structure (one CTA per SM, 192 threads):
//   warp 0      TMA producer: A tile (128 reads x 128 B of K) and B tile
//               (256 index columns x 128 B) per stage, 128-byte swizzle,
//               4-stage mbarrier ring, no multicast.
//   warp 1      TMEM owner + MMA issuer: tcgen05.mma kind::f8f6f4,
//               M=128 N=256 K=32, fp32 accumulators double-buffered in TMEM
//               (2 x 256 of the 512 columns).
//   warps 2..5  epilogue: one thread per read row (TMEM lane); tcgen05.ld of
//               32 columns at a time (the next chunk in flight while one is
//               scored), score transform (fp16 rounding / column scale),
//               group maxima vs the row's threshold, candidates buffered in
//               shared memory and inserted in bulk into a register reservoir
//               of the top KT (score desc, column asc).
// Work unit = (read tile of 128 rows, column split); each unit streams its
// split's column tiles and leaves a sorted partial list per row; a second
// kernel merges the splits.  Every mbarrier wait is bounded; a wait that
// gives up raises a shared abort flag, records a code in the device error
// word and the CTA drains its in-flight work before freeing TMEM.
#include <float.h>
#include <limits.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

#include "common.cuh"

namespace r2m {

constexpr int BM = 128;           // read rows per tile (TMEM lanes)
constexpr int BN = 256;           // index columns per tile at most (TMEM fp32 columns; GemmArgs::bn)
constexpr int BK = 128;           // K bytes per stage (one 128-byte swizzle row)
constexpr int STAGES = 4;
constexpr int A_STAGE = BM * BK;  // 16 KiB
constexpr int B_STAGE = BN * BK;  // 32 KiB
constexpr int TMEM_COLS = 512;
constexpr long long WAIT_LIMIT = 4000000000LL;  // clock cycles (~2 s)
constexpr int MAX_LISTS = 320;  // partial lists per row (column splits x epilogue halves)
// Epilogue forms of both kernels: 4 * H epilogue warps.  With H = 2 two warps
// share each TMEM lane quarter, each draining one half (128 columns) of
// every tile into its own reservoir, so a (read tile, column split) unit
// leaves two partial lists per row.  That halves the per-warp latency chain
// of a tile and the reservoir warm-up at every unit start.  The CTA-pair
// kernel always takes it (k <= 32): its epilogue must drain a tile in the
// time its MMAs take one, and with 4 warps it held the MMAs back (headline
// launch, same box: 1,553 ms per launch with 4 epilogue warps, 1,530 ms with
// 8).  The single-CTA kernel takes it for short units only: on long units
// the extra warps cost clock under the board's power cap.  The host picks H
// per launch (epi_halves_for).  KT = 64 always uses H = 1 (its reservoir
// needs the registers).
__host__ __device__ constexpr int epi_threads(int H) { return 64 + 128 * H; }
// Candidate buffer of the epilogue: 32 KiB per CTA (what the operand stages
// leave of shared memory), entry e of epilogue thread t at [e][t].
constexpr int CAND_BYTES = 32 * 1024;
__host__ __device__ constexpr int cand_cap(int H) { return CAND_BYTES / 8 / (128 * H); }  // entries per thread
// 256-column tiles per work unit at or below which the 8-warp epilogue pays
constexpr int SHORT_UNIT_TILES = 8192;

struct GemmArgs {
  int nb;
  int num_m_tiles;
  long long N;
  int bn;  // columns per tile: 64, 128, 192 or 256
  int n_tiles;
  int splits;
  int num_kb;
  int score_mode;
  int k;     // results wanted per row (<= KT)
  int mpad;  // partial-list row stride, at least nb
  const float *scaleB;
  float *part_vals;
  int *part_cols;
  uint32_t *err;
  long long *pace;  // CTA-pair kernel: per-pair progress (null = no pacing)
  int pace_window;  // column tiles a pair may run ahead of the slowest one
  uint32_t *pub;    // shared row bounds (null = none): key of list l, row r at [l * mpad + r]
  int conc;         // column splits whose lists share a bound
};

__device__ __forceinline__ int split_lo(int s, int n_tiles, int splits) {
  return (int)(((long long)s * n_tiles) / splits);
}

__device__ __forceinline__ float round_f16(float x) { return __half2float(__float2half_rn(x)); }

// The best KT (value, column) pairs of one row, kept sorted in registers:
// larger value first, equal values -> smaller column first.  `thr` is the
// k-th of them: a later column has to beat it to enter the row's top k.
template <int KT>
struct Reservoir {
  float v[KT];
  int c[KT];
  float thr;
  float floor;  // a later column at or below it is not among the row's top k (shared bound)

  __device__ __forceinline__ void reset(float bound) {
#pragma unroll
    for (int i = 0; i < KT; ++i) {
      v[i] = -INFINITY;
      c[i] = INT_MAX;
    }
    thr = floor = bound;
  }
  // Columns arrive in increasing order, so an equal value goes behind the
  // kept one.  x <= v[KT-1] (-inf, a candidate that has since been beaten)
  // changes nothing.  Every slot picks (old, shifted, new) from two compares:
  // no chain through the list.
  __device__ __forceinline__ void insert(float x, int col) {
    bool above = x > v[KT - 1];
#pragma unroll
    for (int i = KT - 1; i > 0; --i) {
      const bool next = x > v[i - 1];
      v[i] = above ? (next ? v[i - 1] : x) : v[i];
      c[i] = above ? (next ? c[i - 1] : col) : c[i];
      above = next;
    }
    if (above) {
      v[0] = x;
      c[0] = col;
    }
  }
  // v[n-1] by selects (a run-time index would move the list to memory)
  __device__ __forceinline__ float best(int n) const {
    float x = v[0];
#pragma unroll
    for (int i = 1; i < KT; ++i) x = i < n ? v[i] : x;
    return x;
  }
  __device__ __forceinline__ void update_thr(int k) { thr = fmaxf(best(k), floor); }
  __device__ __forceinline__ void raise_floor(float f) {
    floor = fmaxf(floor, f);
    thr = fmaxf(thr, f);
  }
};

constexpr int BOUND_LISTS = 16;  // lists that share a bound at most (each reads them all)

// Shared row bounds.  The lists that a row gathers at the same time (the
// epilogue halves of the column splits in one wave) see a fraction of its
// columns each, and their own k-th values say little: n columns in, a list of
// S admits k (1 + ln(n / k)) candidates, S times what the row as a whole
// needs.  So after every flush a list publishes its q-th best value, q =
// ceil(k / S): S lists with q values each hold at least k values no smaller
// than the least of the S published ones, so a column below that is out.  The
// group's bound is read after tiles 1, 2, 3, 4, 6, 8, 12, ... of a unit, and
// the bound of the wave before at the start of one.  Keys are ordered like the
// values, 0 = nothing published; stale reads are only lower bounds, so no
// ordering is needed, and results do not depend on what is seen when.  Measured
// (whole search, own thresholds -> shared bounds): 1,000 reads x 300,007
// columns 489 -> 472 us, 300 x 100,000 124 -> 113, 4,096 x 20,000 185 -> 164; at
// k = 64 100 x 1,000,003 455 -> 411, 1,000 x 300,007 757 -> 654.
__device__ __forceinline__ uint32_t bound_key(float x) {
  const uint32_t u = __float_as_uint(x);
  return (u >> 31) ? ~u : (u | 0x80000000u);
}
// The largest value below the one of `key`: candidates must exceed it.
__device__ __forceinline__ float below_key(uint32_t key) {
  const float x = __uint_as_float((key >> 31) ? key & 0x7FFFFFFFu : ~key);
  if (x == 0.f) return __uint_as_float(0x80000001u);
  return __uint_as_float(__float_as_uint(x) + (x > 0.f ? -1 : 1));
}

struct Bounds {
  uint32_t *pub;             // GemmArgs::pub (null = none)
  int group, mine, stride;   // elements of pub: the group's first key of this row, this list's key
  int lists, q;

  // Unit of column split sp, epilogue half `half` of H, row `row`.
  __device__ __forceinline__ void init(const GemmArgs &g, int sp, int half, int H, int row) {
    const int s0 = sp / g.conc * g.conc, s1 = min(s0 + g.conc, g.splits);
    pub = row < g.nb ? g.pub : nullptr;
    lists = (s1 - s0) * H;
    q = (g.k + lists - 1) / lists;
    stride = g.mpad;
    group = s0 * H * stride + row;
    mine = (sp * H + half) * stride + row;
  }
  // What a candidate must exceed by the n lists whose first key is at `at`.
  __device__ __forceinline__ float bound(int at, int n) const {
    if (pub == nullptr) return -INFINITY;
    uint32_t m = 0xFFFFFFFFu;
#pragma unroll 8
    for (int l = 0; l < n; ++l) {
      uint32_t x;
      asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(x) : "l"(pub + at + l * stride) : "memory");
      m = min(m, x);
    }
    return m == 0 ? -INFINITY : below_key(m);
  }
  __device__ __forceinline__ float group_bound() const { return lists > 1 ? bound(group, lists) : -INFINITY; }
  // The bound of the group before (full: conc splits), or -inf for the first.
  __device__ __forceinline__ float bound_before(int n) const {
    return group >= n * stride ? bound(group - n * stride, n) : -INFINITY;
  }
  __device__ __forceinline__ void publish(float x) const {
    if (pub != nullptr && x > -INFINITY)
      asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(pub + mine), "r"(bound_key(x)) : "memory");
  }
  // Whether to read the group's bound after tile number `done` (1, 2, ...) of the unit.
  static __device__ __forceinline__ bool due(int done) {
    const int top = 31 - __clz(done);
    return top <= 1 || (done & ((1 << (top - 1)) - 1)) == 0;
  }
};

// Candidates of one row waiting to enter its reservoir.  An insertion costs
// a warp ~5 KT instructions whether one lane or all 32 have a candidate, and
// the lanes' rows find theirs in different columns.  So a column that beats
// its row's threshold is appended to the lane's buffer in shared memory (a
// predicated store), and once a lane's buffer could overflow on the next 8
// columns the warp empties all of them together, entry by entry: one
// insertion then serves most of the lanes.  The threshold stands still
// meanwhile, which only lets a few more candidates in; each is compared again
// when it is inserted.  This bounds every search whose units are short: about
// KT ln(columns / KT) insertions a row, against 32 cycles of MMA a column.
// Inserting column by column as they came, rdim 2048, fused kernel alone:
// 1,000 reads x 300,007 columns 2,346 us -> 614 us, 8,192 x 50,000 3,159 ->
// 750, 4,096 x 500,000 at k = 64 50.1 ms -> 5.0 ms, 65,536 x 1,048,576
// 122.0 -> 100.3 ms.
template <int H>
struct Candidates {
  static constexpr uint32_t STRIDE = 128 * H * 8;  // bytes between a thread's entries
  uint32_t base, end, limit;

  __device__ __forceinline__ void init(uint32_t smem_base, int t) {
    base = end = smem_base + 8u * (uint32_t)t;
    limit = base + STRIDE * (uint32_t)(cand_cap(H) - 8);
  }
  __device__ __forceinline__ void append(float x, float thr, int col) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.gt.f32 p, %1, %2;\n\t"
        "@p st.shared.v2.b32 [%0], {%3, %4};\n\t"
        "@p add.u32 %0, %0, %5;\n\t}"
        : "+r"(end)
        : "f"(x), "f"(thr), "r"(__float_as_uint(x)), "r"(col), "n"(STRIDE)
        : "memory");
  }
  // Entry at byte offset o, or a value that no list takes.
  __device__ __forceinline__ void load(uint32_t o, float &x, int &col) const {
    uint32_t xb = 0xFF800000u;
    col = 0;
    if (base + o < end) asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(xb), "=r"(col) : "r"(base + o) : "memory");
    x = __uint_as_float(xb);
  }
  // Called by the whole warp.
  template <int KT>
  __device__ __forceinline__ void flush(Reservoir<KT> &R, const Bounds &S, int k) {
    const unsigned FULL = 0xFFFFFFFFu;
    const uint32_t most = __reduce_max_sync(FULL, end - base);
    float x;
    int col;
    load(0, x, col);
#pragma unroll 1
    for (uint32_t o = 0; o < most; o += STRIDE) {
      float next_x;
      int next_col;
      load(o + STRIDE, next_x, next_col);  // in flight during the insertion
      R.insert(x, col);
      x = next_x;
      col = next_col;
    }
    end = base;
    R.update_thr(k);
    S.publish(R.best(S.q));
  }
};

// Column scales of one 32-column chunk: broadcast loads (every lane of the
// warp reads the same 128 bytes).  Past the index end they read as 1; those
// columns are masked to -inf before scoring.
__device__ __forceinline__ void load_scales(float4 (&s)[8], const float *scaleB, long long c0, long long N,
                                            bool tail) {
  if (!tail) {
    const float4 *p = reinterpret_cast<const float4 *>(scaleB + c0);
#pragma unroll
    for (int q = 0; q < 8; ++q) s[q] = __ldg(p + q);
  } else {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const long long c = c0 + 4 * q;
      s[q].x = c < N ? __ldg(scaleB + c) : 1.f;
      s[q].y = c + 1 < N ? __ldg(scaleB + c + 1) : 1.f;
      s[q].z = c + 2 < N ? __ldg(scaleB + c + 2) : 1.f;
      s[q].w = c + 3 < N ? __ldg(scaleB + c + 3) : 1.f;
    }
  }
}

// (a, b) *= (x, y), one instruction; each half is the scalar product.
__device__ __forceinline__ void mul2(float &a, float &b, float x, float y) {
  asm("{\n\t.reg .b64 p, q;\n\t"
      "mov.b64 p, {%0, %1};\n\t"
      "mov.b64 q, {%2, %3};\n\t"
      "mul.rn.f32x2 p, p, q;\n\t"
      "mov.b64 {%0, %1}, p;\n\t}"
      : "+f"(a), "+f"(b)
      : "f"(x), "f"(y));
}
// max(a, b, c), one instruction; like fmaxf it passes over NaNs.
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

__device__ __forceinline__ void apply_scales(float (&v)[32], const float4 (&s)[8]) {
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    mul2(v[4 * q], v[4 * q + 1], s[q].x, s[q].y);
    mul2(v[4 * q + 2], v[4 * q + 3], s[q].z, s[q].w);
  }
}

// Score one 32-column chunk of this thread's row (columns c0 .. c0+31).  The
// maxima of its four groups of 8 columns against the row's threshold decide,
// for the warp as a whole, which groups have candidates.  Most chunks of a long
// unit have none, so this is the epilogue's steady cost: paired products and
// three-way maxima took it from about 75 instructions to 45 (8,192 reads x
// 50,000 columns 738 -> 569 us, 20,000 x 50,000 1,758 -> 1,642).
template <int KT, int H>
__device__ __forceinline__ void score_chunk(Reservoir<KT> &R, Candidates<H> &Q, const Bounds &S, float (&v)[32], long long c0,
                                            long long N, bool tail, bool f16, int k) {
  const unsigned FULL = 0xFFFFFFFFu;
  if (tail) {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (c0 + j >= N) v[j] = -INFINITY;
  }
  float m[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float *w = v + 8 * q;
    m[q] = max3(max3(w[0], w[1], w[2]), max3(w[3], w[4], w[5]), fmaxf(w[6], w[7]));
  }
  float mx = fmaxf(max3(m[0], m[1], m[2]), m[3]);
  if (f16) mx = round_f16(mx);
  if (!__any_sync(FULL, mx > R.thr)) return;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    if (f16) m[q] = round_f16(m[q]);
    if (__any_sync(FULL, m[q] > R.thr)) {
#pragma unroll
      for (int j = 8 * q; j < 8 * q + 8; ++j) Q.append(f16 ? round_f16(v[j]) : v[j], R.thr, (int)(c0 + j));
      if (__any_sync(FULL, Q.end > Q.limit)) Q.flush(R, S, k);
    }
  }
}

// Drain this warp's `ch` chunks (an even number) of one accumulator tile (TMEM address `taddr`
// = its lane quarter and first chunk; columns c_first .. c_first + 32 ch - 1)
// into the row's reservoir.  Software-pipelined: the TMEM load and the column
// scales of chunk i + 1 are in flight while chunk i is scored.  Every load is
// waited for before returning, so the caller may release the accumulator.
template <int KT, int H>
__device__ __forceinline__ void drain_tile(Reservoir<KT> &R, Candidates<H> &Q, const Bounds &S, uint32_t taddr, int ch, long long c_first, long long N,
                                           const float *scaleB, bool scaled, bool f16, int k) {
  const bool tail = c_first + 32LL * ch > N;
  float va[32], vb[32];
  float4 s[8];
  __syncwarp();
  tmem_ld32(taddr, va);
  if (scaled) load_scales(s, scaleB, c_first, N, tail);
#pragma unroll 1
  for (int i = 0; i < ch; i += 2) {
    const long long c0 = c_first + 32LL * i;
    __syncwarp();
    tmem_wait_ld_tied(va);
    if (scaled) apply_scales(va, s);
    tmem_ld32(taddr + (uint32_t)(i + 1) * 32u, vb);
    if (scaled) load_scales(s, scaleB, c0 + 32, N, tail);
    score_chunk(R, Q, S, va, c0, N, tail, f16, k);
    __syncwarp();
    tmem_wait_ld_tied(vb);
    if (scaled) apply_scales(vb, s);
    if (i + 2 < ch) {
      tmem_ld32(taddr + (uint32_t)(i + 2) * 32u, va);
      if (scaled) load_scales(s, scaleB, c0 + 64, N, tail);
    }
    score_chunk(R, Q, S, vb, c0 + 32, N, tail, f16, k);
  }
}

// The same, one chunk at a time: for the 8-warp form, whose 168-register
// budget has no room for a second chunk (two warps per scheduler cover the
// TMEM latency), and for the 64-entry reservoir.
template <int KT, int H>
__device__ __forceinline__ void drain_tile_serial(Reservoir<KT> &R, Candidates<H> &Q, const Bounds &S, uint32_t taddr, int ch, long long c_first, long long N,
                                                  const float *scaleB, bool scaled, bool f16, int k) {
  const bool tail = c_first + 32LL * ch > N;
#pragma unroll 1
  for (int i = 0; i < ch; ++i) {
    const long long c0 = c_first + 32LL * i;
    float v[32];
    float4 s[8];
    __syncwarp();
    if (scaled) load_scales(s, scaleB, c0, N, tail);
    tmem_ld32(taddr + (uint32_t)i * 32u, v);
    tmem_wait_ld_tied(v);
    if (scaled) apply_scales(v, s);
    score_chunk(R, Q, S, v, c0, N, tail, f16, k);
  }
}

template <int KT, int H>
__device__ __forceinline__ void drain_acc(Reservoir<KT> &R, Candidates<H> &Q, const Bounds &S, uint32_t taddr, int ch, long long c_first, long long N,
                                      const float *scaleB, bool scaled, bool f16, int k) {
  if constexpr (H == 1 && KT < 64)
    drain_tile<KT, H>(R, Q, S, taddr, ch, c_first, N, scaleB, scaled, f16, k);
  else
    drain_tile_serial<KT, H>(R, Q, S, taddr, ch, c_first, N, scaleB, scaled, f16, k);
}

template <int KT, int H, bool NARROW>
__global__ void __launch_bounds__(epi_threads(H), 1)
    k_gemm_topk(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                GemmArgs g) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char *smem =
      reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t *sA = smem;
  uint8_t *sB = smem + STAGES * A_STAGE;
  uint64_t *full = reinterpret_cast<uint64_t *>(sB + STAGES * B_STAGE);
  uint64_t *empty = full + STAGES;
  uint64_t *acc_full = empty + STAGES;
  uint64_t *acc_empty = acc_full + 2;
  uint64_t *drain = acc_empty + 2;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drain + 1);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const uint32_t cand = smem_u32(tmem_slot + 4);  // candidate buffers (CAND_BYTES)

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned FULL = 0xFFFFFFFFu;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], 4 * H);  // epilogue warps
    }
    mbar_init(drain, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 0 && lane == 0) {
    prefetch_tmap(&tmA);
    prefetch_tmap(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  const int num_units = g.num_m_tiles * g.splits;
  const int bn = NARROW ? g.bn : BN;  // columns per tile

  if (warp == 0) {
    // ------------------------------------------------ TMA producer
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      long long issued = 0;
      bool ok = true;
      for (int u = blockIdx.x; ok && u < num_units; u += gridDim.x) {
        const int mt = u % g.num_m_tiles, sp = u / g.num_m_tiles;
        const int t0 = split_lo(sp, g.n_tiles, g.splits), t1 = split_lo(sp + 1, g.n_tiles, g.splits);
        for (int t = t0; ok && t < t1; ++t) {
          for (int kb = 0; kb < g.num_kb; ++kb) {
            if (!mbar_wait_bounded(&empty[stage], phase ^ 1u, abort_flag, WAIT_LIMIT)) {
              if (!*abort_flag) atomicExch(g.err, kErrTimeoutEmpty);
              *abort_flag = 1;
              ok = false;
              break;
            }
            mbar_arrive_expect_tx(&full[stage], A_STAGE + (uint32_t)(bn * BK));
            tma_load_2d(sA + stage * A_STAGE, &tmA, &full[stage], kb * BK, mt * BM);
            tma_load_2d(sB + stage * B_STAGE, &tmB, &full[stage], kb * BK, t * bn);
            ++issued;
            if (++stage == STAGES) {
              stage = 0;
              phase ^= 1u;
            }
          }
        }
      }
      if (!ok) {
        // let the copies already issued land before the CTA can exit
        int nlast = issued < STAGES ? (int)issued : STAGES;
        for (int j = 1; j <= nlast; ++j) {
          int s = stage - j;
          uint32_t ph = phase;
          if (s < 0) {
            s += STAGES;
            ph ^= 1u;
          }
          long long t0 = clock64();
          while (!mbar_try_wait(&full[s], ph) && clock64() - t0 < WAIT_LIMIT) {
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------ MMA issuer
    if (lane == 0) {
      const uint32_t idesc = idesc_e4m3_f32(BM, bn);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int u = blockIdx.x; ok && u < num_units; u += gridDim.x) {
        const int sp = u / g.num_m_tiles;
        const int t0 = split_lo(sp, g.n_tiles, g.splits), t1 = split_lo(sp + 1, g.n_tiles, g.splits);
        for (int t = t0; ok && t < t1; ++t) {
          if (!mbar_wait_bounded(&acc_empty[acc], acc_phase ^ 1u, abort_flag, WAIT_LIMIT)) {
            if (!*abort_flag) atomicExch(g.err, kErrTimeoutAccEmpty);
            *abort_flag = 1;
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + (uint32_t)(acc * BN);
          for (int kb = 0; kb < g.num_kb; ++kb) {
            if (!mbar_wait_bounded(&full[stage], phase, abort_flag, WAIT_LIMIT)) {
              if (!*abort_flag) atomicExch(g.err, kErrTimeoutFull);
              *abort_flag = 1;
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t a0 = smem_u32(sA + stage * A_STAGE);
            const uint32_t b0 = smem_u32(sB + stage * B_STAGE);
#pragma unroll
            for (int kk = 0; kk < BK / 32; ++kk) {
              mma_f8(d_tmem, smem_desc_sw128(a0 + kk * 32), smem_desc_sw128(b0 + kk * 32), idesc,
                     (kb | kk) != 0 ? 1u : 0u);
            }
            mma_commit(&empty[stage]);
            if (++stage == STAGES) {
              stage = 0;
              phase ^= 1u;
            }
          }
          if (!ok) break;
          mma_commit(&acc_full[acc]);
          acc ^= 1;
          if (acc == 0) acc_phase ^= 1u;
        }
      }
      // every MMA issued by this thread has completed once `drain` flips
      mma_commit(drain);
      long long t0 = clock64();
      while (!mbar_try_wait(drain, 0) && clock64() - t0 < WAIT_LIMIT) {
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------ epilogue (top-k)
    const int ch = bn / 32 / H;    // 32-column chunks per warp and tile
    const int quarter = warp & 3;    // TMEM lanes [32*quarter, 32*quarter+32)
    const int half = (warp - 2) >> 2;  // tile chunks [ch half, ch half + ch)
    const int row_in_tile = quarter * 32 + lane;
    const bool f16 = g.score_mode == R2M_SCORE_F16;
    const bool scaled = g.score_mode == R2M_SCORE_SCALED;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    Reservoir<KT> R;
    Candidates<H> Q;
    Bounds S;
    Q.init(cand, threadIdx.x - 64);
    for (int u = blockIdx.x; ok && u < num_units; u += gridDim.x) {
      const int mt = u % g.num_m_tiles, sp = u / g.num_m_tiles;
      const int t0 = split_lo(sp, g.n_tiles, g.splits), t1 = split_lo(sp + 1, g.n_tiles, g.splits);
      S.init(g, sp, half, H, mt * BM + row_in_tile);
      R.reset(u != (int)blockIdx.x ? S.bound_before(g.conc * H) : -INFINITY);
      for (int t = t0; t < t1; ++t) {
        bool w = mbar_wait_bounded(&acc_full[acc], acc_phase, abort_flag, WAIT_LIMIT);
        if (__any_sync(FULL, !w)) {
          if (lane == 0 && !*abort_flag) atomicExch(g.err, kErrTimeoutAccFull);
          *abort_flag = 1;
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * BN + half * ch * 32);
        drain_acc<KT, H>(R, Q, S, taddr, ch, (long long)t * bn + half * ch * 32, g.N, g.scaleB, scaled, f16, g.k);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[acc]);
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1u;
        if (t + 1 < t1 && S.due(t - t0 + 1)) R.raise_floor(S.group_bound());
      }
      if (!ok) break;
      Q.flush(R, S, g.k);
      const int row = mt * BM + row_in_tile;
      if (row < g.nb) {
        const size_t list = (size_t)sp * H + half;
        float *pv = g.part_vals + (list * g.mpad + row) * KT;
        int *pc = g.part_cols + (list * g.mpad + row) * KT;
        // 16 bytes a store: a lane's list is contiguous, its neighbours' are not
#pragma unroll
        for (int j = 0; j < KT; j += 4) {
          *reinterpret_cast<float4 *>(pv + j) = make_float4(R.v[j], R.v[j + 1], R.v[j + 2], R.v[j + 3]);
          *reinterpret_cast<int4 *>(pc + j) = make_int4(R.c[j], R.c[j + 1], R.c[j + 2], R.c[j + 3]);
        }
      }
    }
    __syncwarp();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ------------------------------------------------------------------
// 2-SM variant: a CTA pair (cluster of 2) computes a 256-read x 256-column
// tile with tcgen05.mma.cta_group::2 (M = 256, N = 256, K = 32).  Each CTA
// loads its own 128 read rows and its own 128 of the 256 index columns per
// K chunk (32 KiB instead of 48 KiB per CTA), so a CTA pulls 2/3 of the
// single-CTA kernel's operand bytes per FLOP.  The leader CTA (rank 0)
// issues the MMAs; both CTAs' TMA loads complete on the leader's stage
// barrier; the leader's commits release both CTAs' stages and signal both
// CTAs' accumulators; each CTA's epilogue drains its own 128 TMEM lanes (all
// 256 columns) and arrives on the leader's accumulator-empty barrier.  No
// load uses multicast.
//
// A stage holds two 128-byte K chunks (8 MMAs), and one commit releases it in
// both CTAs (the commit's arrive goes to the barrier at the same offset in
// each CTA of the mask).  The one issuing thread is what bounds this kernel:
// per stage it waits on the stage barrier, forms descriptors, issues the
// MMAs and commits.  With one chunk and two commits per stage that took ~730
// SM clocks against 512 of tensor work (clock64 probes on the headline
// launch, 65,536 reads x 16.8M columns), so the tensor pipe idled ~30% of the
// time.  Same-box A/B, identical results: 1,697 ms per launch -> 1,553 ms
// with two chunks per stage, one commit and precomputed descriptors; three
// chunks per stage (two stages in flight) 1,800 ms; one commit to the leader
// passed on to the peer by the leader's producer (the peer's loads then
// start later) 1,983 ms.
constexpr int HALF_TILE = 128 * BK;            // 16 KiB: one 128-byte K chunk of 128 rows
constexpr int KCH = 2;                         // K chunks per stage
constexpr int STAGES2 = 3;                     // stages in flight (3 x 64 KiB per CTA)
constexpr int STAGE2_BYTES = KCH * HALF_TILE;  // per operand and CTA

// Pair pacing.  Every pair streams the index in column order, and the pairs
// of one wave (units p, p + npairs, ... run side by side) read the same index
// tiles, so a tile comes from DRAM once and from L2 for the other pairs --
// while the pairs stay within an L2's worth of tiles of each other.  Left
// alone they drift apart over a long unit, and then every pair streams the
// index from DRAM itself.  So each pair's producer publishes its position
// (1 + column tiles issued since the launch; 0 = not started, LLONG_MAX = done)
// every PACE_EVERY tiles and, while it is more than `window` tiles ahead of
// the slowest started pair, sleeps -- for at most PACE_CHECKS short naps.
// Pacing only ever delays a pair a little: it never waits for a pair that is
// not running, nor for one more than PACE_LOST windows behind (a pair that
// started late, e.g. on a GPU shared with other work, is outside any shared
// L2 range and cannot be waited out), and it cannot stall the launch.
// Same-box sweep on 65,536 reads x 16.8M columns (mean of two launches):
// no pacing 1,761 ms; window 16 checked every 16 tiles 1,667 ms; windows of
// 32 / 64 / 128 tiles 1,693 / 1,717 / 1,732 ms; tighter windows or checks
// every 8 or 4 tiles 1,698-1,837 ms (the naps and reads start to cost).
constexpr int PACE_EVERY = 16;
constexpr int PACE_CHECKS = 16;
constexpr int PACE_WINDOW = 16;  // tiles of 256 columns: 8 MiB of a 2048-byte index
constexpr int PACE_LOST = 8;     // windows behind which a pair is no longer waited for

__device__ __forceinline__ void pace_pair(long long *pace, int pair, int npairs, long long pos, int window) {
  volatile long long *p = pace;
  p[pair] = ++pos;
  for (int it = 0; it < PACE_CHECKS; ++it) {
    const long long lost = pos - (long long)PACE_LOST * window;
    long long mn = LLONG_MAX;
    for (int q = 0; q < npairs; ++q) {
      const long long v = p[q];
      if (v > 0 && v >= lost && v < mn) mn = v;
    }
    if (pos - mn <= window) return;
    __nanosleep(1000);
  }
}
// CTA-pair kernel: TMA warp, MMA warp and 4 * H epilogue warps (epilogue
// forms above).
template <int KT, int H, bool NARROW>
__global__ void __launch_bounds__(epi_threads(H), 1)
    k_gemm_topk2(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, GemmArgs g) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char *smem =
      reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t *sA = smem;
  uint8_t *sB = smem + STAGES2 * STAGE2_BYTES;
  uint64_t *full = reinterpret_cast<uint64_t *>(sB + STAGES2 * STAGE2_BYTES);
  uint64_t *empty = full + STAGES2;
  uint64_t *acc_full = empty + STAGES2;
  uint64_t *acc_empty = acc_full + 2;
  uint64_t *drain = acc_empty + 2;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drain + 1);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const uint32_t cand = smem_u32(tmem_slot + 4);  // candidate buffers (CAND_BYTES)

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned FULL = 0xFFFFFFFFu;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES2; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], 2 * 4 * H);  // epilogue warps x 2 CTAs (leader's copy is used)
    }
    mbar_init(drain, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 0 && lane == 0) {
    prefetch_tmap(&tmA);
    prefetch_tmap(&tmB);
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, TMEM_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();  // both CTAs' barriers are initialised before any remote arrive
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int num_units = g.num_m_tiles * g.splits;
  const int bn = NARROW ? g.bn : BN;  // columns per tile

  if (warp == 0) {
    // ------------------------------------------------ TMA producer (both CTAs)
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      long long issued = 0;
      long long pos = 0;  // column tiles this pair issued in earlier units
      const bool pacing = leader && g.pace != nullptr;
      bool ok = true;
      for (int u = pair; ok && u < num_units; u += npairs) {
        const int mt = u % g.num_m_tiles, sp = u / g.num_m_tiles;
        const int t0 = split_lo(sp, g.n_tiles, g.splits), t1 = split_lo(sp + 1, g.n_tiles, g.splits);
        for (int t = t0; ok && t < t1; ++t) {
          if (pacing && (t - t0) % PACE_EVERY == 0) pace_pair(g.pace, pair, npairs, pos + (t - t0), g.pace_window);
          for (int kb = 0; kb < g.num_kb; kb += KCH) {
            if (!mbar_wait_bounded(&empty[stage], phase ^ 1u, abort_flag, WAIT_LIMIT)) {
              if (!*abort_flag) atomicExch(g.err, kErrTimeoutEmpty);
              *abort_flag = 1;
              ok = false;
              break;
            }
            const uint32_t fbar = mapa_shared(smem_u32(&full[stage]), 0);
            const int nch = g.num_kb - kb < KCH ? g.num_kb - kb : KCH;
            if (leader) mbar_arrive_expect_tx(&full[stage], (uint32_t)(2 * HALF_TILE + bn * BK) * nch);
            for (int c = 0; c < nch; ++c) {
              tma_load_2d_pair(sA + stage * STAGE2_BYTES + c * HALF_TILE, &tmA, fbar, (kb + c) * BK,
                               mt * 256 + (int)rank * 128);
              tma_load_2d_pair(sB + stage * STAGE2_BYTES + c * HALF_TILE, &tmB, fbar, (kb + c) * BK,
                               t * bn + (int)rank * (bn >> 1));
            }
            ++issued;
            if (++stage == STAGES2) {
              stage = 0;
              phase ^= 1u;
            }
          }
        }
        pos += t1 - t0;
      }
      if (pacing) reinterpret_cast<volatile long long *>(g.pace)[pair] = LLONG_MAX;  // holds no one back
      if (!ok && leader) {
        int nlast = issued < STAGES2 ? (int)issued : STAGES2;
        for (int j = 1; j <= nlast; ++j) {
          int s = stage - j;
          uint32_t ph = phase;
          if (s < 0) {
            s += STAGES2;
            ph ^= 1u;
          }
          long long c0 = clock64();
          while (!mbar_try_wait(&full[s], ph) && clock64() - c0 < WAIT_LIMIT) {
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------ MMA issuer (leader CTA)
    if (lane == 0 && leader) {
      const uint32_t idesc = idesc_e4m3_f32(256, bn);
      // descriptors of stage 0; a stage / chunk / K step offset adds its
      // 16-byte units to the start-address field
      const uint64_t dA0 = smem_desc_sw128(smem_u32(sA)), dB0 = smem_desc_sw128(smem_u32(sB));
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int u = pair; ok && u < num_units; u += npairs) {
        const int sp = u / g.num_m_tiles;
        const int t0 = split_lo(sp, g.n_tiles, g.splits), t1 = split_lo(sp + 1, g.n_tiles, g.splits);
        for (int t = t0; ok && t < t1; ++t) {
          if (!mbar_wait_bounded(&acc_empty[acc], acc_phase ^ 1u, abort_flag, WAIT_LIMIT)) {
            if (!*abort_flag) atomicExch(g.err, kErrTimeoutAccEmpty);
            *abort_flag = 1;
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + (uint32_t)(acc * BN);
          for (int kb = 0; kb < g.num_kb; kb += KCH) {
            if (!mbar_wait_bounded(&full[stage], phase, abort_flag, WAIT_LIMIT)) {
              if (!*abort_flag) atomicExch(g.err, kErrTimeoutFull);
              *abort_flag = 1;
              ok = false;
              break;
            }
            tc_fence_after();
            const int nch = g.num_kb - kb < KCH ? g.num_kb - kb : KCH;
            const uint64_t so = (uint64_t)((stage * STAGE2_BYTES) >> 4);
#pragma unroll
            for (int c = 0; c < KCH; ++c) {
              if (c < nch) {
#pragma unroll
                for (int kk = 0; kk < BK / 32; ++kk) {
                  const uint64_t o = so + (uint64_t)((c * HALF_TILE + kk * 32) >> 4);
                  mma_f8_pair(d_tmem, dA0 + o, dB0 + o, idesc, ((kb + c) | kk) != 0 ? 1u : 0u);
                }
              }
            }
            mma_commit_pair_mask(smem_u32(&empty[stage]), (uint16_t)3);  // both CTAs' stage
            if (++stage == STAGES2) {
              stage = 0;
              phase ^= 1u;
            }
          }
          if (!ok) break;
          const uint32_t fb = smem_u32(&acc_full[acc]);
          mma_commit_pair(mapa_shared(fb, 0));
          mma_commit_pair(mapa_shared(fb, 1));
          acc ^= 1;
          if (acc == 0) acc_phase ^= 1u;
        }
      }
      mma_commit_pair(mapa_shared(smem_u32(drain), 0));
      long long c0 = clock64();
      while (!mbar_try_wait(drain, 0) && clock64() - c0 < WAIT_LIMIT) {
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------ epilogue (both CTAs)
    const int ch = bn / 32 / H;          // 32-column chunks per warp and tile
    const int quarter = warp & 3;          // TMEM lanes this warp may read
    const int half = (warp - 2) >> 2;      // tile chunks [ch half, ch half + ch)
    const int row_in_tile = quarter * 32 + lane;
    const bool f16 = g.score_mode == R2M_SCORE_F16;
    const bool scaled = g.score_mode == R2M_SCORE_SCALED;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    Reservoir<KT> R;
    Candidates<H> Q;
    Bounds S;
    Q.init(cand, threadIdx.x - 64);
    for (int u = pair; ok && u < num_units; u += npairs) {
      const int mt = u % g.num_m_tiles, sp = u / g.num_m_tiles;
      const int t0 = split_lo(sp, g.n_tiles, g.splits), t1 = split_lo(sp + 1, g.n_tiles, g.splits);
      S.init(g, sp, half, H, mt * 256 + (int)rank * 128 + row_in_tile);
      R.reset(u != pair ? S.bound_before(g.conc * H) : -INFINITY);
      for (int t = t0; t < t1; ++t) {
        bool w = mbar_wait_bounded(&acc_full[acc], acc_phase, abort_flag, WAIT_LIMIT);
        if (__any_sync(FULL, !w)) {
          if (lane == 0 && !*abort_flag) atomicExch(g.err, kErrTimeoutAccFull);
          *abort_flag = 1;
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * BN + half * ch * 32);
        drain_acc<KT, H>(R, Q, S, taddr, ch, (long long)t * bn + half * ch * 32, g.N, g.scaleB, scaled, f16, g.k);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(mapa_shared(smem_u32(&acc_empty[acc]), 0));
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1u;
        if (t + 1 < t1 && S.due(t - t0 + 1)) R.raise_floor(S.group_bound());
      }
      if (!ok) break;
      Q.flush(R, S, g.k);
      const int row = mt * 256 + (int)rank * 128 + row_in_tile;
      if (row < g.nb) {
        const size_t list = (size_t)sp * H + half;
        float *pv = g.part_vals + (list * g.mpad + row) * KT;
        int *pc = g.part_cols + (list * g.mpad + row) * KT;
        // 16 bytes a store: a lane's list is contiguous, its neighbours' are not
#pragma unroll
        for (int j = 0; j < KT; j += 4) {
          *reinterpret_cast<float4 *>(pv + j) = make_float4(R.v[j], R.v[j + 1], R.v[j + 2], R.v[j + 3]);
          *reinterpret_cast<int4 *>(pc + j) = make_int4(R.c[j], R.c[j + 1], R.c[j + 2], R.c[j + 3]);
        }
      }
    }
    __syncwarp();
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync();  // the leader's MMAs touch the peer's smem and TMEM until here
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

// Merge the per-split sorted lists of every row into its final top-k: G lanes
// per row, PER lists per lane, k rounds of an arg-max over the list heads.
// Each lane holds the next four entries of its lists in registers, so the
// rounds run without touching memory until a list has given four of the k
// (with one entry held, every round waited for the load of the winner's
// successor: k L2 latencies, 16-20 us whatever the batch).  G follows the
// number of lists, so that a row of a large batch (few lists) does not
// occupy a whole warp: 65,536 rows of 4 lists 308 -> 44 us, 8,192 rows of 32
// lists 39 -> 20, 16 to 200 rows of 128 lists 18 -> 12 (launch included).
// It also puts the launch's row bounds and pacing slots back to zero for the
// next launch.
template <int G, int PER>
__global__ void __launch_bounds__(256) k_merge_splits(const float *__restrict__ pv, const int *__restrict__ pc,
                                                     int lists, int mpad, int KT, int nb, int k,
                                                     const float *__restrict__ scaleA, float *out_v, int *out_l,
                                                     uint32_t *pub, long long *pace, int npace) {
  if (pace != nullptr && blockIdx.x == 0)
    for (int i = threadIdx.x; i < npace; i += 256) pace[i] = 0;
  const int gl = threadIdx.x % G;
  const int row = blockIdx.x * (256 / G) + threadIdx.x / G;
  if (row >= nb) return;  // whole groups
  const unsigned gmask = G == 32 ? 0xFFFFFFFFu : ((1u << G) - 1u) << ((threadIdx.x & 31) / G * G);
  float v[PER][4];
  int c[PER][4], taken[PER];
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    const int s = gl + G * q;
    float4 a = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
    int4 b = make_int4(INT_MAX, INT_MAX, INT_MAX, INT_MAX);
    if (s < lists) {
      const size_t at = ((size_t)s * mpad + row) * KT;
      a = *reinterpret_cast<const float4 *>(pv + at);
      b = *reinterpret_cast<const int4 *>(pc + at);
    }
    v[q][0] = a.x, v[q][1] = a.y, v[q][2] = a.z, v[q][3] = a.w;
    c[q][0] = b.x, c[q][1] = b.y, c[q][2] = b.z, c[q][3] = b.w;
    taken[q] = 0;
  }
  if (pub != nullptr)
    for (int s = gl; s < lists; s += G) pub[(size_t)s * mpad + row] = 0u;
  const float sa = scaleA ? scaleA[row] : 1.0f;
  for (int r = 0; r < k; ++r) {
    float bv = v[0][0];
    int bc = c[0][0], bq = 0;
#pragma unroll
    for (int q = 1; q < PER; ++q) {
      const bool better = v[q][0] > bv || (v[q][0] == bv && c[q][0] < bc);
      bv = better ? v[q][0] : bv;
      bc = better ? c[q][0] : bc;
      bq = better ? q : bq;
    }
    // (value desc, column asc) as unsigned keys; -0 counts as +0
    const uint32_t u = __float_as_uint(bv + 0.0f);
    uint32_t key = (u >> 31) ? ~u : (u | 0x80000000u);
    uint32_t col = (uint32_t)bc;
    const uint32_t mykey = key;
    if constexpr (G == 32) {
      key = __reduce_max_sync(gmask, key);
      col = __reduce_min_sync(gmask, mykey == key ? col : 0xFFFFFFFFu);
    } else {
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) {
        const uint32_t ok = __shfl_xor_sync(gmask, key, o), oc = __shfl_xor_sync(gmask, col, o);
        const bool better = ok > key || (ok == key && oc < col);
        key = better ? ok : key;
        col = better ? oc : col;
      }
    }
    if (col == (uint32_t)INT_MAX) {  // every list is empty
      if (gl == 0) {
        out_v[(size_t)row * k + r] = -INFINITY;
        out_l[(size_t)row * k + r] = 0;
      }
    } else if (mykey == key && (uint32_t)bc == col) {  // columns are distinct: one lane
      out_v[(size_t)row * k + r] = bv * sa;
      out_l[(size_t)row * k + r] = bc + 1;
#pragma unroll
      for (int q = 0; q < PER; ++q) {
        if (q != bq) continue;
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          v[q][e] = v[q][e + 1];
          c[q][e] = c[q][e + 1];
        }
        v[q][3] = -INFINITY;
        c[q][3] = INT_MAX;
        if ((++taken[q] & 3) == 0 && taken[q] < KT) {
          const size_t at = ((size_t)(gl + G * q) * mpad + row) * KT + taken[q];
          const float4 a = *reinterpret_cast<const float4 *>(pv + at);
          const int4 b = *reinterpret_cast<const int4 *>(pc + at);
          v[q][0] = a.x, v[q][1] = a.y, v[q][2] = a.z, v[q][3] = a.w;
          c[q][0] = b.x, c[q][1] = b.y, c[q][2] = b.z, c[q][3] = b.w;
        }
      }
    }
    __syncwarp(gmask);
  }
}

template <int G, int PER>
static void launch_merge_as(const GemmArgs &g, int lists, int KT, const float *scaleA, float *vals, int *locs,
                            int npace, cudaStream_t st) {
  constexpr int rows = 256 / G;
  k_merge_splits<G, PER><<<(g.nb + rows - 1) / rows, 256, 0, st>>>(g.part_vals, g.part_cols, lists, g.mpad, KT, g.nb,
                                                                  g.k, scaleA, vals, locs, g.pub, g.pace, npace);
}

// Merge the `lists` partial lists a launch with arguments g left per row.
static int launch_merge(const GemmArgs &g, int lists, int KT, const float *scaleA, float *vals, int *locs,
                        int npace, cudaStream_t st) {
  static_assert(MAX_LISTS <= 32 * 10, "the widest merge holds 320 lists");
  if (g.score_mode != R2M_SCORE_SCALED) scaleA = nullptr;
  if (lists <= 4) launch_merge_as<4, 1>(g, lists, KT, scaleA, vals, locs, npace, st);
  else if (lists <= 8) launch_merge_as<8, 1>(g, lists, KT, scaleA, vals, locs, npace, st);
  else if (lists <= 16) launch_merge_as<8, 2>(g, lists, KT, scaleA, vals, locs, npace, st);
  else if (lists <= 32) launch_merge_as<32, 1>(g, lists, KT, scaleA, vals, locs, npace, st);
  else if (lists <= 64) launch_merge_as<32, 2>(g, lists, KT, scaleA, vals, locs, npace, st);
  else if (lists <= 128) launch_merge_as<32, 4>(g, lists, KT, scaleA, vals, locs, npace, st);
  else launch_merge_as<32, 10>(g, lists, KT, scaleA, vals, locs, npace, st);
  R2M_CUDA(cudaGetLastError());
  return R2M_OK;
}

// ------------------------------------------------------------------ host

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                  const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static int get_encode_fn(EncodeTiledFn *fn) {
  static std::mutex mu;
  static EncodeTiledFn cached = nullptr;
  std::lock_guard<std::mutex> lk(mu);
  if (!cached) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q);
    if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !p)
      return fail(R2M_ECUDA, "cuTensorMapEncodeTiled is not available from the driver");
    cached = reinterpret_cast<EncodeTiledFn>(p);
  }
  *fn = cached;
  return R2M_OK;
}

// 2-D uint8 tensor of `rows` x `cols` bytes (row stride = cols), box
// `box_rows` x 128 bytes, 128-byte swizzle, zero fill outside.
static int make_map(CUtensorMap *map, const void *base, long long rows, int cols, int box_rows) {
  EncodeTiledFn fn = nullptr;
  int rc = get_encode_fn(&fn);
  if (rc) return rc;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)cols};
  cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(base), dims, strides, box,
                  estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(R2M_ECUDA, "cuTensorMapEncodeTiled failed (code " + std::to_string((int)r) + ")");
  return R2M_OK;
}

static int pick_kt(int k) {
  if (k <= 8) return 8;
  if (k <= 16) return 16;
  if (k <= 20) return 20;
  if (k <= 32) return 32;
  return 64;
}

static size_t gemm_smem_bytes(int H) {
  return 1024 + (size_t)STAGES * (A_STAGE + B_STAGE) + (2 * STAGES + 5) * 8 + 16 +
         CAND_BYTES;
}

// Column splits for a given number of read tiles.
//
// At least half as many read tiles as CTA pairs: the board is power-bound, a
// last wave with a few idle pairs loses little (the busy ones clock higher)
// but every doubling of the splits costs about 9% at equal wave use (20,000
// reads x 300,007 columns, 79 tiles: 13.7 ms with one split, 9.8 with 5, 9.9
// with 10), so the splits maximise units / (waves x pairs) x
// 0.91^log2(splits) over 1..8.
//
// Fewer read tiles: whole waves of equal units decide.  A unit takes its
// column tiles plus about `fixed` more for filling its reservoirs (8 tiles of
// 6.5 us up to 20 entries, 50 at 64), so the splits minimise waves x (tiles +
// fixed); 6% per doubling of the waves covers the index reads that pairs in
// different splits do not share (8,192 x 619,001: 7.2 ms with 2 splits in one
// wave, 7.6 with 9 in four).  Its weight falls as units grow, and 8,192 reads take
// 9 splits again from 3.3 million columns on, where they are the faster: 4,194,304
// 49.0 ms (2 splits 50.7), 16,777,216 193.9 (202.8); 4,096 reads with 9 98.2 (4
// splits 102.7), 5,120 with 11 120.6 (3 splits 132.1), 7,168 with 5 171.9 (2 splits
// 189.5).  Against the rule before (at least four units per CTA, capped at 64
// splits): 100 reads x 1,000,003 columns 489 -> 336 us (148 splits, one per
// SM), 1,000 x 300,007 575 -> 498 (18), 1,000 x 30,000 196 -> 103 (18),
// 4,096 x 20,000 333 -> 182 (4), 4,096 x 500,000 at k = 64 4.9 -> 3.6 ms (4).
static int choose_splits(int m_tiles, int n_tiles, int ctas, int forced, int max_splits, bool pair, int KT) {
  if (forced > 0) {
    int s = forced;
    if (s > n_tiles) s = n_tiles;
    if (s > max_splits) s = max_splits;
    return s < 1 ? 1 : s;
  }
  int cap = n_tiles < max_splits ? n_tiles : max_splits;
  if (cap < 1) cap = 1;
  int best = 1;
  if (pair && 2 * m_tiles >= ctas) {
    double best_score = -1.0;
    for (int s = 1; s <= 8 && s <= cap; ++s) {
      const long long units = (long long)m_tiles * s;
      const long long waves = (units + ctas - 1) / ctas;
      const double score = (double)units / (double)(waves * ctas) * std::pow(0.91, std::log2((double)s));
      if (score > best_score + 1e-9) {
        best_score = score;
        best = s;
      }
    }
    return best;
  }
  const int fixed = KT <= 20 ? 8 : KT <= 32 ? 16 : 50;
  double best_cost = 0.0, weight = 0.0;
  int waves = 0;
  for (int s = 1; s <= cap; ++s) {
    const int w = (m_tiles * s + ctas - 1) / ctas;
    if (w != waves) {
      waves = w;
      weight = w * (1.0 + 0.06 * std::log2((double)w));
    }
    const double cost = weight * ((n_tiles + s - 1) / s + fixed);
    if (s == 1 || cost < best_cost) {
      best_cost = cost;
      best = s;
    }
  }
  return best;
}

// Tiles and splits of a launch over N columns.  When every unit is one or two
// tiles, narrower tiles spread the columns over more SMs: a tile takes its
// columns plus the reads loaded with it again (32 + 3/4 of them, measured in
// columns) in loads and, per column, in first insertions.  256 -> 64 columns: 1
// read x 2,000 31.4 -> 23.1 us, 16 x 5,000 33.3 -> 29.3, 129 x 2,000 42.0 ->
// 28.6; 256 -> 192: 16 x 20,000 41.5 -> 39.4, 1,000 x 5,000 45.6 -> 43.5.
struct ColumnPlan {
  int bn, n_tiles, splits;
};
static ColumnPlan plan_columns(long long N, int nb, int m_tiles, int ctas, int forced, int max_splits, bool pair,
                               int KT, bool narrow = true) {
  ColumnPlan p;
  p.bn = BN;
  p.n_tiles = (int)((N + BN - 1) / BN);
  p.splits = choose_splits(m_tiles, p.n_tiles, ctas, forced, max_splits, pair, KT);
  const int per_unit = (p.n_tiles + p.splits - 1) / p.splits;
  if (!narrow || forced > 0 || m_tiles * p.splits > ctas || per_unit > 2) return p;
  const int most = std::max(1, std::min(ctas / m_tiles, max_splits)), again = 32 + 3 * std::min(nb, BM) / 4;
  int best = per_unit * (BN + again);
  for (int bn = 192; bn >= 64; bn -= 64) {
    const int tiles = (int)((N + bn - 1) / bn), tau = (tiles + most - 1) / most;
    if (tau * (bn + again) >= best) continue;
    best = tau * (bn + again);
    p.bn = bn;
    p.n_tiles = tiles;
    p.splits = (tiles + tau - 1) / tau;
  }
  return p;
}

template <int KT, int H, bool NARROW = false>
static int launch_gemm(const CUtensorMap &mA, const CUtensorMap &mB, const GemmArgs &g, int ctas,
                       cudaStream_t st) {
  size_t smem = gemm_smem_bytes(H);
  // a function attribute is per device: set it on every launch (cheap)
  R2M_CUDA(cudaFuncSetAttribute(k_gemm_topk<KT, H, NARROW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k_gemm_topk<KT, H, NARROW><<<ctas, epi_threads(H), smem, st>>>(mA, mB, g);
  R2M_CUDA(cudaGetLastError());
  return R2M_OK;
}

static size_t gemm2_smem_bytes(int H) {
  return 1024 + (size_t)STAGES2 * 2 * STAGE2_BYTES + (2 * STAGES2 + 5) * 8 + 16 +
         CAND_BYTES;
}

// Epilogue halves of a launch of kernel `kind`: the CTA-pair kernel always
// takes 2 when the reservoir allows (k <= 32), the single-CTA kernel for
// short units only.
static int epi_halves_for(int kind, int KT, int n_tiles, int splits) {
  if (KT > 32) return 1;
  if (kind == 2) return 2;
  return (n_tiles + splits - 1) / splits <= SHORT_UNIT_TILES ? 2 : 1;
}

template <int KT, int H, bool NARROW = false>
static int launch_gemm2(const CUtensorMap &mA, const CUtensorMap &mB, const GemmArgs &g, int pairs,
                        cudaStream_t st) {
  size_t smem = gemm2_smem_bytes(H);
  R2M_CUDA(cudaFuncSetAttribute(k_gemm_topk2<KT, H, NARROW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * pairs, 1, 1);
  cfg.blockDim = dim3(epi_threads(H), 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  R2M_CUDA(cudaLaunchKernelEx(&cfg, k_gemm_topk2<KT, H, NARROW>, mA, mB, g));
  return R2M_OK;
}

// Reservoir size of an engine: the smallest of 8/16/20/32/64 that holds k,
// or tuning.reserved[4] when that is one of them and holds k.
static int kt_for(int k, const r2m_tuning *tune) {
  const int r = tune ? tune->reserved[4] : 0;
  if ((r == 8 || r == 16 || r == 20 || r == 32 || r == 64) && r >= k) return r;
  return pick_kt(k);
}

// Load every fused-kernel instance once per device (and set its shared-
// memory limit) so that no kernel is first loaded while a stream is being
// captured into a graph.
static int preload_kernels() {
  static std::mutex mu;
  static bool done[64] = {};
  int dev = 0;
  R2M_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  if (dev < 0 || dev >= 64 || done[dev]) return R2M_OK;
#define R2M_PRELOAD1(KT, H, NARROW)                                                                    \
  R2M_CUDA(cudaFuncSetAttribute(k_gemm_topk<KT, H, NARROW>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                (int)gemm_smem_bytes(H)))
#define R2M_PRELOAD2(KT, H, NARROW)                                                                     \
  R2M_CUDA(cudaFuncSetAttribute(k_gemm_topk2<KT, H, NARROW>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                (int)gemm2_smem_bytes(H)))
#define R2M_PRELOAD(KT, H, NARROW) \
  R2M_PRELOAD1(KT, H, NARROW);     \
  R2M_PRELOAD2(KT, H, NARROW)
  R2M_PRELOAD(8, 1, false); R2M_PRELOAD(16, 1, false); R2M_PRELOAD(20, 1, false); R2M_PRELOAD(32, 1, false);
  R2M_PRELOAD(8, 2, false); R2M_PRELOAD(16, 2, false); R2M_PRELOAD(20, 2, false); R2M_PRELOAD(32, 2, false);
  R2M_PRELOAD(8, 2, true); R2M_PRELOAD(16, 2, true); R2M_PRELOAD(20, 2, true); R2M_PRELOAD(32, 2, true);
  R2M_PRELOAD(64, 1, false); R2M_PRELOAD(64, 1, true);
#undef R2M_PRELOAD
#undef R2M_PRELOAD1
#undef R2M_PRELOAD2
  cudaFuncAttributes fa;
  R2M_CUDA(cudaFuncGetAttributes(&fa, k_merge_splits<4, 1>));
  R2M_CUDA(cudaFuncGetAttributes(&fa, k_merge_splits<8, 1>));
  R2M_CUDA(cudaFuncGetAttributes(&fa, k_merge_splits<8, 2>));
  R2M_CUDA(cudaFuncGetAttributes(&fa, k_merge_splits<32, 1>));
  R2M_CUDA(cudaFuncGetAttributes(&fa, k_merge_splits<32, 2>));
  R2M_CUDA(cudaFuncGetAttributes(&fa, k_merge_splits<32, 4>));
  R2M_CUDA(cudaFuncGetAttributes(&fa, k_merge_splits<32, 10>));
  done[dev] = true;
  return R2M_OK;
}

// Which kernel a batch of nb reads runs on: 1 = one CTA per 128-read tile,
// 2 = CTA pairs per 256-read tile.  mode 0 (auto) uses pairs above 128 reads.
static int kernel_kind(int mode, int nb) {
  if (mode == 1) return 1;
  if (mode == 2) return 2;
  return nb > BM ? 2 : 1;
}

// Launch the fused kernel of `kind` (1 single-CTA, 2 CTA pairs) with
// `halves` epilogue halves for the reservoir size KT.  Tiles narrower than BN
// have instances of their own (a run-time tile width costs the others 1%), for
// the most halves of a reservoir size.
template <int KT, int H, bool NARROW = false>
static int launch_kind(int kind, const CUtensorMap &mA, const CUtensorMap &mB, const CUtensorMap &mB128,
                       const GemmArgs &g, int ctas, cudaStream_t st) {
  return kind == 2 ? launch_gemm2<KT, H, NARROW>(mA, mB128, g, ctas, st)
                   : launch_gemm<KT, H, NARROW>(mA, mB, g, ctas, st);
}
static int dispatch_gemm(int kind, int halves, int KT, const CUtensorMap &mA, const CUtensorMap &mB,
                         const CUtensorMap &mB128, const GemmArgs &g, int ctas, cudaStream_t st) {
  if (g.bn != BN) {
    if (halves != (KT <= 32 ? 2 : 1)) return fail(R2M_ESTATE, "narrow tiles need the widest epilogue");
    switch (KT) {
      case 8: return launch_kind<8, 2, true>(kind, mA, mB, mB128, g, ctas, st);
      case 16: return launch_kind<16, 2, true>(kind, mA, mB, mB128, g, ctas, st);
      case 20: return launch_kind<20, 2, true>(kind, mA, mB, mB128, g, ctas, st);
      case 32: return launch_kind<32, 2, true>(kind, mA, mB, mB128, g, ctas, st);
      default: return launch_kind<64, 1, true>(kind, mA, mB, mB128, g, ctas, st);
    }
  }
  if (halves == 2) {
    switch (KT) {
      case 8: return launch_kind<8, 2>(kind, mA, mB, mB128, g, ctas, st);
      case 16: return launch_kind<16, 2>(kind, mA, mB, mB128, g, ctas, st);
      case 20: return launch_kind<20, 2>(kind, mA, mB, mB128, g, ctas, st);
      default: return launch_kind<32, 2>(kind, mA, mB, mB128, g, ctas, st);
    }
  }
  switch (KT) {
    case 8: return launch_kind<8, 1>(kind, mA, mB, mB128, g, ctas, st);
    case 16: return launch_kind<16, 1>(kind, mA, mB, mB128, g, ctas, st);
    case 20: return launch_kind<20, 1>(kind, mA, mB, mB128, g, ctas, st);
    case 32: return launch_kind<32, 1>(kind, mA, mB, mB128, g, ctas, st);
    default: return launch_kind<64, 1>(kind, mA, mB, mB128, g, ctas, st);
  }
}

// Progress slots for pair pacing (one per CTA pair of a launch).
constexpr int kPaceSlots = 1024;

// Pacing window of the CTA-pair kernel from tuning.reserved[3]: 0 = the
// default, > 0 = that many column tiles, < 0 = no pacing.
static int pace_window_for(const r2m_tuning *tune) {
  const int r = tune ? tune->reserved[3] : 0;
  return r < 0 ? 0 : r == 0 ? PACE_WINDOW : r;
}

// Column splits whose lists share a row bound: those that run at the same time.
static int bound_splits(int ctas, int m_tiles, int splits, int halves) {
  const int c = std::max(1, std::min(ctas / m_tiles, splits)), most = BOUND_LISTS / halves;
  const int groups = (c + most - 1) / most;
  return (c + groups - 1) / groups;  // groups of equal size
}

// One allocation: the pacing slots and the row bounds (zero between launches),
// then `lists` partial lists of KT values and columns.  `lists` is a multiple
// of 8, which keeps every part 16-byte aligned.
struct Workspace {
  long long *pace;
  uint32_t *pub;
  float *vals;
  int *cols;
  size_t zero_bytes;  // slots and bounds, from `pace` on
  size_t bytes;       // all of it
};
static cudaError_t alloc_workspace(size_t lists, int KT, Workspace *w) {
  unsigned char *p = nullptr;
  const size_t part = lists * KT * sizeof(float), zero = kPaceSlots * sizeof(long long) + lists * sizeof(uint32_t);
  w->bytes = zero + 2 * part;
  cudaError_t e = cudaMalloc(&p, w->bytes);
  if (e != cudaSuccess) return e;
  // The first search may come at once and on any stream, and recycled memory
  // read as row bounds drops results: the zeros are in place before this
  // returns.  A stream of its own, so that work queued elsewhere is not waited for.
  cudaStream_t st = nullptr;
  e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaMemsetAsync(p, 0, zero, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (st) cudaStreamDestroy(st);
  if (e != cudaSuccess) {
    cudaFree(p);
    return e;
  }
  w->pace = reinterpret_cast<long long *>(p);
  w->pub = reinterpret_cast<uint32_t *>(p + kPaceSlots * sizeof(long long));
  w->vals = reinterpret_cast<float *>(p + zero);
  w->cols = reinterpret_cast<int *>(p + zero + part);
  w->zero_bytes = zero;
  return cudaSuccess;
}

// Rows of a partial list (its stride): the batch, rounded up so that the parts
// of the workspace stay aligned.
static int list_rows(int nb) { return (nb + 7) & ~7; }

// Split lists the workspace must hold for any batch height up to rows_cap.
static size_t lists_needed(int rows_cap, long long N, int ctas, int forced, int mode, int KT) {
  size_t lists = 0;
  const int H = KT <= 32 ? 2 : 1;  // either kernel may leave two partial lists per row and split
  for (int nb = 1; nb < rows_cap + BM; nb = nb == 1 ? BM : nb + BM) {
    const int h = nb < rows_cap ? nb : rows_cap;
    const int kind = kernel_kind(mode, h);
    const int tile = kind == 2 ? 256 : BM;
    const int mt = (h + tile - 1) / tile;
    const int c = kind == 2 ? (ctas / 2 > 0 ? ctas / 2 : 1) : ctas;
    const ColumnPlan p = plan_columns(N, h, mt, c, forced, MAX_LISTS / H, kind == 2, KT);
    lists = std::max(lists, (size_t)p.splits * H * list_rows(h));
  }
  return lists;
}

}  // namespace r2m

using namespace r2m;

struct r2m_engine {
  const uint8_t *B;
  const float *scaleB;
  int rdim;
  long long N;
  long long N_cap;  // columns at creation (the workspace is sized for them)
  int k, KT;
  int rows_cap;
  int score_mode;
  int ctas;
  int forced_splits;
  CUtensorMap mapB;
  CUtensorMap mapB128;  // 128-row box for the CTA-pair kernel
  int mode;             // 0 auto, 1 single-CTA kernel, 2 CTA-pair kernel
  int epi;              // CTA-pair epilogue: 0 auto, 1 four warps, 2 eight warps
  Workspace ws;
  size_t part_lists;  // capacity in lists (rows x splits)
  size_t pub_lists;   // row bounds the workspace holds
  bool dirty;         // a launch whose merge did not follow may have left bounds behind, and nothing has cleared them yet
  uint32_t *err;
  int pace_window;    // 0 = no pacing
  bool timing;        // record events around the two kernels of each call
  cudaEvent_t ev[3];
  int last_splits;
};

extern "C" int r2m_engine_create(const uint8_t *d_B, const float *d_scaleB, int rdim, int64_t N, int k,
                                 int rows_cap, int score_mode, const r2m_tuning *tune,
                                 r2m_engine **out) {
  R2M_REQUIRE(out != nullptr, "out is null");
  *out = nullptr;
  R2M_REQUIRE(d_B != nullptr, "B is null");
  R2M_REQUIRE(rdim >= 16 && rdim % 16 == 0, "rdim must be a positive multiple of 16");
  R2M_REQUIRE(N >= 1 && N <= (1LL << 31) - 1 - BN, "N out of range");
  R2M_REQUIRE(k >= 1 && k <= 64 && k <= N, "need 1 <= k <= min(N, 64)");
  R2M_REQUIRE(rows_cap >= 1, "rows_cap must be >= 1");
  R2M_REQUIRE(score_mode >= R2M_SCORE_F16 && score_mode <= R2M_SCORE_SCALED, "bad score_mode");
  R2M_REQUIRE(score_mode != R2M_SCORE_SCALED || d_scaleB, "scaled scores need scaleB");
  R2M_REQUIRE((reinterpret_cast<uintptr_t>(d_B) & 15) == 0, "B must be 16-byte aligned");
  R2M_REQUIRE(score_mode != R2M_SCORE_SCALED || (reinterpret_cast<uintptr_t>(d_scaleB) & 15) == 0,
              "scaleB must be 16-byte aligned");
  int rc = r2m_device_check();
  if (!rc) rc = preload_kernels();
  if (rc) return rc;
  r2m_engine *e = new r2m_engine();
  e->B = d_B;
  e->scaleB = d_scaleB;
  e->rdim = rdim;
  e->N = N;
  e->N_cap = N;
  e->k = k;
  e->KT = kt_for(k, tune);
  e->rows_cap = rows_cap;
  e->score_mode = score_mode;
  e->ctas = (tune && tune->ctas > 0) ? tune->ctas : sm_count();
  e->forced_splits = (tune && tune->splits > 0) ? tune->splits : 0;
  e->timing = tune && tune->reserved[0] != 0;
  e->mode = tune ? tune->reserved[1] : 0;
  if (e->mode < 0 || e->mode > 2) e->mode = 0;
  e->epi = tune ? tune->reserved[2] : 0;
  if (e->epi < 0 || e->epi > 2) e->epi = 0;
  e->pace_window = pace_window_for(tune);
  e->last_splits = 0;
  if (e->timing) {
    for (int i = 0; i < 3; ++i) {
      cudaError_t ce = cudaEventCreate(&e->ev[i]);
      if (ce != cudaSuccess) {
        delete e;
        return cuda_fail(ce, "cudaEventCreate");
      }
    }
  }
  rc = make_map(&e->mapB, d_B, N, rdim, BN);
  if (!rc) rc = make_map(&e->mapB128, d_B, N, rdim, 128);
  if (rc) {
    delete e;
    return rc;
  }
  // workspace: the largest (read tiles x splits) any batch height can ask for
  size_t lists = lists_needed(rows_cap, N, e->ctas, e->forced_splits, e->mode, e->KT);
  e->part_lists = lists;
  if (alloc_workspace(lists, e->KT, &e->ws) != cudaSuccess) {
    delete e;
    return fail(R2M_ENOMEM, "engine workspace allocation failed");
  }
  e->pub_lists = lists;
  e->dirty = false;
  rc = device_error_word(&e->err);
  if (rc) {
    cudaFree(e->ws.pace);
    delete e;
    return rc;
  }
  *out = e;
  return R2M_OK;
}

extern "C" int r2m_engine_destroy(r2m_engine *eng) {
  if (!eng) return R2M_OK;
  cudaFree(eng->ws.pace);  // the whole workspace
  if (eng->timing)
    for (int i = 0; i < 3; ++i) cudaEventDestroy(eng->ev[i]);
  delete eng;
  return R2M_OK;
}

extern "C" int r2m_engine_set_tuning(r2m_engine *eng, const r2m_tuning *tune) {
  R2M_REQUIRE(eng != nullptr && tune != nullptr, "null pointer");
  const int ctas = tune->ctas > 0 ? tune->ctas : sm_count();
  const int forced = tune->splits > 0 ? tune->splits : 0;
  const int mode = (tune->reserved[1] >= 0 && tune->reserved[1] <= 2) ? tune->reserved[1] : 0;
  const int KT = kt_for(eng->k, tune);
  size_t lists = lists_needed(eng->rows_cap, eng->N_cap, ctas, forced, mode, KT);
  if (lists * KT > eng->part_lists * eng->KT) {  // grow the split workspace
    Workspace w;
    if (alloc_workspace(lists, KT, &w) != cudaSuccess)
      return fail(R2M_ENOMEM, "engine workspace allocation failed");
    const cudaError_t ce = cudaDeviceSynchronize();
    if (ce != cudaSuccess) {
      cudaFree(w.pace);
      return cuda_fail(ce, "cudaDeviceSynchronize");
    }
    cudaFree(eng->ws.pace);
    eng->ws = w;
    eng->pub_lists = lists;
    eng->dirty = false;
    eng->part_lists = lists;
  } else {
    eng->part_lists = eng->part_lists * eng->KT / KT;  // the same bytes hold more, shorter lists
  }
  eng->KT = KT;
  eng->ctas = ctas;
  eng->forced_splits = forced;
  eng->mode = mode;
  eng->epi = (tune->reserved[2] >= 0 && tune->reserved[2] <= 2) ? tune->reserved[2] : 0;
  eng->pace_window = pace_window_for(tune);
  return R2M_OK;
}

namespace r2m {
// Point the engine at another B (and scaleB) of at most the columns it was
// created for: the split workspace stays valid, the tensor maps are encoded
// again on the host.  The maps reach the kernels as launch parameters, so
// launches already queued keep the previous B.
int engine_rebind(r2m_engine *eng, const uint8_t *d_B, const float *d_scaleB, int64_t N) {
  R2M_REQUIRE(eng != nullptr && d_B != nullptr, "null pointer");
  R2M_REQUIRE(N >= eng->k && N <= eng->N_cap, "rebind: N must be in k..N at creation");
  R2M_REQUIRE((reinterpret_cast<uintptr_t>(d_B) & 15) == 0, "B must be 16-byte aligned");
  R2M_REQUIRE(eng->score_mode != R2M_SCORE_SCALED || (d_scaleB && (reinterpret_cast<uintptr_t>(d_scaleB) & 15) == 0),
              "scaled scores need a 16-byte aligned scaleB");
  CUtensorMap m, m128;
  int rc = make_map(&m, d_B, N, eng->rdim, BN);
  if (!rc) rc = make_map(&m128, d_B, N, eng->rdim, 128);
  if (rc) return rc;
  eng->B = d_B;
  eng->scaleB = d_scaleB;
  eng->N = N;
  eng->mapB = m;
  eng->mapB128 = m128;
  return R2M_OK;
}
}  // namespace r2m

extern "C" int r2m_engine_info(const r2m_engine *eng, int *k, int *rdim, int *score_mode, int *rows_cap,
                               int64_t *N) {
  R2M_REQUIRE(eng != nullptr, "engine is null");
  if (k) *k = eng->k;
  if (rdim) *rdim = eng->rdim;
  if (score_mode) *score_mode = eng->score_mode;
  if (rows_cap) *rows_cap = eng->rows_cap;
  if (N) *N = eng->N;
  return R2M_OK;
}

extern "C" int64_t r2m_engine_workspace_bytes(const r2m_engine *eng) {
  if (!eng) return 0;
  return (int64_t)eng->ws.bytes;
}

extern "C" int r2m_batch_gemm_topk(r2m_engine *eng, const uint8_t *d_A, const float *d_scaleA, int nb,
                                   float *d_vals, int32_t *d_locs, r2m_stream_t stream) {
  R2M_REQUIRE(eng != nullptr, "engine is null");
  R2M_REQUIRE(nb >= 0 && nb <= eng->rows_cap, "nb must be in 0..rows_cap");
  if (nb == 0) return R2M_OK;
  R2M_REQUIRE(d_A && d_vals && d_locs, "null pointer");
  R2M_REQUIRE((reinterpret_cast<uintptr_t>(d_A) & 15) == 0, "A must be 16-byte aligned");
  R2M_REQUIRE(eng->score_mode != R2M_SCORE_SCALED || d_scaleA, "scaled scores need scaleA");
  cudaStream_t st = as_stream(stream);
  CUtensorMap mapA;
  int rc = make_map(&mapA, d_A, nb, eng->rdim, BM);
  if (rc) return rc;
  const int kind = kernel_kind(eng->mode, nb);
  const int tile = kind == 2 ? 256 : BM;
  const int ctas_eff = kind == 2 ? (eng->ctas / 2 > 0 ? eng->ctas / 2 : 1) : eng->ctas;
  GemmArgs g;
  g.nb = nb;
  g.num_m_tiles = (nb + tile - 1) / tile;
  g.N = eng->N;
  const int hmax = eng->KT <= 32 ? 2 : 1;
  // (a rebound index of fewer columns may prefer more splits than the
  // workspace was sized for)
  const size_t room = eng->part_lists / ((size_t)hmax * list_rows(nb));
  const ColumnPlan plan =
      plan_columns(eng->N, nb, g.num_m_tiles, ctas_eff, eng->forced_splits,
                   (int)std::min<size_t>(MAX_LISTS / hmax, room), kind == 2, eng->KT, eng->epi != 1 || hmax == 1);
  g.bn = plan.bn;
  g.n_tiles = plan.n_tiles;
  g.splits = plan.splits;
  CUtensorMap narrow;
  if (plan.bn != BN && (rc = make_map(&narrow, eng->B, eng->N, eng->rdim, kind == 2 ? plan.bn / 2 : plan.bn))) return rc;
  const int halves =
      eng->epi == 1 ? 1 : eng->epi == 2 ? hmax : epi_halves_for(kind, eng->KT, g.n_tiles, g.splits);
  const int lists_per_row = halves * g.splits;  // partial lists each row leaves
  g.num_kb = (eng->rdim + BK - 1) / BK;
  g.score_mode = eng->score_mode;
  g.k = eng->k;
  g.mpad = list_rows(nb);
  g.scaleB = eng->scaleB;
  g.part_vals = eng->ws.vals;
  g.part_cols = eng->ws.cols;
  g.err = eng->err;
  if ((size_t)lists_per_row * g.mpad > eng->part_lists) return fail(R2M_ESTATE, "engine workspace too small");
  long long units = (long long)g.num_m_tiles * g.splits;
  int ctas = (int)(units < ctas_eff ? units : ctas_eff);
  eng->last_splits = g.splits;
  g.pace = nullptr;
  g.pace_window = 0;
  if (kind == 2 && eng->pace_window > 0 && ctas > 1 && ctas <= kPaceSlots) {
    g.pace = eng->ws.pace;
    g.pace_window = eng->pace_window;
  }
  const size_t bounds = (size_t)lists_per_row * g.mpad;  // indexed with 32 bits
  g.pub = bounds <= eng->pub_lists && bounds <= INT_MAX ? eng->ws.pub : nullptr;
  g.conc = bound_splits(ctas, g.num_m_tiles, g.splits, halves);
  // Bounds and pacing slots are zero here: the merge of the launch before left
  // them so, or the clear that follows a failure did.  Where that failed too,
  // they are cleared first; a clear that is only being captured runs with the
  // graph, so the calls after it clear again.
  auto clear = [&]() { return cudaMemsetAsync(eng->ws.pace, 0, eng->ws.zero_bytes, st); };
  bool still_dirty = false;
  if (eng->dirty) {
    R2M_CUDA(clear());
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    still_dirty = cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone;
  }
  eng->dirty = true;
  auto launch = [&]() -> int {
    if (eng->timing) R2M_CUDA(cudaEventRecord(eng->ev[0], st));
    if (int e = dispatch_gemm(kind, halves, eng->KT, mapA, plan.bn != BN ? narrow : eng->mapB,
                              plan.bn != BN ? narrow : eng->mapB128, g, ctas, st))
      return e;
    if (eng->timing) R2M_CUDA(cudaEventRecord(eng->ev[1], st));
    return launch_merge(g, lists_per_row, eng->KT, d_scaleA, d_vals, d_locs, ctas, st);
  };
  rc = launch();
  if (rc == R2M_OK || clear() == cudaSuccess) eng->dirty = still_dirty;
  if (rc) {
    cudaGetLastError();  // of the clear; rc and its message tell what failed first
    return rc;
  }
  if (eng->timing) R2M_CUDA(cudaEventRecord(eng->ev[2], st));
  return R2M_OK;
}

extern "C" int r2m_engine_kernel_ms(r2m_engine *eng, float *gemm_ms, float *merge_ms, int *splits) {
  R2M_REQUIRE(eng != nullptr, "engine is null");
  R2M_REQUIRE(eng->timing, "engine was created without kernel timing (tuning.reserved[0] = 1)");
  R2M_CUDA(cudaEventSynchronize(eng->ev[2]));
  float a = 0.f, b = 0.f;
  R2M_CUDA(cudaEventElapsedTime(&a, eng->ev[0], eng->ev[1]));
  R2M_CUDA(cudaEventElapsedTime(&b, eng->ev[1], eng->ev[2]));
  if (gemm_ms) *gemm_ms = a;
  if (merge_ms) *merge_ms = b;
  if (splits) *splits = eng->last_splits;
  return R2M_OK;
}

// ------------------------------------------------------------------
// Allocation-free search.
//
// Some callers cannot allocate device memory at the point where they map a
// batch: a serving loop where a cudaMalloc would synchronize the device and
// stall other streams, or a host whose memory pool (CUDA.jl's, PyTorch's
// caching allocator) already owns the free device memory, so a side
// allocation can fail.  This entry point needs no engine: the pacing slots
// and the per-split partial top-k lists live in the file-scope array below,
// whose device address is looked up with cudaGetSymbolAddress by the first
// call on each device (so that first call should come before any stream
// capture) and again whenever the device's current context is a different
// one (after a cudaDeviceReset the module, and with it the array, is loaded
// anew).  Every GPU that loads this library holds the array
// (kNoAllocScratchBytes) until the process exits; all calls share it, so
// calls that overlap on the GPU race.  The schedule is the engine's
// automatic one (the CTA-pair kernel above 128 reads, paced; the epilogue
// form and the column splits the engine would pick), with the splits cut to
// what the array holds.
namespace r2m {

constexpr size_t kNoAllocScratchBytes = 32u << 20;  // 32 MiB
constexpr size_t kNoAllocPaceBytes = kPaceSlots * sizeof(long long);
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];
static __device__ __align__(256) uint32_t g_noalloc_err;

static std::mutex g_noalloc_mu;
static unsigned char *g_noalloc_ptr[64];
static uint32_t *g_noalloc_err_ptr[64];
static unsigned long long g_noalloc_ctx[64];  // id of the context the addresses belong to

typedef CUresult (*CtxGetCurrentFn)(CUcontext *);
typedef CUresult (*CtxGetIdFn)(CUcontext, unsigned long long *);

// Process-unique id of the current context (0 when the driver cannot tell).
static unsigned long long current_ctx_id() {
  static CtxGetCurrentFn get_cur = nullptr;
  static CtxGetIdFn get_id = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_cur = reinterpret_cast<CtxGetCurrentFn>(p);
    p = nullptr;
    if (cudaGetDriverEntryPoint("cuCtxGetId", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_id = reinterpret_cast<CtxGetIdFn>(p);
  }
  CUcontext c = nullptr;
  unsigned long long id = 0;
  if (!get_cur || !get_id || get_cur(&c) != CUDA_SUCCESS || !c || get_id(c, &id) != CUDA_SUCCESS) return 0;
  return id;
}

// Device addresses of the scratch array and error word on the current device
// (looked up on the first call per device and per context).
static int noalloc_setup(unsigned char **scratch, uint32_t **err) {
  int dev = 0;
  R2M_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return fail(R2M_ESTATE, "device ordinal out of range");
  const unsigned long long ctx = current_ctx_id();
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (g_noalloc_ptr[dev] == nullptr || ctx == 0 || ctx != g_noalloc_ctx[dev]) {
    void *p = nullptr, *q = nullptr;
    R2M_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
    R2M_CUDA(cudaGetSymbolAddress(&q, g_noalloc_err));
    g_noalloc_ptr[dev] = static_cast<unsigned char *>(p);
    g_noalloc_err_ptr[dev] = static_cast<uint32_t *>(q);
    g_noalloc_ctx[dev] = current_ctx_id();  // the lookup made the device's context current
  }
  *scratch = g_noalloc_ptr[dev];
  *err = g_noalloc_err_ptr[dev];
  return R2M_OK;
}

// A bounded wait that gave up leaves partial lists unwritten: mark every
// output row invalid (NaN values, location -1) so the caller sees it.
__global__ void k_noalloc_poison(const uint32_t *err, float *vals, int *locs, long long count) {
  if (*err == 0) return;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < count;
       i += (long long)gridDim.x * blockDim.x) {
    vals[i] = __int_as_float(0x7fc00000);
    locs[i] = -1;
  }
}

}  // namespace r2m

extern "C" int r2m_batch_gemm_topk_noalloc(const uint8_t *d_B, const float *d_scaleB, int rdim, int64_t N,
                                           const uint8_t *d_A, const float *d_scaleA, int nb, int k,
                                           int score_mode, float *d_vals, int32_t *d_locs,
                                           r2m_stream_t stream) {
  R2M_REQUIRE(d_B != nullptr, "B is null");
  R2M_REQUIRE(rdim >= 16 && rdim % 16 == 0, "rdim must be a positive multiple of 16");
  R2M_REQUIRE(N >= 1 && N <= (1LL << 31) - 1 - BN, "N out of range");
  R2M_REQUIRE(k >= 1 && k <= 64 && k <= N, "need 1 <= k <= min(N, 64)");
  R2M_REQUIRE(nb >= 0, "nb must be >= 0");
  R2M_REQUIRE(score_mode >= R2M_SCORE_F16 && score_mode <= R2M_SCORE_SCALED, "bad score_mode");
  if (nb == 0) return R2M_OK;
  R2M_REQUIRE(d_A && d_vals && d_locs, "null pointer");
  R2M_REQUIRE(score_mode != R2M_SCORE_SCALED || (d_scaleA && d_scaleB), "scaled scores need scaleA and scaleB");
  R2M_REQUIRE((reinterpret_cast<uintptr_t>(d_B) & 15) == 0 && (reinterpret_cast<uintptr_t>(d_A) & 15) == 0,
              "A and B must be 16-byte aligned");
  R2M_REQUIRE(score_mode != R2M_SCORE_SCALED || (reinterpret_cast<uintptr_t>(d_scaleB) & 15) == 0,
              "scaleB must be 16-byte aligned");
  const int KT = pick_kt(k);
  const int kind = kernel_kind(0, nb);
  const int tile = kind == 2 ? 256 : BM;
  const int m_tiles = (nb + tile - 1) / tile;
  const size_t list_bytes = (size_t)KT * (sizeof(float) + sizeof(int));
  const size_t max_lists = (kNoAllocScratchBytes - kNoAllocPaceBytes) / list_bytes;
  const size_t mpad = (size_t)m_tiles * tile;
  if (mpad > max_lists)
    return fail(R2M_EINVAL, "nb = " + std::to_string(nb) + " exceeds the allocation-free scratch (" +
                                std::to_string(kNoAllocScratchBytes >> 20) + " MiB holds at most " +
                                std::to_string(max_lists / 256 * 256) + " rows at k = " + std::to_string(k) +
                                "); split the batch or use r2m_batch_gemm_topk");
  unsigned char *scratch = nullptr;
  uint32_t *err = nullptr;
  int rc = noalloc_setup(&scratch, &err);
  if (rc) return rc;
  cudaStream_t st = as_stream(stream);
  const int sms = sm_count();
  const int ctas_eff = kind == 2 ? (sms / 2 > 0 ? sms / 2 : 1) : sms;
  const int hmax = KT <= 32 ? 2 : 1;
  // the engine's automatic schedule, with the splits cut to the scratch
  const ColumnPlan plan = plan_columns(N, nb, m_tiles, ctas_eff, 0, MAX_LISTS / hmax, kind == 2, KT);
  CUtensorMap mapA, mapB;
  if ((rc = make_map(&mapB, d_B, N, rdim, kind == 2 ? plan.bn / 2 : plan.bn))) return rc;
  if ((rc = make_map(&mapA, d_A, nb, rdim, BM))) return rc;
  const int n_tiles = plan.n_tiles;
  int splits = plan.splits;
  int halves = epi_halves_for(kind, KT, n_tiles, splits);
  while (splits > 1 && (size_t)halves * splits * mpad > max_lists) {
    --splits;
    halves = epi_halves_for(kind, KT, n_tiles, splits);
  }
  if ((size_t)halves * splits * mpad > max_lists) halves = 1;
  GemmArgs g;
  g.nb = nb;
  g.num_m_tiles = m_tiles;
  g.N = N;
  g.bn = plan.bn;
  g.n_tiles = n_tiles;
  g.splits = splits;
  g.num_kb = (rdim + BK - 1) / BK;
  g.score_mode = score_mode;
  g.k = k;
  g.mpad = (int)mpad;
  g.scaleB = d_scaleB;
  long long *pace = reinterpret_cast<long long *>(scratch);
  unsigned char *lists = scratch + kNoAllocPaceBytes;
  const size_t nlists = (size_t)halves * splits * mpad;
  g.part_vals = reinterpret_cast<float *>(lists);
  g.part_cols = reinterpret_cast<int *>(lists + nlists * KT * sizeof(float));
  g.err = err;
  const long long units = (long long)m_tiles * splits;
  const int ctas = (int)(units < ctas_eff ? units : ctas_eff);
  g.pace = nullptr;
  g.pace_window = 0;
  // the error word, the pacing slots and the row bounds must start at zero;
  // the partial lists are fully rewritten by the kernel before the merge
  // reads them.  Bounds go behind the lists where they fit.
  R2M_CUDA(cudaMemsetAsync(err, 0, sizeof(uint32_t), st));
  if (kind == 2 && ctas > 1 && ctas <= kPaceSlots) {
    R2M_CUDA(cudaMemsetAsync(pace, 0, (size_t)ctas * sizeof(long long), st));
    g.pace = pace;
    g.pace_window = PACE_WINDOW;
  }
  g.pub = nullptr;
  g.conc = bound_splits(ctas, m_tiles, splits, halves);
  if (nlists * (list_bytes + sizeof(uint32_t)) <= kNoAllocScratchBytes - kNoAllocPaceBytes) {
    g.pub = reinterpret_cast<uint32_t *>(lists + nlists * list_bytes);
    R2M_CUDA(cudaMemsetAsync(g.pub, 0, nlists * sizeof(uint32_t), st));
  }
  rc = dispatch_gemm(kind, halves, KT, mapA, mapB, mapB, g, ctas, st);
  if (rc) return rc;
  if ((rc = launch_merge(g, halves * splits, KT, d_scaleA, d_vals, d_locs, ctas, st))) return rc;
  k_noalloc_poison<<<64, 256, 0, st>>>(err, d_vals, d_locs, (long long)nb * k);
  R2M_CUDA(cudaGetLastError());
  return R2M_OK;
}

// The give-up path of the allocation-free search, driven without a fault:
// the kernels' bounded wait, with a short limit, on an mbarrier nothing
// arrives on, records its code in this path's error word; the poison pass
// then marks the caller's rows as the search would.
extern "C" int r2m_selftest_noalloc_timeout(int64_t limit_cycles, int nb, int k, float *d_vals,
                                            int32_t *d_locs, r2m_stream_t stream) {
  R2M_REQUIRE(limit_cycles >= 0 && limit_cycles <= (int64_t)4000000000LL, "limit_cycles must be in 0..4e9");
  R2M_REQUIRE(nb >= 0 && k >= 1, "need nb >= 0 and k >= 1");
  if (nb == 0) return R2M_OK;
  R2M_REQUIRE(d_vals && d_locs, "null pointer");
  unsigned char *scratch = nullptr;
  uint32_t *err = nullptr;
  int rc = noalloc_setup(&scratch, &err);
  if (rc) return rc;
  cudaStream_t st = as_stream(stream);
  R2M_CUDA(cudaMemsetAsync(err, 0, sizeof(uint32_t), st));
  rc = launch_selftest_wait((long long)limit_cycles, 0, err, st);
  if (rc) return rc;
  k_noalloc_poison<<<64, 256, 0, st>>>(err, d_vals, d_locs, (long long)nb * k);
  R2M_CUDA(cudaGetLastError());
  return R2M_OK;
}
