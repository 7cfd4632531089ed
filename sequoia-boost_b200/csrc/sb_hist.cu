// sb_hist.cu — gradient histogram construction (K4) and subtraction (K5).
//
// Replaces CpuBackend::build / accumulate (tree/hist/mod.rs:58-119) and
// `subtracted` / HistogramBackend::subtract (:25-28, :38-44).
//
// Design: a persistent grid (one CTA of 1024 threads per SM, or four of 256
// where four partials fit) divides the concatenated rows of every node to
// build (all frontier nodes of all class trees in one launch; cta_parts). A
// CTA keeps one node's histogram for one feature tile in shared memory, walks
// its rows with two sub-batches of codes in flight per warp (hist_body), adds
// every code of a row into the shared partial, and flushes the non-zero
// entries to the node's HBM histogram with global atomics when it moves to the
// next piece.
//   codes  TILED layout: lane l reads features 4l..4l+3 of the tile (one
//          8-byte load per row) and a code is the entry's index in the tile's
//          partial, where a feature's bins are contiguous. LANES layout: each
//          tile gives lane l `S` (1, 2 or 4) code positions of the row, packed
//          with features so that every lane's entries fit its own column;
//          entry e of lane l sits at word e * 32 + l: the 32 lanes of a warp
//          add into 32 different banks.
//   sums   FP32 form: f32 shared atomics, f64 node histograms. FIXED form:
//          gradients rounded to |q| <= 2^bits with a per-round power-of-two
//          scale; one int32 and one uint32 shared atomic per entry, exact
//          because a CTA flushes at least every fixed_rows_per_flush(bits)
//          rows; int64 node histograms (order independent).
// Each feature also owns one extra "missing" bin (index total_bins + f), so a
// node's missing-value statistics are summed directly instead of being
// recovered as total - present.
#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "sb_internal.cuh"

namespace sb {
namespace {

constexpr int HIST_THREADS = 1024;
// CTA size where four partials fit one SM (HIST_SMALL_SMEM each): a node of
// few rows takes a CTA mostly latency (zeroing, the dependent loads of its
// first rows, flushing), so that four small CTAs per SM take four nodes in the
// time of one.
constexpr int HIST_SMALL_THREADS = 256;
constexpr size_t HIST_SMALL_SMEM = 48 << 10;
constexpr int MAX_TILE_FEATURES = 128;  // 4 features per lane
// rows a CTA adds in about the time it zeroes and flushes a partial
constexpr int FLUSH_ROWS = 1500, FLUSH_ROWS_SMALL = 256;

struct HistDev {
  const uint16_t* bins;  // u16 codes, or null with u8 codes in bins8
  const uint8_t* bins8;
  const uint32_t* foff;
  size_t Fp;             // row stride of bins (u16)
  const int* rbase;      // LANES: first shared word of each feature, and the shift of its bins
  const int* rshift;
  const int* slot_feat;  // LANES: feature of each code position of a row
  size_t n;              // gradient column stride
  int total_bins;
  const void* gpair;
  const HistItem* items;
  const uint64_t* prefix;
  const int* count;
  const FeatureTile* tiles;
  int ntiles;
  uint32_t flush_rows;   // FIXED: max rows per shared partial
  unsigned long long* rows_done;  // sampled rows accumulated (or null)
  const uint32_t* pool_mask;      // [K][FW] features to accumulate (or null: all)
  int FW;
  const uint64_t* parts;          // [2 * CTAs] each CTA's part of the rows (cta_parts), or null: equal shares
};

__device__ __forceinline__ int find_item(const uint64_t* prefix, int count, uint64_t pos) {
  int lo = 0, hi = count;  // last i with prefix[i] <= pos
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (prefix[mid] <= pos) lo = mid; else hi = mid;
  }
  return lo;
}

// One addition into each plane of the shared partial, at the 32-bit shared
// address `a` (g plane) and `a + hoff` (h plane), with `red` (no value
// returned). FIXED: int32 g and uint32 h; FP32: f32 bits.
template <bool FIXED>
__device__ __forceinline__ void add_pair(unsigned a, unsigned hoff, uint32_t vg, uint32_t vh) {
  if (FIXED) {
    asm volatile("red.shared.add.s32 [%0], %1;" ::"r"(a), "r"(vg));
    asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(a + hoff), "r"(vh));
  } else {
    asm volatile("red.shared.add.f32 [%0], %1;" ::"r"(a), "f"(__uint_as_float(vg)));
    asm volatile("red.shared.add.f32 [%0], %1;" ::"r"(a + hoff), "f"(__uint_as_float(vh)));
  }
}

// Loads of the row gather, volatile so that they stay ahead of the adds they
// are meant to overlap (the compiler otherwise sinks them towards their use).
__device__ __forceinline__ uint2 gather(const uint2* p) {
  uint2 v;
  asm volatile("ld.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ uint16_t gather(const uint16_t* p) {
  uint16_t v;
  asm volatile("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t gather(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// The code layouts of a launch (see sb_internal.cuh): TILED with u16 or u8
// codes, LANES with 1, 2 or 4 code positions per lane.
enum { CODES_U16 = 0, CODES_U8 = 1, CODES_LANES1 = 2, CODES_LANES2 = 3, CODES_LANES4 = 4 };
template <int KIND> struct Codes { using T = uint2; };  // 4 u16 codes
template <> struct Codes<CODES_U8> { using T = uint32_t; };      // 4 u8 codes
template <> struct Codes<CODES_LANES1> { using T = uint16_t; };
template <> struct Codes<CODES_LANES2> { using T = uint32_t; };  // 2 u16 codes

__device__ __forceinline__ uint32_t code_word(const uint2& v, int i) { return i ? v.y : v.x; }
__device__ __forceinline__ uint32_t code_word(uint32_t v, int) { return v; }
__device__ __forceinline__ uint32_t code_word(uint16_t v, int) { return v; }

// One CTA's share of a launch. The shared partial is two planes of `words`
// 32-bit words, g then h (FIXED: int32 / uint32 integers; FP32: floats).
//
// What bounds it: the load-store unit. A row costs two shared reductions per
// code position, a load of its codes and three shuffles, and an instruction
// whose lanes hit one bank k times takes k passes. So
//  - the row loop has no predicate or branch at all: a predicated or branched
//    shared reduction compiles to a branch around it, which also keeps loads
//    from moving ahead of adds (100 warp instructions per 100-feature row, 45
//    without; LANES at 10M rows x 100 features, root level, per launch: 756 us
//    with a test per row, 486 without). FP32 tests each position: a shared f32
//    reduction is a compare-and-swap loop, and warps that meet in a lane's
//    unused word retry (10M rows x 100 features, per launch: 1.78 ms, 0.78 with
//    the test), as do the lanes of one instruction that add the zeros of rows past
//    the end to row 0's bins (1000 rows x 10 features, whole call 76 us, 63
//    without those; rounds of 10,000 x 20 337 and 287 us);
//  - LANES, whose 32 lanes hit 32 banks, needs 8 passes for 4 positions per
//    lane where TILED's 25 lanes of random bins need 23.
template <bool FIXED, int KIND, int RL>
__device__ __forceinline__ void hist_body(const HistDev& a, unsigned bx, unsigned gdx) {
  constexpr bool LANES = KIND >= CODES_LANES1, U8 = KIND == CODES_U8;
  constexpr int S = KIND == CODES_LANES1 ? 1 : KIND == CODES_LANES2 ? 2 : 4;  // codes per lane and row
  constexpr int rl = LANES ? 0 : RL;
  constexpr int R = rl == 3 ? 2 : S == 4 ? 4 : 8;  // steps per sub-batch
  constexpr uint32_t SUB = (uint32_t)R << rl;      // rows per sub-batch: two or more fill a block of 32
  using CW = typename Codes<KIND>::T;
  extern __shared__ __align__(16) unsigned long long sh_u64[];  // zeroed 16 bytes at a time
  unsigned* sh_g = reinterpret_cast<unsigned*>(sh_u64);
  __shared__ double s_tot_d[2];
  __shared__ unsigned long long s_tot_u[2];

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int count = *a.count;
  if (count <= 0) return;
  const uint64_t W = a.prefix[count];
  if (W == 0) return;
  const uint64_t U = W * (uint64_t)a.ntiles;
  const uint64_t lo = a.parts ? a.parts[2 * bx] : U * bx / gdx, hi = a.parts ? a.parts[2 * bx + 1] : U * (bx + 1) / gdx;
  uint64_t u = lo;
  while (u < hi) {
    const int t = (int)(u / W);
    const uint64_t pos = u - (uint64_t)t * W;
    const int it = find_item(a.prefix, count, pos);
    const HistItem item = a.items[it];
    const uint64_t item_lo = a.prefix[it], item_hi = a.prefix[it + 1];
    uint64_t piece_hi_u = (uint64_t)t * W + item_hi;
    if (piece_hi_u > hi) piece_hi_u = hi;
    uint64_t n_pos = piece_hi_u - u;
    if (FIXED && n_pos > a.flush_rows) n_pos = a.flush_rows;
    const uint32_t pbeg = item.begin + (uint32_t)(pos - item_lo);
    const FeatureTile tile = a.tiles[t];
    const int nf = tile.f1 - tile.f0;
    const int nent = LANES ? 32 * tile.E : tile.nbins + nf;  // entries of a plane
    // words of a plane. LANES: half a bank turn between an entry's g and h, for
    // the flush. TILED: a word per lane for what is not added; an even count.
    const int words = LANES ? nent + 16 : (nent + 33) & ~1;
    unsigned* sh_h = sh_g + words;
    const unsigned sh_base = (unsigned)__cvta_generic_to_shared(sh_g), hoff = 4u * (unsigned)words;
    const bool want_total = item.root && t == 0;

    // Where the lane's codes of a row sit. TILED: a warp instruction covers
    // 2^rl rows: the lane works on row slot lane >> (5 - rl) and owns the 4
    // consecutive features f0 + 4 * grp .. +3 of the tile, grp = its lane
    // within the row's group (lanes past the tile read its first features and
    // add none). Tiles start at multiples of 4, hold at most 4 * 32 >> rl
    // features, and rows are padded to a multiple of 8 codes, so a row's load
    // is aligned and stays inside it.
    const int grp = lane & ((32 >> rl) - 1), rsub = lane >> (5 - rl);
    const bool past = !LANES && 4 * grp >= nf;
    const int pos0 = LANES ? tile.slot_off + lane * S : tile.f0 + (past ? 0 : 4 * grp);
    // A code is added at `base` + 4 * code. Positions without a feature of the
    // tree's pool read as code 0 and add to a word of the lane's own that the
    // flush leaves out (LANES: entry 0 of its column).
    unsigned base[S];
    uint32_t keep[2] = {0, 0};  // code bits that count
    unsigned pool = 0;          // FP32: the positions that are added, of rows before the end
#pragma unroll
    for (int j = 0; j < S; ++j) {
      int f = LANES ? a.slot_feat[pos0 + j] : pos0 + j;
      if (past || (!LANES && f >= tile.f1)) f = -1;
      const bool in_pool =
          f >= 0 && (!a.pool_mask || ((a.pool_mask[(size_t)item.k * a.FW + (f >> 5)] >> (f & 31)) & 1u));
      base[j] = sh_base;
      pool |= (unsigned)in_pool << j;
      if (!in_pool) base[j] += 4u * (unsigned)(LANES ? lane : nent + lane);
      else if (U8) base[j] += 4u * (a.foff[f] - (unsigned)tile.bin0 + (unsigned)(4 * grp + j));
      if (in_pool) keep[U8 ? 0 : j >> 1] |= U8 ? 0xFFu << (8 * j) : 0xFFFFu << (16 * (j & 1));
    }
    for (int i = threadIdx.x; i < words / 2; i += blockDim.x)
      reinterpret_cast<uint4*>(sh_g)[i] = make_uint4(0u, 0u, 0u, 0u);
    if (threadIdx.x < 2) {
      s_tot_d[threadIdx.x] = 0.0;
      s_tot_u[threadIdx.x] = 0ull;
    }
    __syncthreads();

    // A warp's rows: FIXED, an equal, contiguous part of the piece; FP32, runs
    // of RUN rows dealt to the warps in turn, so that the piece's rows are
    // added in about their own order whatever the load pipeline. They go in
    // blocks of 32: lane i holds row i of a block, its id loaded two blocks
    // ahead and its gradient pair one block ahead. The codes are loaded in
    // sub-batches of SUB rows into two register buffers in turn: the next
    // sub-batch is requested before the wait for the current one, so that two
    // are in flight while a warp waits (with one buffer copied to the other,
    // the copy waited for the newest load: 35 clocks per row instead of 19).
    // Step q of a sub-batch covers its rows (q << rl) + slot; shuffles hand
    // every lane its row's id and pair.
    const size_t gcol = (size_t)item.k * a.n;
    const CW* codes = reinterpret_cast<const CW*>(U8 ? (const void*)(a.bins8 + pos0) : (const void*)(a.bins + pos0));
    const uint32_t row_words = (uint32_t)(a.Fp / (U8 ? 4 : S));
    constexpr uint32_t RUN = LANES ? 8 : 4u << rl;
    const uint32_t m = (uint32_t)n_pos, per = (m + nwarps - 1) / nwarps, round = nwarps * RUN;
    const uint32_t p0 = pbeg + (FIXED ? min(m, warp * per) : warp * RUN);
    const uint32_t nrows = FIXED ? min(m, (warp + 1) * per) - min(m, warp * per)
                                 : m / round * RUN + min(RUN, max(m % round, warp * RUN) - warp * RUN);
    // the warp's row v of the piece, in the item's list
    auto row_at = [&](uint32_t v) { return FIXED ? p0 + v : p0 + v / RUN * round + v % RUN; };
    double tg = 0.0, th = 0.0;
    int tqg = 0;  // a piece has at most flush_rows rows of |q| <= 2^bits: 31 bits hold the sums
    uint32_t tqh = 0;
    auto load_rid = [&](uint32_t q) { return q + lane < nrows ? item.rows[row_at(q + lane)] : 0u; };
    auto load_pair = [&](uint32_t q, uint32_t rid, uint32_t& g, uint32_t& h) {
      uint2 v = make_uint2(0u, 0u);
      if (q + lane < nrows) v = gather(reinterpret_cast<const uint2*>(a.gpair) + gcol + rid);
      g = FIXED ? v.y : v.x;  // FIXED: (q_g << 32) + q_h; FP32: {grad, hess}
      h = FIXED ? v.x : v.y;
    };
    // The codes of rows [s, s + SUB) of a block. Positions past the part's end
    // hold row id 0 and a zero pair: their adds change nothing, and FIXED needs
    // no test per row.
    auto load_codes = [&](uint32_t rid, uint32_t s, CW (&bv)[R]) {
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const uint32_t id = __shfl_sync(0xFFFFFFFFu, rid, s + ((uint32_t)q << rl) + (uint32_t)rsub);
        bv[q] = gather(codes + (uint64_t)id * row_words);
      }
    };
    auto add_codes = [&](uint32_t g, uint32_t h, uint32_t s, uint32_t nr, const CW (&bv)[R]) {
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const uint32_t src = s + ((uint32_t)q << rl) + (uint32_t)rsub;
        const uint32_t vg = __shfl_sync(0xFFFFFFFFu, g, src);
        const uint32_t vh = __shfl_sync(0xFFFFFFFFu, h, src);
        const unsigned on = src < nr ? pool : 0u;
#pragma unroll
        for (int j = 0; j < S; ++j) {
          const uint32_t w = code_word(bv[q], U8 ? 0 : j >> 1) & keep[U8 ? 0 : j >> 1];
          const uint32_t c = U8 ? (w >> (8 * j)) & 0xFFu : (j & 1) ? w >> 16 : w & 0xFFFFu;
          if (FIXED || (on >> j & 1)) add_pair<FIXED>(base[j] + 4u * c, hoff, vg, vh);
        }
      }
    };
    if (nrows) {
      uint32_t p = 0;
      uint32_t rid_c = load_rid(p), g_c, h_c;
      uint32_t rid_n = load_rid(p + 32);
      load_pair(p, rid_c, g_c, h_c);
      uint32_t nr = min(nrows - p, 32u);
      CW buf0[R], buf1[R];
      load_codes(rid_c, 0, buf0);
      for (;;) {
        const uint32_t pn = p + 32;
        const uint32_t nr_n = pn < nrows ? min(nrows - pn, 32u) : 0u;
        uint32_t g_n, h_n;
        load_pair(pn, rid_n, g_n, h_n);
        const uint32_t rid_nn = load_rid(pn + 32);
        if (want_total) {
          if (FIXED) {
            tqg += (int)g_c;
            tqh += h_c;
          } else {
            tg += (double)__uint_as_float(g_c);
            th += (double)__uint_as_float(h_c);
          }
        }
#pragma unroll 1
        for (uint32_t s = 0; s < nr; s += 2 * SUB) {
          load_codes(rid_c, s + SUB, buf1);
          add_codes(g_c, h_c, s, nr, buf0);
          const bool inside = s + 2 * SUB < nr;
          load_codes(inside ? rid_c : rid_n, inside ? s + 2 * SUB : 0u, buf0);
          add_codes(g_c, h_c, s + SUB, nr, buf1);
        }
        if (nr_n == 0) break;
        p = pn;
        nr = nr_n;
        rid_c = rid_n;
        rid_n = rid_nn;
        g_c = g_n;
        h_c = h_n;
      }
    }
    if (a.rows_done && t == 0 && threadIdx.x == 0) atomicAdd(a.rows_done, (unsigned long long)n_pos);
    if (want_total) {  // one add per warp: 64-bit shared adds to one address go one after another
      if (FIXED) {
        tqg = __reduce_add_sync(0xFFFFFFFFu, tqg);
        tqh = __reduce_add_sync(0xFFFFFFFFu, tqh);
      } else {
        for (int o = 16; o > 0; o >>= 1) {
          tg += __shfl_xor_sync(0xFFFFFFFFu, tg, o);
          th += __shfl_xor_sync(0xFFFFFFFFu, th, o);
        }
      }
      if (lane == 0) {
        if (FIXED) {
          atomicAdd(&s_tot_u[0], (unsigned long long)(long long)tqg);
          atomicAdd(&s_tot_u[1], (unsigned long long)tqh);
        } else {
          atomicAdd(&s_tot_d[0], tg);
          atomicAdd(&s_tot_d[1], th);
        }
      }
    }
    __syncthreads();
    // Flush the partial into the node's HBM histogram, two threads per entry:
    // a warp's adds then cover whole sectors (570 G words/s over 148 CTAs of
    // 25,700 entries; g and h in separate instructions 300 G words/s). TILED
    // u16 entries are in histogram order; the others go one sector of each of
    // 8 features at a time (LANES: of 8 neighbouring lanes, 2 threads per
    // bank), their words computed from the feature's place. Four entries per
    // thread and step keep their shared reads in flight together.
    unsigned* plane = (lane & 1) ? sh_h : sh_g;
    auto add_out = [&](int bin, uint32_t v) {
      const size_t gi = 2 * (size_t)bin + (lane & 1);
      if (v == 0u) return;
      if (FIXED) {
        const unsigned long long add =
            (lane & 1) ? (unsigned long long)v : (unsigned long long)(long long)(int)v;
        atomicAdd(reinterpret_cast<unsigned long long*>(item.out) + gi, add);
      } else {
        atomicAdd(reinterpret_cast<double*>(item.out) + gi, (double)__uint_as_float(v));
      }
    };
    if (KIND == CODES_U16) {
      const int step = blockDim.x >> 1;
      for (int i0 = threadIdx.x >> 1; i0 < nent; i0 += 4 * step) {
        uint32_t v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = i0 + j * step < nent ? plane[i0 + j * step] : 0u;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int i = i0 + j * step;
          add_out(i < tile.nbins ? tile.bin0 + i : a.total_bins + tile.f0 + (i - tile.nbins), v[j]);
        }
      }
    } else {
      constexpr int CHUNKS = 8;  // warps that share 8 features
      const int ngroups = LANES ? 4 * S : (nf + 7) / 8, k8 = lane >> 2;
      for (int unit = warp; unit < ngroups * CHUNKS; unit += nwarps) {
        const int grp8 = unit / CHUNKS;
        int f = LANES ? a.slot_feat[tile.slot_off + (8 * (grp8 & 3) + k8) * S + (grp8 >> 2)] : tile.f0 + 8 * grp8 + k8;
        if (!LANES && f >= tile.f1) f = -1;
        int first = 0, nb = -1, word = 0, shift = 0;  // nb: the missing entry
        if (f >= 0) {
          first = (int)a.foff[f];
          nb = (int)a.foff[f + 1] - first;
          word = LANES ? a.rbase[f] : first - tile.bin0 + (f - tile.f0);
          shift = LANES ? a.rshift[f] : 0;
        }
        const int most = __reduce_max_sync(0xFFFFFFFFu, nb);
        for (int s = unit % CHUNKS; 2 * s - 1 <= most; s += 4 * CHUNKS) {
          uint32_t v[4];
          const int b0 = 2 * s + ((lane >> 1) & 1) - (first & 1);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int b = b0 + 2 * CHUNKS * j;
            v[j] = b >= 0 && b <= nb ? plane[word + (b << shift)] : 0u;
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int b = b0 + 2 * CHUNKS * j;
            add_out(b < nb ? first + b : a.total_bins + f, v[j]);
          }
        }
      }
    }
    if (want_total && threadIdx.x == 0) {
      if (FIXED) {
        unsigned long long* o = reinterpret_cast<unsigned long long*>(item.total);
        atomicAdd(o, s_tot_u[0]);
        atomicAdd(o + 1, s_tot_u[1]);
      } else {
        double* o = reinterpret_cast<double*>(item.total);
        atomicAdd(o, s_tot_d[0]);
        atomicAdd(o + 1, s_tot_d[1]);
      }
    }
    __syncthreads();
    u += n_pos;
  }
}

template <bool FIXED, int KIND, int RL, int THREADS = HIST_THREADS>
__global__ void __launch_bounds__(THREADS, HIST_THREADS / THREADS) k_hist(HistDev a) {
  follow_launch();
  hist_body<FIXED, KIND, RL>(a, blockIdx.x, gridDim.x);
}

// Many indexes' histogram launches as one (sb_train_many): the x-blocks are
// every job's own persistent grid laid end to end; block x belongs to job j
// when xoff[j] <= x < xoff[j + 1], and runs job j's launch description.
struct HistJobs {
  const HistDev* devs;   // [njobs]
  const unsigned* xoff;  // [njobs + 1]
  int njobs;
};

__device__ __forceinline__ int hist_job_of(const unsigned* xoff, int njobs, unsigned x) {
  int lo = 0, hi = njobs;  // the last job whose first block is <= x
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (xoff[mid] <= x) lo = mid; else hi = mid;
  }
  return lo;
}

template <bool FIXED, int KIND, int RL, int THREADS>
__global__ void __launch_bounds__(THREADS, HIST_THREADS / THREADS) k_hist_jobs(HistJobs H) {
  const int j = hist_job_of(H.xoff, H.njobs, blockIdx.x);
  __shared__ HistDev s_dev;  // the job's description, as near as a launch's own parameters
  for (unsigned i = threadIdx.x; i < sizeof(HistDev) / 4; i += blockDim.x)
    reinterpret_cast<uint32_t*>(&s_dev)[i] = reinterpret_cast<const uint32_t*>(H.devs + j)[i];
  __syncthreads();
  hist_body<FIXED, KIND, RL>(s_dev, blockIdx.x - H.xoff[j], H.xoff[j + 1] - H.xoff[j]);
}

// The TILED kernels for a precision, rows per warp instruction (log2), code
// width and CTA size: alone, or batched over jobs.
template <bool FIXED, int KIND, int RL>
const void* tiled_pick(int threads, bool jobs) {
  if (threads == HIST_SMALL_THREADS)
    return jobs ? (const void*)k_hist_jobs<FIXED, KIND, RL, HIST_SMALL_THREADS>
                : (const void*)k_hist<FIXED, KIND, RL, HIST_SMALL_THREADS>;
  return jobs ? (const void*)k_hist_jobs<FIXED, KIND, RL, HIST_THREADS> : (const void*)k_hist<FIXED, KIND, RL>;
}
template <bool FIXED, int KIND>
const void* tiled_pick(int rl, int threads, bool jobs) {
  switch (rl) {
    case 1: return tiled_pick<FIXED, KIND, 1>(threads, jobs);
    case 2: return tiled_pick<FIXED, KIND, 2>(threads, jobs);
    case 3: return tiled_pick<FIXED, KIND, 3>(threads, jobs);
    default: return tiled_pick<FIXED, KIND, 0>(threads, jobs);
  }
}
const void* tiled_kernel(bool fixed, const Ghist* g, bool jobs) {
  const int rl = g->tiled_rl, th = g->hist_threads;
  if (g->code_bytes == 1) return fixed ? tiled_pick<true, CODES_U8>(rl, th, jobs) : tiled_pick<false, CODES_U8>(rl, th, jobs);
  return fixed ? tiled_pick<true, CODES_U16>(rl, th, jobs) : tiled_pick<false, CODES_U16>(rl, th, jobs);
}

const void* lanes_kernel(bool fixed, int slots) {
  switch (slots) {
    case 1: return fixed ? (const void*)k_hist<true, CODES_LANES1, 0> : (const void*)k_hist<false, CODES_LANES1, 0>;
    case 2: return fixed ? (const void*)k_hist<true, CODES_LANES2, 0> : (const void*)k_hist<false, CODES_LANES2, 0>;
    default: return fixed ? (const void*)k_hist<true, CODES_LANES4, 0> : (const void*)k_hist<false, CODES_LANES4, 0>;
  }
}

// The parts of a launch's CTAs in the tile-major list of (tile, item) row
// ranges, into parts[2 * CTA] and [2 * CTA + 1]; run by one block of
// ZERO_THREADS. An equal share of all rows, or, where zeroing and flushing a
// second partial would cost more than the longer share of whole-range CTAs, a
// part of one range only: every range gets one CTA and its share of the
// others. (2M x 200 multiclass lossguide, 20 ranges a launch: 45 us with equal
// shares, 23 us with one range per CTA.) With min_units set, a launch holding
// few rows uses fewer CTAs of at least that many (row, tile) units, so that a
// partial is paid for by enough rows; the others get nothing.
constexpr int ZERO_THREADS = 256, MAX_RANGES = 1024;
__device__ void cta_parts(const HistParts& p, int count) {
  __shared__ uint32_t s_end[MAX_RANGES];  // CTAs of the ranges up to and including each
  const int tid = threadIdx.x, lane = tid & 31;
  const uint64_t W = count > 0 ? p.prefix[count] : 0, U = W * (uint64_t)p.ntiles;
  const uint64_t ranges = (uint64_t)max(count, 0) * p.ntiles;
  const uint64_t mu = p.min_units ? p.min_units : 1;
  const uint32_t act = (uint32_t)min((uint64_t)p.ctas, max((uint64_t)1, (U + mu - 1) / mu));
  if (ranges >= act || ranges > MAX_RANGES || U * ranges >= (uint64_t)p.flush_rows * act * (act - ranges)) {
    for (uint32_t c = tid; c < (uint32_t)p.ctas; c += ZERO_THREADS) {
      p.parts[2 * c] = c < act ? U * c / act : 0;
      p.parts[2 * c + 1] = c < act ? U * (c + 1) / act : 0;
    }
    return;
  }
  const uint32_t nr = (uint32_t)ranges, nc = max(count, 1);
  for (uint32_t r = tid; r < nr; r += ZERO_THREADS) {  // the CTAs beyond one per range, in proportion, rounded down
    const uint32_t i = r % nc, len = (uint32_t)(p.prefix[i + 1] - p.prefix[i]);
    s_end[r] = 1 + (U ? (uint32_t)((double)len * ((double)(act - nr) * (1.0 - 1e-12) / (double)U)) : 0u);
  }
  __syncthreads();
  if (tid < 32) {
    uint32_t before = 0;
    for (uint32_t r0 = 0; r0 < nr; r0 += 32) {
      uint32_t v = r0 + lane < nr ? s_end[r0 + lane] : 0u;
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= o) v += y;
      }
      v += before;
      if (r0 + lane < nr) s_end[r0 + lane] = v;
      before = __shfl_sync(0xFFFFFFFFu, v, 31);
    }
  }
  __syncthreads();
  for (uint32_t c = tid; c < (uint32_t)p.ctas; c += ZERO_THREADS) {
    uint64_t b = 0, e = 0;
    if (nr && c < s_end[nr - 1]) {
      uint32_t lo = 0, hi = nr - 1;  // the first range whose CTAs reach past c
      while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (s_end[mid] > c) hi = mid; else lo = mid + 1;
      }
      const uint32_t c0 = lo ? s_end[lo - 1] : 0u, n = s_end[lo] - c0, q = c - c0;
      const uint32_t t = lo / nc, i = lo - t * nc;
      const uint32_t len = (uint32_t)(p.prefix[i + 1] - p.prefix[i]), each = len / n, more = len % n;
      b = p.prefix[i] + (uint64_t)t * W + (uint64_t)each * q + min(q, more);
      e = b + each + (q < more ? 1u : 0u);
    }
    p.parts[2 * c] = b;
    p.parts[2 * c + 1] = e;
  }
}

// Zeroes the node histograms (and root totals) of a launch's items, one grid
// row per item; the last row divides the rows over the histogram's CTAs.
__device__ __forceinline__ void zero_items_body(const HistItem* items, const int* count, size_t words,
                                                const HistParts& parts, unsigned bx, unsigned gdx) {
  const int it = blockIdx.y, n = *count;
  if (it == (int)gridDim.y - 1) {
    if (bx == 0 && parts.parts) cta_parts(parts, n);
    return;
  }
  if (it >= n) return;
  unsigned long long* o = reinterpret_cast<unsigned long long*>(items[it].out);
  for (size_t i = (size_t)bx * blockDim.x + threadIdx.x; i < words; i += (size_t)gdx * blockDim.x) o[i] = 0ull;
  if (items[it].root && bx == 0 && threadIdx.x < 2)
    reinterpret_cast<unsigned long long*>(items[it].total)[threadIdx.x] = 0ull;
}

__global__ void k_zero_items(const HistItem* items, const int* count, size_t words, HistParts parts) {
  follow_launch();
  zero_items_body(items, count, words, parts, blockIdx.x, gridDim.x);
}

// k_zero_items for many jobs: job j's blocks are xoff[j] .. xoff[j + 1] - 1.
__global__ void k_zero_items_jobs(const ZeroJob* __restrict__ zj, const unsigned* __restrict__ xoff, int njobs) {
  const int j = hist_job_of(xoff, njobs, blockIdx.x);
  const ZeroJob z = zj[j];
  zero_items_body(z.items, z.count, z.words, z.parts, blockIdx.x - xoff[j], xoff[j + 1] - xoff[j]);
}

__global__ void k_subtract(const double2* __restrict__ p, const double2* __restrict__ c,
                           double2* __restrict__ o, size_t n) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    double2 a = p[i], b = c[i];
    o[i] = make_double2(__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y));
  }
}

__global__ void k_fixed_to_f64(const longlong2* __restrict__ in, double2* __restrict__ out, size_t n,
                               double sg, double sh) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    longlong2 v = in[i];
    out[i] = make_double2(__dmul_rn((double)v.x, sg), __dmul_rn((double)v.y, sh));
  }
}

}  // namespace

namespace {

// TILED layout: contiguous feature ranges whose bins and missing entries fit
// the shared-memory budget, at most 128 features (4 per lane), starting at
// multiples of 4 features.
// Rows per warp instruction of the TILED kernel (as log2): a narrow matrix
// leaves most of a warp's lanes without features when one row takes the
// whole warp (4 features per lane), so up to 8 rows share an instruction:
// at most 128 >> rl features per tile. SB_HIST_ROWS (1, 2, 4, 8) forces it.
static int tiled_rows_log(size_t F) {
  if (const char* e = std::getenv("SB_HIST_ROWS")) {
    const int v = std::atoi(e);
    if (v == 1) return 0;
    if (v == 2) return 1;
    if (v == 4) return 2;
    if (v == 8) return 3;
  }
  return F <= 16 ? 3 : F <= 32 ? 2 : F <= 64 ? 1 : 0;
}

int plan_tiled(Ghist* g, size_t budget, int rl) {
  g->tiles.clear();
  const size_t F = g->F;
  g->tiled_rl = rl >= 0 ? rl : tiled_rows_log(F);
  const size_t max_tile = (size_t)MAX_TILE_FEATURES >> g->tiled_rl;
  size_t f0 = 0, maxb = 0;
  while (f0 < F) {
    size_t f1 = f0;
    while (f1 < F && f1 - f0 < max_tile) {
      size_t bins = g->h_foff[f1 + 1] - g->h_foff[f0];
      if ((bins + (f1 + 1 - f0) + 33) / 2 * 16 > budget) break;
      f1++;
    }
    SB_REQUIRE(f1 > f0, SB_ERR_UNSUPPORTED, "feature %zu has too many bins for shared memory", f0);
    if (f1 < F && f1 - f0 >= 4) f1 -= (f1 - f0) % 4;  // next tile starts on a multiple of 4
    SB_REQUIRE(f1 == F || (f1 - f0) % 4 == 0, SB_ERR_UNSUPPORTED,
               "features %zu.. need more shared memory than one CTA has", f0);
    FeatureTile t{};
    t.f0 = (int)f0;
    t.f1 = (int)f1;
    t.bin0 = (int)g->h_foff[f0];
    t.nbins = (int)(g->h_foff[f1] - g->h_foff[f0]);
    maxb = std::max(maxb, (size_t)(t.nbins + (t.f1 - t.f0) + 33) / 2 * 16);
    SB_REQUIRE(t.nbins + (t.f1 - t.f0) < 0xFFFF, SB_ERR_UNSUPPORTED, "histogram tile too large");
    g->tiles.push_back(t);
    f0 = f1;
  }
  g->layout = HIST_LAYOUT_TILED;
  g->slots = 0;
  g->Fp = (F + 7) / 8 * 8;
  // one-byte codes when every feature's local bins and its missing code fit
  // (SB_HIST_CODES=2 keeps two bytes)
  size_t max_nb = 0;
  for (size_t f = 0; f < F; ++f) max_nb = std::max<size_t>(max_nb, g->h_foff[f + 1] - g->h_foff[f]);
  const char* cb = std::getenv("SB_HIST_CODES");
  g->code_bytes = (max_nb <= 255 && !(cb && std::atoi(cb) == 2)) ? 1 : 2;
  g->h_rpos.assign(F, 0);
  g->h_rbase.assign(F, 0);
  g->h_rmiss.assign(F, 0);
  g->h_rshift.assign(F, 0);
  for (FeatureTile& t : g->tiles) {
    for (int f = t.f0; f < t.f1; ++f) {
      g->h_rpos[f] = f;
      if (g->code_bytes == 1) {  // the local bin; the bin count when missing
        g->h_rbase[f] = 0;
        g->h_rmiss[f] = (int)(g->h_foff[f + 1] - g->h_foff[f]);
      } else {  // the entry in the tile's partial: bins, then one missing entry per feature
        g->h_rbase[f] = (int)g->h_foff[f] - t.bin0;
        g->h_rmiss[f] = t.nbins + (f - t.f0);
      }
    }
  }
  g->hist_smem_bytes = maxb;
  return SB_OK;
}

// One feature's place in the LANES layout: bin b at shared word
// word + (b << shift) (shift 5 in the lane's own column, else 0).
struct LanePlace {
  int lane, slot, word, shift;
};

// Longest-processing-time packing of features [f0, f1) into 32 lanes of
// `slots` positions, at most `emax` rows of 32 words. Row 0 of every lane's
// column takes what is not a feature's. Features whose bins fit no column any
// more (the fourth 257-bin feature of a lane) get consecutive words in rows
// below the columns: a few lanes' adds to random banks cost less than another
// tile. Returns the rows used, or -1 when the features do not fit.
int pack_lanes(const Ghist* g, size_t f0, size_t f1, int slots, int emax, std::vector<LanePlace>* out) {
  const size_t m = f1 - f0;
  if (m > (size_t)32 * slots) return -1;
  std::vector<int> order(m);
  for (size_t i = 0; i < m; ++i) order[i] = (int)(f0 + i);
  auto ent = [&](int f) { return (int)(g->h_foff[f + 1] - g->h_foff[f]) + 1; };
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return ent(a) > ent(b); });
  for (int reserve = 0;;) {  // rows kept for the features outside the columns
    int load[32], used[32] = {0};
    for (int& l : load) l = 1;
    out->assign(m, LanePlace{0, 0, 0, 5});
    std::vector<int> rest;
    int rows = 1, rest_words = 0;
    for (int f : order) {
      int best = -1;
      for (int l = 0; l < 32; ++l)
        if (used[l] < slots && (best < 0 || load[l] < load[best])) best = l;
      if (best < 0 || load[best] + ent(f) > emax - reserve) {
        rest.push_back(f);
        rest_words += ent(f);
        continue;
      }
      (*out)[f - f0] = LanePlace{best, used[best]++, load[best] * 32 + best, 5};
      load[best] += ent(f);
      rows = std::max(rows, load[best]);
    }
    const int rest_rows = (rest_words + 31) / 32;
    if (rows + rest_rows <= emax) {
      int word = rows * 32;
      for (int f : rest) {
        const int l = (int)(std::min_element(used, used + 32) - used);
        (*out)[f - f0] = LanePlace{l, used[l]++, word, 0};
        word += ent(f);
      }
      return rows + rest_rows;
    }
    if (rest_rows <= reserve) return -1;
    reserve = rest_rows;
  }
}

// LANES layout: the fewest tiles of near-equal feature counts whose features
// all pack into the 32 lanes (a last tile of few features would cost a pass
// over the rows of its own).
int plan_lanes(Ghist* g, size_t budget, int slots, std::vector<std::vector<LanePlace>>* places) {
  const size_t F = g->F;
  const int emax = (int)std::min<size_t>((budget / 8 - 16) / 32, 0xFFFF / 32);
  for (size_t T = (F + 32 * slots - 1) / (32 * slots); T <= F; ++T) {
    std::vector<FeatureTile> tiles;
    places->clear();
    for (size_t i = 0; i < T; ++i) {
      FeatureTile t{};
      t.f0 = (int)(F * i / T);
      t.f1 = (int)(F * (i + 1) / T);
      std::vector<LanePlace> at;
      t.E = pack_lanes(g, t.f0, t.f1, slots, emax, &at);
      if (t.E < 0) break;
      t.bin0 = (int)g->h_foff[t.f0];
      t.nbins = (int)(g->h_foff[t.f1] - g->h_foff[t.f0]);
      t.slot_off = (int)i * 32 * slots;
      tiles.push_back(t);
      places->push_back(at);
    }
    if (tiles.size() == T) {
      g->tiles = tiles;
      return SB_OK;
    }
  }
  return SB_ERR_UNSUPPORTED;  // one feature's bins exceed the partial
}

size_t lanes_smem(const Ghist* g) {
  size_t m = 0;
  for (const FeatureTile& t : g->tiles) m = std::max(m, ((size_t)t.E * 32 + 16) * 8);
  return m;
}

}  // namespace

namespace {

size_t smem_budget(const sb_ctx* ctx) {
  return ctx->smem_optin > 8192 ? ctx->smem_optin - 4096 : ctx->smem_optin;
}

}  // namespace

// Plans the histogram's bin-code layout and feature tiles for one choice
// (HIST_LAYOUT_TILED, or HIST_LAYOUT_LANES with 1, 2 or 4 code positions per
// lane and tile). SB_ERR_UNSUPPORTED when a feature's entries do not fit the
// partial.
int hist_prepare(sb_ctx* ctx, Ghist* g, HistChoice c) {
  const size_t budget = smem_budget(ctx);
  const size_t F = g->F;
  if (c.layout == HIST_LAYOUT_TILED) {
    SB_TRY(plan_tiled(g, budget, c.rl));
  } else {
    const int slots = c.slots;
    SB_REQUIRE(slots == 1 || slots == 2 || slots == 4, SB_ERR_INVALID_ARG, "internal: %d slots", slots);
    std::vector<std::vector<LanePlace>> places;
    SB_REQUIRE(plan_lanes(g, budget, slots, &places) == SB_OK, SB_ERR_UNSUPPORTED,
               "a feature has too many bins for the lane layout");
    g->layout = HIST_LAYOUT_LANES;
    g->slots = slots;
    g->code_bytes = 2;
    g->Fp = g->tiles.size() * 32 * slots;
    g->h_rpos.assign(F, 0);
    g->h_rbase.assign(F, 0);
    g->h_rmiss.assign(F, 0);
    g->h_rshift.assign(F, 0);
    std::vector<int> sf(g->Fp, -1);
    for (size_t ti = 0; ti < g->tiles.size(); ++ti) {
      const FeatureTile& t = g->tiles[ti];
      for (int f = t.f0; f < t.f1; ++f) {
        const LanePlace& pl = places[ti][f - t.f0];
        g->h_rpos[f] = t.slot_off + pl.lane * slots + pl.slot;
        g->h_rbase[f] = pl.word;
        g->h_rshift[f] = pl.shift;
        g->h_rmiss[f] = pl.word + ((int)(g->h_foff[f + 1] - g->h_foff[f]) << pl.shift);
        sf[g->h_rpos[f]] = f;
      }
    }
    SB_TRY(g->slot_feat.alloc(ctx, sf.size()));
    SB_CUDA(cudaMemcpyAsync(g->slot_feat.p, sf.data(), sf.size() * 4, cudaMemcpyHostToDevice, ctx->stream));
    SB_CUDA(cudaStreamSynchronize(ctx->stream));  // the pageable copy must finish before sf goes away
    g->hist_smem_bytes = lanes_smem(g);
  }
  g->hist_threads =
      g->layout == HIST_LAYOUT_TILED && g->hist_smem_bytes <= HIST_SMALL_SMEM ? HIST_SMALL_THREADS : HIST_THREADS;
  if (g->layout == HIST_LAYOUT_TILED)
    for (int fixed = 0; fixed < 2; ++fixed) SB_TRY(raise_smem_limit(tiled_kernel(fixed != 0, g, false), g->hist_smem_bytes));
  for (int fixed = 0; fixed < 2; ++fixed)
    for (int slots : {1, 2, 4}) SB_TRY(raise_smem_limit(lanes_kernel(fixed != 0, slots), g->hist_smem_bytes));
  return SB_OK;
}

// Device memory that an allocation on the context can still get: what is free
// on the device and what the pool holds unused.
static int memory_left(const sb_ctx* ctx, size_t* left) {
  size_t free_b = 0, total_b = 0;
  uint64_t reserved = 0, used = 0;
  cudaMemPool_t pool;
  SB_CUDA(cudaMemGetInfo(&free_b, &total_b));
  SB_CUDA(cudaDeviceGetDefaultMemPool(&pool, ctx->device));
  SB_CUDA(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved));
  SB_CUDA(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used));
  *left = free_b + (size_t)(reserved - used);
  return SB_OK;
}

// The layout an index takes without timing, or what SB_HIST_LAYOUT ("tiled"
// or "lanes") in the environment forces. Wide matrices (more than 64 features)
// of 200k rows and more take LANES with 4 positions per lane where it packs:
// its adds never meet in a bank. Measured per launch, root / deepest level, us:
// 10M x 100 x 256 bins 481 / 255 against TILED's 955 / 403; 300k x 100 48 / 80
// against 71 / 79; 3M x 70 x 64 bins (TILED u8) 141 / 72 against 252 / 115.
// Two bounds on that:
//  - at least LANES_MIN_ROWS_PER_BIN rows to a histogram entry. A partial's flush
//    is dearer than TILED's and there are more tiles of wide features, which few
//    rows do not pay for (rounds of depth 8, 200k rows, LANES / TILED, ms: 300 x
//    512 bins, 1.3 rows to an entry, 2.38 / 2.13; 128 x 1024, 1.5, 2.20 / 1.96; 100
//    x 512, 3.9, 1.17 / 1.07; 80 x 512, 4.9, 1.01 / 1.02; 65 x 512, 6.0, 0.91 /
//    0.94; 129 x 256, 6.0, 0.78 / 0.86; 100 x 256, 7.8, 0.79 / 0.70);
//  - its codes take up to five times the memory (256 bytes per row and tile). An
//    index whose extra codes are more than an eighth of the memory that a TILED
//    index would leave stays TILED, so that what fits beside such an index fits.
// Smaller indexes take TILED, the layout that batched jobs share.
constexpr size_t LANES_MIN_ROWS_PER_BIN = 4, LANES_MEMORY_SHARE = 8;
constexpr size_t LANES_SMALL_EXTRA = 256 << 20;  // not worth asking the driver: its answer takes 0.09 ms
int hist_default_choice(sb_ctx* ctx, Ghist* g, HistChoice* out) {
  const size_t F = g->F;
  const char* force = std::getenv("SB_HIST_LAYOUT");
  const bool force_lanes = force && std::strcmp(force, "lanes") == 0;
  *out = HistChoice{HIST_LAYOUT_TILED, 0};
  if (!force_lanes && (force || std::getenv("SB_HIST_ROWS") || F <= 64 || g->n < TUNE_MIN_ROWS ||
                       g->n < LANES_MIN_ROWS_PER_BIN * (g->total_bins + F)))
    return SB_OK;
  const int slots = F <= 32 ? 1 : (F <= 64 ? 2 : 4);
  std::vector<std::vector<LanePlace>> places;
  const std::vector<FeatureTile> keep = g->tiles;
  const bool ok = plan_lanes(g, smem_budget(ctx), slots, &places) == SB_OK;
  const size_t lanes_row = g->tiles.size() * 32 * slots * 2;
  g->tiles = keep;
  SB_REQUIRE(ok || !force_lanes, SB_ERR_UNSUPPORTED, "SB_HIST_LAYOUT=lanes: a feature has too many bins");
  if (!ok) return SB_OK;
  const size_t tiled_row = (F + 7) / 8 * 8 * (g->max_feature_bins <= 255 ? 1 : 2);
  const size_t extra = lanes_row > tiled_row ? g->n * (lanes_row - tiled_row) : 0;
  if (!force_lanes && extra > LANES_SMALL_EXTRA) {
    size_t left = 0;
    SB_TRY(memory_left(ctx, &left));
    const size_t tiled = g->n * (tiled_row + 2 * F);  // with the feature-major bins
    if (left < tiled || (left - tiled) / LANES_MEMORY_SHARE < extra) return SB_OK;
  }
  *out = HistChoice{HIST_LAYOUT_LANES, slots};
  return SB_OK;
}

// The choices the autotuner times for up to 64 features: TILED with 1, 2, 4
// or 8 rows per instruction (one row per instruction keeps at most 16 of a
// warp's lanes busy) and LANES with 1 and 2 positions per lane where the
// features pack. Wider matrices take hist_default_choice's rule.
std::vector<HistChoice> hist_candidates(sb_ctx* ctx, Ghist* g) {
  std::vector<HistChoice> out{HistChoice{HIST_LAYOUT_TILED, 0, 0}};
  if (g->F > 64) return out;
  // TILED with 2, 4, 8 rows per warp instruction while a tile still holds
  // every feature (128 >> rl features)
  for (int rl = 1; rl <= 3 && (size_t)(MAX_TILE_FEATURES >> rl) >= g->F; ++rl)
    out.push_back(HistChoice{HIST_LAYOUT_TILED, 0, rl});
  const std::vector<FeatureTile> keep = g->tiles;
  for (int slots : {1, 2}) {
    std::vector<std::vector<LanePlace>> places;
    if (plan_lanes(g, smem_budget(ctx), slots, &places) == SB_OK) out.push_back(HistChoice{HIST_LAYOUT_LANES, slots});
  }
  g->tiles = keep;
  return out;
}

namespace {

const void* hist_kernel(const Ghist* g, bool fixed) {
  if (g->layout == HIST_LAYOUT_LANES) return lanes_kernel(fixed, g->slots);
  return tiled_kernel(fixed, g, false);
}

}  // namespace

// The persistent grid: every resident CTA, or for a launch known to hold few
// rows one CTA per `rows_per_cta` (row, tile) units (a batched job leaves SMs
// to the other batches' launches).
int hist_grid(sb_ctx* ctx, const Ghist* g, size_t rows_bound, size_t rows_per_cta) {
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, hist_kernel(g, true), g->hist_threads,
                                                g->hist_smem_bytes);
  if (per_sm < 1) per_sm = 1;
  const size_t full = (size_t)ctx->num_sms * per_sm;
  if (rows_bound == 0) return (int)full;
  const size_t want = (rows_bound * g->tiles.size() + rows_per_cta - 1) / rows_per_cta;
  return (int)std::max<size_t>(1, std::min(full, want));
}

// The kernel's description of one launch.
static HistDev hist_dev(const HistLaunch& L) {
  HistDev a;
  a.bins = L.g->code_bytes == 1 ? nullptr : L.g->bins.p;
  a.bins8 = L.g->code_bytes == 1 ? L.g->bins8.p : nullptr;
  a.foff = L.g->foff.p;
  a.Fp = L.g->Fp;
  a.rbase = L.g->rbase.p;
  a.rshift = L.g->rshift.p;
  a.slot_feat = L.g->slot_feat.p;
  a.n = L.g->n;
  a.total_bins = (int)L.g->total_bins;
  a.gpair = L.gpair;
  a.items = L.items;
  a.prefix = L.prefix;
  a.count = L.count;
  a.tiles = L.tiles;
  a.ntiles = L.ntiles;
  a.flush_rows = fixed_rows_per_flush(L.quant_bits);
  a.rows_done = L.rows_done;
  a.pool_mask = L.pool_mask;
  a.FW = (int)((L.g->F + 31) / 32);
  a.parts = L.parts;
  return a;
}

int launch_hist(sb_ctx* ctx, const HistLaunch& L) {
  const HistDev a = hist_dev(L);
  const int grid = hist_grid(ctx, L.g, L.rows_bound, L.rows_per_cta);
  const size_t sm = L.g->hist_smem_bytes;
  void (*kern)(HistDev) = reinterpret_cast<void (*)(HistDev)>(const_cast<void*>(hist_kernel(L.g, L.fixed != 0)));
  SB_LAUNCH_NEXT(ctx, kern, grid, L.g->hist_threads, sm, a);
  return SB_OK;
}

// The division of a launch's rows over its CTAs (cta_parts).
static HistParts hist_parts(sb_ctx* ctx, const HistLaunch& L) {
  HistParts p;
  p.prefix = L.prefix;
  p.ntiles = L.ntiles;
  p.ctas = hist_grid(ctx, L.g, L.rows_bound, L.rows_per_cta);
  p.min_units = L.min_units;
  p.flush_rows = L.g->hist_threads == HIST_SMALL_THREADS ? FLUSH_ROWS_SMALL : FLUSH_ROWS;
  p.parts = L.parts;
  return p;
}

int launch_zero_items(sb_ctx* ctx, const HistLaunch& L) {
  if (L.max_items <= 0) return SB_OK;
  const size_t words = (L.g->total_bins + L.g->F) * 2;
  dim3 grid((unsigned)std::min<size_t>((words + 255) / 256, 64), (unsigned)L.max_items + 1);
  SB_LAUNCH_NEXT(ctx, k_zero_items, grid, ZERO_THREADS, 0, L.items, L.count, words, hist_parts(ctx, L));
  return SB_OK;
}

int hist_jobs_prepare(sb_ctx* ctx, const std::vector<HistLaunch>& Ls, HistJobsPlan* P) {
  const int nj = (int)Ls.size();
  SB_REQUIRE(nj > 0, SB_ERR_INVALID_ARG, "internal: no jobs");
  std::vector<HistDev> devs(nj);
  std::vector<ZeroJob> zero(nj);
  P->fixed = Ls[0].fixed;
  P->smem = 0;
  P->hist_grid.assign(nj, 0);
  P->zero_grid.assign(nj, 0);
  for (int j = 0; j < nj; ++j) {
    const HistLaunch& L = Ls[j];
    SB_REQUIRE(L.g->layout == HIST_LAYOUT_TILED && L.fixed == P->fixed && L.g->tiled_rl == Ls[0].g->tiled_rl &&
                   L.g->code_bytes == Ls[0].g->code_bytes && L.g->hist_threads == Ls[0].g->hist_threads,
               SB_ERR_INVALID_ARG,
               "internal: batched histograms need the TILED layout, one precision, one row grouping, one "
               "code width and one CTA size");
    devs[j] = hist_dev(L);
    const size_t words = (L.g->total_bins + L.g->F) * 2;
    zero[j] = ZeroJob{L.items, L.count, words, hist_parts(ctx, L)};
    P->hist_grid[j] = (unsigned)hist_grid(ctx, L.g, L.rows_bound, L.rows_per_cta);
    P->zero_grid[j] = (unsigned)std::min<size_t>((words + 255) / 256, 64);
    P->smem = std::max(P->smem, L.g->hist_smem_bytes);
  }
  P->njobs = nj;
  cudaStream_t st = ctx->stream;
  SB_TRY(P->devs.alloc(ctx, nj * sizeof(HistDev)));
  SB_TRY(P->zero.alloc(ctx, nj));
  SB_CUDA(cudaMemcpyAsync(P->devs.p, devs.data(), nj * sizeof(HistDev), cudaMemcpyHostToDevice, st));
  SB_CUDA(cudaMemcpyAsync(P->zero.p, zero.data(), nj * sizeof(ZeroJob), cudaMemcpyHostToDevice, st));
  P->kernel = tiled_kernel(P->fixed != 0, Ls[0].g, true);
  P->threads = Ls[0].g->hist_threads;
  SB_TRY(raise_smem_limit(P->kernel, P->smem));
  SB_CUDA(cudaStreamSynchronize(st));  // the host tables are released on return
  return SB_OK;
}

int launch_hist_jobs(sb_ctx* ctx, const HistJobsPlan& P, const unsigned* d_xoff, unsigned hist_blocks,
                     const unsigned* d_zoff, unsigned zero_blocks, int max_items) {
  if (max_items <= 0 || hist_blocks == 0) return SB_OK;
  SB_LAUNCH(ctx, k_zero_items_jobs, dim3(zero_blocks, (unsigned)max_items + 1), ZERO_THREADS, 0, P.zero.p, d_zoff, P.njobs);
  HistJobs H;
  H.devs = reinterpret_cast<const HistDev*>(P.devs.p);
  H.xoff = d_xoff;
  H.njobs = P.njobs;
  void (*kern)(HistJobs) =
      reinterpret_cast<void (*)(HistJobs)>(const_cast<void*>(P.kernel));
  SB_LAUNCH(ctx, kern, hist_blocks, P.threads, P.smem, H);
  return SB_OK;
}

// Device time of fixed-point histogram launches over min(n, 2^20) rows
// spread over the whole matrix (one row drawn from each of m equal strides,
// ascending): the gathers of a round's deeper levels, on codes mostly
// outside L2. Best of two after a warm-up launch: the autotuner's measure.
int hist_time(sb_ctx* ctx, const Ghist* g, float* ms) {
  const size_t m = std::min<size_t>(g->n, (size_t)1 << 20);
  const size_t HB = g->total_bins + g->F;
  cudaStream_t st = ctx->stream;
  DBuf<uint32_t> rows;
  DBuf<unsigned long long> gp;
  DBuf<longlong2> out;
  DBuf<HistItem> item;
  DBuf<uint64_t> prefix;
  DBuf<int> count;
  DBuf<FeatureTile> tiles;
  SB_TRY(rows.alloc(ctx, m));
  SB_TRY(gp.alloc_zero(ctx, g->n));
  SB_TRY(out.alloc(ctx, HB));
  SB_TRY(item.alloc(ctx, 1));
  SB_TRY(prefix.alloc(ctx, 2));
  SB_TRY(count.alloc(ctx, 1));
  SB_TRY(tiles.alloc(ctx, g->tiles.size()));
  std::vector<uint32_t> h_rows(m);
  const size_t stride = g->n / m;
  for (size_t i = 0; i < m; ++i) h_rows[i] = (uint32_t)(i * stride + sb_mix64(i) % stride);
  HistItem it{};
  it.rows = rows.p;
  it.begin = 0;
  it.end = (uint32_t)m;
  it.out = out.p;
  const uint64_t h_prefix[2] = {0, (uint64_t)m};
  const int one = 1;
  SB_CUDA(cudaMemcpyAsync(rows.p, h_rows.data(), m * 4, cudaMemcpyHostToDevice, st));
  SB_CUDA(cudaMemcpyAsync(item.p, &it, sizeof(it), cudaMemcpyHostToDevice, st));
  SB_CUDA(cudaMemcpyAsync(prefix.p, h_prefix, sizeof(h_prefix), cudaMemcpyHostToDevice, st));
  SB_CUDA(cudaMemcpyAsync(count.p, &one, sizeof(one), cudaMemcpyHostToDevice, st));
  SB_CUDA(cudaMemcpyAsync(tiles.p, g->tiles.data(), g->tiles.size() * sizeof(FeatureTile), cudaMemcpyHostToDevice,
                          st));
  HistLaunch L;
  L.g = g;
  L.gpair = gp.p;
  L.fixed = 1;
  L.quant_bits = 16;
  L.items = item.p;
  L.prefix = prefix.p;
  L.count = count.p;
  L.max_items = 1;
  L.tiles = tiles.p;
  L.ntiles = (int)g->tiles.size();
  L.rows_done = nullptr;
  L.pool_mask = nullptr;
  cudaEvent_t e0, e1;
  SB_CUDA(cudaEventCreate(&e0));
  SB_CUDA(cudaEventCreate(&e1));
  float best = 1e30f;
  int rc = SB_OK;
  for (int rep = 0; rep < 3 && rc == SB_OK; ++rep) {
    cudaMemsetAsync(out.p, 0, out.bytes(), st);
    cudaEventRecord(e0, st);
    rc = launch_hist(ctx, L);
    cudaEventRecord(e1, st);
    if (cudaEventSynchronize(e1) != cudaSuccess) rc = SB_ERR_CUDA;
    float t = 0.0f;
    cudaEventElapsedTime(&t, e0, e1);
    if (rep > 0) best = std::min(best, t);
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  *ms = best;
  return rc;
}

// The CTAs of a fixed-point launch over m rows by itself (the seam): for few
// rows one per SM, for more one per 128 (row, tile) units up to the full grid.
// More CTAs zero and flush more partials than the rows pay for (256 bins, whole
// call, full grid of 592 / this: 3000 rows x 20 features 115 / 110 us, 50,000 x 30
// 217 / 204). FP32 keeps the full grid: fewer CTAs put more rows into an f32
// partial (1000 rows x 8 features: error against 64 bits 1.3e-9, 5.6e-9 with 148).
static void seam_grid(sb_ctx* ctx, HistLaunch* L, size_t m) {
  if (!L->fixed) return;
  const size_t units = m * (size_t)L->ntiles, sms = (size_t)ctx->num_sms;
  L->rows_bound = m;
  L->rows_per_cta = std::max<size_t>(1, std::min<size_t>(128, units / sms));
}

// per-node seam helpers (defined in sb_grow.cu)
int quantize_pairs(sb_ctx* ctx, const float2* d_gp, size_t n, int bits, unsigned long long* d_packed,
                   int* h_shift_g, int* h_shift_h);

}  // namespace sb

extern "C" {

int sb_hist_build(sb_ctx* ctx, const sb_ghist* g, const uint32_t* rows, size_t m,
                  const sb_gradpair* gpair, size_t n, int precision, int quantize_bits,
                  sb_gradstats* out, size_t total_bins) {
  using namespace sb;
  SB_REQUIRE(ctx && g && gpair && out, SB_ERR_INVALID_ARG, "NULL argument");
  SB_SAME_DEVICE(ctx, g);
  SB_REQUIRE(m == 0 || rows, SB_ERR_INVALID_ARG, "rows is NULL");
  SB_REQUIRE(total_bins == g->total_bins, SB_ERR_DIMENSION,
             "dimension mismatch: out length expected %zu, got %zu", g->total_bins, total_bins);
  SB_REQUIRE(n == g->n, SB_ERR_DIMENSION, "dimension mismatch: gpair length expected %zu, got %zu",
             g->n, n);
  SB_REQUIRE(precision == SB_HIST_FP32 || precision == SB_HIST_FIXED, SB_ERR_INVALID_ARG,
             "unknown precision %d", precision);
  int bits = quantize_bits ? quantize_bits : 16;
  SB_REQUIRE(bits >= 8 && bits <= 23, SB_ERR_INVALID_ARG, "quantize_bits must be in [8, 23]");
  for (size_t i = 0; i < m; ++i)
    SB_REQUIRE(rows[i] < n, SB_ERR_INVALID_ARG, "row %u out of range", rows[i]);
  SB_CUDA(cudaSetDevice(ctx->device));
  cudaStream_t st = ctx->stream;
  const size_t HB = g->total_bins + g->F;
  DBuf<uint32_t> d_rows;
  DBuf<float2> d_gp;
  DBuf<unsigned long long> d_packed;
  DBuf<double2> d_hist, d_out;
  DBuf<HistItem> d_item;
  DBuf<uint64_t> d_prefix;
  DBuf<int> d_count;
  DBuf<FeatureTile> d_tiles;
  SB_TRY(d_rows.alloc(ctx, std::max<size_t>(m, 1)));
  SB_TRY(d_gp.alloc(ctx, n));
  SB_TRY(d_hist.alloc(ctx, HB));
  SB_TRY(d_out.alloc(ctx, HB));
  SB_TRY(d_item.alloc(ctx, 1));
  SB_TRY(d_prefix.alloc(ctx, 2));
  SB_TRY(d_count.alloc(ctx, 1));
  SB_TRY(d_tiles.alloc(ctx, g->tiles.size()));
  if (m) SB_CUDA(cudaMemcpyAsync(d_rows.p, rows, m * 4, cudaMemcpyHostToDevice, st));
  SB_CUDA(cudaMemcpyAsync(d_gp.p, gpair, n * 8, cudaMemcpyHostToDevice, st));
  SB_CUDA(cudaMemcpyAsync(d_tiles.p, g->tiles.data(), g->tiles.size() * sizeof(FeatureTile),
                          cudaMemcpyHostToDevice, st));
  int sg = 0, shh = 0;
  const void* gsrc = d_gp.p;
  if (precision == SB_HIST_FIXED) {
    SB_TRY(d_packed.alloc(ctx, n));
    SB_TRY(quantize_pairs(ctx, d_gp.p, n, bits, d_packed.p, &sg, &shh));
    gsrc = d_packed.p;
  }
  HistItem it;
  it.rows = d_rows.p;
  it.begin = 0;
  it.end = (uint32_t)m;
  it.k = 0;
  it.root = 0;
  it.out = d_hist.p;
  it.total = nullptr;
  uint64_t prefix[2] = {0, (uint64_t)m};
  int one = 1;
  SB_CUDA(cudaMemcpyAsync(d_item.p, &it, sizeof(it), cudaMemcpyHostToDevice, st));
  SB_CUDA(cudaMemcpyAsync(d_prefix.p, prefix, sizeof(prefix), cudaMemcpyHostToDevice, st));
  SB_CUDA(cudaMemcpyAsync(d_count.p, &one, sizeof(int), cudaMemcpyHostToDevice, st));
  SB_CUDA(cudaMemsetAsync(d_hist.p, 0, d_hist.bytes(), st));
  HistLaunch L;
  L.g = g;
  L.gpair = gsrc;
  L.fixed = precision == SB_HIST_FIXED;
  L.quant_bits = bits;
  L.items = d_item.p;
  L.prefix = d_prefix.p;
  L.count = d_count.p;
  L.max_items = 1;
  L.tiles = d_tiles.p;
  L.ntiles = (int)g->tiles.size();
  L.rows_done = nullptr;
  L.pool_mask = nullptr;
  seam_grid(ctx, &L, m);
  if (m) SB_TRY(launch_hist(ctx, L));
  const double2* res = d_hist.p;
  if (L.fixed) {
    SB_LAUNCH(ctx, k_fixed_to_f64, 256, 256, 0, reinterpret_cast<const longlong2*>(d_hist.p), d_out.p,
              HB, std::ldexp(1.0, -sg), std::ldexp(1.0, -shh));
    res = d_out.p;
  }
  SB_CUDA(cudaMemcpyAsync(out, res, total_bins * sizeof(double2), cudaMemcpyDeviceToHost, st));
  SB_CUDA(cudaStreamSynchronize(st));
  return SB_OK;
}

int sb_hist_subtract(sb_ctx* ctx, const sb_gradstats* parent, const sb_gradstats* child,
                     sb_gradstats* out, size_t total_bins) {
  using namespace sb;
  SB_REQUIRE(ctx && parent && child && out, SB_ERR_INVALID_ARG, "NULL argument");
  if (total_bins == 0) return SB_OK;
  SB_CUDA(cudaSetDevice(ctx->device));
  cudaStream_t st = ctx->stream;
  DBuf<double2> p, c, o;
  SB_TRY(p.alloc(ctx, total_bins));
  SB_TRY(c.alloc(ctx, total_bins));
  SB_TRY(o.alloc(ctx, total_bins));
  SB_CUDA(cudaMemcpyAsync(p.p, parent, p.bytes(), cudaMemcpyHostToDevice, st));
  SB_CUDA(cudaMemcpyAsync(c.p, child, c.bytes(), cudaMemcpyHostToDevice, st));
  unsigned blocks = (unsigned)std::min<size_t>((total_bins + 255) / 256, (size_t)ctx->num_sms * 8);
  SB_LAUNCH(ctx, k_subtract, blocks, 256, 0, p.p, c.p, o.p, total_bins);
  SB_CUDA(cudaMemcpyAsync(out, o.p, o.bytes(), cudaMemcpyDeviceToHost, st));
  SB_CUDA(cudaStreamSynchronize(st));
  return SB_OK;
}

}  // extern "C"
