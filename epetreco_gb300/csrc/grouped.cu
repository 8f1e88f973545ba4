// grouped.cu -- a reconstruction's system matrix as row groups with
// group-local column ids, and the one-pass MLEM iteration over it.
//
// The rows (in the reconstruction's crystal-pair order) are cut into groups
// of consecutive rows whose distinct columns fit a per-warp table in shared
// memory.  Consecutive rows in that order are a fan of lines through nearly
// one point, so a group touches few voxels, and two consecutive rows (a
// strip) touch few more than one of them.  A strip is stored as the merged list
// of its rows' columns: per entry the two rows' values (zero where a row
// does not touch the column) and a 2-byte rank of the column among the
// group's sorted distinct columns (the group's table), 10 bytes in FP32 and 6
// in the 16-bit forms for about 1.7 non-zeros, instead of a CSR plus a
// column-major copy (16 bytes per non-zero).
//
// One iteration reads every entry once (k_group_mlem): a warp takes a group,
// gathers x at the table into shared memory, and strip by strip forms A x from
// the shared copy, e = y / (A x) and adds the strip times e into the group's
// shared correction; a strip's columns are distinct, so the lanes never write
// the same word and each column's sum runs in row order.  The group's
// corrections go to one slot per (group, column); the slots of each column,
// listed in group order (built once: the column-major order of the table's
// entries), are summed in that order by the slot-sum kernel (k_sums), whose
// epilogue applies x*c/s.  Every sum has an input-determined order, so
// results are deterministic (where an entry lies in memory does not matter).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "internal.h"
#include "mlem_internal.h"
#include "spmv.cuh"

namespace epet {

constexpr int kGroupFirstRows = 32;  // rows of a first-cut group (split while too wide)
constexpr int kGroupThreads = 256;   // threads of the table-building kernels
// Shared tables are indexed by rank (the word of rank r sits in bank r % 32);
// a group's padding entries have the rank after its last column.
constexpr int kColsumWarps = 8;  // warps of the column-sum kernel
constexpr int kMaxStride = kGroupCap + 4;  // floats of the largest shared table
constexpr size_t kMaxPassSmem = 227 * 1024;
// Floats of each of a warp's two tables with `warps` warps in a block: fixed, so
// that a rank's place in the second is the first's plus a constant (with a
// run-time stride the full-size iteration took 79 ms instead of 73), and no
// larger than the matrices with that many warps need: what is left of the
// SM's memory caches the gathers of x (17.1 -> 16.0 ms for 16 small problems).
__host__ __device__ constexpr int pass_stride(int warps) {
  return warps == 20 ? 1088 : warps == 16 ? 1312 : kMaxStride;
}
constexpr size_t kColsumSmem = (size_t)kColsumWarps * kMaxStride * 4;
static_assert(kGroupFirstRows <= 64 && kGroupFirstRows % kStrip == 0, "row masks, strips");
constexpr int kGroupStrips = kGroupFirstRows / kStrip;  // strips of a first cut

// Row r of the source: its columns and values, and its length.
struct RowSpan {
  const int32_t* col;
  const float* val;
  int64_t n;
};
__device__ __forceinline__ RowSpan row_span(const RowSource& A, int64_t r) {
  if (A.segs) {
    const int64_t q = A.idx[r];
    const SegDev sg = A.segs[q / A.ch];
    const int64_t b = A.rp[q] - sg.e0;
    return RowSpan{sg.col + b, sg.val + b, A.rp[q + 1] - A.rp[q]};
  }
  const int64_t b = A.rp[r];
  return RowSpan{A.col + b, A.val + b, A.rp[r + 1] - b};
}

// The spans of rows r0 .. r1 - 1 (at most kGroupFirstRows) in shared memory;
// the loads run in parallel, a thread per row.  Ends with a block barrier.
struct GroupSpans {
  const int32_t* col[kGroupFirstRows];
  const float* val[kGroupFirstRows];
  int n[kGroupFirstRows];
};
__device__ __forceinline__ void load_spans(const RowSource& A, int r0, int r1, GroupSpans* S) {
  const int nr = r1 - r0;
  int n = 0;
  if ((int)threadIdx.x < nr) {
    const RowSpan rs = row_span(A, r0 + threadIdx.x);
    S->col[threadIdx.x] = rs.col;
    S->val[threadIdx.x] = rs.val;
    n = (int)rs.n;
  }
  if ((int)threadIdx.x < nr) S->n[threadIdx.x] = n;
  __syncthreads();
}

// A warp's walk along a row's columns, four consecutive ones per lane (16-byte
// loads): f(c, k) gets k of them, ascending.  Neighbouring columns fall into
// the same bitmap word, so a lane ORs its four together before it touches
// shared memory, and the lanes of a warp spread over a few words more: with a
// column per lane a dozen lanes hit one word at a time, and these atomics'
// replays held the table kernel at 71 % of the L1's throughput.
template <class F>
__device__ __forceinline__ void for_row4(const int32_t* __restrict__ col, int n, F&& f) {
  const int lane = threadIdx.x & 31;
  // entries before the first 16-byte boundary, whole 16-byte pieces, the rest
  const int head = min(n, (int)((0u - (unsigned)(reinterpret_cast<uintptr_t>(col) >> 2)) & 3u));
  const int nv = (n - head) >> 2, tail = n - head - 4 * nv;
  const int4* v = reinterpret_cast<const int4*>(col + head);
  if (lane < 2 && (lane ? tail : head) > 0) {
    const int32_t* p = lane ? col + n - tail : col;
    const int k = lane ? tail : head;
    const int c[4] = {p[0], k > 1 ? p[1] : 0, k > 2 ? p[2] : 0, 0};
    f(c, k);
  }
  for (int j = lane; j < nv; j += 64) {
    const bool two = j + 32 < nv;
    const int4 q = v[j];
    int4 r = q;
    if (two) r = v[j + 32];
    {
      const int c[4] = {q.x, q.y, q.z, q.w};
      f(c, 4);
    }
    if (two) {
      const int c[4] = {r.x, r.y, r.z, r.w};
      f(c, 4);
    }
  }
}

// ORs the bits of k ascending positions into a bitmap.
__device__ __forceinline__ void or_bits(const int* c, int k, unsigned* words) {
  int w = c[0] >> 5;
  unsigned m = 1u << (c[0] & 31);
#pragma unroll
  for (int t = 1; t < 4; t++) {
    if (t < k) {
      const int wt = c[t] >> 5;
      if (wt != w) {
        atomicOr(&words[w], m);
        w = wt;
        m = 0u;
      }
      m |= 1u << (c[t] & 31);
    }
  }
  atomicOr(&words[w], m);
}

// Sets the group's columns in the bitmap bm, a warp per row.
__device__ __forceinline__ void set_group_columns(const GroupSpans& S, int nr, unsigned* bm) {
  for (int r = threadIdx.x >> 5; r < nr; r += kGroupThreads / 32)
    for_row4(S.col[r], S.n[r], [&](const int* c, int k) { or_bits(c, k, bm); });
}

// Distinct columns of the candidate groups cand[g] = {r0, r1}: a bitmap over
// the columns in shared memory (nwords 32-bit words).
__global__ void __launch_bounds__(kGroupThreads)
k_group_distinct(RowSource A, const int2* __restrict__ cand, int nwords,
                 int32_t* __restrict__ nd) {
  extern __shared__ unsigned gbm[];
  __shared__ int wsum[kGroupThreads / 32];
  __shared__ GroupSpans S;
  for (int i = threadIdx.x; i < nwords; i += kGroupThreads) gbm[i] = 0u;
  const int2 c = cand[blockIdx.x];
  load_spans(A, c.x, c.y, &S);
  set_group_columns(S, c.y - c.x, gbm);
  __syncthreads();
  int n = 0;
  for (int i = threadIdx.x; i < nwords; i += kGroupThreads) n += __popc(gbm[i]);
  for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
  if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = n;
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0;
    for (int w = 0; w < kGroupThreads / 32; w++) t += wsum[w];
    nd[blockIdx.x] = t;
  }
}

// Words of a row's or strip's bitmap over the group's ranks.
constexpr int kRankWords = kGroupCap / 32;
static_assert(kGroupCap % 32 == 0, "rank bitmaps");

// A warp's strip while its entries are made: per row and for the strip the
// bitmap over the ranks and the exclusive prefix of its words.
struct StripBits {
  uint32_t row[kStrip][kRankWords];
  uint16_t rpre[kStrip][kRankWords], apre[kRankWords];
  __device__ uint32_t all(int w) const { return row[0][w] | row[1][w]; }
};
static_assert(kStrip == 2, "StripBits::all");
constexpr int kListEntries = 1024;  // ranks of a warp's strip, in order, that many at a time
static_assert(kListEntries % 128 == 0, "whole rounds of the pass");

// Sets a row's ranks in its bitmap.
__device__ __forceinline__ void set_row_ranks(const int32_t* __restrict__ col, int n,
                                              const unsigned* bm, const uint16_t* pre,
                                              uint32_t* words) {
  for_row4(col, n, [&](const int* c, int k) {
    int rk[4];
#pragma unroll
    for (int t = 0; t < 4; t++) {
      const unsigned v = (unsigned)c[t];
      rk[t] = t < k ? pre[v >> 5] + __popc(bm[v >> 5] & ((1u << (v & 31)) - 1u)) : 0;
    }
    or_bits(rk, k, words);
  });
}

// Exclusive prefixes of the popcounts of the rows' words and of their unions
// over the first `words` words, packed in one scan (each below 2^10 a round);
// returns the union's total.
__device__ __forceinline__ int rank_prefixes(StripBits& Q, int words) {
  const int lane = threadIdx.x & 31;
  int run = 0, run0 = 0, run1 = 0;
  for (int w0 = 0; w0 < words; w0 += 32) {
    const int w = w0 + lane;
    const bool ok = w < words;
    const uint32_t r0 = ok ? Q.row[0][w] : 0u, r1 = ok ? Q.row[1][w] : 0u;
    // (a round's totals are at most 1024 each: 10 + 1 bits)
    const int n0 = __popc(r0), n1 = __popc(r1), n = __popc(r0 | r1);
    const int inc01 = warp_incl_scan(n0 | (n1 << 16)), inc = warp_incl_scan(n);
    if (ok) {
      Q.rpre[0][w] = (uint16_t)(run0 + (inc01 & 0xffff) - n0);
      Q.rpre[1][w] = (uint16_t)(run1 + (inc01 >> 16) - n1);
      Q.apre[w] = (uint16_t)(run + inc - n);
    }
    const int t01 = __shfl_sync(0xffffffffu, inc01, 31);
    run0 += t01 & 0xffff;
    run1 += t01 >> 16;
    run += __shfl_sync(0xffffffffu, inc, 31);
  }
  return run;
}

// Strips are padded to whole 4-entry chunks.  Chunk 32 r + l is lane l's in
// round r of the pass, and an access takes one entry of every lane's chunk,
// so the entries are stored for it to take consecutive ones (ascending
// ranks): round r (cq = min(32, chunks left) chunks) holds entry 128 r + t cq
// + l at chunk l, position t.  FP32 values of a round: the first two entries
// of every chunk (16 bytes each), then the last two, so that each of a lane's
// two loads is part of one contiguous run (side by side, every 32-byte sector
// was fetched twice).  Padding: zero values on the group's spare rank.  A wide row's
// strip (n > kGroupCap) is a plain list.
__host__ __device__ constexpr int strip_pad(int n) { return (n + 3) & ~3; }

// Where the entries go: the arrays' capacity and the cursor (entries
// reserved so far: each block takes its strips' share with one atomic add, so
// the place of a group's entries in memory varies, their contents do not).
struct EntryOut {
  unsigned long long* cursor;
  int64_t cap;
  StripF* val;
  uint16_t* loc;
  StripDesc* strips;
};

// Tables and entries of groups (one block per group, a warp per strip): the
// group's distinct columns, ascending, at table[tb ..]; per strip its entries
// in column order.
//
// Three uses.  Counting (entries.val null): block b takes the first cut
// b * every and only adds its strips' entries to the cursor.  First cuts
// (nd_out set): block b takes the rows [R b, min(m, R b + R)), writes the
// cut's count of distinct columns to nd_out[b] and, for a cut that fits the
// shared tables, its table to ftab + b * kGroupCap and its entries, with the
// strip descriptors at [R / kStrip * b ..] (scratch, like ftab).  Final groups: a
// first cut kept whole copies its table and strip descriptors to their
// places; a group made by splitting a wider cut is laid out in full; a
// single row wider than the shared tables (a "wide" group) keeps its own
// columns as its table, its entries in that order (ranks unused).
__global__ void __launch_bounds__(kGroupThreads)
k_group_tables(RowSource A, const GroupDesc* __restrict__ groups, int64_t m, int nwords,
               int64_t every, int32_t* __restrict__ table, const int32_t* __restrict__ ftab,
               const StripDesc* __restrict__ fstrips, int32_t* __restrict__ nd_out, EntryOut out) {
  extern __shared__ __align__(16) unsigned gsh[];
  StripBits* sbits = reinterpret_cast<StripBits*>(gsh);
  unsigned* bm = gsh + sizeof(StripBits) * kGroupStrips / 4;
  // per bitmap word the rank of its first column (< kGroupCap where read)
  uint16_t* pre = reinterpret_cast<uint16_t*>(bm + nwords);
  __shared__ int wtot[kGroupThreads / 32], sn[kGroupStrips];
  __shared__ int s_nd;
  __shared__ unsigned long long s_base;
  const bool count = out.val == nullptr, first = count || nd_out != nullptr;
  GroupDesc gd;
  if (first) {
    const int64_t r0 = (int64_t)blockIdx.x * every * kGroupFirstRows;
    gd = GroupDesc{(int32_t)r0, (int32_t)min(m, r0 + kGroupFirstRows), 0, 0,
                   (int32_t)(blockIdx.x * kGroupStrips)};
  } else {
    gd = groups[blockIdx.x];
    if (gd.nd <= kGroupCap && gd.r0 % kGroupFirstRows == 0 &&
        gd.r1 == min(m, (int64_t)gd.r0 + kGroupFirstRows)) {
      // a first cut kept whole: laid out by the first launch
      const int64_t cut = gd.r0 / kGroupFirstRows;
      const int32_t* src = ftab + cut * kGroupCap;
      for (int j = threadIdx.x; j < gd.nd; j += kGroupThreads) table[gd.tb + j] = src[j];
      if ((int)threadIdx.x < (gd.r1 - gd.r0 + kStrip - 1) / kStrip)
        out.strips[gd.qb + threadIdx.x] = fstrips[cut * kGroupStrips + threadIdx.x];
      return;
    }
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (!first && gd.nd > kGroupCap) {  // wide: one row
    const RowSpan rs = row_span(A, gd.r0);
    const int np = strip_pad((int)rs.n);
    if (threadIdx.x == 0) s_base = atomicAdd(out.cursor, (unsigned long long)np);
    __syncthreads();
    const int64_t base = (int64_t)s_base;
    if (threadIdx.x == 0) out.strips[gd.qb] = StripDesc{base, (int32_t)rs.n, gd.r0};
    for (int64_t j = threadIdx.x; j < np; j += kGroupThreads) {
      if (j < rs.n) table[gd.tb + j] = rs.col[j];
      if (base + np <= out.cap) {
        StripF v = {};
        v.v[0] = j < rs.n ? rs.val[j] : 0.f;
        out.val[base + j] = v;
        out.loc[base + j] = 0;
      }
    }
    return;
  }
  __shared__ GroupSpans S;
  const int nr = gd.r1 - gd.r0;
  for (int i = threadIdx.x; i < nwords; i += kGroupThreads) bm[i] = 0u;
  load_spans(A, gd.r0, gd.r1, &S);
  set_group_columns(S, nr, bm);
  __syncthreads();
  // exclusive prefix of the words' popcounts: thread t owns a contiguous
  // range of words
  const int per = (nwords + kGroupThreads - 1) / kGroupThreads;
  const int wb = min(nwords, (int)threadIdx.x * per), we = min(nwords, wb + per);
  int cnt = 0;
  for (int w = wb; w < we; w++) cnt += __popc(bm[w]);
  const int inc = warp_incl_scan(cnt);
  if (lane == 31) wtot[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    const int t = lane < kGroupThreads / 32 ? wtot[lane] : 0;
    const int ti = warp_incl_scan(t);
    if (lane < kGroupThreads / 32) wtot[lane] = ti - t;
    if (lane == kGroupThreads / 32 - 1) s_nd = ti;
  }
  __syncthreads();
  const int nd = s_nd;  // (uniform across the block)
  if (first && !count && threadIdx.x == 0) nd_out[blockIdx.x] = nd;
  if (nd > kGroupCap) {
    // split by the host, laid out by the last launch; while counting, taken
    // as if each row had its own entries
    if (count) {
      for (int r = threadIdx.x; r < nr; r += kGroupThreads)
        atomicAdd(out.cursor, (unsigned long long)strip_pad(S.n[r]));
    }
    return;
  }
  // (the first launch's table is its cut's share of the scratch ftab)
  int32_t* const tab = first ? table + (int64_t)blockIdx.x * kGroupCap : table + gd.tb;
  int run = wtot[wid] + inc - cnt;
  for (int w = wb; w < we; w++) {
    pre[w] = (uint16_t)run;
    run += __popc(bm[w]);
  }
  const int words = (nd + 31) / 32;  // of the ranks
  for (int i = threadIdx.x; i < kGroupStrips * kStrip * kRankWords; i += kGroupThreads) {
    const int s = i / (kStrip * kRankWords);
    (&sbits[s].row[0][0])[i - s * kStrip * kRankWords] = 0u;
  }
  __syncthreads();
  if (!count) {
    // the table, 32 words at a time per warp: a lane per column of each word
    // that has any
    for (int w0 = 32 * wid; w0 < nwords; w0 += kGroupThreads) {
      const unsigned mine = w0 + lane < nwords ? bm[w0 + lane] : 0u;
      unsigned left = __ballot_sync(0xffffffffu, mine != 0u);
      while (left) {
        const int l = __ffs(left) - 1;
        left &= left - 1u;
        const unsigned word = __shfl_sync(0xffffffffu, mine, l);
        if ((word >> lane) & 1u)
          tab[pre[w0 + l] + __popc(word & ((1u << lane) - 1u))] = (w0 + l) * 32 + lane;
      }
    }
  }
  // the strips' rows as bitmaps over the ranks, and their unions, a warp per
  // strip
  const int ns = (nr + kStrip - 1) / kStrip;
  for (int s = wid; s < kGroupStrips; s += kGroupThreads / 32) {
    StripBits& Q = sbits[s];
    int n = 0;
    if (s < ns) {  // (uniform in the warp)
      for (int r = 0; r < kStrip && kStrip * s + r < nr; r++)
        set_row_ranks(S.col[kStrip * s + r], S.n[kStrip * s + r], bm, pre, Q.row[r]);
      __syncwarp();
      n = rank_prefixes(Q, words);
    }
    if (lane == 0) sn[s] = n;
  }
  __syncthreads();
  int total = 0;
  for (int s = 0; s < kGroupStrips; s++) total += strip_pad(sn[s]);
  if (threadIdx.x == 0) s_base = atomicAdd(out.cursor, (unsigned long long)total);
  if (count) return;
  __syncthreads();
  int64_t base = (int64_t)s_base;
  const bool fits = base + total <= out.cap;  // (else the host sees the cursor and starts again)
  const unsigned below = (1u << lane) - 1u;
  // (the columns' bitmap is not needed any more: the lists take its place)
  uint16_t* list = reinterpret_cast<uint16_t*>(bm) + wid * kListEntries;
  for (int s = 0; s < ns; base += strip_pad(sn[s]), s++) {
    if (s % (kGroupThreads / 32) != wid) continue;
    const int n = sn[s], np = strip_pad(n);
    if (lane == 0) out.strips[gd.qb + s] = StripDesc{base, n, gd.r0 + kStrip * s};
    if (!fits) continue;
    const StripBits& Q = sbits[s];
    const float* val[kStrip];
#pragma unroll
    for (int r = 0; r < kStrip; r++) val[r] = kStrip * s + r < nr ? S.val[kStrip * s + r] : nullptr;
    for (int e0 = 0; e0 < n; e0 += kListEntries) {
      for (int w = 0; w < words; w++) {
        const uint32_t all = Q.all(w);
        const unsigned i = Q.apre[w] + __popc(all & below) - e0;
        if (((all >> lane) & 1u) && i < (unsigned)kListEntries) list[i] = (uint16_t)(32 * w + lane);
      }
      __syncwarp();
      // a chunk per lane, in the storage order
      for (int c = e0 / 4 + lane; c < min(np, e0 + kListEntries) / 4; c += 32) {
        const int first_e = c & ~31, cq = min(32, np / 4 - first_e);  // chunks of this round
        StripF v[4];
        unsigned rk[4];
  #pragma unroll
        for (int t = 0; t < 4; t++) {
          const int i = 4 * first_e + t * cq + lane;
          rk[t] = i < n ? list[i - e0] : nd;
          const int w = min((int)rk[t] >> 5, kRankWords - 1), bit = rk[t] & 31;
          const uint32_t lower = (1u << bit) - 1u;
  #pragma unroll
          for (int r = 0; r < kStrip; r++) {
            const uint32_t mine = Q.row[r][w];
            const bool has = i < n && ((mine >> bit) & 1u);
            v[t].v[r] = has ? val[r][Q.rpre[r][w] + __popc(mine & lower)] : 0.f;
          }
        }
        float4* q = reinterpret_cast<float4*>(out.val + base + 4 * first_e) + lane;
        q[0] = make_float4(v[0].v[0], v[0].v[1], v[1].v[0], v[1].v[1]);
        q[cq] = make_float4(v[2].v[0], v[2].v[1], v[3].v[0], v[3].v[1]);
        *reinterpret_cast<uint2*>(out.loc + base + 4 * c) =
            make_uint2(rk[0] | (rk[1] << 16), rk[2] | (rk[3] << 16));
      }
      __syncwarp();
    }
  }
}

// First cuts counted to size the entries' arrays, and the non-zeros from which
// they are.
constexpr int64_t kSampleCuts = 2048, kSampleCutsFew = 512;
constexpr int64_t kSampleNnz = int64_t(1) << 24;

// Dynamic shared memory of k_group_tables: the strips' bitmaps, the group's
// bitmap and its word ranks, later a list of ranks per warp.
static size_t table_smem(int nwords) {
  return sizeof(StripBits) * kGroupStrips +
         std::max((size_t)nwords * 6, (size_t)(kGroupThreads / 32) * kListEntries * 2);
}

__global__ void k_fill_f32(float* __restrict__ p, int64_t n, float v) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = v;
}

epet_status grouped_ones(GroupedMatrix* G, cudaStream_t st) {
  if (G->ones) return EPET_OK;
  const int64_t ns = std::max<int64_t>(G->nslots, 1);
  EPET_CUDA(dev_alloc((void**)&G->ones, ns * 4, st));
  if (G->nslots > 0) {
    k_fill_f32<<<ceil_div(G->nslots, 256), 256, 0, st>>>(G->ones, G->nslots, 1.f);
    EPET_LAUNCHED();
  }
  return EPET_OK;
}

// 16-bit values: q = the 16-bit float of value / scale, scale = the row's
// largest value (the 16-bit forms' quantisation), a warp per row.
template <int FMT>
__device__ __forceinline__ uint16_t gq_to(float v) {
  if (FMT == 1) return __bfloat16_as_ushort(__float2bfloat16_rn(v));
  return __half_as_ushort(__float2half_rn(v));
}
template <int FMT>
__device__ __forceinline__ float gq_from(uint32_t q) {
  if (FMT == 1) return __uint_as_float(q << 16);
  return __half2float(__ushort_as_half((unsigned short)q));
}

// Whether a row touches an entry's column, from its value there: absent is +0
// (values are positive; those that a 16-bit form rounds to zero are kept as -0,
// which adds nothing either, but an infinite x or ratio must meet them).
__device__ __forceinline__ bool touches(float v) { return __float_as_uint(v) != 0u; }

// 16-bit values of a strip's rows and their scales, a warp per strip.
template <int FMT>
__global__ void k_group_quantise(const StripDesc* __restrict__ strips, int64_t nstrips,
                                 const StripF* __restrict__ val, int64_t m,
                                 float* __restrict__ scale, StripH* __restrict__ q) {
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (i >= nstrips) return;
  const StripDesc d = strips[i];
  // (strips are in row order: this one ends where the next begins)
  const int nr = (int)((i + 1 < nstrips ? strips[i + 1].r0 : m) - d.r0);
  const bool wide = d.n > kGroupCap;
  float mx[kStrip] = {};
  for (int64_t k = d.start + lane; k < d.start + strip_pad(d.n); k += 32) {
    // (pairs of values: the same two rows whatever the order of the entries)
    const StripF v = val[k];
#pragma unroll
    for (int j = 0; j < kStrip; j++) mx[j] = fmaxf(mx[j], fabsf(v.v[j]));
  }
  float sc[kStrip];
#pragma unroll
  for (int j = 0; j < kStrip; j++) {
    for (int o = 16; o > 0; o >>= 1) mx[j] = fmaxf(mx[j], __shfl_xor_sync(0xffffffffu, mx[j], o));
    sc[j] = mx[j] > 0.f ? mx[j] : 1.f;
    if (lane == 0 && j < nr) scale[d.r0 + j] = sc[j];
  }
  for (int k = lane; k < strip_pad(d.n); k += 32) {
    const StripF v = val[d.start + k];
    StripH b;
#pragma unroll
    for (int j = 0; j < kStrip; j++) {
      b.v[j] = gq_to<FMT>(__fdiv_rn(v.v[j], sc[j]));
      if (touches(v.v[j]) && b.v[j] == 0) b.v[j] = 0x8000;
    }
    // FP32 position k of round u: half h, chunk l, entry 2 h + e of it; the
    // 16-bit values of a chunk lie together
    int to = k;
    if (!wide) {
      const int u = k >> 7, cq = min(32, strip_pad(d.n) / 4 - 32 * u);
      const int i = k & 127, h = i >= 2 * cq ? 1 : 0, r = i - 2 * cq * h;
      to = 128 * u + 4 * (r >> 1) + 2 * h + (r & 1);
    }
    q[d.start + to] = b;
  }
}

// A strip's entries as the pass holds them: chunk 32 r + lane in slot r (up to
// 128 ROUNDS entries of a strip), four
// entries of two values (FP32: two float4, 16-bit: 8 x 16 bits) and their
// ranks (4 x 16 bits).
static_assert(kStrip == 2, "a chunk's loads");
struct Chunk32 {
  float4 a, b;
};
template <int FMT>
using ChunkV = typename std::conditional<FMT == 0, Chunk32, uint4>::type;
template <int FMT, int ROUNDS>
struct StripBuf {
  ChunkV<FMT> v[ROUNDS];
  uint2 l[ROUNDS];
};
// Row j's value of entry t.
template <int FMT>
__device__ __forceinline__ float cvalue(const ChunkV<FMT>& c, int t, int j) {
  if constexpr (FMT == 0) {
    const float4& q = t < 2 ? c.a : c.b;
    const int k = 2 * (t & 1) + j;
    return k == 0 ? q.x : k == 1 ? q.y : k == 2 ? q.z : q.w;
  } else {
    const uint32_t w = t == 0 ? c.x : t == 1 ? c.y : t == 2 ? c.z : c.w;
    return gq_from<FMT>(j ? w >> 16 : w & 0xffffu);
  }
}
__device__ __forceinline__ int crank(const uint2& c, int t) {
  const uint32_t w = t < 2 ? c.x : c.y;
  return (int)((t & 1) ? (w >> 16) : (w & 0xffffu));
}

struct GroupIterArgs {
  const GroupDesc* groups;
  int64_t ngroups;
  const StripDesc* strips;
  const void* val;     // StripF (FP32) or StripH (16-bit) per entry
  const float* scale;  // per row (16-bit forms)
  const uint16_t* loc;
  const int32_t* table;
  const float* x;
  const float* y;
  float* ybar;
  float* partial;
};

// The chunk of lane `lane` in round u of the strip of nq chunks at `start`.
template <int FMT>
__device__ __forceinline__ void gload(const void* val, const uint16_t* loc, int64_t start, int nq,
                                      int u, int lane, ChunkV<FMT>* v, uint2* l) {
  const int64_t k = start + 128 * u;
  if constexpr (FMT == 0) {
    const float4* p =
        reinterpret_cast<const float4*>(static_cast<const StripF*>(val) + k) + lane;
    v->a = __ldcs(p);
    v->b = __ldcs(p + min(32, nq - 32 * u));
  } else {
    *v = __ldcs(reinterpret_cast<const uint4*>(static_cast<const StripH*>(val) + k) + lane);
  }
  *l = __ldcs(reinterpret_cast<const uint2*>(loc + k) + lane);
}

// What a group's pass needs before its first strip: its counts and scales, a
// row per lane, and its strips, one per lane (a group has at most 32 rows),
// loaded one group ahead.
static_assert(kGroupFirstRows <= 32, "a row per lane");
struct GroupHead {
  GroupDesc gd;
  int64_t qs;
  int qn;
  float y, sc;
};

template <int FMT>
__device__ __forceinline__ GroupHead group_head(const GroupIterArgs& a, const GroupDesc& gd,
                                                int lane) {
  GroupHead h;
  h.gd = gd;
  const int nr = gd.r1 - gd.r0;
  h.qs = 0;
  h.qn = 0;
  if (lane < (nr + kStrip - 1) / kStrip) {
    const StripDesc q = a.strips[gd.qb + lane];
    h.qs = q.start;
    h.qn = q.n;
  }
  h.y = lane < nr ? a.y[gd.r0 + lane] : 0.f;
  h.sc = FMT != 0 && lane < nr ? a.scale[gd.r0 + lane] : 1.f;
  return h;
}

// One group of the MLEM pass (a warp): per row ybar = A x, e = y / ybar (0
// where ybar == 0, the fused epilogue's guard) and the strip's share of A^T e
// added, strip after strip, to the group's shared correction, written to
// partial[slot] at the end.
//
// Merging two rows per entry cuts what the pass issues per non-zero: one read
// of x and one read and write of the correction per entry (0.6 per non-zero),
// the ranks' decoding, and one warp sum, division and broadcast per two rows.
// The next strip's entries are in flight while a strip is reduced and added.
// Bound by the latency of those loads and of the chain from a strip's sums to
// its corrections.  One row at a time: 120 M instructions, 279 us for the
// first 400,000 channels of the full workload, 4.17 ms an iteration at full
// size (the slot sums included); in strips of two 87 M, 238 us, 3.59 ms.  Where
// few channels are measured rows share few columns and strips lose: the full
// geometry with 1 % of the channels 221 us an iteration for 199, with 10 % 691
// for 742.
// Tried: strips of four (more registers than a thread has), a ring in shared
// memory filled by asynchronous copies ahead of the pass (5.2 ms: a third of
// the tables' room and twice the instructions).
template <int FMT, int ROUNDS>
__device__ __forceinline__ void group_pass(const GroupIterArgs& a, const GroupHead& H, float* xs,
                                           float* cs, int lane) {
  const GroupDesc& gd = H.gd;
  const int nr = gd.r1 - gd.r0;
  const int ns = (nr + kStrip - 1) / kStrip;
  using V = ChunkV<FMT>;
  // (a batch's descriptors are read where they lie: held in registers, they
  // would push entries out)
  const void* const val = a.val;
  const uint16_t* const loc = a.loc;
  auto load_strip = [&](int k, StripBuf<FMT, ROUNDS>& B) {
    const int64_t start = __shfl_sync(0xffffffffu, H.qs, k);
    const int nq = (__shfl_sync(0xffffffffu, H.qn, k) + 3) >> 2;
#pragma unroll
    for (int u = 0; u < ROUNDS; u++)
      if (lane + 32 * u < nq) gload<FMT>(val, loc, start, nq, u, lane, &B.v[u], &B.l[u]);
  };
  StripBuf<FMT, ROUNDS> b0, b1;
  load_strip(0, b0);
  // x at the table: batches of 8 independent table loads, then their x
  // gathers.  An entry's zeros (a row that does not touch its column) must
  // not meet an infinite x or ratio: such groups or strips take the tested
  // form below.
  bool odd = false;
  for (int j0 = 0; j0 < gd.nd; j0 += 8 * 32) {
    int col[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const int j = j0 + 32 * k + lane;
      col[k] = j < gd.nd ? __ldg(a.table + gd.tb + j) : 0;
    }
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const int j = j0 + 32 * k + lane;
      const float xv = __ldg(a.x + col[k]);
      if (j < gd.nd) {
        xs[j] = xv;
        cs[j] = 0.f;
        odd = odd || !(fabsf(xv) <= 3.402823466e38f);
      }
    }
  }
  if (lane == 0) xs[gd.nd] = 0.f;  // (the padding's rank)
  odd = __any_sync(0xffffffffu, odd);
  __syncwarp();
  float yb_l = 0.f;
  auto process = [&](int k, const StripBuf<FMT, ROUNDS>& B) {
    const int n = __shfl_sync(0xffffffffu, H.qn, k);
    const int nq = (n + 3) >> 2;
    float s0[2] = {0.f, 0.f}, s1[2] = {0.f, 0.f};
    auto dot = [&](const V& v, const uint2& l) {
      float xv[4];
#pragma unroll
      for (int t = 0; t < 4; t++) xv[t] = xs[crank(l, t)];
#pragma unroll
      for (int t = 0; t < 4; t++) {
        s0[t & 1] = fmaf(cvalue<FMT>(v, t, 0), xv[t], s0[t & 1]);
        s1[t & 1] = fmaf(cvalue<FMT>(v, t, 1), xv[t], s1[t & 1]);
      }
    };
    if (!odd) {
#pragma unroll
      for (int u = 0; u < ROUNDS; u++)
        if (lane + 32 * u < nq) dot(B.v[u], B.l[u]);
      if (nq > 32 * ROUNDS) {
        const int64_t start = __shfl_sync(0xffffffffu, H.qs, k);
        for (int u = ROUNDS; 32 * u + lane < nq; u++) {
          V v;
          uint2 l;
          gload<FMT>(val, loc, start, nq, u, lane, &v, &l);
          dot(v, l);
        }
      }
    } else {
      const int64_t start = __shfl_sync(0xffffffffu, H.qs, k);
      for (int u = 0; 32 * u + lane < nq; u++) {
        V v;
        uint2 l;
        gload<FMT>(val, loc, start, nq, u, lane, &v, &l);
        for (int t = 0; t < 4; t++) {
          const float xv = xs[crank(l, t)];
          const float v0 = cvalue<FMT>(v, t, 0), v1 = cvalue<FMT>(v, t, 1);
          if (touches(v0)) s0[0] = fmaf(v0, xv, s0[0]);
          if (touches(v1)) s1[0] = fmaf(v1, xv, s1[0]);
        }
      }
    }
    // both rows' sums over the warp: lane l gets that of row l % 2
    const float a0 = fadd(s0[0], s0[1]), a1 = fadd(s1[0], s1[1]);
    const bool odd_lane = lane & 1;
    float d = fadd(odd_lane ? a1 : a0, __shfl_xor_sync(0xffffffffu, odd_lane ? a0 : a1, 1));
#pragma unroll
    for (int o = 2; o < 32; o <<= 1) d = fadd(d, __shfl_xor_sync(0xffffffffu, d, o));
    const int rl = kStrip * k + (lane & 1);
    const float sc = FMT == 0 ? 1.f : __shfl_sync(0xffffffffu, H.sc, rl);
    const float yb = FMT == 0 ? d : fmul(d, sc);
    // e = y / (A x) (mlemOperations.hpp:22-32; 0 where A x == 0)
    const float yr = __shfl_sync(0xffffffffu, H.y, rl);
    const float er = yb > 0.f ? __fdiv_rn(yr, yb) : 0.f;
    const float f = FMT == 0 ? er : fmul(er, sc);
    if (lane / kStrip == k) yb_l = yb;  // lane = row of the group
    const float f0 = __shfl_sync(0xffffffffu, f, 0), f1 = __shfl_sync(0xffffffffu, f, 1);
    // the strip's rows added, in row order, to the group's correction, a
    // chunk at a time: its four columns are distinct (as all of a strip's;
    // padding goes to the trash slot), so the four sums are read before any
    // is written
    auto add = [&](const V& v, const uint2& l) {
      float c[4];
#pragma unroll
      for (int t = 0; t < 4; t++) c[t] = cs[crank(l, t)];
#pragma unroll
      for (int t = 0; t < 4; t++)
        cs[crank(l, t)] = fmaf(cvalue<FMT>(v, t, 1), f1, fmaf(cvalue<FMT>(v, t, 0), f0, c[t]));
    };
    if (!odd && fabsf(f0) <= 3.402823466e38f && fabsf(f1) <= 3.402823466e38f) {
#pragma unroll
      for (int u = 0; u < ROUNDS; u++)
        if (lane + 32 * u < nq) add(B.v[u], B.l[u]);
      if (nq > 32 * ROUNDS) {
        const int64_t start = __shfl_sync(0xffffffffu, H.qs, k);
        for (int u = ROUNDS; 32 * u + lane < nq; u++) {
          V v;
          uint2 l;
          gload<FMT>(val, loc, start, nq, u, lane, &v, &l);
          add(v, l);
        }
      }
    } else {
      const int64_t start = __shfl_sync(0xffffffffu, H.qs, k);
      for (int u = 0; 32 * u + lane < nq; u++) {
        V v;
        uint2 l;
        gload<FMT>(val, loc, start, nq, u, lane, &v, &l);
        for (int t = 0; t < 4; t++) {
          const float v0 = cvalue<FMT>(v, t, 0), v1 = cvalue<FMT>(v, t, 1);
          float c = cs[crank(l, t)];
          if (touches(v0)) c = fmaf(v0, f0, c);
          if (touches(v1)) c = fmaf(v1, f1, c);
          cs[crank(l, t)] = c;
        }
      }
    }
    __syncwarp();
  };
  for (int k = 0; k < ns; k += 2) {
    if (k + 1 < ns) load_strip(k + 1, b1);
    process(k, b0);
    if (k + 1 < ns) {
      if (k + 2 < ns) load_strip(k + 2, b0);
      process(k + 1, b1);
    }
  }
  if (lane < nr) a.ybar[gd.r0 + lane] = yb_l;
  for (int j = lane; j < gd.nd; j += 32) a.partial[gd.tb + j] = cs[j];
  __syncwarp();
}

// Entry k of a wide row.
template <int FMT>
__device__ __forceinline__ float evalue(const GroupIterArgs& a, int64_t k) {
  if constexpr (FMT == 0) return static_cast<const StripF*>(a.val)[k].v[0];
  else return gq_from<FMT>(static_cast<const StripH*>(a.val)[k].v[0]);
}

// A wide group (one row, its own columns as its table, in the entries' order).
template <int FMT>
__device__ __forceinline__ void wide_pass(const GroupIterArgs& a, const GroupDesc& gd, int lane) {
  const StripDesc q = a.strips[gd.qb];
  float s = 0.f;
  for (int i = lane; i < q.n; i += 32)
    s = fmaf(evalue<FMT>(a, q.start + i), __ldg(a.x + a.table[gd.tb + i]), s);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s = fadd(s, __shfl_xor_sync(0xffffffffu, s, o));
  const float sc = FMT == 0 ? 1.f : a.scale[gd.r0];
  const float yb = FMT == 0 ? s : fmul(s, sc);
  const float er = yb > 0.f ? __fdiv_rn(a.y[gd.r0], yb) : 0.f;
  const float f = FMT == 0 ? er : fmul(er, sc);
  if (lane == 0) a.ybar[gd.r0] = yb;
  for (int i = lane; i < q.n; i += 32)
    a.partial[gd.tb + i] = fmul(evalue<FMT>(a, q.start + i), f);
}

// A warp per group, a persistent grid striding over the groups; each warp
// holds its group's tables (x and the correction at the distinct columns) in
// its share of the block's shared memory.  The next group's head is loaded one group ahead, descriptors two ahead.
template <int FMT, int ROUNDS, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 1)
k_group_mlem(GroupIterArgs a) {
  extern __shared__ __align__(16) float gsm[];
  constexpr int kStride = pass_stride(WARPS);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* xs = gsm + (size_t)w * 2 * kStride;
  float* cs = xs + kStride;
  const int64_t step = (int64_t)gridDim.x * WARPS;
  int64_t g = (int64_t)blockIdx.x * WARPS + w;
  if (g >= a.ngroups) return;
  GroupHead cur = group_head<FMT>(a, a.groups[g], lane);
  GroupDesc nxt = g + step < a.ngroups ? a.groups[g + step] : GroupDesc{0, 0, 0, 0, 0};
  for (; g < a.ngroups; g += step) {
    const GroupDesc nn =
        g + 2 * step < a.ngroups ? a.groups[g + 2 * step] : GroupDesc{0, 0, 0, 0, 0};
    GroupHead head_next{};
    if (g + step < a.ngroups) head_next = group_head<FMT>(a, nxt, lane);
    // (wide groups: k_group_mlem_wide)
    if (cur.gd.nd <= kGroupCap) group_pass<FMT, ROUNDS>(a, cur, xs, cs, lane);
    cur = head_next;
    nxt = nn;
  }
}

// The wide groups (ids in wide[0 .. nwide)), a warp each.
template <int FMT>
__global__ void __launch_bounds__(128)
k_group_mlem_wide(GroupIterArgs a, const int32_t* __restrict__ wide, int64_t nwide) {
  const int lane = threadIdx.x & 31;
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i >= nwide) return;
  wide_pass<FMT>(a, a.groups[wide[i]], lane);
}

// The same over the groups of many reconstructions (batched form): global
// group g belongs to problem p with gstart[p] <= g < gstart[p + 1].
template <int ROUNDS, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 1)
k_group_mlem_batch(const GroupIterArgs* __restrict__ desc, const int64_t* __restrict__ gstart,
                   int np) {
  extern __shared__ __align__(16) float gsm[];
  constexpr int kStride = pass_stride(WARPS);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* xs = gsm + (size_t)w * 2 * kStride;
  float* cs = xs + kStride;
  const int64_t total = gstart[np];  // (gstart[0]: the groups of the runs before)
  const int64_t step = (int64_t)gridDim.x * WARPS;
  auto locate = [&](int64_t g) {  // gstart[lo] <= g < gstart[lo + 1]
    int lo = 0, hi = np;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (__ldg(gstart + mid) <= g) lo = mid;
      else hi = mid;
    }
    return lo;
  };
  int64_t g = gstart[0] + (int64_t)blockIdx.x * WARPS + w;
  if (g >= total) return;
  // the next group's problem and head loaded one group ahead
  int p = locate(g);
  GroupHead cur = group_head<0>(desc[p], desc[p].groups[g - gstart[p]], lane);
  for (; g < total; g += step) {
    int pn = p;
    GroupHead hn{};
    if (g + step < total) {
      pn = locate(g + step);
      const GroupIterArgs& an = desc[pn];
      hn = group_head<0>(an, an.groups[g + step - gstart[pn]], lane);
    }
    // (wide groups: k_group_mlem_batch_wide)
    if (cur.gd.nd <= kGroupCap) group_pass<0, ROUNDS>(desc[p], cur, xs, cs, lane);
    p = pn;
    cur = hn;
  }
}

// The wide groups of a batch (global group ids wide[0 .. nwide)), a warp each.
__global__ void __launch_bounds__(128)
k_group_mlem_batch_wide(const GroupIterArgs* __restrict__ desc, const int64_t* __restrict__ gstart,
                        int np, const int32_t* __restrict__ wide, int64_t nwide) {
  const int lane = threadIdx.x & 31;
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i >= nwide) return;
  const int64_t g = wide[i];
  int lo = 0, hi = np;  // gstart[lo] <= g < gstart[lo + 1]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(gstart + mid) <= g) lo = mid;
    else hi = mid;
  }
  const GroupIterArgs a = desc[lo];
  wide_pass<0>(a, a.groups[g - gstart[lo]], lane);
}

// Column sums of the grouped matrix's values (the 16-bit forms dequantised)
// over its rows, by the same group / slot structure as the pass: a warp per
// group adds its strips' values, in row order, into the group's shared sums
// (the slots); the slot sums per column then run on the slot-sum kernel.
template <int FMT>
__global__ void __launch_bounds__(kColsumWarps * 32)
k_group_colsum(GroupIterArgs a) {
  extern __shared__ __align__(16) float gsm[];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* cs = gsm + (size_t)w * kMaxStride;
  for (int64_t g = (int64_t)blockIdx.x * kColsumWarps + w; g < a.ngroups;
       g += (int64_t)gridDim.x * kColsumWarps) {
    const GroupDesc gd = a.groups[g];
    const bool wide = gd.nd > kGroupCap;
    if (!wide) {
      for (int j = lane; j < gd.nd; j += 32) cs[j] = 0.f;
      __syncwarp();
    }
    for (int r = gd.r0, q = gd.qb; r < gd.r1; r += kStrip, q++) {
      const StripDesc d = a.strips[q];
      float sc[kStrip];
#pragma unroll
      for (int j = 0; j < kStrip; j++) sc[j] = FMT != 0 && r + j < gd.r1 ? a.scale[r + j] : 1.f;
      auto with = [&](float c, const float* v) {
#pragma unroll
        for (int j = 0; j < kStrip; j++) c = fadd(c, FMT == 0 ? v[j] : fmul(v[j], sc[j]));
        return c;
      };
      if (wide) {
        for (int i = lane; i < d.n; i += 32) {
          const float v[kStrip] = {evalue<FMT>(a, d.start + i), 0.f};
          a.partial[gd.tb + i] = with(0.f, v);
        }
      } else {
        const int nq = strip_pad(d.n) / 4;
        for (int u = 0; 32 * u + lane < nq; u++) {
          ChunkV<FMT> vv;
          uint2 l;
          gload<FMT>(a.val, a.loc, d.start, nq, u, lane, &vv, &l);
          for (int t = 0; t < 4; t++) {  // (padding: the trash slot)
            const float v[kStrip] = {cvalue<FMT>(vv, t, 0), cvalue<FMT>(vv, t, 1)};
            cs[crank(l, t)] = with(cs[crank(l, t)], v);
          }
        }
      }
      __syncwarp();
    }
    if (!wide) {
      for (int j = lane; j < gd.nd; j += 32) a.partial[gd.tb + j] = cs[j];
      __syncwarp();
    }
  }
}

// ---------------------------------------------------------------- host

static int bitmap_words(int64_t V) { return (int)((V + 31) / 32); }

// A bitmap over the columns and its prefix in a table block's shared memory.
constexpr int64_t kMaxColumns = 819200;

bool grouped_supported(int64_t V, int64_t m) {  // (int32 rows)
  return V > 0 && V <= kMaxColumns && m < INT32_MAX;
}

void grouped_free(GroupedMatrix* G, cudaStream_t st) {
  for (void* p : {(void*)G->groups, (void*)G->table, (void*)G->loc, (void*)G->wide,
                  (void*)G->cg_ptr,
                  (void*)G->cg_slot, (void*)G->ones, (void*)G->partial, (void*)G->val16,
                  (void*)G->val32, (void*)G->strips, (void*)G->scale})
    if (p) dev_free(p, st);
  *G = GroupedMatrix{};
}

void grouped_drop_fp32(GroupedMatrix* G, cudaStream_t st) {
  if (G->fmt != EPET_VALUES_FP32 && G->val32) {
    dev_free(G->val32, st);
    G->val32 = nullptr;
  }
}

// Groups of consecutive rows of A (row pointers on the device) whose
// distinct columns fit kGroupCap: first cuts of kGroupFirstRows rows, halved
// while too wide; a single row wider than that is a group of its own, its
// table the row's columns.  The first round measures the first cuts and lays
// out those that fit (k_group_tables' first launch: tables in ftab, strips in
// fstrips, entries in out); the halves are measured by k_group_distinct.
static epet_status form_groups(const RowSource& A, int64_t m, int64_t ncols, int32_t* ftab,
                               const EntryOut& entries, std::vector<GroupDesc>* out,
                               cudaStream_t st) {
  const int nwords = bitmap_words(ncols);
  const int64_t ncut = (m + kGroupFirstRows - 1) / kGroupFirstRows;
  EPET_CUDA(cudaFuncSetAttribute(k_group_distinct, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 bitmap_words(kMaxColumns) * 4));
  // every first cut counted, those that fit laid out
  std::vector<int32_t> cut_nd(ncut);
  {
    int32_t* nd = nullptr;
    cudaError_t e = dev_alloc((void**)&nd, std::max<int64_t>(ncut, 1) * 4, st);
    if (e == cudaSuccess && ncut > 0) {
      k_group_tables<<<(unsigned)ncut, kGroupThreads, table_smem(nwords), st>>>(
          A, nullptr, m, nwords, 1, ftab, nullptr, nullptr, nd, entries);
      note_launch();
      e = cudaGetLastError();
      if (e == cudaSuccess)
        e = cudaMemcpyAsync(cut_nd.data(), nd, ncut * 4, cudaMemcpyDeviceToHost, st);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (nd) dev_free(nd, st);
    if (e != cudaSuccess) return cuda_status(e, "row groups");
  }
  // The wider cuts, halved until their pieces fit or are one row; only
  // those pieces are counted again.  A split cut s keeps its pieces as bits
  // of mask[s] (a piece starting at row j of the cut) and their counts at
  // sub[kGroupFirstRows s + j].
  std::vector<int32_t> slot(ncut, -1);
  std::vector<uint64_t> mask;
  std::vector<int32_t> sub;
  std::vector<int2> pend, nextp;
  for (int64_t c = 0; c < ncut; c++) {
    const int32_t r0 = (int32_t)(c * kGroupFirstRows);
    const int32_t r1 = (int32_t)std::min<int64_t>(m, r0 + kGroupFirstRows);
    if (cut_nd[c] > kGroupCap && r1 - r0 > 1) {
      slot[c] = (int32_t)mask.size();
      mask.push_back(0);
      const int32_t mid = r0 + (r1 - r0) / 2;
      pend.push_back(make_int2(r0, mid));
      pend.push_back(make_int2(mid, r1));
    }
  }
  sub.assign(mask.size() * kGroupFirstRows, 0);
  std::vector<int32_t> hn;
  for (int round = 1; !pend.empty(); round++) {
    if (round > 40) return set_error(EPET_ERR_INVALID, "internal: row groups unmeasured");
    const size_t n = pend.size();
    hn.resize(n);
    int2* cand = nullptr;
    int32_t* nd = nullptr;
    cudaError_t e = dev_alloc((void**)&cand, n * sizeof(int2), st);
    if (e == cudaSuccess) e = dev_alloc((void**)&nd, n * 4, st);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(cand, pend.data(), n * sizeof(int2), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
      k_group_distinct<<<(unsigned)n, kGroupThreads, nwords * 4, st>>>(A, cand, nwords, nd);
      note_launch();
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(hn.data(), nd, n * 4, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (cand) dev_free(cand, st);
    if (nd) dev_free(nd, st);
    if (e != cudaSuccess) return cuda_status(e, "row groups");
    nextp.clear();
    for (size_t k = 0; k < n; k++) {
      const int2 p = pend[k];
      if (hn[k] > kGroupCap && p.y - p.x > 1) {
        const int32_t mid = p.x + (p.y - p.x) / 2;
        nextp.push_back(make_int2(p.x, mid));
        nextp.push_back(make_int2(mid, p.y));
      } else {
        const int32_t s = slot[p.x / kGroupFirstRows], j = p.x % kGroupFirstRows;
        mask[s] |= uint64_t(1) << j;
        sub[(size_t)s * kGroupFirstRows + j] = hn[k];
      }
    }
    pend.swap(nextp);
  }
  // the groups in row order: the cuts kept whole, and a split cut's pieces
  out->clear();
  out->reserve(ncut + sub.size() / 8);
  int64_t tb = 0, qb = 0;
  for (int64_t c = 0; c < ncut; c++) {
    const int32_t r0 = (int32_t)(c * kGroupFirstRows);
    const int32_t r1 = (int32_t)std::min<int64_t>(m, r0 + kGroupFirstRows);
    uint64_t msk = slot[c] < 0 ? 1u : mask[slot[c]];
    if (!(msk & 1u)) return set_error(EPET_ERR_INVALID, "internal: row groups unmeasured");
    while (msk) {
      const int j = __builtin_ctzll(msk);
      msk &= msk - 1u;
      const int32_t e = msk ? r0 + __builtin_ctzll(msk) : r1;
      const int32_t ndv = slot[c] < 0 ? cut_nd[c] : sub[(size_t)slot[c] * kGroupFirstRows + j];
      const int32_t nq = (e - (r0 + j) + kStrip - 1) / kStrip;
      if (tb + ndv > INT32_MAX || qb + nq > INT32_MAX)
        return set_error(EPET_ERR_UNSUPPORTED, "row-group tables exceed int32");
      out->push_back(GroupDesc{r0 + j, e, (int32_t)tb, ndv, (int32_t)qb});
      tb += ndv;
      qb += nq;
    }
  }
  return EPET_OK;
}

// Launch shape of the pass: chunks per lane in registers (two sets of 10
// registers each) and warps of a block (one per SM), by the mean entries of a
// strip and the widest group.  Long strips want them whole in registers (what
// is beyond is loaded twice, on the warp's path), short ones more warps.
// Measured: 52^3 voxels, 100 rays (510 entries a strip; 20 iterations of 5.1M
// rows): 5 chunks and 12 warps 73.2 ms, 4 and 12 80.4, 4 and 16 84.0, 6 and 12
// (spilling) 94; 24^3 and 32^3, 20 to 100 rays (16 problems, 10 iterations):
// 5 and 12 20.1 ms, 4 and 12 17.5, by this rule 16.5; 24^3, 20 rays (one
// iteration): 5 and 12 67 us, 2 and 20 55.
struct PassShape {
  int rounds, warps;
  size_t smem() const { return (size_t)warps * 2 * pass_stride(warps) * 4; }
};
static PassShape pass_shape(int64_t entries, int64_t strips, int max_nd) {
  const double mean = strips > 0 ? (double)entries / strips : 0.0;
  // (the tables hold the group's columns and the padding's rank)
  if (mean <= 220 && max_nd < pass_stride(20)) return PassShape{2, 20};
  if (mean <= 340 && max_nd < pass_stride(16)) return PassShape{3, 16};
  return PassShape{5, 12};
}
static_assert(pass_stride(12) > kGroupCap, "the largest groups");
static_assert(12 * 8 * (size_t)pass_stride(12) <= kMaxPassSmem, "shared tables");
static_assert(16 * 8 * (size_t)pass_stride(16) <= kMaxPassSmem, "shared tables");
static_assert(20 * 8 * (size_t)pass_stride(20) <= kMaxPassSmem, "shared tables");

// f(integral_constant<ROUNDS>, integral_constant<WARPS>) for the shape.
template <class F>
static void dispatch_shape(const PassShape& s, F&& f) {
  using std::integral_constant;
  if (s.rounds == 2) f(integral_constant<int, 2>{}, integral_constant<int, 20>{});
  else if (s.rounds == 3) f(integral_constant<int, 3>{}, integral_constant<int, 16>{});
  else f(integral_constant<int, 5>{}, integral_constant<int, 12>{});
}

// Shared memory of every instantiation (set when a layout is built: the
// launches may be captured in a graph).
static cudaError_t allow_pass_smem() {
  cudaError_t e = cudaSuccess;
  auto allow = [&](const void* k, size_t bytes) {
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  };
  for (int r : {2, 3, 5})
    dispatch_shape(PassShape{r, 0}, [&](auto R, auto W) {
      constexpr int rounds = decltype(R)::value, warps = decltype(W)::value;
      allow((const void*)k_group_mlem<0, rounds, warps>, kMaxPassSmem);
      allow((const void*)k_group_mlem<1, rounds, warps>, kMaxPassSmem);
      allow((const void*)k_group_mlem<2, rounds, warps>, kMaxPassSmem);
      allow((const void*)k_group_mlem_batch<rounds, warps>, kMaxPassSmem);
    });
  allow((const void*)k_group_colsum<0>, kColsumSmem);
  allow((const void*)k_group_colsum<1>, kColsumSmem);
  allow((const void*)k_group_colsum<2>, kColsumSmem);
  return e;
}

epet_status grouped_build(const RowSource& A, int64_t m, int64_t ncols, int64_t nnz,
                          int value_format, GroupedMatrix* G, cudaStream_t st) {
  *G = GroupedMatrix{};
  G->fmt = value_format;
  G->n = ncols;
  if (!grouped_supported(ncols, m))
    return set_error(EPET_ERR_UNSUPPORTED, "grouped layout: %lld columns", (long long)ncols);
  int32_t* ftab = nullptr;              // first cuts' tables (scratch)
  StripDesc* fstrips = nullptr;         // first cuts' strips (scratch)
  unsigned long long* cursor = nullptr; // entries reserved
  auto drop_scratch = [&]() {
    for (void* p : {(void*)ftab, (void*)fstrips, (void*)cursor})
      if (p) dev_free(p, st);
    ftab = nullptr;
    fstrips = nullptr;
    cursor = nullptr;
  };
  auto fail = [&](epet_status rc) {
    drop_scratch();
    grouped_free(G, st);
    return rc;
  };
#define GALLOC(ptr, bytes)                                                        \
  do {                                                                            \
    cudaError_t e_ = dev_alloc((void**)&(ptr), std::max<size_t>((bytes), 16), st); \
    if (e_ != cudaSuccess) return fail(cuda_status(e_, "grouped allocation " #ptr)); \
  } while (0)
  const int nwords = bitmap_words(ncols);
  // (limits for any grid: another thread may be between its own and its launch)
  cudaError_t e = cudaFuncSetAttribute(k_group_tables, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)table_smem(bitmap_words(kMaxColumns)));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_group_tables, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  if (e == cudaSuccess) e = allow_pass_smem();
  if (e != cudaSuccess) return fail(cuda_status(e, "grouped kernels"));
  const int64_t ncut = ceil_div(std::max<int64_t>(m, 1), (int64_t)kGroupFirstRows);
  GALLOC(cursor, 8);
  GALLOC(ftab, ncut * kGroupCap * 4);
  GALLOC(fstrips, ncut * kGroupStrips * sizeof(StripDesc));
  auto read_cursor = [&](int64_t* n) -> epet_status {
    unsigned long long v = 0;
    EPET_CUDA(cudaMemcpyAsync(&v, cursor, 8, cudaMemcpyDeviceToHost, st));
    EPET_CUDA(cudaStreamSynchronize(st));
    *n = (int64_t)v;
    return EPET_OK;
  };
  // The entries' arrays: how far the rows of a strip share columns is only
  // known once they are merged (0.6 entries per non-zero in scans).  A sample of
  // the first cuts sizes them, one wave of blocks for up to 2^26 non-zeros, where
  // it weighs; should the entries not fit after all, the layout is made again at
  // the size it asked for.  Up to 2^24 non-zeros the arrays are sized as if no
  // columns were shared (0.17 GB at most), and the entries move into smaller ones
  // afterwards.  16 problems of 24^3 and 32^3 hold 7.6 bytes per non-zero (11.6
  // in arrays for unshared columns).  Whole reconstructions of 36M, 49M (two
  // iterations) and 55M non-zeros, in ms, with the sample 3.70, 4.82, 6.00, moved
  // 3.74, 4.79, 6.01 to 6.08, in arrays for unshared columns 3.71, 4.76, 5.95.
  int64_t cap = nnz + 3 * std::max<int64_t>(m, 1);
  if (m > 0 && nnz > kSampleNnz) {
    const bool few = nnz <= (int64_t(1) << 26);
    const int64_t every = std::max<int64_t>(1, ncut / (few ? kSampleCutsFew : kSampleCuts));
    const int64_t sampled = (ncut + every - 1) / every;
    e = cudaMemsetAsync(cursor, 0, 8, st);
    if (e == cudaSuccess) {
      k_group_tables<<<(unsigned)sampled, kGroupThreads, table_smem(nwords), st>>>(
          A, nullptr, m, nwords, every, nullptr, nullptr, nullptr, nullptr,
          EntryOut{cursor, 0, nullptr, nullptr, nullptr});
      note_launch();
      e = cudaGetLastError();
    }
    int64_t n = 0;
    const epet_status rc = e == cudaSuccess ? read_cursor(&n) : cuda_status(e, "group sample");
    if (rc != EPET_OK) return fail(rc);
    cap = (int64_t)((double)n / sampled * ncut * (few ? 1.08 : 1.03)) + 65536;
  }
  std::vector<GroupDesc> hg;
  for (int attempt = 0;; attempt++) {
    GALLOC(G->val32, cap * sizeof(StripF));
    GALLOC(G->loc, cap * 2);
    e = cudaMemsetAsync(cursor, 0, 8, st);
    if (e != cudaSuccess) return fail(cuda_status(e, "group entries"));
    // the groups; the first cuts that fit are laid out on the way
    epet_status rc = form_groups(A, m, ncols, ftab, EntryOut{cursor, cap, G->val32, G->loc, fstrips},
                                 &hg, st);
    if (rc != EPET_OK) return fail(rc);
    G->ngroups = (int64_t)hg.size();
    G->nslots = hg.empty() ? 0 : (int64_t)hg.back().tb + hg.back().nd;
    G->nstrips =
        hg.empty() ? 0 : (int64_t)hg.back().qb + (hg.back().r1 - hg.back().r0 + kStrip - 1) / kStrip;
    if (attempt == 0) {  // (the groups do not depend on the entries' place)
      GALLOC(G->groups, hg.size() * sizeof(GroupDesc));
      GALLOC(G->strips, std::max<int64_t>(G->nstrips, 1) * sizeof(StripDesc));
      GALLOC(G->table, std::max<int64_t>(G->nslots, 1) * 4);
    }
    // the tables and strips at their places and the layout of the groups
    // split from wider cuts
    if (!hg.empty()) {
      e = cudaMemcpyAsync(G->groups, hg.data(), hg.size() * sizeof(GroupDesc),
                          cudaMemcpyHostToDevice, st);
      if (e == cudaSuccess) {
        k_group_tables<<<(unsigned)hg.size(), kGroupThreads, table_smem(nwords), st>>>(
            A, G->groups, m, nwords, 1, G->table, ftab, fstrips, nullptr,
            EntryOut{cursor, cap, G->val32, G->loc, G->strips});
        note_launch();
        e = cudaGetLastError();
      }
      if (e != cudaSuccess) return fail(cuda_status(e, "group tables"));
    }
    rc = read_cursor(&G->nent);
    if (rc != EPET_OK) return fail(rc);
    if (G->nent <= cap) break;
    if (attempt > 0) return fail(set_error(EPET_ERR_INVALID, "internal: group entries"));
    dev_free(G->val32, st);
    dev_free(G->loc, st);
    G->val32 = nullptr;
    G->loc = nullptr;
    cap = G->nent;
  }
  drop_scratch();
  // (arrays that are too large are kept where there is no memory for the move)
  auto fit = [&](auto*& a) -> cudaError_t {
    auto* was = a;
    void* p = nullptr;
    if (dev_alloc(&p, std::max<size_t>(G->nent * sizeof(*a), 16), st) != cudaSuccess) {
      cudaGetLastError();
      return cudaSuccess;
    }
    a = static_cast<decltype(was)>(p);
    const cudaError_t c =
        cudaMemcpyAsync(a, was, G->nent * sizeof(*a), cudaMemcpyDeviceToDevice, st);
    dev_free(was, st);
    return c;
  };
  if (G->nent < cap - cap / 8) {
    e = fit(G->val32);
    if (e == cudaSuccess) e = fit(G->loc);
    if (e != cudaSuccess) return fail(cuda_status(e, "group entries"));
  }
  for (const GroupDesc& g : hg)
    if (g.nd <= kGroupCap) G->max_nd = std::max(G->max_nd, g.nd);
  const int64_t ns = std::max<int64_t>(G->nslots, 1);
  GALLOC(G->partial, ns * 4);
  GALLOC(G->cg_ptr, (ncols + 1) * 8);
  {
    std::vector<int32_t> wide;
    for (size_t i = 0; i < hg.size(); i++)
      if (hg[i].nd > kGroupCap) wide.push_back((int32_t)i);
    G->nwide = (int64_t)wide.size();
    G->wide_h = wide;
    if (!wide.empty()) {
      GALLOC(G->wide, wide.size() * 4);
      e = cudaMemcpyAsync(G->wide, wide.data(), wide.size() * 4, cudaMemcpyHostToDevice, st);
      if (e == cudaSuccess) e = cudaStreamSynchronize(st);  // (the host vector goes)
      if (e != cudaSuccess) return fail(cuda_status(e, "wide groups"));
    }
  }
  // the slots of each column in group order: the column-major order of the
  // (group x column) table's entries, i.e. their positions
  GALLOC(G->cg_slot, ns * 4);
  {
    const epet_status rc = csr_to_csc_positions(G->nslots, ncols, G->table, G->cg_ptr,
                                                reinterpret_cast<uint32_t*>(G->cg_slot), st);
    if (rc != EPET_OK) return fail(rc);
  }
  if (value_format != EPET_VALUES_FP32) {
    GALLOC(G->val16, std::max<int64_t>(G->nent, 1) * sizeof(StripH));
    GALLOC(G->scale, std::max<int64_t>(m, 1) * 4);
    if (m > 0) {
      const unsigned nb = (unsigned)ceil_div(G->nstrips * 32, 256);
      if (value_format == EPET_VALUES_BF16)
        k_group_quantise<1><<<nb, 256, 0, st>>>(G->strips, G->nstrips, G->val32, m, G->scale,
                                                G->val16);
      else
        k_group_quantise<2><<<nb, 256, 0, st>>>(G->strips, G->nstrips, G->val32, m, G->scale,
                                                G->val16);
      note_launch();
      if (cudaGetLastError() != cudaSuccess) return fail(set_error(EPET_ERR_CUDA, "quantise"));
    }
  }
#undef GALLOC
  G->plan_cols = default_plan(ncols ? (double)G->nslots / ncols : 0.0);
  return EPET_OK;
}

static GroupIterArgs iter_args(const GroupedMatrix& G, const float* x, const float* y,
                               float* ybar) {
  return GroupIterArgs{G.groups, G.ngroups, G.strips,
                       G.fmt == EPET_VALUES_FP32 ? (const void*)G.val32 : (const void*)G.val16,
                       G.scale, G.loc, G.table, x, y, ybar, G.partial};
}

size_t grouped_batch_desc_bytes() { return sizeof(GroupIterArgs); }

void grouped_batch_desc(const GroupedMatrix& G, const float* x, const float* y, float* ybar,
                        void* out) {
  *static_cast<GroupIterArgs*>(out) = iter_args(G, x, y, ybar);
}

static unsigned pass_grid(int64_t ngroups, int warps) {
  return (unsigned)std::max<int64_t>(
      1, std::min<int64_t>((ngroups + warps - 1) / warps, (int64_t)num_sms()));
}

// The launches of a batch's pass: the problems of one launch shape together,
// a problem with kAloneWaves groups or more for every warp of the device in a
// launch of its own (it fills the device by itself, and its descriptor is then
// a kernel parameter: in memory, its loads stand before every strip's).
// Measured, 10 iterations: 64 problems of 24^3 to 64^3 and up to 5.1M rows, one
// launch for all in the shape of the widest 691 ms, a launch a shape 654, alone
// from 1, 4, 16 waves 578, 577, 579; 64 of 24^3 and 32^3, 8 angles: 66.9, 50.7,
// and 56.8, 50.7, 50.7.
constexpr int kAloneWaves = 4;

std::vector<int> grouped_batch_order(const std::vector<const GroupedMatrix*>& G,
                                     std::vector<BatchRun>* runs) {
  runs->clear();
  std::vector<int> order;
  auto shape = [&](int i) { return pass_shape(G[i]->nent, G[i]->nstrips, G[i]->max_nd); };
  auto alone = [&](int i) {
    return G[i]->ngroups >= (int64_t)kAloneWaves * shape(i).warps * num_sms();
  };
  for (int rounds : {5, 3, 2}) {
    BatchRun run{(int)order.size(), 0, 0, nullptr};
    for (int i = 0; i < (int)G.size(); i++) {
      if (G[i]->ngroups == 0 || alone(i) || shape(i).rounds != rounds) continue;
      order.push_back(i);
      run.np++;
      run.groups += G[i]->ngroups;
      run.rep = G[i];
    }
    if (run.np > 0) runs->push_back(run);
  }
  for (int i = 0; i < (int)G.size(); i++) {
    if (G[i]->ngroups > 0 && !alone(i)) continue;  // (without groups: last, in no run)
    if (G[i]->ngroups > 0) runs->push_back(BatchRun{(int)order.size(), 1, G[i]->ngroups, G[i]});
    order.push_back(i);
  }
  return order;
}

epet_status grouped_pass_batch(const void* desc, const void* desc_h, const int64_t* gstart, int np,
                               const std::vector<BatchRun>& runs, const int32_t* wide,
                               int64_t nwide, cudaStream_t st) {
  for (const BatchRun& run : runs) {
    const PassShape s = pass_shape(run.rep->nent, run.rep->nstrips, run.rep->max_nd);
    const unsigned grid = pass_grid(run.groups, s.warps), T = s.warps * 32;
    dispatch_shape(s, [&](auto R, auto W) {
      constexpr int rounds = decltype(R)::value, warps = decltype(W)::value;
      if (run.np == 1)
        k_group_mlem<0, rounds, warps><<<grid, T, s.smem(), st>>>(
            static_cast<const GroupIterArgs*>(desc_h)[run.p0]);
      else
        k_group_mlem_batch<rounds, warps><<<grid, T, s.smem(), st>>>(
            static_cast<const GroupIterArgs*>(desc) + run.p0, gstart + run.p0, run.np);
    });
    EPET_LAUNCHED();
  }
  if (nwide > 0) {
    k_group_mlem_batch_wide<<<(unsigned)ceil_div(nwide * 32, (int64_t)128), 128, 0, st>>>(
        static_cast<const GroupIterArgs*>(desc), gstart, np, wide, nwide);
    EPET_LAUNCHED();
  }
  return EPET_OK;
}

epet_status grouped_column_sums(const GroupedMatrix& G, bool quantised, float* out,
                                cudaStream_t st) {
  if (G.ngroups > 0) {
    GroupIterArgs a = iter_args(G, nullptr, nullptr, nullptr);
    int fmt = G.fmt;
    if (!quantised) {
      if (!G.val32) return set_error(EPET_ERR_INVALID, "internal: FP32 values released");
      a.val = G.val32;
      fmt = EPET_VALUES_FP32;
    }
    const unsigned grid = 3 * pass_grid(G.ngroups, kColsumWarps), T = kColsumWarps * 32;
    switch (fmt) {
      case EPET_VALUES_BF16: k_group_colsum<1><<<grid, T, kColsumSmem, st>>>(a); break;
      case EPET_VALUES_FP16: k_group_colsum<2><<<grid, T, kColsumSmem, st>>>(a); break;
      default: k_group_colsum<0><<<grid, T, kColsumSmem, st>>>(a);
    }
    EPET_LAUNCHED();
  }
  return launch_sums(G.plan_cols, G.cg_ptr, G.cg_slot, G.partial, G.n, EpiKeep{out},
                     nullptr, st);
}

int grouped_pass_kernels(const GroupedMatrix& G) {
  return G.ngroups == 0 ? 0 : (G.nwide > 0 ? 2 : 1);
}

epet_status grouped_pass(const GroupedMatrix& G, const float* x, const float* y, float* ybar,
                         cudaStream_t st) {
  if (G.ngroups == 0) return EPET_OK;
  const GroupIterArgs a = iter_args(G, x, y, ybar);
  const PassShape s = pass_shape(G.nent, G.nstrips, G.max_nd);
  const unsigned grid = pass_grid(G.ngroups, s.warps), T = s.warps * 32;
  dispatch_shape(s, [&](auto R, auto W) {
    constexpr int rounds = decltype(R)::value, warps = decltype(W)::value;
    switch (G.fmt) {
      case EPET_VALUES_BF16:
        k_group_mlem<1, rounds, warps><<<grid, T, s.smem(), st>>>(a);
        break;
      case EPET_VALUES_FP16:
        k_group_mlem<2, rounds, warps><<<grid, T, s.smem(), st>>>(a);
        break;
      default: k_group_mlem<0, rounds, warps><<<grid, T, s.smem(), st>>>(a);
    }
  });
  EPET_LAUNCHED();
  if (G.nwide > 0) {
    const unsigned wgrid = (unsigned)ceil_div(G.nwide * 32, (int64_t)128);
    switch (G.fmt) {
      case EPET_VALUES_BF16: k_group_mlem_wide<1><<<wgrid, 128, 0, st>>>(a, G.wide, G.nwide); break;
      case EPET_VALUES_FP16: k_group_mlem_wide<2><<<wgrid, 128, 0, st>>>(a, G.wide, G.nwide); break;
      default: k_group_mlem_wide<0><<<wgrid, 128, 0, st>>>(a, G.wide, G.nwide);
    }
    EPET_LAUNCHED();
  }
  return EPET_OK;
}

}  // namespace epet
