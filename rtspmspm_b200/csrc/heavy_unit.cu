// Heavy-row numeric pass: one CTA per unit, a run of 2^kTileShift-column
// tiles of one output row, with accumulators for exactly the unit's output
// entries.
//
// The unit's columns are a bitmap in shared memory with the number of output
// entries before each of its 32-bit words, so a product's accumulator is that
// number + popc(word & the lower columns).  Compact accumulators let a unit span
// as many tiles as its entries fit (R-MAT rows fill a few percent of their
// columns), so a row of A is walked once per some ten thousand output entries
// instead of once per 2,048 columns and its B-row segments stay long.
//
// Bound: barriers (6.4 stalls an issue) and issue slots (50 % at IPC 2), not
// memory (8 % of the copy peak): R-MAT rows meet 15 M segments at scale 17,
// two thirds of them under 32 products.  Against one warp per (row, 2,048
// columns), which rescanned its row of A 64 to 128 times and took segments of
// a few products: R-MAT 16 7.0 -> 3.6 ms, R-MAT 18 35.4 -> 22.7 ms.
// Measured and dropped (R-MAT 17, 7.0 ms as kept): units of 6,800 / 9,000
// words 7.6 / 8.7 ms (fewer CTAs an SM), 256 threads 9.3, 64 threads 8.0, one
// warp per unit about 1.9 times the CTA (R-MAT 16), every run of short segments
// added by one warp 8.0 (kPackSegment), no barrier between two segments of at most
// 32 products 1.02 to 1.03 times, mbarriers in place of the CTA barrier 7.7 (more
// instructions than the waits they take away).
//
// Reference counterpart: the any-hit multiply-accumulate into a dense row
// (optixSpMSpM/src/optixSpMSpM/optixSpMSpM.cu:234-260).
#include <algorithm>

#include "common.cuh"
#include "kernels.hpp"

namespace spg {

// Shared words of one tile: its bitmap and a count per bitmap word, side by
// side so that one load brings both.
constexpr int kTileCost = 2 * kTileWords;
constexpr int kUnitWarps = kUnitThreads / 32;
// A unit that marks its columns itself leaves segments of at most this many
// products to one lane each (6,479 rows of which 900 have 3,000 segments, most of
// 2 or 3 products in a unit, call 6.75 -> 6.48 ms).
constexpr int kLaneSegment = 16;
// Where three of four segments of the walk's 128 hold at most this many products,
// runs of them are added by one warp, 32 products a step: a step of the whole CTA
// for 2 or 3 products costs its four warps 160 instructions (the product above
// 5.36 -> 2.86 ms, its new values, with columns from C, 5.14 -> 2.78).
constexpr int kPackSegment = 8;
// Rows of A of more entries than this are cut first and taken first: their
// units run longest.
constexpr int64_t kLongRow = 1024;

static_assert(kTileCost + kTileCols <= kUnitCost, "a full tile fits a unit");
static_assert(kUnitCost < 65536, "a unit's entries are a 16-bit field");

// Cuts every heavy row into units, greedily from its first tile with output
// entries: a unit takes tiles while their bitmaps, counts and entries fit
// kUnitCost words.  One warp per row, 32 tiles at a time (a scan of their
// entries and a ballot find the first tile that no longer fits): a sweep to
// count the units, one atomic for their place in the list, a sweep to write
// them.  Units of long rows of A fill the list from its front, the others from
// its back; *nunits counts them in its low and its high half.  Unit: {row, first
// tile, (tiles << 16) | entries, entries of the row before it}.  A tile holds at
// most kTileCols entries and so fits a unit of its own.  The list has room for
// every unit of rows that hold the entries they were said to; row pointers of
// C that say otherwise raise a flag.
__global__ void k_cut_units(const int32_t* heavy_rows, int64_t nheavy, const int32_t* big_slot, const int32_t* tile_cnt,
                            int ntiles, const int64_t* a_rp, int4* units, int64_t room, unsigned long long* nunits,
                            int* flags) {
  const int lane = lane_id();
  const int64_t gw = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t h = gw; h < nheavy; h += nw) {
    const int32_t row = heavy_rows[h];
    const int32_t* cnt = tile_cnt + (int64_t)big_slot[row] * ntiles;
    int4* out = nullptr;
    for (int sweep = 0; sweep < 2; ++sweep) {
      // the open unit: tiles from `start`, its first entry the `first`-th of the row
      int made = 0, start = 0, end = 0, first = 0, done = 0;
      for (int t0 = 0; t0 < ntiles; t0 += 32) {
        const int t = t0 + lane;
        const int v = t < ntiles ? cnt[t] : 0;
        const int incl = done + warp_incl_scan(v);  // entries of the row through tile t
        const unsigned filled = __ballot_sync(kFull, v > 0);
        for (unsigned todo = filled; todo;) {
          const int next = __ffs(todo) - 1;
          const int before = __shfl_sync(kFull, incl - v, next);
          if (first == before) start = t0 + next;  // the unit opens here
          const unsigned over =
              __ballot_sync(kFull, v > 0 && lane >= next && (t - start + 1) * kTileCost + incl - first > kUnitCost);
          if (!over) break;
          const int stop = __ffs(over) - 1;
          const int upto = __shfl_sync(kFull, incl - v, stop);
          const unsigned inside = filled & ((1u << stop) - 1u);
          if (inside) end = t0 + 32 - __clz(inside);
          if (out && lane == 0) out[made] = make_int4(row, start, ((end - start) << 16) | (upto - first), first);
          ++made;
          first = upto;
          todo &= ~0u << stop;
        }
        done = __shfl_sync(kFull, incl, 31);
        if (filled) end = t0 + 32 - __clz(filled);
      }
      if (done > first) {
        if (out && lane == 0) out[made] = make_int4(row, start, ((end - start) << 16) | (done - first), first);
        ++made;
      }
      if (sweep == 0) {
        const bool back = a_rp[row + 1] - a_rp[row] <= kLongRow;
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(nunits, (unsigned long long)made << (back ? 32 : 0));
        base = __shfl_sync(kFull, base, 0);
        const int64_t front = (int64_t)(base & 0xffffffffu), behind = (int64_t)(base >> 32);
        if (front + behind + made > room) {  // the units' kernel sees the count and takes none
          if (lane == 0) raise_flag(flags, kFlagCountDiff);
          break;
        }
        out = back ? units + (room - behind - made) : units + front;
      }
    }
  }
}

// First position in [bs, be) whose column is >= c.
template <typename Off>
__device__ __forceinline__ Off first_at_least(const int32_t* col, Off bs, Off be, int64_t c) {
  while (bs < be) {
    const Off m = bs + (be - bs) / 2;
    if (col[m] < c) bs = m + 1;
    else be = m;
  }
  return bs;
}

// The part of B row A.col[p] inside tiles [t0, t1), and A.val[p].
template <bool R32>
__device__ __forceinline__ void unit_segment(const DCsr& A, const DCsr& B, int64_t p, int64_t e, int t0, int t1,
                                             int ntiles, const int32_t* bidx, typename RowOff<R32>::T& bs, int& len,
                                             float& a) {
  using Off = typename RowOff<R32>::T;
  bs = 0;
  len = 0;
  a = 0.f;
  if (p >= e) return;
  const int32_t k = A.col[p];
  a = A.val[p];
  Off rs = RowOff<R32>::at(B, k), re;
  if (bidx) {
    const int32_t* bi = bidx + (int64_t)k * (ntiles + 1);
    re = rs + (Off)bi[t1];
    rs += (Off)bi[t0];
  } else {
    re = RowOff<R32>::at(B, k + 1);
    if (t0 > 0) rs = first_at_least<Off>(B.col, rs, re, (int64_t)t0 << kTileShift);
    if (t1 < ntiles) re = first_at_least<Off>(B.col, rs, re, (int64_t)t1 << kTileShift);
  }
  bs = rs;
  len = (int)(re - rs);
}

// A segment of the CTA's list: the part of a B row inside the unit and A's
// value.
template <typename Off>
__device__ __forceinline__ int4 pack_segment(Off bs, int len, float a) {
  const int64_t b = (int64_t)bs;
  return make_int4((int)(uint32_t)b, (int)(b >> 32), len, __float_as_int(a));
}
template <typename Off>
__device__ __forceinline__ Off segment_start(const int4& s) {
  return (Off)(((int64_t)s.y << 32) | (uint32_t)s.x);
}

// What the CTA walks at a time: the non-empty segments of kUnitThreads
// entries of A's row, in order, and empty ones behind them.
struct SegmentList {
  int4 seg[kUnitThreads + 5];
  int cnt[kUnitWarps];         // a warp's segments; those of at most kPackSegment products << 16
  unsigned small[kUnitWarps];  // one bit a segment: such a one (small_segments)
};

// Fills `sl` with A entries [base, base + kUnitThreads) of the unit; returns
// the number of segments (and the small ones << 16).
template <bool R32>
__device__ __forceinline__ int list_segments(const DCsr& A, const DCsr& B, int64_t base, int64_t e, int t0, int t1,
                                             int ntiles, const int32_t* bidx, SegmentList& sl) {
  using Off = typename RowOff<R32>::T;
  const int lane = lane_id(), wib = threadIdx.x >> 5;
  Off bs;
  int len;
  float a;
  unit_segment<R32>(A, B, base + threadIdx.x, e, t0, t1, ntiles, bidx, bs, len, a);
  const unsigned m = __ballot_sync(kFull, len > 0);
  const unsigned few = __ballot_sync(kFull, len > 0 && len <= kPackSegment);
  if (lane == 0) sl.cnt[wib] = __popc(m) | __popc(few) << 16;
  __syncthreads();  // also: the previous list has been walked
  int at = 0, cnt = 0;
#pragma unroll
  for (int w = 0; w < kUnitWarps; ++w) {
    at += w < wib ? sl.cnt[w] : 0;
    cnt += sl.cnt[w];
  }
  at &= 0xffff;
  if (len > 0) sl.seg[at + __popc(m & ((1u << lane) - 1u))] = pack_segment<Off>(bs, len, a);
  if (threadIdx.x < 5) sl.seg[(cnt & 0xffff) + threadIdx.x] = make_int4(0, 0, 0, 0);
  __syncthreads();
  return cnt;
}

// A column's accumulator in a unit; one outside its columns, or with CHECK not
// one of C's, is noted in `far` (and lands on any).
template <bool CHECK>
__device__ __forceinline__ int locate_column(const uint2* bits, int32_t c, int32_t c0, uint32_t span, uint32_t& far) {
  uint32_t off = (uint32_t)(c - c0);
  far = max(far, off);
  off = min(off, span - 1u);
  const uint2 w = bits[off >> 5];
  const uint32_t bit = 1u << (off & 31);
  if (CHECK && !(w.x & bit)) far = 0xffffffffu;
  return (int)w.y + __popc(w.x & (bit - 1u));
}

// What an accumulator holds before its first product where every one has to get
// one: a NaN that no sum is (adds give 0x7fffffff).
constexpr uint32_t kUntouched = 0xffabcdefu;
template <bool CHECK>
__device__ __forceinline__ float added_to(float s, float p) {
  if (CHECK && __float_as_uint(s) == kUntouched) s = 0.f;
  return add_rn(s, p);
}

// Adds the products of a list of mostly small segments, in order: runs of small
// ones by one warp, 32 products a step, the others by the CTA.  The unit's bitmap
// of `words` words and its accumulators are in sm_unit.  Returns locate_column's
// `far`.  Not inlined: in the kernel its registers would cost every unit one or
// two of nine CTAs an SM (R-MAT 18, 3 edges: 4.72 -> 4.91 ms a call).
template <typename Off, bool CHECK>
__device__ __noinline__ uint32_t add_small_segments(const int32_t* col, const float* val, int words, SegmentList& sl,
                                                    int cnt, int32_t c0, uint32_t span) {
  extern __shared__ __align__(16) uint32_t sm_unit[];
  const uint2* bits = reinterpret_cast<const uint2*>(sm_unit);
  float* acc = reinterpret_cast<float*>(sm_unit) + 2 * words;
  const int tid = threadIdx.x, lane = lane_id(), wib = tid >> 5;
  uint32_t far = 0;
  const int mine = tid < cnt ? sl.seg[tid].z : 0;
  const unsigned few = __ballot_sync(kFull, mine > 0 && mine <= kPackSegment);
  if (lane == 0) sl.small[wib] = few;
  __syncthreads();
  for (int i = 0; i < cnt;) {
    const unsigned rest = ~(sl.small[i >> 5] >> (i & 31));
    const int run = min(rest ? __ffs(rest) - 1 : 32, 32 - (i & 31));
    if (run == 0) {
      const int4 sg = sl.seg[i];
      const Off sb = segment_start<Off>(sg);
      const float a = __int_as_float(sg.w);
      for (int q = tid; q < sg.z; q += kUnitThreads) {
        const int at = locate_column<CHECK>(bits, col[sb + q], c0, span, far);
        acc[at] = added_to<CHECK>(acc[at], prod_rn(a, val[sb + q]));
      }
      ++i;
    } else {
      if (wib == 0) {
        const int4 own = lane < run ? sl.seg[i + lane] : make_int4(0, 0, 0, 0);
        const Off ob = segment_start<Off>(own);
        const int incl = warp_incl_scan(own.z);
        const int total = __shfl_sync(kFull, incl, 31);
        for (int p0 = 0; p0 < total; p0 += 4 * 32) {
          int32_t c4[4];
          float p4[4];
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            if (p0 + x * 32 >= total) break;
            // lanes past the end take the last product and drop it
            const int t = min(p0 + x * 32 + lane, total - 1);
            const int from = warp_upper_bound(incl, t);
            const Off q = __shfl_sync(kFull, ob, from) + (Off)(t - __shfl_sync(kFull, incl - own.z, from));
            c4[x] = col[q];
            p4[x] = prod_rn(__int_as_float(__shfl_sync(kFull, own.w, from)), val[q]);
          }
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            if (p0 + x * 32 >= total) break;
            const int at = locate_column<CHECK>(bits, c4[x], c0, span, far);
            const bool act = p0 + x * 32 + lane < total;
            // products on one column: the first lane adds them in their order
            const unsigned grp = __match_any_sync(kFull, act ? at : -1 - lane);
            const bool lead = act && (grp & ((1u << lane) - 1u)) == 0u;
            unsigned later = grp & ~(1u << lane);
            float s = 0.f;
            if (lead) s = added_to<CHECK>(acc[at], p4[x]);
            while (__any_sync(kFull, lead && later)) {
              const int next = later ? __ffs(later) - 1 : lane;
              const float v = __shfl_sync(kFull, p4[x], next);
              if (lead && later) s = add_rn(s, v);
              later &= later - 1;
            }
            if (lead) acc[at] = s;
            __syncwarp();
          }
        }
      }
      i += run;
    }
    __syncthreads();
  }
  return far;
}

// Where a unit's columns come from.
enum UnitColumns {
  kStored,  // the rows' bitmaps of the symbolic pass (big_slot order, `stride` words a row)
  kFromC,   // c_col (value-only recompute)
  kMarked,  // a walk over its products; compared with tile_cnt, tile by tile
};

// One CTA per unit, one atomic ticket each.  With columns from C every product
// has to fall on one of them and every accumulator, kUntouched at first, has to
// get one; a unit where that fails raises a flag, its columns as they were.  For
// rows of at most whole_max entries the walk over the products also takes in the
// empty tiles up to the next unit, or the row's ends, so that no product of such
// a row goes unseen (kFromC, kMarked).  Then A's
// row is walked in canonical order, segment by segment with a barrier after
// each: a segment's columns are distinct, so the CTA's threads add its
// products at once.  A thread's first two products of segment i + 2 are
// loaded and those of segment i + 1 located while segment i is added.
template <bool R32, UnitColumns FROM>
__global__ void __launch_bounds__(kUnitThreads, R32 ? 9 : 8) k_num_unit(DCsr A, DCsr B, const int4* units, int64_t room,
                                                           const unsigned long long* nunits, int ntiles,
                                                           const int64_t* c_rp, int32_t* c_col, float* c_val,
                                                           const int32_t* bidx, const uint32_t* bitmap,
                                                           int64_t stride, const int32_t* big_slot,
                                                           const int32_t* tile_cnt, int64_t whole_max,
                                                           unsigned long long* ticket, int* flags) {
  using Off = typename RowOff<R32>::T;
  extern __shared__ __align__(16) uint32_t sm_unit[];
  __shared__ SegmentList sl;
  __shared__ int warp_cnt[kUnitWarps];
  __shared__ unsigned long long sh_ticket;
  const int tid = threadIdx.x, lane = lane_id(), wib = tid >> 5;
  uint2* bits = reinterpret_cast<uint2*>(sm_unit);  // {columns, entries before them}
  const int64_t nfront = (int64_t)(*nunits & 0xffffffffu), total_units = nfront + (int64_t)(*nunits >> 32);
  if (total_units > room) return;
  for (;;) {
    if (tid == 0) sh_ticket = atomicAdd(ticket, 1ull);
    __syncthreads();
    const int64_t u = (int64_t)sh_ticket;
    if (u >= total_units) break;
    const int4 un = units[u < nfront ? u : room - 1 - (u - nfront)];
    const int32_t row = un.x;
    const int t0 = un.y, nt = un.z >> 16, n = un.z & 0xffff, t1 = t0 + nt;
    const int32_t c0 = t0 << kTileShift;
    const uint32_t span = (uint32_t)nt << kTileShift;
    const int words = nt * kTileWords;
    float* acc = reinterpret_cast<float*>(bits + words);
    const int64_t s = A.rp[row], e = A.rp[row + 1];
    int g0 = t0, g1 = t1;  // the tiles looked at
    bool whole = false;
    if (FROM != kStored) {
      const int64_t entries = c_rp[row + 1] - c_rp[row];
      whole = entries <= whole_max;
      if (whole) {
        const int32_t* tc = tile_cnt + (int64_t)big_slot[row] * ntiles;
        while (g0 > 0) {
          const int t = g0 - 1 - lane;
          const unsigned filled = __ballot_sync(kFull, t >= 0 && tc[t] > 0);
          g0 = filled ? g0 - (__ffs(filled) - 1) : max(0, g0 - 32);
          if (filled) break;
        }
        if (un.w + n == entries) g1 = ntiles;
      }
    }
    const int64_t out = c_rp[row] + un.w;
    // the columns
    if (FROM == kStored) {
      const uint32_t* bm = bitmap + (int64_t)big_slot[row] * stride + (int64_t)t0 * kTileWords;
      for (int i = tid; i < words; i += kUnitThreads) bits[i].x = bm[i];
    } else {
      for (int i = tid; i < words; i += kUnitThreads) bits[i].x = 0u;
    }
    if (FROM == kFromC) {
      __syncthreads();
      for (int i = tid; i < n; i += kUnitThreads) {
        const uint32_t off = (uint32_t)(c_col[out + i] - c0);
        if (off < span) atomicOr(&bits[off >> 5].x, 1u << (off & 31));
        else raise_flag(flags, kFlagCountDiff);
      }
    }
    if (FROM == kMarked) {
      for (int64_t base = s; base < e; base += kUnitThreads) {
        const int cnt = list_segments<R32>(A, B, base, e, g0, g1, ntiles, bidx, sl) & 0xffff;
        auto mark = [&](int32_t c) {
          const uint32_t off = (uint32_t)(c - c0);
          if (off < span) {
            const uint32_t bit = 1u << (off & 31);
            if (!(bits[off >> 5].x & bit)) atomicOr(&bits[off >> 5].x, bit);
          } else {
            raise_flag(flags, whole ? kFlagCountDiff : kFlagBadIndex);
          }
        };
        // the warp's segments, one a lane: short ones by their lane, the others by
        // the warp
        const int mine = lane * kUnitWarps + wib;
        const int4 own = mine < cnt ? sl.seg[mine] : make_int4(0, 0, 0, 0);
        const Off ob = segment_start<Off>(own);
        if (own.z <= kLaneSegment) {
#pragma unroll 4
          for (int q = 0; q < own.z; ++q) mark(B.col[ob + q]);
        }
        for (unsigned todo = __ballot_sync(kFull, own.z > kLaneSegment); todo; todo &= todo - 1) {
          const int from = __ffs(todo) - 1;
          const int len = __shfl_sync(kFull, own.z, from);
          const Off sb = __shfl_sync(kFull, ob, from);
#pragma unroll 4
          for (int q = lane; q < len; q += 32) mark(B.col[sb + q]);
        }
      }
    }
    __syncthreads();
    // entries before each bitmap word: warp w owns a run of words
    const int per = (words + kUnitThreads - 1) / kUnitThreads * 32;
    const int p0 = min(words, wib * per), p1 = min(words, p0 + per);
    int sum = 0;
    for (int i = p0 + lane; i < p1; i += 32) sum += __popc(bits[i].x);
    sum = __reduce_add_sync(kFull, sum);
    if (lane == 0) warp_cnt[wib] = sum;
    __syncthreads();
    int before = 0, found = 0;
#pragma unroll
    for (int w = 0; w < kUnitWarps; ++w) {
      before += w < wib ? warp_cnt[w] : 0;
      found += warp_cnt[w];
    }
    for (int i0 = p0; i0 < p1; i0 += 32) {
      const int c = __popc(bits[i0 + lane].x);
      const int inc = warp_incl_scan(c);
      bits[i0 + lane].y = (uint32_t)(before + inc - c);
      before += __shfl_sync(kFull, inc, 31);
    }
    if (found != n) {
      if (tid == 0) raise_flag(flags, kFlagCountDiff);
      __syncthreads();
      continue;
    }
    for (int i = tid; i < n; i += kUnitThreads) acc[i] = FROM == kFromC ? __uint_as_float(kUntouched) : 0.f;
    __syncthreads();
    if (FROM == kMarked) {
      // C's columns of such a unit stay as they are: a second look at the row
      // counts them again
      const int32_t* tc = tile_cnt + (int64_t)big_slot[row] * ntiles + t0;
      bool differ = false;
      for (int j = tid; j < nt; j += kUnitThreads) {
        const uint32_t upto = j + 1 < nt ? bits[(j + 1) * kTileWords].y : (uint32_t)found;
        differ |= (int)(upto - bits[j * kTileWords].y) != tc[j];
      }
      if (__syncthreads_or(differ)) {
        if (tid == 0) raise_flag(flags, kFlagCountDiff);
        continue;
      }
    }
    uint32_t far = 0;
    auto locate = [&](int32_t c) { return locate_column<FROM == kFromC>(bits, c, c0, span, far); };
    auto added = [&](int at, float p) { return added_to<FROM == kFromC>(acc[at], p); };
    const int first = wib << 5;  // the warp's first product of a segment
    for (int64_t base = s; base < e; base += kUnitThreads) {
      const int listed = FROM == kFromC ? list_segments<R32>(A, B, base, e, g0, g1, ntiles, bidx, sl)
                                        : list_segments<R32>(A, B, base, e, t0, t1, ntiles, bidx, sl);
      const int cnt = listed & 0xffff;
      if (cnt >= 32 && (listed >> 16) * 4 >= cnt * 3) {
        far = max(far, add_small_segments<Off, FROM == kFromC>(B.col, B.val, words, sl, cnt, c0, span));
        continue;
      }
      // products tid and kUnitThreads + tid of three segments: one being
      // added, one located, one on its way
      int4 sg[3];
      int at[3][2];
      int32_t cc[3][2];
      float vv[3][2];
      // threads past a segment's end take its last product and drop it
      auto load = [&](int u, int i) {
        sg[u] = sl.seg[i];
        const int len = sg[u].z;
        if (first >= len) return;
        const Off sb = segment_start<Off>(sg[u]);
        const Off q = sb + (Off)min(tid, len - 1);
        cc[u][0] = B.col[q];
        vv[u][0] = B.val[q];
        if (first + kUnitThreads < len) {
          const Off q1 = sb + (Off)min(tid + kUnitThreads, len - 1);
          cc[u][1] = B.col[q1];
          vv[u][1] = B.val[q1];
        }
      };
      auto place = [&](int u) {
        if (first >= sg[u].z) return;
        at[u][0] = locate(cc[u][0]);
        if (first + kUnitThreads < sg[u].z) at[u][1] = locate(cc[u][1]);
      };
      auto add = [&](int u) {
        const int len = sg[u].z;
        if (first >= len) return;
        const float a = __int_as_float(sg[u].w);
        const float r0 = added(at[u][0], prod_rn(a, vv[u][0]));
        if (tid < len) acc[at[u][0]] = r0;
        if (first + kUnitThreads >= len) return;
        const float r1 = added(at[u][1], prod_rn(a, vv[u][1]));
        if (tid + kUnitThreads < len) acc[at[u][1]] = r1;
        if (first + 2 * kUnitThreads >= len) return;
        const Off sb = segment_start<Off>(sg[u]);
        for (int q0 = first + 2 * kUnitThreads; q0 < len; q0 += 4 * kUnitThreads) {
          int32_t c4[4];
          float v4[4];
          int a4[4];
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            const Off q = sb + (Off)min(q0 + x * kUnitThreads + lane, len - 1);
            c4[x] = B.col[q];
            v4[x] = B.val[q];
          }
#pragma unroll
          for (int x = 0; x < 4; ++x) a4[x] = locate(c4[x]);
          float cur[4];
#pragma unroll
          for (int x = 0; x < 4; ++x) cur[x] = added(a4[x], prod_rn(a, v4[x]));
#pragma unroll
          for (int x = 0; x < 4; ++x)
            if (q0 + x * kUnitThreads + lane < len) acc[a4[x]] = cur[x];
        }
      };
      load(0, 0);
      load(1, 1);
      place(0);
      for (int i = 0; i < cnt; i += 3) {
#pragma unroll
        for (int u = 0; u < 3; ++u) {
          load((u + 2) % 3, i + u + 2);
          place((u + 1) % 3);
          add(u);
          __syncthreads();
        }
      }
    }
    if (far >= span) raise_flag(flags, kFlagBadIndex);
    // values, then the columns laid out in the accumulators' place
    for (int i = tid; i < n; i += kUnitThreads) {
      c_val[out + i] = acc[i];
      if (FROM == kFromC && __float_as_uint(acc[i]) == kUntouched) raise_flag(flags, kFlagCountDiff);
    }
    __syncthreads();
    if (FROM == kFromC) continue;
    int32_t* cols = reinterpret_cast<int32_t*>(acc);
    for (int i = tid; i < words; i += kUnitThreads) {
      const uint2 w = bits[i];
      int at = (int)w.y;
      const int32_t c = c0 + i * 32 - 1;
      for (uint32_t b = w.x; b; b &= b - 1) cols[at++] = c + __ffs(b);
    }
    __syncthreads();
    for (int i = tid; i < n; i += kUnitThreads) c_col[out + i] = cols[i];
    __syncthreads();
  }
}

int64_t heavy_unit_bound(int64_t nheavy, int ntiles, int64_t entries) {
  // of two consecutive units of a row, the first and the second's first tile
  // exceed kUnitCost together (and the list's two 32-bit counts hold it: at
  // 16 bytes a unit, 2^31 of them are 32 GB)
  return 2 * (entries + (int64_t)kTileCost * ntiles * nheavy) / kUnitCost + nheavy + 1;
}

template <bool R32, UnitColumns FROM>
static void num_unit_one(const DCsr& A, const DCsr& B, const int4* units, int64_t room,
                         const unsigned long long* nunits, int ntiles,
                         const int64_t* c_rp, int32_t* c_col, float* c_val, const int32_t* bidx,
                         const uint32_t* bitmap, int64_t stride, const int32_t* big_slot, const int32_t* tile_cnt,
                         int64_t whole_max, unsigned long long* ticket, int* flags, const LaunchCtx& lc) {
  const size_t smem = (size_t)kUnitWords * 4;
  cudaFuncSetAttribute(k_num_unit<R32, FROM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_num_unit<R32, FROM>, kUnitThreads, smem);
  k_num_unit<R32, FROM><<<lc.sms * std::max(1, per_sm), kUnitThreads, smem, lc.stream>>>(
      A, B, units, room, nunits, ntiles, c_rp, c_col, c_val, bidx, bitmap, stride, big_slot, tile_cnt, whole_max,
      ticket, flags);
}

void launch_num_units(const DCsr& A, const DCsr& B, const int32_t* heavy_rows, int64_t nheavy, const int32_t* big_slot,
                      const int32_t* tile_cnt, int ntiles, const int64_t* c_rp, int32_t* c_col, float* c_val,
                      const int32_t* bidx, const uint32_t* bitmap, int64_t stride, bool c_known, int64_t whole_max,
                      int4* units, int64_t room, unsigned long long* counters, int* flags, const LaunchCtx& lc) {
  if (nheavy == 0) return;
  cudaMemsetAsync(counters, 0, 2 * sizeof(unsigned long long), lc.stream);
  const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((nheavy + 7) / 8, (int64_t)lc.sms * 8));
  k_cut_units<<<blocks, 256, 0, lc.stream>>>(heavy_rows, nheavy, big_slot, tile_cnt, ntiles, A.rp, units, room,
                                             counters, flags);
#define SPG_NU(R, F)                                                                                            \
  num_unit_one<R, F>(A, B, units, room, counters, ntiles, c_rp, c_col, c_val, bidx, bitmap, stride, big_slot,   \
                     tile_cnt, whole_max, counters + 1, flags, lc)
  if (B.rp32) {
    if (bitmap) SPG_NU(true, kStored);
    else if (c_known) SPG_NU(true, kFromC);
    else SPG_NU(true, kMarked);
  } else {
    if (bitmap) SPG_NU(false, kStored);
    else if (c_known) SPG_NU(false, kFromC);
    else SPG_NU(false, kMarked);
  }
#undef SPG_NU
}

}  // namespace spg
