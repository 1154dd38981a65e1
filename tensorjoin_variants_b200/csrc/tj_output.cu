// Canonical output order: emitted keys -> pairs sorted by (i, j), kept as row ends and columns.
//
// The screens and the refinement append pair keys in no order.  The canonical order is by row first,
// so instead of sorting whole keys (five 8-bit passes, 16 bytes of traffic and one ranking of every
// key per pass) the keys are
//   1. counted per row        (row_count: one read of the keys, one atomic per run of equal rows),
//   2. placed in their row    (exclusive scan of the counts, then row_scatter: each run of equal
//                              rows takes its slots by one atomic; 4 bytes written per pair),
//   3. put in order per row   (row_rank, row_sort_mid, row_sort_long: rows are short, so a warp ranks or
//                              sorts them on chip; a block sorts the long ones).
// The result stays in that form, four bytes per pair and four per row, and pairs, keys or a neighbour
// table are written from it directly.  What bounds it: the scattered 4-byte writes and the returning
// atomics of step 2 in L2 (keys of one row come from few tiles, close in time, so most writes of a
// sector merge there).
//
#include <algorithm>
#include <cstring>

#include "tj_emit.cuh"
#include "tj_internal.h"

namespace tj {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kChunk = 256;              // consecutive slots a warp takes at a time
constexpr unsigned kWarpSortMax = kMidRow;   // longest row a warp sorts in registers
constexpr unsigned kStage = 1024;        // pairs a warp stages in shared memory
constexpr unsigned kRankMax = 64;        // longest row ranked by counting

// Join of a key or row: the last entry of off that is <= v (off ascending).
TJ_DEV int find_join(const unsigned long long* off, int n, unsigned long long v) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (off[mid] <= v) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// key -> (row over all joins, column).  `hint` carries the join from call to call: a warp's slots
// mostly come from one join.
// False for a key that names no row of the joins (no screen writes one): nothing is counted or written.
TJ_DEV bool split_key(const RowTables& t, uint32_t nrows, uint64_t key, int& hint, uint32_t& row, uint32_t& col) {
    RowTable e = t.first;
    if (t.njoins > 1) {
        if (key < t.key_off[hint] || (hint + 1 < t.njoins && key >= t.key_off[hint + 1]))
            hint = find_join(t.key_off, t.njoins, key);
        e = t.tab[hint];
    }
    // quotient by the reciprocal floor((2^64 - 1) / n_cols): at most two too small
    const uint64_t v = key - e.key_off;
    uint64_t q = __umul64hi(v, e.recip);
    uint64_t r = v - q * e.n_cols;
    while (r >= e.n_cols) {
        r -= e.n_cols;
        ++q;
    }
    row = (uint32_t)(e.row_off + q);
    col = (uint32_t)r;
    return e.row_off + q < nrows;
}

// Runs of equal rows among a warp's 32 slots (invalid slots are runs of their own that nobody counts).
struct Run {
    unsigned head, len;   // first lane of this lane's run, and the run's lanes
};
TJ_DEV Run find_run(uint32_t row, bool valid) {
    const unsigned lane = lane_id();
    const uint32_t before = __shfl_up_sync(0xffffffffu, row, 1);
    const unsigned vm = __ballot_sync(0xffffffffu, valid);
    const bool lead = lane == 0 || !valid || !((vm >> (lane - 1)) & 1u) || before != row;
    const unsigned heads = __ballot_sync(0xffffffffu, lead);
    const unsigned upto = 0xFFFFFFFFu >> (31 - lane);   // lanes 0..lane
    const unsigned after = heads & ~upto;
    const unsigned head = 31 - __clz(heads & upto);
    return Run{head, (after ? __ffs(after) - 1 : 32) - head};
}

__global__ void fill_u32(uint32_t* p, size_t n, uint32_t v) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) p[i] = v;
}

// Step 1.  kDirected: both directions of every (i < j) key (the self pairs are in the initial counts).
template <bool kDirected>
__global__ void __launch_bounds__(kThreads) row_count(const uint64_t* keys, const Counters* ctr, unsigned long long cap,
                                                      const RowTables t, uint32_t nrows, uint32_t* cnt) {
    const unsigned long long n = ctr->acc_reserved, pairs = ctr->acc_valid;
    if (n > cap || !rows_may_fit(kDirected ? 2 * pairs + nrows : pairs, nrows)) return;   // as the host reads them
    const unsigned lane = lane_id();
    const unsigned long long nw = (unsigned long long)gridDim.x * kWarps;
    int hint = 0;
    for (unsigned long long c = (unsigned long long)blockIdx.x * kWarps + (threadIdx.x >> 5); c * kChunk < n; c += nw) {
        uint64_t key[kChunk / 32];
#pragma unroll
        for (int u = 0; u < kChunk / 32; ++u) {
            const unsigned long long p = c * kChunk + u * 32 + lane;
            key[u] = p < n ? keys[p] : kSentinel;
        }
#pragma unroll
        for (int u = 0; u < kChunk / 32; ++u) {
            uint32_t row = 0xFFFFFFFFu, col = 0;
            const bool valid = key[u] != kSentinel && split_key(t, nrows, key[u], hint, row, col);
            const Run r = find_run(row, valid);
            if (valid && r.head == lane) atomicAdd(cnt + row, r.len);
            if (kDirected && valid) atomicAdd(cnt + col, 1u);
        }
    }
}

// Step 2: `cursor` holds every row's first position and ends as its end.
template <bool kDirected>
__global__ void __launch_bounds__(kThreads) row_scatter(const uint64_t* keys, unsigned long long n, const RowTables t,
                                                        uint32_t* cursor, uint32_t* cols, uint32_t total,
                                                        uint32_t nrows, unsigned long long* status) {
    const unsigned lane = lane_id();
    const unsigned long long nw = (unsigned long long)gridDim.x * kWarps;
    int hint = 0;
    bool outside = false;   // cannot happen with consistent counts; checked so that nothing lands outside
    constexpr int kU = 4;
    auto put = [&](uint32_t pos, uint32_t col) {
        if (pos < total) cols[pos] = col;
        else outside = true;
    };
    for (unsigned long long c = (unsigned long long)blockIdx.x * kWarps + (threadIdx.x >> 5); c * kChunk < n; c += nw) {
        for (int u0 = 0; u0 < kChunk / 32; u0 += kU) {
            uint64_t key[kU];
            uint32_t row[kU], col[kU], base[kU], back[kU];
            Run run[kU];
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                const unsigned long long p = c * kChunk + (u0 + u) * 32 + lane;
                key[u] = p < n ? keys[p] : kSentinel;
            }
            // all four slots' atomics are in flight before the first result is used
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                row[u] = 0xFFFFFFFFu;
                col[u] = base[u] = back[u] = 0;
                const bool valid = key[u] != kSentinel && split_key(t, nrows, key[u], hint, row[u], col[u]);
                outside |= key[u] != kSentinel && !valid;
                if (!valid) key[u] = kSentinel;
                run[u] = find_run(row[u], valid);
                if (valid && run[u].head == lane) base[u] = atomicAdd(cursor + row[u], run[u].len);
                if (kDirected && valid) back[u] = atomicAdd(cursor + col[u], 1u);
            }
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                const uint32_t b = __shfl_sync(0xffffffffu, base[u], run[u].head);
                if (key[u] == kSentinel) continue;
                put(b + lane - run[u].head, col[u]);
                if (kDirected) put(back[u], row[u]);
            }
        }
    }
    if (kDirected)   // the self pairs
        for (uint32_t r = blockIdx.x * kThreads + threadIdx.x; r < nrows; r += gridDim.x * kThreads)
            put(atomicAdd(cursor + r, 1u), r);
    if (outside) atomicOr(status, (unsigned long long)kStatusGuard);
}

// ------------------------------------------------------------------ step 3
// Ascending order of one row of len <= 32 kE columns, by a bitonic network over registers: element
// lane * kE + e in register e, so steps of less than kE stay inside a lane.
template <int kE>
TJ_DEV void warp_sort(uint32_t* p, unsigned len, uint32_t* buf) {
    const unsigned lane = lane_id();
    uint32_t x[kE];
#pragma unroll
    for (int e = 0; e < kE; ++e) x[e] = (unsigned)(e * 32) + lane < len ? p[e * 32 + lane] : 0xFFFFFFFFu;
#pragma unroll
    for (int k = 2; k <= 32 * kE; k <<= 1) {
#pragma unroll
        for (int s = k >> 1; s > 0; s >>= 1) {
            if (s >= kE) {
                const bool keep_min = ((lane * kE & k) == 0) == ((lane & (s / kE)) == 0);
#pragma unroll
                for (int e = 0; e < kE; ++e) {
                    const uint32_t y = __shfl_xor_sync(0xffffffffu, x[e], s / kE);
                    x[e] = keep_min ? min(x[e], y) : max(x[e], y);
                }
            } else {
#pragma unroll
                for (int e = 0; e < kE; ++e) {
                    if (e & s) continue;
                    const uint32_t a = min(x[e], x[e | s]), b = max(x[e], x[e | s]);
                    const bool up = k < kE ? (e & k) == 0 : (lane * kE & k) == 0;
                    x[e] = up ? a : b;
                    x[e | s] = up ? b : a;
                }
            }
        }
    }
    // through shared memory (one word of padding per 32), so that the row is written in full lines
    __syncwarp();
#pragma unroll
    for (int e = 0; e < kE; ++e) {
        const unsigned q = lane * kE + e;
        buf[q + (q >> 5)] = x[e];
    }
    __syncwarp();
#pragma unroll
    for (int e = 0; e < kE; ++e) {
        const unsigned q = e * 32 + lane;
        if (q < len) p[q] = buf[q + (q >> 5)];
    }
    __syncwarp();
}

// Rows that row_rank leaves to the other two kernels: medium ones (a warp each) and long ones (a block each).
struct RowLists {
    uint32_t *mid, *lng;
    unsigned *n_mid, *n_lng;
};

// A warp takes `group` (1..32, a power of two) consecutive rows, stages the columns of the short ones
// together and writes each to its place, the number of smaller columns in its row.  Kept apart from the
// register sorts below, which hold three times the registers: with them in one kernel 24 warps of an SM
// ran here, and ranking is bound by the latency of its shared-memory reads.
__global__ void __launch_bounds__(kThreads) row_rank(const uint32_t* row_end, uint32_t nrows, unsigned group,
                                                     uint32_t* cols, const RowLists lists) {
    __shared__ uint32_t stage[kWarps][kStage];
    const unsigned lane = lane_id();
    uint32_t* buf = stage[threadIdx.x >> 5];
    const unsigned long long r0 = ((unsigned long long)blockIdx.x * kWarps + (threadIdx.x >> 5)) * group;
    if (r0 >= nrows) return;   // warp-uniform
    const unsigned ng = (unsigned)min((unsigned long long)group, nrows - r0);
    const uint32_t beg = r0 ? row_end[r0 - 1] : 0u;
    const uint32_t end = row_end[r0 + min(lane, ng - 1)];
    uint32_t start = __shfl_up_sync(0xffffffffu, end, 1);   // lanes past the last row: an empty row at its end
    if (lane == 0) start = beg;
    unsigned len = end - start;
    const unsigned longest = __reduce_max_sync(0xffffffffu, len);
    if (longest <= 1) return;
    unsigned total = __shfl_sync(0xffffffffu, end, 31) - beg, off = start - beg;
    bool packed = true;   // the staged columns are consecutive in memory
    if (longest > kRankMax || total > kStage) {
        // longer rows go to the lists; 32 rows of at most 32 columns always fit the stage
        unsigned lim = kRankMax;
        off = warp_excl_scan(len <= lim ? len : 0u, total);
        if (total > kStage) {
            lim = 32;
            off = warp_excl_scan(len <= lim ? len : 0u, total);
        }
        if (len > kWarpSortMax) lists.lng[atomicAdd(lists.n_lng, 1u)] = (uint32_t)r0 + lane;
        const bool mid = len > lim && len <= kWarpSortMax;
        const unsigned m = __ballot_sync(0xffffffffu, mid);
        unsigned base = 0;
        if (lane == 0 && m) base = atomicAdd(lists.n_mid, __popc(m));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (mid) lists.mid[base + __popc(m & ((1u << lane) - 1u))] = (uint32_t)r0 + lane;
        if (len > lim) len = 0;
        packed = false;
    }
    // row of staged position p: the last one whose first position is <= p (empty rows share the first
    // position of the row after them)
    auto row_of = [&](unsigned p) {
        unsigned r = 0;
#pragma unroll
        for (int s = 16; s > 0; s >>= 1)
            if (__shfl_sync(0xffffffffu, off, r + s) <= p) r += s;
        return r;
    };
    for (unsigned p0 = 0; p0 < total; p0 += 32) {
        const unsigned p = p0 + lane;
        uint32_t src = beg + p;
        if (!packed) {
            const unsigned r = row_of(p);
            src = __shfl_sync(0xffffffffu, start - off, r) + p;
        }
        if (p < total) buf[p] = cols[src];
    }
    __syncwarp();
    for (unsigned p0 = 0; p0 < total; p0 += 32) {
        const unsigned p = p0 + lane, r = row_of(p);
        const unsigned o = __shfl_sync(0xffffffffu, off, r), l = __shfl_sync(0xffffffffu, len, r);
        const uint32_t dst = __shfl_sync(0xffffffffu, start, r);
        if (p >= total) continue;
        const uint32_t x = buf[p];
        unsigned rank = 0;
#pragma unroll 8
        for (unsigned q = o; q < o + l; ++q) rank += buf[q] < x ? 1u : 0u;
        cols[dst + rank] = x;
    }
}

// Medium rows, one warp each.
__global__ void __launch_bounds__(kThreads) row_sort_mid(const uint32_t* row_end, uint32_t* cols, const RowLists lists) {
    __shared__ uint32_t stage[kWarps][kWarpSortMax + kWarpSortMax / 32];
    uint32_t* buf = stage[threadIdx.x >> 5];
    const unsigned n = *lists.n_mid;
    for (unsigned k = blockIdx.x * kWarps + (threadIdx.x >> 5); k < n; k += gridDim.x * kWarps) {
        const uint32_t r = lists.mid[k], beg = r ? row_end[r - 1] : 0u, len = row_end[r] - beg;
        uint32_t* p = cols + beg;
        if (len <= 64) warp_sort<2>(p, len, buf);
        else if (len <= 128) warp_sort<4>(p, len, buf);
        else if (len <= 256) warp_sort<8>(p, len, buf);
        else warp_sort<16>(p, len, buf);
    }
}

// Long rows (kWarpSortMax < len <= kLongRow), one block each: a bitonic network in shared memory.
constexpr int kLongThreads = 512;
__global__ void __launch_bounds__(kLongThreads) row_sort_long(const uint32_t* row_end, uint32_t* cols,
                                                              const RowLists lists) {
    extern __shared__ uint32_t sm[];
    const unsigned count = *lists.n_lng;
    for (unsigned q = blockIdx.x; q < count; q += gridDim.x) {
        const uint32_t r = lists.lng[q], beg = r ? row_end[r - 1] : 0u, len = row_end[r] - beg;
        unsigned n = 2 * kWarpSortMax;
        while (n < len) n <<= 1;
        for (unsigned i = threadIdx.x; i < n; i += kLongThreads) sm[i] = i < len ? cols[beg + i] : 0xFFFFFFFFu;
        __syncthreads();
        for (unsigned k = 2; k <= n; k <<= 1)
            for (unsigned s = k >> 1; s > 0; s >>= 1) {
                for (unsigned i = threadIdx.x; i < n / 2; i += kLongThreads) {
                    const unsigned a = 2 * i - (i & (s - 1)), b = a + s;   // the pair of step s
                    const uint32_t x = sm[a], y = sm[b];
                    if ((x > y) == ((a & k) == 0)) {
                        sm[a] = y;
                        sm[b] = x;
                    }
                }
                __syncthreads();
            }
        for (unsigned i = threadIdx.x; i < len; i += kLongThreads) cols[beg + i] = sm[i];
        __syncthreads();
    }
}

// ------------------------------------------------------------------ results from rows and columns
enum { kOutPairs = 0, kOutKeys = 1, kOutCols = 2 };

// A warp takes `group` consecutive rows and writes their pairs 32 at a time; each position finds its
// row by a shuffle search over the rows' first positions.
template <int kOut>
__global__ void __launch_bounds__(kThreads) rows_out(const uint32_t* row_end, const uint32_t* cols, uint32_t nrows,
                                                     unsigned group, const RowTables t, int64_t* a, int64_t* b) {
    const unsigned lane = lane_id();
    const unsigned long long r0 = ((unsigned long long)blockIdx.x * kWarps + (threadIdx.x >> 5)) * group;
    if (r0 >= nrows) return;   // warp-uniform
    const unsigned ng = (unsigned)min((unsigned long long)group, nrows - r0);
    const uint32_t beg = r0 ? row_end[r0 - 1] : 0u;
    const uint32_t end = row_end[r0 + min(lane, ng - 1)];
    uint32_t start = __shfl_up_sync(0xffffffffu, end, 1);
    if (lane == 0) start = beg;
    const unsigned total = __shfl_sync(0xffffffffu, end, 31) - beg, off = start - beg;
    uint32_t i = (uint32_t)r0 + lane;
    uint64_t key0 = 0;
    if (kOut != kOutCols) {
        RowTable e = t.first;
        if (t.njoins > 1) e = t.tab[find_join(t.row_off, t.njoins, min((unsigned long long)i, (unsigned long long)nrows - 1))];
        i -= (uint32_t)e.row_off;
        key0 = e.key_off + (uint64_t)i * e.n_cols;
    }
    for (unsigned p0 = 0; p0 < total; p0 += 32) {
        const unsigned p = p0 + lane;
        unsigned r = 0;
        if (kOut != kOutCols) {
#pragma unroll
            for (int s = 16; s > 0; s >>= 1)
                if (__shfl_sync(0xffffffffu, off, r + s) <= p) r += s;
        }
        const uint32_t iv = __shfl_sync(0xffffffffu, i, r);
        const uint64_t kv = kOut == kOutKeys ? __shfl_sync(0xffffffffu, key0, r) : 0;
        if (p >= total) continue;
        const uint32_t c = cols[beg + p];
        if (kOut == kOutPairs) {
            a[beg + p] = iv;
            b[beg + p] = c;
        } else {
            a[beg + p] = kOut == kOutKeys ? (int64_t)(kv + c) : (int64_t)c;
        }
    }
}

// The same by positions, for one join with rows of any length (direct joins: of up to 2^20 columns, where
// the few warps that had them took 0.6 us per 32 pairs: a join of 16 x 1,048,576 with 8.9M pairs
// 11.0 -> 0.73 ms).  A block finds the rows of its first and last position, and every position its row
// between them.
constexpr unsigned kFlat = 2048;
template <int kOut>
__global__ void __launch_bounds__(kThreads) rows_out_flat(const uint32_t* row_end, const uint32_t* cols, uint32_t nrows,
                                                          uint32_t total, unsigned long long n_cols, int64_t* a,
                                                          int64_t* b) {
    __shared__ uint32_t lim[2];
    const uint32_t p0 = blockIdx.x * kFlat;   // (< total)
    auto row_of = [&](uint32_t p, uint32_t lo, uint32_t hi) {   // the first row that ends beyond p
        while (lo < hi) {
            const uint32_t mid = lo + (hi - lo) / 2;
            if (row_end[mid] > p) hi = mid; else lo = mid + 1;
        }
        return lo;
    };
    if (threadIdx.x < 2)
        lim[threadIdx.x] = row_of(threadIdx.x ? p0 + min(kFlat, total - p0) - 1 : p0, 0u, nrows - 1);
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < min(kFlat, total - p0); k += kThreads) {
        const uint32_t p = p0 + k, c = cols[p];
        if (kOut == kOutCols) {
            a[p] = c;
            continue;
        }
        const uint32_t i = row_of(p, lim[0], lim[1]);
        if (kOut == kOutPairs) {
            a[p] = i;
            b[p] = c;
        } else {
            a[p] = (int64_t)(i * n_cols + c);
        }
    }
}

__global__ void rows_counts(const uint32_t* row_end, uint32_t nrows, uint32_t* out) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < nrows) out[r] = row_end[r] - (r ? row_end[r - 1] : 0u);
}

__global__ void rows_offsets(const uint32_t* row_end, const unsigned long long* row_off, int njoins, long long n,
                             long long* out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k > njoins) return;
    const unsigned long long r = k < njoins ? row_off[k] : 0;
    out[k] = k == njoins ? n : r ? (long long)row_end[r - 1] : 0;
}

// Rows per warp: 32, or fewer where that would leave the chip without warps.
unsigned rows_per_warp(uint32_t nrows) {
    unsigned g = 32;
    while (g > 1 && nrows / g < (uint32_t)num_sms() * 32) g >>= 1;
    return g;
}
unsigned warp_blocks(uint32_t nrows, unsigned group) {
    return (unsigned)(((unsigned long long)nrows + (unsigned long long)group * kWarps - 1) /
                      ((unsigned long long)group * kWarps));
}
unsigned slot_blocks(unsigned long long slots) {
    const unsigned long long per = (unsigned long long)kChunk * kWarps;
    return (unsigned)std::max<unsigned long long>(1, std::min<unsigned long long>((slots + per - 1) / per,
                                                                                  (unsigned long long)num_sms() * 16));
}

}  // namespace

RowTable make_row_table(unsigned long long key_off, unsigned long long row_off, unsigned long long n_cols) {
    return RowTable{key_off, row_off, std::max(n_cols, 1ull), n_cols > 1 ? ~0ull / n_cols : ~0ull};
}

void count_rows(const uint64_t* keys, Counters* ctr, unsigned long long cap, const RowTables& t, bool directed,
                uint32_t nrows, uint32_t* cnt, uint32_t* first, uint32_t* ws, cudaStream_t st) {
    if (directed)   // every row's self pair
        launch(fill_u32, std::max(1u, std::min((nrows + 255) / 256, (unsigned)num_sms() * 8)), 256, 0, st, cnt,
               (size_t)nrows, 1u);
    else
        TJ_CUDA(cudaMemsetAsync(cnt, 0, (size_t)nrows * sizeof(uint32_t), st));
    const unsigned blocks = slot_blocks(cap);
    if (directed)
        launch(row_count<true>, blocks, kThreads, 0, st, keys, (const Counters*)ctr, cap, t, nrows, cnt);
    else
        launch(row_count<false>, blocks, kThreads, 0, st, keys, (const Counters*)ctr, cap, t, nrows, cnt);
    static_assert(offsetof(Counters, long_pairs) == offsetof(Counters, longest_row) + 8, "the scan's two words");
    exclusive_scan_u32(cnt, first, nrows, nullptr, ws, st, &ctr->longest_row);
}

void order_rows(const uint64_t* keys, unsigned long long slots, const RowTables& t, bool directed, uint32_t nrows,
                uint32_t total, unsigned long long longest, uint32_t* cursor, uint32_t* cols,
                unsigned long long* status, cudaStream_t st) {
    const unsigned blocks = slot_blocks(std::max<unsigned long long>(slots, directed ? nrows : 0));
    if (directed)
        launch(row_scatter<true>, blocks, kThreads, 0, st, keys, slots, t, cursor, cols, total, nrows, status);
    else
        launch(row_scatter<false>, blocks, kThreads, 0, st, keys, slots, t, cursor, cols, total, nrows, status);
    if (longest <= 1) return;
    const unsigned g = rows_per_warp(nrows);
    RowLists lists{};
    DBuf<uint32_t> mem;
    if (longest > 32) {   // else every row is ranked
        const size_t nm = total / 33 + 1, nl = total / (kWarpSortMax + 1) + 1;
        mem = DBuf<uint32_t>(2 + nm + nl, st);
        lists = RowLists{mem.p + 2, mem.p + 2 + nm, mem.p, mem.p + 1};
        TJ_CUDA(cudaMemsetAsync(mem.p, 0, 2 * sizeof(uint32_t), st));
    }
    launch(row_rank, warp_blocks(nrows, g), kThreads, 0, st, (const uint32_t*)cursor, nrows, g, cols, lists);
    if (longest > 32)
        launch(row_sort_mid, std::min((total / 33 + kWarps) / kWarps, (unsigned)num_sms() * 8), kThreads, 0, st,
               (const uint32_t*)cursor, cols, lists);
    if (longest > kWarpSortMax) {
        size_t n = 2 * kWarpSortMax;
        while (n < longest) n <<= 1;
        TJ_CUDA(cudaFuncSetAttribute(row_sort_long, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(n * 4)));
        launch(row_sort_long, std::min(total / (kWarpSortMax + 1) + 1, (unsigned)num_sms() * 4), kLongThreads, n * 4,
               st, (const uint32_t*)cursor, cols, lists);
    }
}

template <int kOut>
static void write_rows(const RowsView& v, int64_t* a, int64_t* b, cudaStream_t st) {
    if (v.longest > kLongRow && v.tabs->njoins == 1) {
        launch(rows_out_flat<kOut>, (unsigned)((v.total + kFlat - 1) / kFlat), kThreads, 0, st, v.row_end, v.cols, v.nrows,
               (uint32_t)v.total, v.tabs->first.n_cols, a, b);
        return;
    }
    const unsigned g = rows_per_warp(v.nrows);
    launch(rows_out<kOut>, warp_blocks(v.nrows, g), kThreads, 0, st, v.row_end, v.cols, v.nrows, g, *v.tabs, a, b);
}
void rows_pairs(const RowsView& v, int64_t* i_out, int64_t* j_out, cudaStream_t st) {
    write_rows<kOutPairs>(v, i_out, j_out, st);
}
void rows_keys(const RowsView& v, uint64_t* out, cudaStream_t st) {
    write_rows<kOutKeys>(v, (int64_t*)out, nullptr, st);
}
void rows_neighbors(const RowsView& v, uint32_t* counts, int64_t* flat, cudaStream_t st) {
    launch(rows_counts, (v.nrows + 255) / 256, 256, 0, st, v.row_end, v.nrows, counts);
    if (flat) write_rows<kOutCols>(v, flat, nullptr, st);
}
void rows_batch_offsets(const uint32_t* row_end, const unsigned long long* row_off, int njoins, long long n,
                        long long* out, cudaStream_t st) {
    launch(rows_offsets, (unsigned)(njoins / 256 + 1), 256, 0, st, row_end, row_off, njoins, n, out);
}

}  // namespace tj
