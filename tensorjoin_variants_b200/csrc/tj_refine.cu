// FP64 band refinement, the plain FP32 direct-difference join, and the
// canonical-output helpers (directed expansion, pair decoding).
//
// Refinement reproduces the oracle's predicate exactly: for every band pair,
//   acc = 0; for k = 0..d-1: t = dbl(x_k) - dbl(y_k); acc = acc + t*t   (one rounding each, no FMA)
//   accept iff acc <= T
// which is the reference's FP64 terminal (src/run_g2a_tensorjoin.py:194-232,
// src/run_d1_triton.py:206-248) with its summation order fixed to sequential k
// (the reference summed 256-wide blocks in tree order), so the emitted pair set is
// bit-identical to the CPU oracle.
//
// The plain join is the "plain GPU method" baseline: FP32 direct difference over
// the same candidate tile pairs (no tensor cores), a rigorous FP32 error band, and
// the same FP64 refinement of band pairs.  It plays the role of the reference's
// GDS-Join FP64 grid join / FP32-first control (adapters/gds_g2a/kernel.cu:314-386,
// g15_strong_control_20260905/src/fp32_first.py:104-157).
#include <algorithm>
#include <cstring>
#include <vector>

#include "tj_emit.cuh"
#include "tj_internal.h"

namespace tj {

namespace {

// Squared distance in the oracle's order: sequential k, one FP64 rounding per operation.
TJ_DEV double seq_d2(const float* x, const float* y, int d) {
    double acc = 0.0;
    if ((d & 3) == 0 && ((((uintptr_t)x) | ((uintptr_t)y)) & 15) == 0) {
        const float4* x4 = (const float4*)x;
        const float4* y4 = (const float4*)y;
        for (int k = 0; k < d / 4; ++k) {
            const float4 a = __ldg(x4 + k), b = __ldg(y4 + k);
            double t;
            t = __dsub_rn((double)a.x, (double)b.x); acc = __dadd_rn(acc, __dmul_rn(t, t));
            t = __dsub_rn((double)a.y, (double)b.y); acc = __dadd_rn(acc, __dmul_rn(t, t));
            t = __dsub_rn((double)a.z, (double)b.z); acc = __dadd_rn(acc, __dmul_rn(t, t));
            t = __dsub_rn((double)a.w, (double)b.w); acc = __dadd_rn(acc, __dmul_rn(t, t));
        }
    } else {
        for (int k = 0; k < d; ++k) {
            const double t = __dsub_rn((double)__ldg(x + k), (double)__ldg(y + k));
            acc = __dadd_rn(acc, __dmul_rn(t, t));
        }
    }
    return acc;
}

// ------------------------------------------------------------------ plain FP32 join
// A unit is 128 R rows x 64 S rows (a quarter of a candidate tile pair); a CTA of 16 x 16 threads
// holds 8 x 4 pairs per thread, each as two running sums (even and odd k) in one FP32x2 register
// pair, so a row's (k, k + 1) read from shared memory is a packed operand as it lies there.
//
// What bounds it: FP32 issue (a packed subtract and a packed FMA per two elements of a pair; the
// packed pipe alone needs 180 us for the 202M pairs of a 20,000 x 16 self-join), with the per-pair
// sum and classification on top of it below d = 16.  With 8 x 16 pairs per thread, one CTA per SM,
// unpipelined loads and a branch per pair it was latency: 31,000 cycles per 128 x 256 tile pair at d = 16
// and at d = 2 alike.  Hence two CTAs of 8 warps per SM, operand
// chunks brought in two stages ahead by cp.async (across unit and tile borders), one minimum over a
// thread's 32 pairs in front of the per-pair tests, and an even cut of all units over the CTAs
// (chunks of 64 tile pairs left half of them idle on 20,000 rows).  Measured (one B200): 20,000 x 16
// self-join 702 -> 376 us; 100,000 x 2 self-join with 13.7M pairs 643 -> 290 us.
constexpr int kPT = 256;                // threads: 16 x 16
constexpr int kPI = 8, kPJ = 4;         // pairs per thread: rows i * 16 + ty, columns j * 16 + tx
constexpr int kPCols = 64;              // columns of a unit
constexpr int kPUnits = kTileS / kPCols;
constexpr int kPK = 16;                 // k chunk (elements per stage)
constexpr int kPLd = kPK + 4;           // shared row stride: 16-byte reads of 8 rows hit distinct banks
constexpr int kPStages = 3;
constexpr int kPRows = kTileR + kPCols; // staged rows: R tile, then the unit's S rows

struct PlainClass {
    const float* rx;     // [rows, ld] FP32 rows (R side of the class)
    const float* sx;     // [rows, ld] FP32 rows (S side)
    const uint32_t* r_emit;
    const uint32_t* s_emit;
    int d, ld;           // elements of a row, and from one row to the next
    int vec;             // rows are 16-byte aligned, with zeros up to a multiple of four elements
};

// Direct joins (kDirect below): every pair of one small join, straight from the caller's rows.
struct DirectArgs {
    unsigned nR, nS;            // rows
    unsigned cols64;            // units per R tile: ceil(nS / 64)
    int upper;                  // 1: self-join, columns above the row only
    int diagonal;               // 1: self-join with self pairs (always accepted, not counted as decided)
    unsigned long long* bits;   // [nR][cols64] accepted pairs, bit c of word u: column 64 u + c
    uint32_t* cnt;              // [nR] accepted pairs per row (zeroed)
    unsigned long long* band;   // [2] pairs decided in FP64, and those of them accepted (zeroed)
    double T;
    float2 thr;
};

struct PlainArgs {
    DirectArgs dir;
    const uint32_t* off;        // [ntR] first candidate of each R tile
    const uint32_t* total;      // candidates
    int ntR;
    unsigned run;               // candidates that a CTA takes at a time, in turn (0: one run each, an even cut)
    const uint32_t* jlist;
    const uint4* rtiles;        // (row0, nvalid, join, class) per global R tile
    const uint4* stiles;
    const JoinParams* jps;
    const float2* thr;          // per join: certified-in / certified-out thresholds on the FP32 sum
    PlainClass cls[kMaxClass];
    uint64_t* acc;
    unsigned long long acc_cap;
    uint64_t* band;
    unsigned long long band_cap;
    Counters* ctr;
};

TJ_DEV void cp_async4_zfill(void* dst, const void* src, bool real) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;"
                 :: "r"(smem_u32(dst)), "l"((uint64_t)src), "r"(real ? 4u : 0u) : "memory");
}
TJ_DEV void cp_async16_zfill(void* dst, const void* src, bool real) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                 :: "r"(smem_u32(dst)), "l"((uint64_t)src), "r"(real ? 16u : 0u) : "memory");
}
// acc += (r - s)^2 in both halves, each rounded as the scalar subtract and fmaf
TJ_DEV void sqdiff_x2(unsigned long long r, unsigned long long s, unsigned long long& acc) {
    asm("{\n\t.reg .b64 t;\n\t"
        "sub.rn.f32x2 t, %1, %2;\n\t"
        "fma.rn.f32x2 %0, t, t, %0;\n\t}"
        : "+l"(acc) : "l"(r), "l"(s));
}
TJ_DEV float sum_x2(unsigned long long v) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
    return lo + hi;
}

// What the compute side needs to know of a stage (written by thread 0 when the stage is issued).
struct PlainStage {
    unsigned r0, nvI, c0, nvJ;   // rows of the R tile, columns of the unit
    unsigned join;
    int kc;                      // elements in the stage (0: no more stages)
    int first, last;             // first / last k chunk of the unit
    float2 th;                   // the join's thresholds
};

// R tile of candidate e: the last one whose first candidate is <= e (warp-collective).
TJ_DEV int find_rtile(const uint32_t* off, int n, uint32_t e) {
    int lo = 0, hi = n;
    while (hi - lo > 1) {
        const int step = (hi - lo + 31) / 32;
        const int p = lo + (int)lane_id() * step;
        const unsigned m = __ballot_sync(0xffffffffu, p < hi && off[p] <= e);   // lane 0 always passes
        lo += (31 - __clz(m)) * step;
        hi = min(hi, lo + step);
    }
    return lo;
}

// kDirect: the units are all quarters of the join's own grid, taken in turn by the CTAs; a unit's
// accepted pairs go to a bitmap instead of the emit buffers, and the few pairs the FP32 sum cannot decide
// are decided by the thread that finds them, in FP64 from the rows.  Of an upper join only the units with a
// pair above the diagonal (2 I and later of tile I) are counted, so that every CTA gets as many of them
// (dealt out with the others, some CTAs had none and some twice the mean: 18,918 x 4 423 -> 321 us, 4,634 x 192
// 461 -> 293).  R rows past the last one are zeros in shared memory and nothing else:
// as copies of it they sent every CTA to the same few lines of L2 (one row against 262,144 x 64: 1,284 us
// against 209 for 128 rows).
template <bool kDirect>
__global__ void __launch_bounds__(kPT, 2) plain_kernel(const PlainArgs a) {
    __shared__ __align__(16) float sm[kPStages][kPRows][kPLd];
    __shared__ PlainStage info[kPStages];
    __shared__ uint32_t ids[kPStages][kPRows];   // emitted row ids of the unit's rows and columns
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    // this CTA's run of all candidates' quarters, in candidate order: candidate e, quarter p, `left` units
    // (direct: e is the unit, left counts this CTA's)
    const unsigned nT = (a.dir.nR + kTileR - 1) / kTileR;
    const unsigned long long units = kDirect ? (unsigned long long)nT * (a.dir.cols64 - (a.dir.upper ? nT - 1 : 0u))
                                             : (unsigned long long)*a.total * kPUnits;
    const unsigned long long u0 = units * blockIdx.x / gridDim.x;
    unsigned left = kDirect ? (unsigned)(units > blockIdx.x ? (units - 1 - blockIdx.x) / gridDim.x + 1 : 0)
                            : (unsigned)(units * (blockIdx.x + 1) / gridDim.x - u0);
    uint32_t e = kDirect ? blockIdx.x : (uint32_t)(u0 / kPUnits);
    unsigned p = kDirect ? 0u : (unsigned)(u0 % kPUnits) * kPCols;
    if (!kDirect && a.run) {
        e = blockIdx.x * a.run;
        p = 0;
        left = e < *a.total ? min(a.run, *a.total - e) * kPUnits : 0u;
    }
    __shared__ WarpAppender apps[kPT / 32][2];   // accept and band of each warp: touched by hits only
    WarpAppender* app = apps[threadIdx.x >> 5];
    if (lane_id() < 2) app[lane_id()] = WarpAppender();
    __syncwarp();
    unsigned n_screen_acc = 0, n_items = 0;

    // issue side: the stage that comes next
    int k0 = 0;
    unsigned up_tile = 0, up_first = 0;   // upper direct joins: R tile of unit e, and its first unit
    uint32_t e_end = 0;   // first candidate beyond the R tile of the last one (0: no tile yet)
    bool fresh = true;    // candidate e's tiles are not taken yet
    uint4 rt = make_uint4(0, 0, 0, 0);
    // the S tile (first row, rows) of candidate e, and the next one's, whose two dependent loads are
    // issued a quarter apart so that neither is waited for
    uint2 stt = make_uint2(0, 0), stn = stt;
    uint32_t jn = 0;
    const uint32_t total = kDirect ? 0u : *a.total;
    bool self_join = false, first = true;
    float2 th = make_float2(0.f, 0.f);
    auto s_tile = [&](uint32_t j) { return *reinterpret_cast<const uint2*>(a.stiles + j); };
    const float *pr0 = nullptr, *pr1 = nullptr, *ps = nullptr;   // 16-byte copies: this thread's R and S elements
    const unsigned lr = threadIdx.x >> 2, lq = (threadIdx.x & 3) * 4;
    auto step = [&] {
        --left;
        if (kDirect) {
            e += gridDim.x;
            return;
        }
        p += kPCols;
        if (p == (unsigned)kTileS) {
            p = 0;
            ++e;
            fresh = true;
            if (a.run && left == 0) {   // the next run
                const unsigned long long at = (unsigned long long)e + (unsigned long long)(gridDim.x - 1) * a.run;
                if (at < total) {
                    e = (uint32_t)at;
                    left = min(a.run, total - e) * kPUnits;
                    first = true;
                }
            }
        }
    };
    auto issue = [&](int buf) {
        // the unit's tiles (units without a column, or at or below a self-join's diagonal, are passed over)
        if (kDirect && k0 == 0 && left) {
            unsigned I = e / a.dir.cols64, u = e - I * a.dir.cols64;
            if (a.dir.upper) {
                for (unsigned n; e - up_first >= (n = a.dir.cols64 - 2 * up_tile); ++up_tile) up_first += n;
                I = up_tile;
                u = e - up_first + 2 * up_tile;
            }
            rt = make_uint4(I * kTileR, min((unsigned)kTileR, a.dir.nR - I * kTileR), 0u, 0u);
            stt = make_uint2(u * kPCols, min((unsigned)kPCols, a.dir.nS - u * kPCols));
            th = a.dir.thr;
            const PlainClass& pc = a.cls[0];
            pr0 = pc.rx + (size_t)(rt.x + min(lr, rt.y - 1)) * pc.ld + lq;
            pr1 = pc.rx + (size_t)(rt.x + min(lr + 64, rt.y - 1)) * pc.ld + lq;
        }
        while (!kDirect && k0 == 0 && left) {
            if (fresh) {
                fresh = false;
                if (e >= e_end) {
                    const int I = find_rtile(a.off, a.ntR, e);
                    e_end = I + 1 < a.ntR ? a.off[I + 1] : 0xFFFFFFFFu;
                    rt = a.rtiles[I];
                    // rows past a tile's points repeat its last one, so no read leaves the side
                    const PlainClass& pc = a.cls[rt.w];
                    pr0 = pc.rx + (size_t)(rt.x + min(lr, rt.y - 1)) * pc.ld + lq;
                    pr1 = pc.rx + (size_t)(rt.x + min(lr + 64, rt.y - 1)) * pc.ld + lq;
                    self_join = a.jps[rt.z].self_join != 0;
                    th = a.thr[rt.z];
                }
                stt = stn;
                if (first) {
                    first = false;
                    stt = s_tile(a.jlist[e] & kJMask);
                    if (p != 0) jn = a.jlist[min(e + 1, total - 1)] & kJMask;
                }
            }
            if (p == 0) {
                ++n_items;
                jn = a.jlist[min(e + 1, total - 1)] & kJMask;
            }
            if (p == kTileS - kPCols) stn = s_tile(jn);
            if (p < stt.y && !(self_join && stt.x + p + kPCols <= rt.x + 1)) break;
            step();
        }
        if (!left) {
            if (threadIdx.x == 0) info[buf].kc = 0;
            cp_async_commit();
            return;
        }
        const unsigned c0 = stt.x + p, nvJ = min(stt.y - p, (unsigned)kPCols);
        const PlainClass& pc = a.cls[rt.w];
        const int d = pc.d, kc = min(kPK, d - k0);
        if (!kDirect || pc.vec) {
            if (k0 == 0) ps = pc.sx + (size_t)(c0 + min(lr, nvJ - 1)) * pc.ld + lq;
            if ((int)lq < kc) {
                if (kDirect) {
                    cp_async16_zfill(&sm[buf][lr][lq], pr0 + k0, lr < rt.y);
                    cp_async16_zfill(&sm[buf][lr + 64][lq], pr1 + k0, lr + 64 < rt.y);
                } else {
                    cp_async16(&sm[buf][lr][lq], pr0 + k0);
                    cp_async16(&sm[buf][lr + 64][lq], pr1 + k0);
                }
                cp_async16(&sm[buf][kTileR + lr][lq], ps + k0);
            }
        } else if (kc > kPK / 2) {   // rows of any alignment: element k of every 16th row
            const int k = threadIdx.x & (kPK - 1), r = threadIdx.x / kPK;
            const bool real = k < kc;
            const float* R = pc.rx + (size_t)rt.x * d + k0 + min(k, kc - 1);
            const float* S = pc.sx + (size_t)c0 * d + k0 + min(k, kc - 1);
#pragma unroll
            for (int i = 0; i < kTileR; i += kPT / kPK)
                cp_async4_zfill(&sm[buf][r + i][k], R + min((unsigned)(r + i), rt.y - 1) * (unsigned)d,
                                real && (unsigned)(r + i) < rt.y);
#pragma unroll
            for (int i = 0; i < kPCols; i += kPT / kPK)
                cp_async4_zfill(&sm[buf][kTileR + r + i][k], S + min((unsigned)(r + i), nvJ - 1) * (unsigned)d, real);
        } else {   // elements up to the next power of two, zero beyond kc
            const int lk = kc <= 2 ? 1 : kc <= 4 ? 2 : 3;
            for (int idx = threadIdx.x; idx < kPRows << lk; idx += kPT) {
                const int r = idx >> lk, k = idx & ((1 << lk) - 1);
                const float* row = r < kTileR ? pc.rx + (size_t)(rt.x + min((unsigned)r, rt.y - 1)) * d
                                              : pc.sx + (size_t)(c0 + min((unsigned)(r - kTileR), nvJ - 1)) * d;
                cp_async4_zfill(&sm[buf][r][k], row + k0 + min(k, kc - 1), k < kc && (r >= kTileR || (unsigned)r < rt.y));
            }
        }
        if (threadIdx.x == 0)
            info[buf] = PlainStage{rt.x, rt.y, c0, nvJ, rt.z, kc, k0 == 0, k0 + kc >= d, th};
        if (!kDirect && k0 + kc >= d && threadIdx.x < kPRows) {
            const unsigned t = threadIdx.x;
            cp_async4_zfill(&ids[buf][t], t < kTileR ? pc.r_emit + rt.x + min(t, rt.y - 1)
                                                     : pc.s_emit + c0 + min(t - kTileR, nvJ - 1), true);
        }
        k0 += kPK;
        if (k0 >= d) {
            k0 = 0;
            step();
        }
        cp_async_commit();
    };

    unsigned long long acc[kPI][kPJ];
    issue(0);
    issue(1);
    for (int buf = 0;; buf = buf == kPStages - 1 ? 0 : buf + 1) {
        cp_async_wait<1>();
        __syncthreads();   // this stage has landed and the one before it is no longer read
        const PlainStage in = info[buf];
        if (in.kc == 0) break;
        issue(buf == 0 ? kPStages - 1 : buf - 1);
        if (in.first) {
#pragma unroll
            for (int i = 0; i < kPI; ++i)
#pragma unroll
                for (int j = 0; j < kPJ; ++j) acc[i][j] = 0ull;
        }
        const float(&sR)[kPRows][kPLd] = sm[buf];
        const float(*sS)[kPLd] = sm[buf] + kTileR;
        const int quads = (in.kc + 1) >> 2;   // 3 left over: a whole quad (its last element is 0 on both sides)
        for (int q = 0; q < quads; ++q) {
            ulonglong2 sv[kPJ];
#pragma unroll
            for (int j = 0; j < kPJ; ++j) sv[j] = *reinterpret_cast<const ulonglong2*>(&sS[j * 16 + tx][q * 4]);
#pragma unroll
            for (int i = 0; i < kPI; ++i) {
                const ulonglong2 rv = *reinterpret_cast<const ulonglong2*>(&sR[i * 16 + ty][q * 4]);
#pragma unroll
                for (int j = 0; j < kPJ; ++j) {
                    sqdiff_x2(rv.x, sv[j].x, acc[i][j]);
                    sqdiff_x2(rv.y, sv[j].y, acc[i][j]);
                }
            }
        }
        if (in.kc > quads * 4) {   // one or two elements left over
            unsigned long long sv[kPJ];
#pragma unroll
            for (int j = 0; j < kPJ; ++j)
                sv[j] = *reinterpret_cast<const unsigned long long*>(&sS[j * 16 + tx][quads * 4]);
#pragma unroll
            for (int i = 0; i < kPI; ++i) {
                const unsigned long long rv = *reinterpret_cast<const unsigned long long*>(&sR[i * 16 + ty][quads * 4]);
#pragma unroll
                for (int j = 0; j < kPJ; ++j) sqdiff_x2(rv, sv[j], acc[i][j]);
            }
        }
        if (!in.last) continue;
        // classify the thread's 32 pairs: bit i * kPJ + j
        float v[kPI * kPJ];
#pragma unroll
        for (int b = 0; b < kPI * kPJ; ++b) v[b] = sum_x2(acc[b / kPJ][b % kPJ]);
        // least sum of each of the thread's rows: one vote while no pair is near the threshold, then the
        // rows that hold a near pair in some lane, and only their pairs one by one
        float rm[kPI];
#pragma unroll
        for (int i = 0; i < kPI; ++i) {
            rm[i] = fminf(fmin3(v[i * kPJ], v[i * kPJ + 1], v[i * kPJ + 2]), v[i * kPJ + 3]);
            if (kDirect && (unsigned)(i * 16 + ty) >= in.nvI) rm[i] = INFINITY;   // (no row: zeros)
        }
        const float m = fmin3(fmin3(rm[0], rm[1], rm[2]), fmin3(rm[3], rm[4], rm[5]), fminf(rm[6], rm[7]));
        const bool near = __any_sync(0xffffffffu, !(m > in.th.y));
        if (!kDirect && !near) continue;
        unsigned long long word = 0;   // direct: columns accepted in row tx * 16 + ty (tx < 8)
        unsigned rows = 0;
#pragma unroll
        for (int i = 0; i < kPI; ++i) rows |= rm[i] > in.th.y ? 0u : 1u << i;
        rows = near ? __reduce_or_sync(0xffffffffu, rows) : 0u;
        uint32_t cand = 0, amask = 0;
#pragma unroll
        for (int i = 0; i < kPI; ++i) {
            if (!(rows & (1u << i))) continue;
#pragma unroll
            for (int b = i * kPJ; b < (i + 1) * kPJ; ++b) {
                cand |= v[b] > in.th.y ? 0u : 1u << b;
                amask |= v[b] <= in.th.x ? 1u << b : 0u;
            }
        }
        // valid rows and columns of this thread
        const int ni = min(max((int)in.nvI - ty + 15, 0) >> 4, kPI), nj = min(max((int)in.nvJ - tx + 15, 0) >> 4, kPJ);
        const uint32_t rmask = ni == kPI ? 0xFFFFFFFFu : (1u << (kPJ * ni)) - 1u;
        cand &= rmask & (((1u << nj) - 1u) * 0x11111111u);
        const bool above = kDirect ? a.dir.upper != 0 : a.jps[in.join].self_join != 0;
        if (above && in.c0 <= in.r0 + kTileR - 1) {   // keep (sorted) column > (sorted) row only
            uint32_t w = cand;
            while (w) {
                const int b = __ffs(w) - 1;
                w &= w - 1;
                if (in.c0 + (b % kPJ) * 16 + tx <= in.r0 + (b / kPJ) * 16 + ty) cand &= ~(1u << b);
            }
        }
        amask &= cand;
        const uint32_t bmask = cand & ~amask;
        if (kDirect) {
            if (near) {
                uint32_t w = bmask;
                while (w) {   // the oracle's own sum
                    const int b = __ffs(w) - 1;
                    w &= w - 1;
                    const PlainClass& pc = a.cls[0];
                    if (a.dir.diagonal && in.r0 + (b / kPJ) * 16 + ty == in.c0 + (b % kPJ) * 16 + tx) {
                        amask |= 1u << b;
                        continue;
                    }
                    const bool ok = seq_d2(pc.rx + (size_t)(in.r0 + (b / kPJ) * 16 + ty) * pc.d,
                                           pc.sx + (size_t)(in.c0 + (b % kPJ) * 16 + tx) * pc.d, pc.d) <= a.dir.T;
                    if (ok) amask |= 1u << b;
                    atomicAdd(a.dir.band, 1ull);
                    if (ok) atomicAdd(a.dir.band + 1, 1ull);
                }
                __syncwarp();
#pragma unroll
                for (int i = 0; i < kPI; ++i) {
                    if (!(rows & (1u << i))) continue;
                    unsigned long long wi = 0;
#pragma unroll
                    for (int j = 0; j < kPJ; ++j) {
                        const unsigned bal = __ballot_sync(0xffffffffu, (amask >> (i * kPJ + j)) & 1u);
                        wi |= (unsigned long long)((bal >> (threadIdx.x & 16)) & 0xFFFFu) << (16 * j);
                    }
                    word = tx == i ? wi : word;
                }
            }
            const unsigned row = tx * 16 + ty;
            if (tx < kPI && row < in.nvI) {
                a.dir.bits[(size_t)(in.r0 + row) * a.dir.cols64 + in.c0 / kPCols] = word;
                if (word) atomicAdd(a.dir.cnt + in.r0 + row, (unsigned)__popcll(word));
            }
            continue;
        }
        const JoinParams& jp = a.jps[in.join];
        unsigned tot;
        const unsigned pre = warp_excl_scan(__popc(amask) | (__popc(bmask) << 16), tot);
        const unsigned ta = tot & 0xFFFFu, tb = tot >> 16;
        auto put = [&](uint32_t w, uint64_t* out, unsigned long long pos, unsigned long long cap) {
            while (w) {
                const int b = __ffs(w) - 1;
                w &= w - 1;
                const uint32_t oi = ids[buf][(b / kPJ) * 16 + ty], oj = ids[buf][kTileR + (b % kPJ) * 16 + tx];
                if (pos < cap) out[pos] = pair_key(jp, oi, oj);
                ++pos;
            }
        };
        auto reserve = [&](int which, unsigned n, unsigned long long* reserved, uint64_t* buf, unsigned long long cap) {
            WarpAppender ap = app[which];
            const unsigned long long pos = ap.reserve(n, reserved, buf, cap);
            __syncwarp();
            if (lane_id() == 0) app[which] = ap;
            __syncwarp();
            return pos;
        };
        if (ta) {
            put(amask, a.acc, reserve(0, ta, &a.ctr->acc_reserved, a.acc, a.acc_cap) + (pre & 0xFFFFu), a.acc_cap);
            n_screen_acc += __popc(amask);
        }
        if (tb)
            put(bmask, a.band, reserve(1, tb, &a.ctr->band_reserved, a.band, a.band_cap) + (pre >> 16), a.band_cap);
    }
    cp_async_wait<0>();
    if (kDirect) return;
    WarpAppender app_acc = app[0], app_band = app[1];
    app_acc.pad(a.acc, a.acc_cap);
    app_band.pad(a.band, a.band_cap);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n_screen_acc += __shfl_xor_sync(0xffffffffu, n_screen_acc, o);
    if (lane_id() == 0) {
        if (app_acc.valid) atomicAdd(&a.ctr->acc_valid, app_acc.valid);
        if (app_band.valid) atomicAdd(&a.ctr->band_valid, app_band.valid);
        if (n_screen_acc) atomicAdd(&a.ctr->screen_accept, (unsigned long long)n_screen_acc);
        if (threadIdx.x == 0 && n_items) atomicAdd(&a.ctr->items, (unsigned long long)n_items);
    }
}

// ------------------------------------------------------------------ FP64 refinement
struct RefineArgs {
    const uint64_t* band;
    unsigned long long band_cap;
    const JoinParams* jps;              // per join
    const unsigned long long* key_off;  // ascending key offset of each join
    int njoins;
    const void* const* rsrc;            // caller's rows of each join, original order
    const void* const* ssrc;
    uint64_t* acc;
    unsigned long long acc_cap;
    Counters* ctr;
    const float2* thr;                  // per join FP32-sum thresholds (the FP32 band stage)
    long long T_int;                    // int14 rows: exact integer distances against this
};

// FP32 sum of squared FP32 differences in four FMA chains (tree depth <= d / 4 + 2), the FP32
// band stage's value; certified against the FP64 oracle by fp32_sum_thresholds.
TJ_DEV float fp32_d2(const float* x, const float* y, int d) {
    float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
    if ((d & 3) == 0 && ((((uintptr_t)x) | ((uintptr_t)y)) & 15) == 0) {
        const float4* x4 = (const float4*)x;
        const float4* y4 = (const float4*)y;
        for (int k = 0; k < d / 4; ++k) {
            const float4 a = __ldg(x4 + k), b = __ldg(y4 + k);
            float t;
            t = a.x - b.x; a0 = fmaf(t, t, a0);
            t = a.y - b.y; a1 = fmaf(t, t, a1);
            t = a.z - b.z; a2 = fmaf(t, t, a2);
            t = a.w - b.w; a3 = fmaf(t, t, a3);
        }
    } else {
        for (int k = 0; k < d; ++k) {
            const float t = __ldg(x + k) - __ldg(y + k);
            a0 = fmaf(t, t, a0);
        }
    }
    return (a0 + a1) + (a2 + a3);
}

// Exact squared distance of two int16 rows in int64: each difference fits int32 and its square
// int64, so no order of the sum can round (the oracle's exact integer predicate).
TJ_DEV long long exact_d2_i16(const int16_t* x, const int16_t* y, int d) {
    long long acc = 0;
    auto add2 = [&](int a, int b) {   // two elements
        const int t0 = (int)(short)(a & 0xffff) - (int)(short)(b & 0xffff), t1 = (a >> 16) - (b >> 16);
        acc += (long long)t0 * t0 + (long long)t1 * t1;
    };
    const uintptr_t at = (uintptr_t)x | (uintptr_t)y;
    int k = 0;
    if ((at & 15) == 0) {
        for (; k + 16 <= d; k += 16) {
            const int4 a0 = __ldg((const int4*)(x + k)), a1 = __ldg((const int4*)(x + k + 8));
            const int4 b0 = __ldg((const int4*)(y + k)), b1 = __ldg((const int4*)(y + k + 8));
            add2(a0.x, b0.x), add2(a0.y, b0.y), add2(a0.z, b0.z), add2(a0.w, b0.w);
            add2(a1.x, b1.x), add2(a1.y, b1.y), add2(a1.z, b1.z), add2(a1.w, b1.w);
        }
    }
    if ((at & 7) == 0) {
        for (; k + 16 <= d; k += 16) {
            int2 a[4], b[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) a[u] = __ldg((const int2*)(x + k) + u), b[u] = __ldg((const int2*)(y + k) + u);
#pragma unroll
            for (int u = 0; u < 4; ++u) add2(a[u].x, b[u].x), add2(a[u].y, b[u].y);
        }
    }
    if ((at & 3) == 0) {
        for (; k + 8 <= d; k += 8) {
            int a[4], b[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) a[u] = __ldg((const int*)(x + k) + u), b[u] = __ldg((const int*)(y + k) + u);
#pragma unroll
            for (int u = 0; u < 4; ++u) add2(a[u], b[u]);
        }
    }
    for (; k + 4 <= d; k += 4) {
        int a[4], b[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) a[u] = __ldg(x + k + u), b[u] = __ldg(y + k + u);
#pragma unroll
        for (int u = 0; u < 4; ++u) acc += (long long)(a[u] - b[u]) * (a[u] - b[u]);
    }
    for (; k < d; ++k) {
        const int t = (int)__ldg(x + k) - (int)__ldg(y + k);
        acc += (long long)t * t;
    }
    return acc;
}

// Band pairs -> accept buffer.  kFp32: each pair is first decided, where it can be, by the
// certified FP32 sum (the FP32 band stage); only the rest pay the sequential FP64 terminal.
// kInt: int14 rows.  Their own instance: its wider loads want more registers than the FP64 sums, which lose by
// them (666,000 pairs of a 50,021 x 100 int14 join, rows of 200 bytes read by element: 198 us; by 8 bytes, 78 us;
// FP32 rows by whole sectors: 1M x 1M mixture 441 -> 519 us, so they keep to 16 bytes at a time).
template <bool kFp32, bool kInt>
__global__ void refine_kernel(const RefineArgs a) {
    const unsigned long long n = min(a.ctr->band_reserved, a.band_cap);
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    const unsigned long long start = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long n_acc = 0, n_fp64 = 0;
    // loop count is warp-uniform so the ballot below is well formed
    const unsigned long long warp_start = start & ~31ull;
    for (unsigned long long w = warp_start; w < n; w += stride) {
        const unsigned long long idx = w + lane_id();
        bool ok = false;
        uint64_t key = kSentinel;
        if (idx < n) {
            key = a.band[idx];
            if (key != kSentinel) {
                int lo = 0, hi = a.njoins - 1;   // join owning the key: last offset <= key
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (a.key_off[mid] <= key) lo = mid; else hi = mid - 1;
                }
                const JoinParams& jp = a.jps[lo];
                const uint64_t local = key - jp.key_off;
                const uint64_t i = local / (uint64_t)jp.n_cols, j = local - i * (uint64_t)jp.n_cols;
                if (i >= (uint64_t)jp.n_rows) {   // not a key the screen wrote: flagged, no row is read
                    atomicOr(&a.ctr->status, (unsigned long long)kStatusGuard);
                } else if (kInt) {   // int14 rows: the exact integer predicate decides every pair
                    const int16_t* xi = (const int16_t*)a.rsrc[lo] + (size_t)i * jp.d;
                    const int16_t* yi = (const int16_t*)a.ssrc[lo] + (size_t)j * jp.d;
                    ok = exact_d2_i16(xi, yi, jp.d) <= a.T_int;
                } else {
                const float* x = (const float*)a.rsrc[lo] + (size_t)i * jp.d;
                const float* y = (const float*)a.ssrc[lo] + (size_t)j * jp.d;
                bool decided = false;
                if (kFp32) {
                    const float s = fp32_d2(x, y, jp.d);
                    const float2 th = a.thr[lo];
                    if (s <= th.x) { ok = true; decided = true; }
                    else if (s > th.y) { decided = true; }
                }
                if (!decided) {
                    ok = seq_d2(x, y, jp.d) <= jp.T;
                    ++n_fp64;
                }
                }
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, ok);
        if (m) {
            unsigned long long base = 0;
            if (lane_id() == 0) base = atomicAdd(&a.ctr->acc_reserved, (unsigned long long)__popc(m));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (ok) {
                const unsigned long long pos = base + __popc(m & ((1u << lane_id()) - 1u));
                if (pos < a.acc_cap) a.acc[pos] = key;
            }
            n_acc += (lane_id() == 0) ? __popc(m) : 0;
        }
    }
    if (lane_id() == 0 && n_acc) {
        atomicAdd(&a.ctr->acc_valid, n_acc);
        atomicAdd(&a.ctr->refine_accept, n_acc);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n_fp64 += __shfl_xor_sync(0xffffffffu, n_fp64, o);
    if (lane_id() == 0 && n_fp64) atomicAdd(&a.ctr->band_fp64, n_fp64);
}

// ------------------------------------------------------------------ canonical output helpers
__global__ void expand_directed_kernel(const uint64_t* upper, unsigned long long slots, uint64_t* out, long long N) {
    const unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < slots) {
        const uint64_t k = upper[i];
        out[2 * i] = k;
        if (k == kSentinel) {
            out[2 * i + 1] = kSentinel;
        } else {
            const uint64_t lo = k / (uint64_t)N, hi = k - lo * (uint64_t)N;
            out[2 * i + 1] = hi * (uint64_t)N + lo;
        }
    }
    if (i < (unsigned long long)N) out[2 * slots + i] = i * (uint64_t)N + i;
}

__global__ void decode_kernel(const uint64_t* keys, long long n, long long n_cols, int64_t* io, int64_t* jo) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const uint64_t k = keys[t];
    const uint64_t i = k / (uint64_t)n_cols;
    io[t] = (int64_t)i;
    jo[t] = (int64_t)(k - i * (uint64_t)n_cols);
}

__global__ void decode_batched_kernel(const uint64_t* keys, long long n, const unsigned long long* key_off,
                                     const long long* n_cols, int njoins, int64_t* io, int64_t* jo) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const uint64_t k = keys[t];
    int lo = 0, hi = njoins - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (key_off[mid] <= k) lo = mid; else hi = mid - 1;
    }
    const uint64_t local = k - key_off[lo];
    const uint64_t i = local / (uint64_t)n_cols[lo];
    io[t] = (int64_t)i;
    jo[t] = (int64_t)(local - i * (uint64_t)n_cols[lo]);
}

// offsets[k] = first position of a key >= key_off[k] in the sorted keys; offsets[njoins] = n.
__global__ void batch_offsets_kernel(const uint64_t* keys, long long n, const unsigned long long* key_off,
                                     int njoins, long long* offsets) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k > njoins) return;
    if (k == njoins) { offsets[k] = n; return; }
    long long lo = 0, hi = n;
    const uint64_t v = key_off[k];
    while (lo < hi) {
        const long long mid = (lo + hi) >> 1;
        if (keys[mid] < v) lo = mid + 1; else hi = mid;
    }
    offsets[k] = lo;
}

}  // namespace

// Per join, thresholds on an FP32 sum s of the d squared FP32 differences (FMA accumulation, any
// summation tree of depth <= d + 2): s <= x certifies the FP64 oracle value <= T, s > y certifies
// it > T.  |s - D| <= gamma_{d+4} D + (d + 4) 2^-147 with u = 2^-24 (one rounding in each
// difference, one in each FMA or add along the tree, subnormal products absolutely).
static float2 fp32_sum_threshold(const JoinParams& jp) {
    const double u = 0x1p-24, nu = (double)(jp.d + 4) * u;
    const double gam = nu / (1.0 - nu);
    const double tiny = (double)(jp.d + 4) * 0x1p-147;
    const double tin = (jp.Tm - tiny) * (1.0 - gam) * (1.0 - 0x1p-30);
    const double tout = (jp.Tp + tiny) * (1.0 + gam) * (1.0 + 0x1p-30) + tiny;
    float fin = tin > 0 ? (float)tin : -1.f;   // nearest, then nudged to stay a lower bound
    if (fin > 0 && (double)fin > tin) fin = nextafterf(fin, 0.f);
    float fout = (float)tout;
    if ((double)fout < tout) fout = nextafterf(fout, INFINITY);
    return make_float2(fin, fout);
}
static void fp32_sum_thresholds(const ScreenInput& g, float2* dst, cudaStream_t st) {
    const JoinParams* hj = g.h_jps;
    if (!hj) fail(-1, "the FP32 thresholds need the host join parameters");
    std::vector<float2> th((size_t)g.njoins);
    for (int k = 0; k < g.njoins; ++k) th[k] = fp32_sum_threshold(hj[k]);
    upload(dst, th.data(), g.njoins * sizeof(float2), st);
}

namespace {

// Direct joins, before the distances: every element within `limit` in magnitude (NaN and infinities are
// not), and the row counts and band counters zeroed.  One flag per block, so that nothing needs to be
// zeroed for this kernel itself.
__global__ void __launch_bounds__(256) direct_check(const float* R, size_t nr, const float* S, size_t ns, float limit,
                                                    uint32_t* cnt, unsigned nR, unsigned long long* band,
                                                    uint32_t* bad) {
    const size_t stride = (size_t)gridDim.x * blockDim.x, t0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool ok = true;
    for (size_t i = t0; i < nr; i += stride) ok &= fabsf(R[i]) <= limit;
    for (size_t i = t0; i < ns; i += stride) ok &= fabsf(S[i]) <= limit;
    for (size_t i = t0; i < nR; i += stride) cnt[i] = 0;
    if (t0 < 2) band[t0] = 0;
    const int any = __syncthreads_or(!ok);
    if (threadIdx.x == 0) bad[blockIdx.x] = any ? 1u : 0u;
}

// Exclusive scan of the row counts by one block, and what the host reads: pairs, longest row, whether an
// element was out of range, and the band counters.
__global__ void __launch_bounds__(1024) direct_scan(uint32_t* cnt, unsigned nR, const uint32_t* bad, unsigned nbad,
                                                    const unsigned long long* band, unsigned long long* hdr) {
    __shared__ unsigned wt[32];
    unsigned flag = 0, longest = 0;
    for (unsigned i = threadIdx.x; i < nbad; i += 1024) flag |= bad[i];
    unsigned long long carry = 0;
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    constexpr unsigned kEach = 8;   // consecutive rows per thread
    for (unsigned t = 0; t < nR; t += 1024 * kEach) {
        unsigned v[kEach], sum = 0;
#pragma unroll
        for (unsigned k = 0; k < kEach; ++k) {
            const unsigned i = t + threadIdx.x * kEach + k;
            v[k] = i < nR ? cnt[i] : 0u;
            sum += v[k];
            longest = max(longest, v[k]);
        }
        unsigned tot, all;
        const unsigned pre = warp_excl_scan(sum, tot);
        __syncthreads();
        if (lane == 0) wt[warp] = tot;
        __syncthreads();
        const unsigned wpre = warp_excl_scan(wt[lane], all);
        const unsigned before = __shfl_sync(0xffffffffu, wpre, warp);
        unsigned run = (uint32_t)carry + before + pre;
#pragma unroll
        for (unsigned k = 0; k < kEach; ++k) {
            const unsigned i = t + threadIdx.x * kEach + k;
            run += v[k];
            if (i < nR) cnt[i] = run;   // the row's end
        }
        carry += all;
    }
    longest = __reduce_max_sync(0xffffffffu, longest);
    __syncthreads();
    if (lane == 0) wt[warp] = longest;
    const int any = __syncthreads_or(flag != 0);
    if (threadIdx.x == 0) {
        for (int w = 1; w < 32; ++w) longest = max(longest, wt[w]);
        hdr[0] = carry;
        hdr[1] = longest;
        hdr[2] = any ? 1 : 0;
        hdr[3] = band[0];
        hdr[4] = band[1];
    }
}

// Columns of every row in order, from the bitmap, 32 words at a time: kW = 1 warp per row, or a block, its
// warps on consecutive parts of the words (rows of kEmitWords words and more, where there are too few of them
// to fill the device: 16 dense rows of 2^20 columns 13.4 -> 11.0 ms in all).
constexpr unsigned kEmitWords = 512;
template <int kW>
__global__ void __launch_bounds__(256) direct_emit(const unsigned long long* bits, unsigned nR, unsigned cols64,
                                                   const uint32_t* row_end, uint32_t* cols) {
    const unsigned row = (blockIdx.x * 256 + threadIdx.x) / (32 * kW), lane = lane_id(), warp = threadIdx.x >> 5;
    if (row >= nR) return;   // uniform over the row's warps
    uint32_t pos = row ? row_end[row - 1] : 0u;
    const uint32_t end = row_end[row];
    unsigned first = 0, last = cols64;   // this warp's words
    if (kW > 1) {
        __shared__ unsigned before[kW];
        const unsigned part = (cols64 + kW - 1) / kW;
        first = min(warp * part, cols64);
        last = min(first + part, cols64);
        unsigned n = 0;
        for (unsigned u = first + lane; u < last; u += 32) n += (unsigned)__popcll(bits[(size_t)row * cols64 + u]);
        n = __reduce_add_sync(0xffffffffu, n);
        if (lane == 0) before[warp] = n;
        __syncthreads();
        for (unsigned w = 0; w < warp; ++w) pos += before[w];
    }
    for (unsigned u0 = first; u0 < last && pos < end; u0 += 32) {
        const unsigned u = u0 + lane;
        unsigned long long w = u < last ? bits[(size_t)row * cols64 + u] : 0ull;
        unsigned tot;
        uint32_t p = pos + warp_excl_scan((unsigned)__popcll(w), tot);
        for (; w; w &= w - 1) cols[p++] = u * 64 + (unsigned)__ffsll((long long)w) - 1;
        pos += tot;
    }
}

}  // namespace

bool join_direct(const float* R, unsigned nR, const float* S, unsigned nS, Mode mode, const JoinParams& jp, float limit,
                 DBuf<uint32_t>& rows, DBuf<uint32_t>& cols, unsigned long long (&hdr)[5], cudaStream_t st,
                 cudaEvent_t screen0, cudaEvent_t screen1) {
    // (R-S sides may share their first row and differ in length: only the mode says that S is R)
    const bool self = mode != kModeRS, upper = mode == kModeUpper;
    const unsigned cols64 = (nS + kPCols - 1) / kPCols;
    rows = DBuf<uint32_t>::result(nR, st);
    DBuf<unsigned long long> bits((size_t)nR * cols64, st), band(2 + 5, st);
    const size_t er = (size_t)nR * jp.d, es = self ? 0 : (size_t)nS * jp.d;
    const unsigned nb = (unsigned)std::min<size_t>((size_t)num_sms() * 2, (er + es + nR + 1023) / 1024);
    DBuf<uint32_t> bad(nb, st);
    if (upper) TJ_CUDA(cudaMemsetAsync(bits.p, 0, bits.bytes(), st));   // units below the diagonal are passed over
    launch(direct_check, nb, 256, 0, st, R, er, S, es, limit, rows.p, nR, band.p, bad.p);
    PlainArgs a;
    memset(&a, 0, sizeof(a));
    a.cls[0] = PlainClass{R, S, nullptr, nullptr, jp.d, jp.d,
                          jp.d % 4 == 0 && ((((uintptr_t)R) | ((uintptr_t)S)) & 15) == 0 ? 1 : 0};
    a.dir = DirectArgs{nR, nS, cols64, upper ? 1 : 0, mode == kModeDirected ? 1 : 0, bits.p, rows.p, band.p, jp.T, fp32_sum_threshold(jp)};
    const unsigned nT = (nR + kTileR - 1) / kTileR, units = nT * (cols64 - (upper ? nT - 1 : 0u));
    cudaEventRecord(screen0, st);
    launch(plain_kernel<true>, std::min(units, (unsigned)num_sms() * 2), kPT, 0, st, a);
    cudaEventRecord(screen1, st);
    launch(direct_scan, 1, 1024, 0, st, rows.p, nR, (const uint32_t*)bad.p, nb, (const unsigned long long*)band.p,
           band.p + 2);
    TJ_CUDA(cudaMemcpyAsync(hdr, band.p + 2, sizeof(hdr), cudaMemcpyDeviceToHost, st));
    TJ_CUDA(cudaStreamSynchronize(st));
    if (hdr[2]) {
        rows.reset();
        return false;
    }
    cols = DBuf<uint32_t>::result(std::max<size_t>((size_t)hdr[0], 1), st);
    if (hdr[0] && cols64 >= kEmitWords && nR <= (unsigned)num_sms() * 8)
        launch(direct_emit<8>, nR, 256, 0, st, (const unsigned long long*)bits.p, nR, cols64, (const uint32_t*)rows.p,
               cols.p);
    else if (hdr[0])
        launch(direct_emit<1>, (nR + 7) / 8, 256, 0, st, (const unsigned long long*)bits.p, nR, cols64,
               (const uint32_t*)rows.p, cols.p);
    return true;
}

void screen_plain(const ScreenInput& g, const EmitBuffers& eb, cudaStream_t st) {
    PlainArgs a;
    memset(&a, 0, sizeof(a));
    for (int c = 0; c < g.ncls; ++c) {
        const Side& R = *g.R[c];
        const Side& S = *g.S[c];
        if (R.screen != kScreenPlain || S.screen != kScreenPlain) fail(-1, "screen_plain needs FP32 sides");
        a.cls[c].rx = R.xs.p;
        a.cls[c].sx = S.xs.p;
        a.cls[c].r_emit = R.emit;
        a.cls[c].s_emit = S.emit;
        a.cls[c].d = R.d;
        a.cls[c].ld = plain_ld(R.d);
        a.cls[c].vec = 1;
    }
    DBuf<float2> dth((size_t)g.njoins, st);
    fp32_sum_thresholds(g, dth.p, st);
    a.off = g.cand->off.p;
    a.total = g.cand->dev_counts.p;
    a.ntR = g.ntR_total;
    a.jlist = g.cand->jlist.p;
    a.rtiles = g.rtiles;
    a.stiles = g.stiles;
    a.jps = g.jps;
    a.thr = dth.p;
    a.acc = eb.acc;
    a.acc_cap = eb.acc_cap;
    a.band = eb.band;
    a.band_cap = eb.band_cap;
    a.ctr = eb.ctr;
    // Rows of one length: an even cut of the candidates.  Batches of several lengths, whose candidates cost up
    // to 16 times each other's and come class by class: short runs in turn, so that every CTA has its share of
    // each class (400 joins of up to 65,536 rows, d = 32 and 128: 131 -> 82 ms; under the even cut the CTAs with
    // the long rows came last).
    a.run = g.ncls > 1 ? 4 : 0;
    launch(plain_kernel<false>, num_sms() * 2, kPT, 0, st, a);
}

void refine_band(const ScreenInput& g, const EmitBuffers& eb, bool fp32_stage, cudaStream_t st) {
    RefineArgs a;
    a.band = eb.band;
    a.band_cap = eb.band_cap;
    a.jps = g.jps;
    a.key_off = g.key_off;
    a.njoins = g.njoins;
    a.rsrc = g.rsrc;
    a.ssrc = g.ssrc;
    a.acc = eb.acc;
    a.acc_cap = eb.acc_cap;
    a.ctr = eb.ctr;
    a.thr = nullptr;
    const bool is_int = g.R[0]->dtype == kI16;
    a.T_int = g.T_int;
    if (is_int && g.njoins != 1) fail(-7, "int16 band refinement runs one join at a time");
    if (is_int) {
        launch(refine_kernel<false, true>, num_sms() * 8, 256, 0, st, a);
    } else if (fp32_stage) {
        DBuf<float2> dth((size_t)g.njoins, st);
        fp32_sum_thresholds(g, dth.p, st);
        a.thr = dth.p;
        launch(refine_kernel<true, false>, num_sms() * 8, 256, 0, st, a);
    } else {
        launch(refine_kernel<false, false>, num_sms() * 8, 256, 0, st, a);
    }
}

void expand_directed(const uint64_t* upper, unsigned long long slots, uint64_t* out, long long N, cudaStream_t st) {
    const unsigned long long n = slots > (unsigned long long)N ? slots : (unsigned long long)N;
    if (n == 0) return;
    launch(expand_directed_kernel, (unsigned)((n + 255) / 256), 256, 0, st, upper, slots, out, N);
    TJ_CUDA(cudaGetLastError());
}

void decode_pairs_batched(const uint64_t* keys, long long n, const unsigned long long* key_off,
                          const long long* n_cols, int njoins, int64_t* i_out, int64_t* j_out, cudaStream_t st) {
    if (n <= 0) return;
    launch(decode_batched_kernel, (unsigned)((n + 255) / 256), 256, 0, st, keys, n, key_off, n_cols, njoins, i_out,
           j_out);
}

void batch_offsets(const uint64_t* keys, long long n, const unsigned long long* key_off, int njoins,
                   long long* offsets, cudaStream_t st) {
    launch(batch_offsets_kernel, (unsigned)((njoins + 1 + 255) / 256), 256, 0, st, keys, n, key_off, njoins, offsets);
}

void decode_pairs(const uint64_t* keys, long long n, long long n_cols, int64_t* i_out, int64_t* j_out,
                  cudaStream_t st) {
    if (n <= 0) return;
    launch(decode_kernel, (unsigned)((n + 255) / 256), 256, 0, st, keys, n, n_cols, i_out, j_out);
    TJ_CUDA(cudaGetLastError());
}

}  // namespace tj
