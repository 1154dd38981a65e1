// Exact int14 screen on the tensor cores (tcgen05 kind::i8, sm_100a).
//
// Every int14 coordinate q in [-8192, 8191] is split into two signed int8 limbs
// q = 128 h + l, h = floor((q + 64) / 128) in [-64, 64], l in [-64, 63].  For a tile
// pair the kernel accumulates, exactly in INT32 TMEM accumulators,
//     hh = sum h h',   x = sum (h l' + l h'),   ll = sum l l'
// (|hh|, |ll| <= 4096 d, |x| <= 8192 d: no INT32 overflow for any order) and
// recombines q.q' = 16384 hh + 128 x + ll in INT64, so d2 = |q|^2 + |q'|^2 - 2 q.q'
// and the predicate d2 <= T are exact: there is no band and no refinement.
// This is the reference's limb decomposition and exact recombination
// (src/g9_tc_kernels.py:45-66 limb_dot; NUMERICS_G9_INT14.md:5-18), applied to the
// whole screen instead of a refinement subset.
//
// Fast path: q.q' <= 16384 hh + M with M >= |128 x + ll|.  By Cauchy-Schwarz on the limb vectors,
// |x| <= |h||l'| + |l||h'| and |ll| <= |l||l'|, so per (row i, S tile J)
//     M_iJ = 128 (|h_i| L_J + |l_i| H_J) + |l_i| L_J,   H_J, L_J = tile maxima of |h'|, |l'|
// (FP32 upper bounds of the norms, the sum taken in FP64 and rounded up to an integer), and a pair
// is certainly out when 32768 hh + 2 M_iJ < |q|^2 + |q'|^2 - T.  With
// a_iJ = floor((|q_i|^2 - T - 2 M_iJ) / 2^15) and b_j = floor(|q_j|^2 / 2^15) this is the integer
// test  hh - b_j < a_iJ  (two INT32 ops per pair).  Pairs failing it read x and ll and take the
// exact INT64 test.  (The data-independent bound M = d (128 * 8192 + 4096) is ~3x looser on
// uniform int14 rows and sent ~10x more pairs to the exact test.)
//
// TMEM: hh double-buffered (columns 0..255), x and ll single (256..511).  The hh products of an
// item are committed on their own barrier, and the epilogue's fast path (hh only) runs first; each
// epilogue warp then says whether any of its pairs needs the exact test, and with one k-block per
// item (d <= 128) the UMMA issuer computes x / ll only for items where one does (after issuing the
// next item's hh products), so most items cost one limb product instead of four.  With several
// k-blocks x / ll are computed with hh.
// Warp roles (320 threads): warp 0 TMA producer, warp 1 UMMA issuer, warps 2..9 epilogue
// (warp w reads TMEM lanes 32*(w%4).. and columns 64*((w-2)/4)..).
#include <algorithm>
#include <cstddef>

#include <climits>

#include "tj_emit.cuh"
#include "tj_internal.h"

namespace tj {

namespace {

constexpr int kI8Stages = 3;
constexpr int kI8Epi = 8;
constexpr int kI8Threads = (2 + kI8Epi) * 32;
constexpr int kI8N = 128;                        // S tile rows (UMMA N)
constexpr unsigned kPart = 128u * 128u;          // one 128-row x 128-byte swizzled box (16 KB)
constexpr unsigned kI8Stage = 4 * kPart;         // A_h, A_l, B_h, B_l
constexpr unsigned kColHH0 = 0, kColX = 256, kColLL = 384;

constexpr int kI8Meta = 3;

// Column metadata of one 128-row S tile, loaded with one bulk copy per item.
struct ColMetaI8 {
    int bq[kI8N];           // floor(|q_j|^2 / 2^15); 2^30 for rows beyond the tile's points
    uint32_t perm[kI8N];    // original row id
    long long norm[kI8N];   // exact |q_j|^2
    int gminb[kI8N / 8];    // per 8-column group: min of bq (the group-wise fast test)
    uint32_t c0, nvJ;
    float HJ, LJ;           // >= max |h'|, max |l'| over the tile's rows
};
static_assert(sizeof(ColMetaI8) % 16 == 0, "bulk copies need 16-byte multiples");
static_assert(offsetof(ColMetaI8, gminb) % 16 == 0, "group minima are read four at a time");

struct I8Ctl {
    uint64_t full[kI8Stages];
    uint64_t empty[kI8Stages];
    uint64_t acc_full[2];
    uint64_t hh_empty[2];
    uint64_t xl_empty;
    uint64_t xl_full;      // x and ll of the current item are in TMEM (or were skipped)
    uint64_t xl_dec;       // every epilogue warp has said whether it needs x and ll of the item
    uint64_t meta_full[kI8Meta];
    uint64_t meta_empty[kI8Meta];
    uint64_t drain;
    unsigned tmem_base;
    int abort_flag;
    int need[2];           // item parity: some epilogue warp needs x and ll
};

constexpr size_t kI8Smem = 1024 + (size_t)kI8Stages * kI8Stage + kI8Meta * sizeof(ColMetaI8) + sizeof(I8Ctl);

struct I8Args {
    const uint4* chunks;
    const uint32_t* nchunks;
    const uint32_t* jlist;
    const uint32_t* r_row0;
    const uint32_t* r_nvalid;
    const uint32_t* r_perm;
    const long long* r_norm;   // exact |q|^2
    const float* r_hn;         // >= |h| per row
    const float* r_ln;         // >= |l| per row
    const uint32_t* s_row0;
    const ColMetaI8* s_meta;
    int kblocks;               // kpad / 128
    int kpad;
    unsigned idesc;
    long long T;               // integer threshold
    JoinParams jp;
    uint64_t* acc;
    unsigned long long acc_cap;
    Counters* ctr;
    unsigned long long wait_ns;   // limit of every pipeline wait (drains keep kDrainLimitNs)
};

TJ_DEV int floor_shift15(long long v) { return (int)(v >> 15); }   // arithmetic shift = floor division
// a_iJ = floor(v / 2^15) clamped to [-2^30, 2^31 - 1]: |hh - b_j| < 2^30 for every d the screen takes,
// so the clamp never turns a candidate into a rejection (a huge T makes every real pair a candidate)
TJ_DEV int clamp_shift15(long long v) {
    const long long f = v >> 15;
    return f < -(1ll << 30) ? -(1 << 30) : f > 0x7FFFFFFFll ? 0x7FFFFFFF : (int)f;
}
// columns of a 32-column block at and beyond the tile's valid count carry no point
TJ_DEV uint32_t valid_cols(unsigned nv, unsigned cc) {
    return nv >= cc + 32 ? 0xFFFFFFFFu : nv > cc ? ((1u << (nv - cc)) - 1u) : 0u;
}

// r[k] for a runtime k without local memory (fixed 31-select tree).
TJ_DEV uint32_t pick32(const uint32_t (&r)[32], int k) {
    uint32_t a16[16], a8[8], a4[4], a2[2];
#pragma unroll
    for (int i = 0; i < 16; ++i) a16[i] = (k & 16) ? r[i + 16] : r[i];
#pragma unroll
    for (int i = 0; i < 8; ++i) a8[i] = (k & 8) ? a16[i + 8] : a16[i];
#pragma unroll
    for (int i = 0; i < 4; ++i) a4[i] = (k & 4) ? a8[i + 4] : a8[i];
#pragma unroll
    for (int i = 0; i < 2; ++i) a2[i] = (k & 2) ? a4[i + 2] : a4[i];
    return (k & 1) ? a2[1] : a2[0];
}

TJ_DEV uint32_t pick16(const uint32_t* r, int k) {   // r: 16 registers
    uint32_t a8[8], a4[4], a2[2];
#pragma unroll
    for (int i = 0; i < 8; ++i) a8[i] = (k & 8) ? r[i + 8] : r[i];
#pragma unroll
    for (int i = 0; i < 4; ++i) a4[i] = (k & 4) ? a8[i + 4] : a8[i];
#pragma unroll
    for (int i = 0; i < 2; ++i) a2[i] = (k & 2) ? a4[i + 2] : a4[i];
    return (k & 1) ? a2[1] : a2[0];
}

__global__ void __launch_bounds__(kI8N) build_col_meta_i8(const uint32_t* row0, const uint32_t* nvalid,
                                                         const uint32_t* perm, const long long* norm,
                                                         const float* maxH, const float* maxL, ColMetaI8* out) {
    const unsigned J = blockIdx.x, t = threadIdx.x;
    const unsigned c0 = row0[J], nv = nvalid[J];
    ColMetaI8& m = out[J];
    const bool ok = t < nv;
    const int bq = ok ? floor_shift15(norm[c0 + t]) : 0x40000000;
    m.bq[t] = bq;
    int gb = bq;   // min over the 8 columns t & ~7 .. (t | 7)
    gb = min(gb, __shfl_xor_sync(0xffffffffu, gb, 1));
    gb = min(gb, __shfl_xor_sync(0xffffffffu, gb, 2));
    gb = min(gb, __shfl_xor_sync(0xffffffffu, gb, 4));
    if ((t & 7) == 0) m.gminb[t >> 3] = gb;
    m.perm[t] = ok ? perm[c0 + t] : 0u;
    m.norm[t] = ok ? norm[c0 + t] : 0ll;
    if (t == 0) { m.c0 = c0; m.nvJ = nv; m.HJ = maxH[J]; m.LJ = maxL[J]; }
}

__global__ void __launch_bounds__(kI8Threads, 1)
    screen_i8_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                     const I8Args a) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    ColMetaI8* meta = (ColMetaI8*)(smem + (size_t)kI8Stages * kI8Stage);
    I8Ctl* ctl = (I8Ctl*)(meta + kI8Meta);
    const unsigned warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned long long* status = &a.ctr->status;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kI8Stages; ++s) {
            mbar_init(&ctl->full[s], 1);
            mbar_init(&ctl->empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&ctl->acc_full[b], 1);
            mbar_init(&ctl->hh_empty[b], kI8Epi);
        }
        mbar_init(&ctl->xl_empty, kI8Epi);
        mbar_init(&ctl->xl_full, 1);
        mbar_init(&ctl->xl_dec, kI8Epi);
        ctl->need[0] = ctl->need[1] = 0;
        for (int m = 0; m < kI8Meta; ++m) {
            mbar_init(&ctl->meta_full[m], 1);
            mbar_init(&ctl->meta_empty[m], kI8Epi);
        }
        mbar_init(&ctl->drain, 1);
        ctl->abort_flag = 0;
        fence_barrier_init();
        prefetch_tmap(&tmA);
        prefetch_tmap(&tmB);
    }
    if (warp == 1) tmem_alloc(&ctl->tmem_base, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = ctl->tmem_base;
    const unsigned nchunks = *a.nchunks;

    if (warp == 0) {
        if (lane == 0) {
            unsigned stage = 0, phase = 0;
            unsigned long long n = 0;
            bool ok = true;
            for (unsigned c = blockIdx.x; c < nchunks && ok; c += gridDim.x) {
                const uint4 ch = a.chunks[c];
                const int rrow = (int)a.r_row0[ch.x];
                for (unsigned e = ch.y; e < ch.z && ok; ++e, ++n) {
                    const unsigned J = a.jlist[e];
                    const int srow = (int)a.s_row0[J];
                    const unsigned slot = (unsigned)(n % kI8Meta), mph = (unsigned)((n / kI8Meta) & 1);
                    if (!mbar_wait(&ctl->meta_empty[slot], mph ^ 1, status, a.wait_ns)) { ok = false; break; }
                    mbar_arrive_expect_tx(&ctl->meta_full[slot], (unsigned)sizeof(ColMetaI8));
                    bulk_load(&meta[slot], a.s_meta + J, (unsigned)sizeof(ColMetaI8), &ctl->meta_full[slot]);
                    for (int kb = 0; kb < a.kblocks; ++kb) {
                        if (!mbar_wait(&ctl->empty[stage], phase ^ 1, status, a.wait_ns)) { ok = false; break; }
                        if (*(volatile int*)&ctl->abort_flag) { ok = false; break; }
                        uint8_t* st = smem + (size_t)stage * kI8Stage;
                        mbar_arrive_expect_tx(&ctl->full[stage], kI8Stage);
                        tma_load_2d(st, &tmA, &ctl->full[stage], kb * 128, rrow);
                        tma_load_2d(st + kPart, &tmA, &ctl->full[stage], a.kpad + kb * 128, rrow);
                        tma_load_2d(st + 2 * kPart, &tmB, &ctl->full[stage], kb * 128, srow);
                        tma_load_2d(st + 3 * kPart, &tmB, &ctl->full[stage], a.kpad + kb * 128, srow);
                        if (++stage == kI8Stages) { stage = 0; phase ^= 1; }
                    }
                }
            }
            if (!ok) ctl->abort_flag = 1;
            for (int s = 0; s < kI8Stages; ++s) {
                const unsigned ph = ((unsigned)s < stage) ? phase : (phase ^ 1u);
                mbar_wait(&ctl->full[s], ph, status, kDrainLimitNs);
            }
            for (int s = 0; s < kI8Meta; ++s) {
                if (n <= (unsigned long long)s) continue;
                const unsigned long long last = ((n - 1 - s) / kI8Meta) * kI8Meta + s;
                mbar_wait(&ctl->meta_full[s], (unsigned)((last / kI8Meta) & 1), status, kDrainLimitNs);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            unsigned stage = 0, phase = 0;
            unsigned long long n = 0;   // item counter of this CTA
            bool ok = true;
            // One k-block per item (d <= 128): the x / ll products are issued lazily, only when an
            // epilogue warp's fast test leaves a pair for the exact test.  The item's operand stage
            // is held until that decision, which is taken after the next item's hh products are
            // issued, so the tensor pipe keeps working meanwhile.  Several k-blocks: x / ll are
            // issued with hh (their stages cannot all be held).
            const bool lazy = a.kblocks == 1;
            bool pending = false;
            unsigned long long pn = 0;
            unsigned pstage = 0;
            unsigned long long n_xl = 0;   // items that took the low-limb products
            auto resolve = [&](unsigned long long mi, unsigned si) -> bool {
                if (!mbar_wait(&ctl->xl_dec, (unsigned)(mi & 1), status, a.wait_ns)) return false;
                volatile int* need = &ctl->need[mi & 1];
                const int needed = *need;
                *need = 0;   // the item two ahead writes it only after this resolve (acc_full order)
                if (needed) {
                    ++n_xl;
                    tc_fence_after();
                    const uint8_t* st = smem + (size_t)si * kI8Stage;
                    const uint8_t *Ah = st, *Al = st + kPart, *Bh = st + 2 * kPart, *Bl = st + 3 * kPart;
                    const unsigned t_x = tmem + kColX, t_ll = tmem + kColLL;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        umma_i8(t_x, desc_sw128(Ah, k * 32), desc_sw128(Bl, k * 32), a.idesc, k != 0);
                        umma_i8(t_x, desc_sw128(Al, k * 32), desc_sw128(Bh, k * 32), a.idesc, 1u);
                        umma_i8(t_ll, desc_sw128(Al, k * 32), desc_sw128(Bl, k * 32), a.idesc, k != 0);
                    }
                }
                umma_commit(&ctl->xl_full);
                umma_commit(&ctl->empty[si]);
                return true;
            };
            for (unsigned c = blockIdx.x; c < nchunks && ok; c += gridDim.x) {
                const uint4 ch = a.chunks[c];
                for (unsigned e = ch.y; e < ch.z && ok; ++e, ++n) {
                    const unsigned b = (unsigned)(n & 1);
                    const unsigned use = (unsigned)((n >> 1) & 1);   // parity of this buffer's use
                    if (!mbar_wait(&ctl->hh_empty[b], use ^ 1, status, a.wait_ns)) { ok = false; break; }
                    tc_fence_after();
                    const unsigned t_hh = tmem + kColHH0 + b * 128, t_x = tmem + kColX, t_ll = tmem + kColLL;
                    if (lazy) {
                        if (!mbar_wait(&ctl->full[stage], phase, status, a.wait_ns)) { ok = false; break; }
                        if (*(volatile int*)&ctl->abort_flag) { ok = false; break; }
                        tc_fence_after();
                        const uint8_t* st = smem + (size_t)stage * kI8Stage;
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            umma_i8(t_hh, desc_sw128(st, k * 32), desc_sw128(st + 2 * kPart, k * 32), a.idesc, k != 0);
                        umma_commit(&ctl->acc_full[b]);
                        if (pending && !resolve(pn, pstage)) { ok = false; break; }
                        pending = true;
                        pn = n;
                        pstage = stage;
                        if (++stage == kI8Stages) { stage = 0; phase ^= 1; }
                        continue;
                    }
                    for (int kb = 0; kb < a.kblocks; ++kb) {
                        if (!mbar_wait(&ctl->full[stage], phase, status, a.wait_ns)) { ok = false; break; }
                        if (*(volatile int*)&ctl->abort_flag) { ok = false; break; }
                        tc_fence_after();
                        const uint8_t* st = smem + (size_t)stage * kI8Stage;
                        const uint8_t *Ah = st, *Al = st + kPart, *Bh = st + 2 * kPart, *Bl = st + 3 * kPart;
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            umma_i8(t_hh, desc_sw128(Ah, k * 32), desc_sw128(Bh, k * 32), a.idesc, (kb | k) != 0);
                        // hh is complete after the last k-block's hh products: release it to the
                        // epilogue now, so its fast path overlaps this item's x / ll products
                        if (kb == a.kblocks - 1) umma_commit(&ctl->acc_full[b]);
                        if (kb == 0) {   // x / ll of the previous item must have been read
                            if (!mbar_wait(&ctl->xl_empty, (unsigned)(n & 1) ^ 1u, status, a.wait_ns)) { ok = false; break; }
                            tc_fence_after();
                        }
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            umma_i8(t_x, desc_sw128(Ah, k * 32), desc_sw128(Bl, k * 32), a.idesc, (kb | k) != 0);
                            umma_i8(t_x, desc_sw128(Al, k * 32), desc_sw128(Bh, k * 32), a.idesc, 1u);
                            umma_i8(t_ll, desc_sw128(Al, k * 32), desc_sw128(Bl, k * 32), a.idesc, (kb | k) != 0);
                        }
                        umma_commit(&ctl->empty[stage]);
                        if (++stage == kI8Stages) { stage = 0; phase ^= 1; }
                    }
                    if (!ok) break;
                    umma_commit(&ctl->xl_full);
                }
            }
            if (ok && pending) ok = resolve(pn, pstage);
            if (!lazy) n_xl = n;
            if (n_xl) atomicAdd(&a.ctr->xl_items, n_xl);
            if (!ok) ctl->abort_flag = 1;
            umma_commit(&ctl->drain);
            mbar_wait(&ctl->drain, 0, status, kDrainLimitNs);
        }
    } else {
        const unsigned ew = warp - 2;                 // 0..7
        const unsigned q = warp & 3;                  // TMEM lane quarter
        const unsigned half = ew >> 2;                // column half (0: 0..63, 1: 64..127)
        const unsigned row = q * 32 + lane;
        const JoinParams& jp = a.jp;
        WarpAppender app;
        unsigned long long n = 0, n_acc = 0, n_rare = 0, n_items = 0;
        bool ok = true;
        for (unsigned c = blockIdx.x; c < nchunks && ok; c += gridDim.x) {
            const uint4 ch = a.chunks[c];
            const unsigned I = ch.x;
            const unsigned r0 = a.r_row0[I];
            const bool rvalid = row < a.r_nvalid[I];
            const unsigned rs = r0 + row;
            const long long Ai = rvalid ? a.r_norm[rs] : 0;
            const double hi_n = rvalid ? (double)a.r_hn[rs] : 0.0, li_n = rvalid ? (double)a.r_ln[rs] : 0.0;
            const uint32_t oi = rvalid ? a.r_perm[rs] : 0u;
            for (unsigned e = ch.y; e < ch.z; ++e, ++n) {
                const unsigned b = (unsigned)(n & 1);
                const unsigned slot = (unsigned)(n % kI8Meta), mph = (unsigned)((n / kI8Meta) & 1);
                {   // warp-uniform: the TMEM loads below are warp-collective
                    const bool got = mbar_wait(&ctl->meta_full[slot], mph, status, a.wait_ns) &&
                                     mbar_wait(&ctl->acc_full[b], (unsigned)((n >> 1) & 1), status, a.wait_ns);
                    if (!__all_sync(0xffffffffu, got)) { ok = false; break; }
                }
                tc_fence_after();
                const ColMetaI8& m = meta[slot];
                const unsigned c0 = m.c0;
                // a_iJ with M_iJ >= |128 x + ll| for this row and S tile (every term non-negative;
                // the 2^-40 factor and +2 cover the FP64 rounding of the sum and of the ceil)
                int ai = 0x7FFFFFFF;
                if (rvalid) {
                    const double HJ = m.HJ, LJ = m.LJ;
                    const double Md = (128.0 * (hi_n * LJ + li_n * HJ) + li_n * LJ) * (1.0 + 0x1p-40) + 2.0;
                    const long long M = (long long)ceil(Md);
                    ai = clamp_shift15(Ai - a.T - 2 * M);
                }
                const unsigned lane_off = (q * 32u) << 16;
                const unsigned col0 = half * 64;
                uint32_t cms[2] = {0u, 0u};   // pairs left for the exact test, per 32-column block
                uint32_t hv2[2][32];          // both blocks' hh loads in flight together
                tmem_ld32(tmem + lane_off + kColHH0 + b * 128 + col0, hv2[0]);
                tmem_ld32(tmem + lane_off + kColHH0 + b * 128 + col0 + 32, hv2[1]);
                tmem_ld_wait();
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const unsigned cc = col0 + h * 32;
                    const uint32_t (&hv)[32] = hv2[h];
                    // fast path, one integer test per 8-column group: hh_j - b_j <= max hh - min b, so
                    // max hh - min b < a_iJ proves every pair of the group out (seven maxes and one
                    // subtract per 8 pairs); only the groups that reach the threshold (in any lane) are
                    // examined pair by pair
                    const int4 gb = *reinterpret_cast<const int4*>(&m.gminb[cc >> 3]);
                    const int gbv[4] = {gb.x, gb.y, gb.z, gb.w};
                    int vx[4];
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        const uint32_t* h8 = hv + 8 * g;
                        const int m01 = max((int)h8[0], (int)h8[1]), m23 = max((int)h8[2], (int)h8[3]);
                        const int m45 = max((int)h8[4], (int)h8[5]), m67 = max((int)h8[6], (int)h8[7]);
                        vx[g] = max(max(m01, m23), max(m45, m67)) - gbv[g];
                    }
                    const unsigned gmask = (vx[0] >= ai ? 1u : 0u) | (vx[1] >= ai ? 2u : 0u) |
                                           (vx[2] >= ai ? 4u : 0u) | (vx[3] >= ai ? 8u : 0u);
                    const unsigned gunion = __reduce_or_sync(0xffffffffu, gmask);
                    if (!gunion) continue;
                    uint32_t cmask = 0;
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        if (!(gunion & (1u << g))) continue;
                        if (gmask & (1u << g)) {
#pragma unroll
                            for (int k = 8 * g; k < 8 * g + 8; ++k)
                                cmask |= ((int)hv[k] - m.bq[cc + k] >= ai ? 1u : 0u) << k;
                        }
                    }
                    cmask &= valid_cols(m.nvJ, cc);
                    if (jp.self_join && cmask) {   // keep sorted column > sorted row only
                        const int lim = (int)rs - (int)(c0 + cc);
                        if (lim >= 31) cmask = 0;
                        else if (lim >= 0) cmask &= ~((2u << lim) - 1u);
                    }
                    cms[h] = cmask;
                }
                // tell the MMA issuer whether this item's x / ll products are needed at all (it skips
                // them when no warp needs them), then wait for them, or for the skip, in every warp:
                // each epilogue warp observes every phase of xl_full, so the parity names this item
                const bool any = __any_sync(0xffffffffu, (cms[0] | cms[1]) != 0);
                if (lane == 0) {
                    if (any) atomicOr(&ctl->need[n & 1], 1);
                    mbar_arrive(&ctl->xl_dec);
                }
                {
                    const bool xl_ok = mbar_wait(&ctl->xl_full, (unsigned)(n & 1), status, a.wait_ns);
                    if (!__all_sync(0xffffffffu, xl_ok)) { ok = false; break; }   // warp-uniform exit
                }
                tc_fence_after();
#pragma unroll 1
                for (int h = 0; h < 2 && any; ++h) {
                    const uint32_t cmask = cms[h];
                    if (!__any_sync(0xffffffffu, cmask != 0)) continue;
                    const unsigned cc = col0 + h * 32;
                    uint32_t hv[32], xv[32], lv[32];
                    tmem_ld32(tmem + lane_off + kColHH0 + b * 128 + cc, hv);
                    tmem_ld32(tmem + lane_off + kColX + cc, xv);
                    tmem_ld32(tmem + lane_off + kColLL + cc, lv);
                    tmem_ld_wait();
                    uint32_t amask = 0, mk = cmask;
                    while (mk) {   // exact INT64 test, one copy of the code
                        const int k = __ffs(mk) - 1;
                        mk &= mk - 1;
                        ++n_rare;
                        const long long dot = (long long)(int)pick32(hv, k) * 16384ll +
                                              (long long)(int)pick32(xv, k) * 128ll + (long long)(int)pick32(lv, k);
                        const long long d2 = Ai + m.norm[cc + k] - 2 * dot;
                        if (d2 <= a.T) amask |= 1u << k;
                    }
                    unsigned ta;
                    const unsigned pa = warp_excl_scan(__popc(amask), ta);
                    if (ta) {
                        unsigned long long pos = app.reserve(ta, &a.ctr->acc_reserved, a.acc, a.acc_cap) + pa;
                        uint32_t mk = amask;
                        while (mk) {
                            const int k = __ffs(mk) - 1;
                            mk &= mk - 1;
                            if (pos < a.acc_cap) a.acc[pos] = pair_key(jp, oi, m.perm[cc + k]);
                            ++pos;
                        }
                        n_acc += __popc(amask);
                    }
                }
                if (!ok) break;
                // this item's hh buffer, the shared x / ll and the metadata slot are free again
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&ctl->hh_empty[b]);
                    mbar_arrive(&ctl->xl_empty);
                    mbar_arrive(&ctl->meta_empty[slot]);
                }
                ++n_items;
            }
        }
        if (!ok) ctl->abort_flag = 1;
        app.pad(a.acc, a.acc_cap);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            n_acc += __shfl_xor_sync(0xffffffffu, n_acc, o);
            n_rare += __shfl_xor_sync(0xffffffffu, n_rare, o);
        }
        if (lane == 0) {
            if (app.valid) atomicAdd(&a.ctr->acc_valid, app.valid);
            if (n_acc) atomicAdd(&a.ctr->screen_accept, n_acc);
            if (n_rare) atomicAdd(&a.ctr->rare_checks, n_rare);
            if (ew == 0 && n_items) atomicAdd(&a.ctr->items, n_items);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_dealloc(tmem, 512);
}

// ------------------------------------------------------------------ high-limb screen
// One tensor-core product per pair: hh = sum h h' (exact INT32), and the rest of q.q' bounded by
// Cauchy-Schwarz on the limb vectors, |128 x + ll| <= M_ij = 128 (|h||l'| + |l||h'|) + |l||l'|.  A pair
// whose interval [A_i + B_j - 32768 hh -+ 2 M_ij] lies above T is out, one whose interval lies at or below
// T is in (exact INT64 test per candidate), and the rest go to the band buffer, where the integer
// refinement decides them from the int16 rows.
//
// The column term and the bound ride in the product.  Every row carries 32 more int8 elements
// (I8Fold): on the S side digits of -floor(B_j / 2^15) and the norms L_j, G_j, on the R side the
// digits' weights and the norms H_i, L_i, so that one more K = 32 step leaves
//     v = hh - b_j + H_i L_j + L_i G_j,      H_i L_j + L_i G_j >= M_ij / 2^14
// in the accumulator (norms in units of sqrt(128), rounded up), and v < floor((A_i - T) / 2^15) proves
// the pair out: one maximum per row over any number of columns, against a constant of the row.
//
// What bounds it.  A 128 x 128 item needs 256 cycles of MMAs and took 1,300 with one R tile per CTA and
// per-column tests.  Builds that skip work showed why, one limit behind the other:
//  - the S limbs streamed from L2, 20 KB per item and 7 TB/s in all: a CTA holds kRT R tiles and
//    every S tile brought in meets all of them;
//  - the issuing thread's own instructions, 700 cycles per step with one MMA in it: two S tiles share
//    an N = 256 MMA (and a commit, two barriers and each A fragment read), loops are unrolled, and a
//    descriptor is a constant added to a base;
//  - the epilogue, three warps per SM sub-partition and everything in it latency: the test is one
//    maximum per row and 64 columns, waits first look at the barrier without suspending (290 -> 100
//    cycles for one that is open already), and candidates are queued and tested 32 at a time.
// Now (cycles per item at 1M rows): MMAs and copies alone 420, with the epilogue's tests 600, with the
// candidates of a 24-neighbour threshold 775.
// Candidates come as lists per group of kRT R tiles whose entries say which of them they are for.
// Measured (one B200, self-joins with 24 neighbours per row, this kernel alone): 2M x 128 554 -> 335 ms,
// 50,021 x 100 1.00 -> 0.57 ms.
//
// Warp roles (512 threads): warps 0 and 2 TMA producers (limbs; folds), warp 1 TMEM
// allocator + UMMA issuer, warp 3 idle, warps 4..15 epilogue in three groups of four that take the live 128 x 128 items in turn (warp w
// reads TMEM lanes 32 (w % 4).., all 128 columns in two passes of 64).
constexpr int kHHAcc = 2;                         // TMEM accumulators of 256 columns (two items)
// An epilogue group takes every third item, so its next one may be three steps on (steps of one item),
// and with a barrier per accumulator it would test the phase of the step after next while that of the
// step before it is still open: the parities are equal.  Four barriers keep a step's predecessor on its
// barrier four steps back, which a group has always seen complete.
constexpr int kHHSteps = 4;
constexpr int kHHEpi = 12;
constexpr int kHHGroups = kHHEpi / 4;
constexpr int kHHEpiFirst = 4;
constexpr int kHHThreads = (kHHEpiFirst + kHHEpi) * 32;
constexpr unsigned kFoldBytes = 128u * kI8Fold;   // fold elements of one 128-row tile (32-byte swizzle box)
constexpr unsigned kHHStageBytes = 2 * kPart + 2 * kFoldBytes;   // one k-block of two S tiles (+ their fold)
static_assert(kI8N == 128 && kTileR == 128, "R and S tiles of one size share the row records");

// Shared-memory plan per k-block count: the R tiles with their fold, and the stages (a pair of S tiles
// holds one per k-block until its last R tile is done).
template <int kMaxKb> struct HHCfg {
    static constexpr int kRT = i8_rtiles(kMaxKb);                        // R tiles per CTA
    static constexpr int kStages = 3;
    static constexpr unsigned kATile = kMaxKb * kPart + kFoldBytes;      // one R tile
};
// Candidates a warp collects (value, sorted row and column) before it tests them, a lane each: with one
// test per hit the warp stood 1,300 cycles on it, and with it, two accumulators deep, the whole pipeline.
constexpr unsigned kHHQueue = 64;

template <int kStages> struct HHCtl {
    uint64_t a_full;
    uint64_t a_empty;
    uint64_t full[kStages];
    uint64_t empty[kStages];
    uint64_t acc_full[kHHSteps];   // by step, not by accumulator: see kHHSteps
    uint64_t acc_empty[kHHAcc];
    uint64_t drain;
    unsigned tmem_base;
    int abort_flag;
};

template <int kMaxKb> constexpr size_t hh_smem() {
    using C = HHCfg<kMaxKb>;
    return 1024 + C::kRT * (size_t)C::kATile + (size_t)C::kStages * kHHStageBytes + kHHEpi * kHHQueue * 12 +
           sizeof(HHCtl<C::kStages>);
}
static_assert(hh_smem<1>() <= 232448 && hh_smem<2>() <= 232448, "227 KB of shared memory per CTA at most");

struct HHArgs {
    const uint4* chunks;       // (R tile group, first and last + 1 list entry)
    const uint32_t* nchunks;
    const uint32_t* jlist;     // S tile | live R tiles of the group << (32 - kRT)
    const I8Row *rrec, *srec;  // row records of the sides, in tile order
    unsigned ntR;              // 128-row R tiles
    unsigned nR, nS;           // rows that are points
    unsigned idesc1, idesc2;   // N = 128: one S tile; N = 256: two
    long long T;               // integer threshold
    JoinParams jp;
    uint64_t* acc;
    unsigned long long acc_cap;
    uint64_t* band;
    unsigned long long band_cap;
    Counters* ctr;
    unsigned long long wait_ns;   // limit of every pipeline wait (drains keep kDrainLimitNs)
};

// One lane waits for the warp.
TJ_DEV bool warp_wait(uint64_t* bar, unsigned parity, unsigned long long* status, unsigned long long limit) {
    if (__all_sync(0xffffffffu, mbar_test(bar, parity))) return true;
    int ok = 1;
    if (lane_id() == 0) ok = mbar_wait(bar, parity, status, limit) ? 1 : 0;
    ok = __shfl_sync(0xffffffffu, ok, 0);
    __syncwarp();
    return ok != 0;
}

template <int kMaxKb>
__global__ void __launch_bounds__(kHHThreads, 1)
    screen_i8_hh_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                        const __grid_constant__ CUtensorMap tmFA, const __grid_constant__ CUtensorMap tmFB,
                        const __grid_constant__ CUtensorMap tmB2, const __grid_constant__ CUtensorMap tmFB2,
                        const HHArgs a) {
    using Cfg = HHCfg<kMaxKb>;
    constexpr int kStages = Cfg::kStages, kRT = Cfg::kRT;
    constexpr unsigned kATile = Cfg::kATile;
    constexpr uint32_t kFoldDesc = desc_hi_for_rows(kI8Fold);
    constexpr unsigned kMaskShift = 32 - kRT, kTileMask = (1u << kMaskShift) - 1u;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* abuf = smem;                                       // kRT x (k-blocks, fold)
    uint8_t* bbuf = abuf + kRT * kATile;                        // kStages x kHHStageBytes
    uint32_t* queues = (uint32_t*)(bbuf + (size_t)kStages * kHHStageBytes);   // [kHHEpi][3][kHHQueue]
    auto* ctl = (HHCtl<kStages>*)(queues + kHHEpi * 3 * kHHQueue);
    const unsigned warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned long long* status = &a.ctr->status;

    if (threadIdx.x == 0) {
        mbar_init(&ctl->a_full, 2);             // both producers
        mbar_init(&ctl->a_empty, 1);
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&ctl->full[s], 2);
            mbar_init(&ctl->empty[s], 1);
        }
        for (int b = 0; b < kHHSteps; ++b) mbar_init(&ctl->acc_full[b], 1);
        for (int b = 0; b < kHHAcc; ++b)
            mbar_init(&ctl->acc_empty[b], 8);   // the four warps of each item (twice where there is one)
        mbar_init(&ctl->drain, 1);
        ctl->abort_flag = 0;
        fence_barrier_init();
        prefetch_tmap(&tmA);
        prefetch_tmap(&tmB);
        prefetch_tmap(&tmFA);
        prefetch_tmap(&tmFB);
        prefetch_tmap(&tmB2);
        prefetch_tmap(&tmFB2);
    }
    if (warp == 1) tmem_alloc(&ctl->tmem_base, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = ctl->tmem_base;
    const unsigned nchunks = *a.nchunks;
    constexpr int kblocks = kMaxKb;

    if (warp == 0 || warp == 2) {
        // ------------------------------------------------------------ TMA producers
        // Both walk the same sequence and arrive on every full barrier: warp 0 with the R and S limbs, warp
        // 2 with the folded elements.  S tiles that follow one another (the usual case of a dense list) come
        // in boxes of 256 rows.
        if (lane == 0) {
            const bool limbs = warp == 0;
            unsigned stage = 0, phase = 0, nc = 0;   // nc: chunks issued
            bool ok = true;
            for (unsigned c = blockIdx.x; c < nchunks && ok; c += gridDim.x, ++nc) {
                const uint4 ch = a.chunks[c];
                const unsigned rt0 = ch.x * kRT, rtn = min((unsigned)kRT, a.ntR - rt0);
                if (!mbar_wait(&ctl->a_empty, (nc & 1u) ^ 1u, status, a.wait_ns)) { ok = false; break; }
                mbar_arrive_expect_tx(&ctl->a_full, rtn * (limbs ? (unsigned)kblocks * kPart : kFoldBytes));
                for (unsigned r = 0; r < rtn; ++r) {
                    uint8_t* at = abuf + r * kATile;
                    if (limbs) {
                        for (int kb = 0; kb < kblocks; ++kb)
                            tma_load_2d(at + kb * kPart, &tmA, &ctl->a_full, kb * 128, (int)((rt0 + r) * 128));
                    } else {
                        tma_load_2d(at + kMaxKb * kPart, &tmFA, &ctl->a_full, 0, (int)((rt0 + r) * 128));
                    }
                }
                for (unsigned e = ch.y; e < ch.z && ok; e += 2) {
                    const unsigned two = e + 1 < ch.z ? 2u : 1u;
                    const unsigned J0 = a.jlist[e] & kTileMask, J1 = two == 2 ? a.jlist[e + 1] & kTileMask : 0u;
                    const bool joined = two == 2 && J1 == J0 + 1;
                    for (int kb = 0; kb < kblocks; ++kb) {
                        if (!mbar_wait(&ctl->empty[stage], phase ^ 1, status, a.wait_ns)) { ok = false; break; }
                        if (*(volatile int*)&ctl->abort_flag) { ok = false; break; }
                        uint8_t* sb = bbuf + (size_t)stage * kHHStageBytes;
                        uint64_t* full = &ctl->full[stage];
                        if (limbs) {
                            mbar_arrive_expect_tx(full, two * kPart);
                            if (joined) {
                                tma_load_2d(sb, &tmB2, full, kb * 128, (int)(J0 * 128));
                            } else {
                                tma_load_2d(sb, &tmB, full, kb * 128, (int)(J0 * 128));
                                if (two == 2) tma_load_2d(sb + kPart, &tmB, full, kb * 128, (int)(J1 * 128));
                            }
                        } else if (kb > 0) {
                            mbar_arrive(full);
                        } else {
                            uint8_t* sf = sb + 2 * kPart;
                            mbar_arrive_expect_tx(full, two * kFoldBytes);
                            if (joined) {
                                tma_load_2d(sf, &tmFB2, full, 0, (int)(J0 * 128));
                            } else {
                                tma_load_2d(sf, &tmFB, full, 0, (int)(J0 * 128));
                                if (two == 2) tma_load_2d(sf + kFoldBytes, &tmFB, full, 0, (int)(J1 * 128));
                            }
                        }
                        if (++stage == (unsigned)kStages) { stage = 0; phase ^= 1; }
                    }
                }
            }
            if (!ok) ctl->abort_flag = 1;
            // drain: the last copy issued into every buffer lands before exit
            for (unsigned s = 0; s < (unsigned)kStages; ++s)
                mbar_wait(&ctl->full[s], s < stage ? phase : (phase ^ 1u), status, kDrainLimitNs);
            if (nc) mbar_wait(&ctl->a_full, (nc - 1) & 1u, status, kDrainLimitNs);
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ UMMA issuer
        // One thread, and its own instructions between MMAs add up: with runtime k-block loops and descriptors
        // built from pointers a step took 700 cycles to issue with a single MMA in it.  So the loops are
        // unrolled and a descriptor is a constant added to the low word of a base.
        if (lane == 0) {
            constexpr uint32_t kSw128Hi = desc_hi_for_rows(128);
            auto lo = [](const void* p) { return ((smem_u32(p) >> 4) & 0x3FFFu) | (1u << 16); };
            auto desc = [](uint32_t l, uint32_t hi) { return ((uint64_t)hi << 32) | l; };
            const uint32_t a0 = lo(abuf), b0 = lo(bbuf);
            unsigned stage = 0, phase = 0, step = 0;   // step: accumulators filled
            unsigned long long n = 0;
            unsigned nc = 0;
            bool ok = true;
            for (unsigned c = blockIdx.x; c < nchunks && ok; c += gridDim.x, ++nc) {
                const uint4 ch = a.chunks[c];
                uint32_t j0 = a.jlist[ch.y], j1 = ch.y + 1 < ch.z ? a.jlist[ch.y + 1] : 0u;
                if (!mbar_wait(&ctl->a_full, nc & 1u, status, a.wait_ns)) { ok = false; break; }
                tc_fence_after();
                for (unsigned e = ch.y; e < ch.z && ok; e += 2) {
                    const unsigned m0 = j0 >> kMaskShift, m1 = j1 >> kMaskShift;
                    j0 = e + 2 < ch.z ? a.jlist[e + 2] : 0u;   // the next pair's entries, on their way
                    j1 = e + 3 < ch.z ? a.jlist[e + 3] : 0u;
                    const unsigned any = m0 | m1;
                    const unsigned rlast = 31 - __clz(any);   // the last R tile of the group with a live item
                    unsigned sg[kMaxKb], bl[kMaxKb];          // the pair's stages, and their descriptors
#pragma unroll
                    for (int kb = 0; kb < kMaxKb; ++kb) {
                        sg[kb] = stage;
                        bl[kb] = b0 + stage * (kHHStageBytes >> 4);
                        if (ok && !mbar_wait(&ctl->full[stage], phase, status, a.wait_ns)) ok = false;
                        if (++stage == (unsigned)kStages) { stage = 0; phase ^= 1; }
                    }
                    if (!ok || *(volatile int*)&ctl->abort_flag) { ok = false; break; }
#pragma unroll
                    for (unsigned r = 0; r < (unsigned)kRT; ++r) {
                        if (!((any >> r) & 1u)) continue;
                        const unsigned b = step & (kHHAcc - 1);
                        if (!mbar_wait(&ctl->acc_empty[b], ((step / kHHAcc) & 1u) ^ 1u, status, a.wait_ns)) { ok = false; break; }
                        tc_fence_after();
                        // both S tiles, or the one that is live
                        uint32_t idesc = a.idesc2, d_tmem = tmem + b * 256u, rows = 0, frows = 0;
                        if (!((m0 & m1) >> r & 1u)) {
                            const unsigned second = (m1 >> r) & 1u;
                            idesc = a.idesc1;
                            d_tmem += second * 128u;
                            rows = second * (kPart >> 4);
                            frows = second * (kFoldBytes >> 4);
                            --n;
                        }
                        n += 2;
                        constexpr uint32_t kFoldA = (kMaxKb * kPart) >> 4, kFoldB = (2 * kPart) >> 4;
                        const uint32_t ar = a0 + r * (kATile >> 4);
                        umma_i8(d_tmem, desc(ar + kFoldA, kFoldDesc), desc(bl[0] + kFoldB + frows, kFoldDesc), idesc, 0u);
#pragma unroll
                        for (int kb = 0; kb < kMaxKb; ++kb) {
#pragma unroll
                            for (unsigned k = 0; k < 4; ++k)
                                umma_i8(d_tmem, desc(ar + kb * (kPart >> 4) + 2 * k, kSw128Hi),
                                        desc(bl[kb] + rows + 2 * k, kSw128Hi), idesc, 1u);
                            if (r == rlast) umma_commit(&ctl->empty[sg[kb]]);
                        }
                        umma_commit(&ctl->acc_full[step & (kHHSteps - 1)]);
                        ++step;
                    }
                }
                umma_commit(&ctl->a_empty);   // the R tiles are free once this chunk's MMAs complete
            }
            if (n) atomicAdd(&a.ctr->items, n);
            if (!ok) ctl->abort_flag = 1;
            umma_commit(&ctl->drain);
            mbar_wait(&ctl->drain, 0, status, kDrainLimitNs);
        }
    } else if (warp >= kHHEpiFirst) {
        // ------------------------------------------------------------ epilogue
        const unsigned group = (warp - kHHEpiFirst) >> 2;   // item i goes to group i mod 3
        const unsigned q = warp & 3;                   // TMEM lane quarter
        const unsigned row = q * 32 + lane;
        const unsigned lane_off = (q * 32u) << 16;
        const JoinParams& jp = a.jp;
        uint32_t* qv = queues + (warp - kHHEpiFirst) * 3 * kHHQueue;   // value, sorted row, sorted column
        uint32_t *qr = qv + kHHQueue, *qc = qr + kHHQueue;
        unsigned qn = 0;   // queued candidates
        const unsigned lt = (1u << lane) - 1u;
        WarpAppender app_acc, app_band;
        unsigned step = 0, turn = 0;   // accumulator step; item mod 3
        unsigned n_acc = 0, n_rare = 0;
        bool ok = true;
        // Tests the oldest queued candidates (at most 32, a lane each): exact INT64 interval, in / out / band.
        auto flush = [&](unsigned from) {
            const unsigned m = min(qn - from, 32u);
            const bool has = lane < m;
            const unsigned at = from + min(lane, m - 1);
            const int v = (int)qv[at];
            const I8Row me = a.rrec[qr[at]], cj = a.srec[qc[at]];
            const int m14 = me.H * cj.L + me.L * cj.G;                          // as folded
            const int hh = v + (int)min(cj.norm >> 15, (long long)kI8FoldMax) - m14;
            const long long mid = me.norm + cj.norm - 32768ll * (long long)hh;
            const long long M2 = 32768ll * (long long)m14;
            const bool in = has && mid + M2 <= a.T, band = has && !in && mid - M2 <= a.T;
            const unsigned im = __ballot_sync(0xffffffffu, in), bm = __ballot_sync(0xffffffffu, band);
            n_rare += has ? 1 : 0;
            const uint64_t key = pair_key(jp, me.id, cj.id);
            if (im) {
                const unsigned long long pos =
                    app_acc.reserve(__popc(im), &a.ctr->acc_reserved, a.acc, a.acc_cap) + __popc(im & lt);
                if (in && pos < a.acc_cap) a.acc[pos] = key;
                n_acc += in ? 1 : 0;
            }
            if (bm) {
                const unsigned long long pos =
                    app_band.reserve(__popc(bm), &a.ctr->band_reserved, a.band, a.band_cap) + __popc(bm & lt);
                if (band && pos < a.band_cap) a.band[pos] = key;
            }
        };
        for (unsigned c = blockIdx.x; c < nchunks && ok; c += gridDim.x) {
            const uint4 ch = a.chunks[c];
            // list entries 32 at a time, the next 32 on their way
            unsigned eb = ch.y;
            uint32_t cur = a.jlist[min(eb + lane, ch.z - 1)], nxt = a.jlist[min(eb + 32 + lane, ch.z - 1)];
            // floor((A_i - T) / 2^15) of this lane's row of every R tile (no point: rejects everything; the same
            // once the join is to be done with four products instead, as the host will see by the counter)
            const bool given_up = *(volatile unsigned long long*)&a.ctr->band_reserved >
                                  i8_band_stop(a.ctr->pairs_screened, a.band_cap);
            int c15[kRT];
#pragma unroll
            for (unsigned r = 0; r < (unsigned)kRT; ++r) {
                const unsigned gr = (ch.x * kRT + r) * 128 + row;
                c15[r] = gr < a.nR && !given_up ? clamp_shift15(a.rrec[gr].norm - a.T) : 0x7FFFFFFF;
            }
            for (unsigned e = ch.y; e < ch.z && ok; e += 2) {
                if (e - eb == 32) {
                    eb = e;
                    cur = nxt;
                    nxt = a.jlist[min(eb + 32 + lane, ch.z - 1)];
                }
                const uint32_t j0 = __shfl_sync(0xffffffffu, cur, e - eb);
                const uint32_t j1 = e + 1 < ch.z ? __shfl_sync(0xffffffffu, cur, e + 1 - eb) : 0u;
#pragma unroll 1
                for (unsigned r = 0; r < (unsigned)kRT && ok; ++r) {
                    const unsigned live = ((j0 >> (kMaskShift + r)) & 1u) | (((j1 >> (kMaskShift + r)) & 1u) << 1);
                    if (!live) continue;
                    const unsigned st = step++, b = st & (kHHAcc - 1);
                    // this group's item of the step, if it has one (two items go to two groups)
                    const unsigned items = live == 3u ? 2u : 1u;
                    const unsigned behind = group >= turn ? group - turn : group + kHHGroups - turn;
                    turn += items;
                    if (turn >= (unsigned)kHHGroups) turn -= kHHGroups;
                    if (behind >= items) continue;
                    const unsigned h2 = live == 3u ? behind : live - 1u;
                    int ci = c15[0];
#pragma unroll
                    for (unsigned k = 1; k < (unsigned)kRT; ++k) ci = r == k ? c15[k] : ci;
                    // warp-uniform: the TMEM loads below are warp-collective
                    if (!warp_wait(&ctl->acc_full[st & (kHHSteps - 1)], (st / kHHSteps) & 1u, status, a.wait_ns)) { ok = false; break; }
                    tc_fence_after();
                    const unsigned t0 = tmem + lane_off + b * 256u + h2 * 128u;
#pragma unroll 1
                    for (unsigned pass = 0; pass < 2; ++pass) {
                        uint32_t hv2[2][32];
                        tmem_ld32(t0 + pass * 64, hv2[0]);
                        tmem_ld32(t0 + pass * 64 + 32, hv2[1]);
                        tmem_ld_wait();
                        if (pass == 1) {   // the accumulator is in registers
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive_cnt(&ctl->acc_empty[b], items == 2 ? 1u : 2u);
                        }
                        int gm[4];   // maxima of 16 columns each
#pragma unroll
                        for (int g = 0; g < 4; ++g) {
                            const uint32_t* x = hv2[g / 2] + 16 * (g % 2);
                            const int p0 = __vimax3_s32((int)x[0], (int)x[1], (int)x[2]);
                            const int p1 = __vimax3_s32((int)x[3], (int)x[4], (int)x[5]);
                            const int p2 = __vimax3_s32((int)x[6], (int)x[7], (int)x[8]);
                            const int p3 = __vimax3_s32((int)x[9], (int)x[10], (int)x[11]);
                            const int p4 = __vimax3_s32((int)x[12], (int)x[13], (int)x[14]);
                            gm[g] = __vimax3_s32(__vimax3_s32(p0, p1, p2), __vimax3_s32(p3, p4, (int)x[15]), p4);
                        }
                        const bool hit = max(__vimax3_s32(gm[0], gm[1], gm[2]), gm[3]) >= ci;
                        if (!__any_sync(0xffffffffu, hit)) continue;
                        const unsigned gr = (ch.x * kRT + r) * 128 + row;
                        const unsigned c0 = ((h2 ? j1 : j0) & kTileMask) * 128 + pass * 64;
                        unsigned gb = 0;   // groups of 16 columns with a candidate in some row
#pragma unroll
                        for (int g = 0; g < 4; ++g) gb |= __any_sync(0xffffffffu, gm[g] >= ci) ? 1u << g : 0u;
#pragma unroll 1
                        for (; gb; gb &= gb - 1) {
                            // the group's 16 registers (g is not a constant here: one copy of the code below)
                            const int g = __ffs(gb) - 1;
                            uint32_t x[16];
#pragma unroll
                            for (int k = 0; k < 16; ++k)
                                x[k] = g < 2 ? (g == 0 ? hv2[0][k] : hv2[0][16 + k]) : (g == 2 ? hv2[1][k] : hv2[1][16 + k]);
                            unsigned cm = 0;
#pragma unroll
                            for (int k = 0; k < 16; ++k) cm |= ((int)x[k] >= ci ? 1u : 0u) << k;
                            // real columns; self-joins keep sorted column > sorted row only
                            const unsigned cg = c0 + 16 * g;
                            if (cg + 16 > a.nS) cm &= cg < a.nS ? (1u << (a.nS - cg)) - 1u : 0u;
                            if (jp.self_join && cg <= gr) cm &= gr - cg >= 15 ? 0u : ~((2u << (gr - cg)) - 1u);
                            unsigned bal;
                            while ((bal = __ballot_sync(0xffffffffu, cm != 0)) != 0) {
                                if (cm) {
                                    const int k = __ffs(cm) - 1;
                                    cm &= cm - 1;
                                    const unsigned at = qn + __popc(bal & lt);
                                    qv[at] = pick16(x, k);
                                    qr[at] = gr;
                                    qc[at] = cg + k;
                                }
                                qn += __popc(bal);
                                if (qn >= 32) {
                                    __syncwarp();   // the queue is written
                                    flush(0);
                                    __syncwarp();   // and read
                                    qn -= 32;
                                    if (lane < qn) {   // the rest to the front
                                        const uint32_t v = qv[32 + lane], rr = qr[32 + lane], cc = qc[32 + lane];
                                        qv[lane] = v;
                                        qr[lane] = rr;
                                        qc[lane] = cc;
                                    }
                                    __syncwarp();
                                }
                            }
                        }
                    }
                }
            }
        }
        if (!ok) ctl->abort_flag = 1;
        __syncwarp();
        if (qn) flush(0);
        app_acc.pad(a.acc, a.acc_cap);
        app_band.pad(a.band, a.band_cap);
        unsigned long long t_acc = n_acc, t_rare = n_rare;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            t_acc += __shfl_xor_sync(0xffffffffu, t_acc, o);
            t_rare += __shfl_xor_sync(0xffffffffu, t_rare, o);
        }
        if (lane == 0) {
            if (app_acc.valid) atomicAdd(&a.ctr->acc_valid, app_acc.valid);
            if (app_band.valid) atomicAdd(&a.ctr->band_valid, app_band.valid);
            if (t_acc) atomicAdd(&a.ctr->screen_accept, t_acc);
            if (t_rare) atomicAdd(&a.ctr->rare_checks, t_rare);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_dealloc(tmem, 512);
}

}  // namespace

void make_tmap_2d(CUtensorMap* m, const void* base, long long rows, long long cols, int esize, int box_rows,
                  CUtensorMapDataType dt, int box_bytes);

namespace {

void screen_i8_hh(const ScreenInput& g, const EmitBuffers& eb, const CUtensorMap& tmA, const CUtensorMap& tmB,
                  cudaStream_t st) {
    const Side& R = *g.R[0];
    const Side& S = *g.S[0];
    if (!R.foldR.p || !S.foldS.p) fail(-1, "the high-limb screen needs folded sides");
    CUtensorMap tmFA, tmFB;
    make_tmap_2d(&tmFA, R.foldR.p, R.rows_pad, kI8Fold, 1, 128, CU_TENSOR_MAP_DATA_TYPE_UINT8, kI8Fold);
    make_tmap_2d(&tmFB, S.foldS.p, S.rows_pad, kI8Fold, 1, 128, CU_TENSOR_MAP_DATA_TYPE_UINT8, kI8Fold);
    HHArgs a;
    a.chunks = g.cand->chunks.p;
    a.nchunks = g.cand->dev_counts.p + 1;
    a.jlist = g.cand->jlist.p;
    a.rrec = R.rec.p;
    a.srec = S.rec.p;
    a.ntR = (unsigned)g.tR[0]->ntiles;
    a.nR = (unsigned)R.n;
    a.nS = (unsigned)S.n;
    a.idesc1 = make_idesc(2u, 1u, 128, kI8N);
    a.idesc2 = make_idesc(2u, 1u, 128, 2 * kI8N);
    a.T = g.T_int;
    a.jp = g.jp0;
    a.acc = eb.acc;
    a.acc_cap = eb.acc_cap;
    a.band = eb.band;
    a.band_cap = eb.band_cap;
    a.ctr = eb.ctr;
    a.wait_ns = pipeline_wait_ns();
    CUtensorMap tmB2, tmFB2;   // two tiles at once
    make_tmap_2d(&tmB2, S.op8.p, S.rows_pad, 2 * (long long)S.kpad, 1, 256, CU_TENSOR_MAP_DATA_TYPE_UINT8, 128);
    make_tmap_2d(&tmFB2, S.foldS.p, S.rows_pad, kI8Fold, 1, 256, CU_TENSOR_MAP_DATA_TYPE_UINT8, kI8Fold);
    auto run = [&](auto kern, size_t smem) {
        TJ_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        launch(kern, num_sms(), kHHThreads, smem, st, tmA, tmB, tmFA, tmFB, tmB2, tmFB2, a);
    };
    if (R.kpad == 128) run(screen_i8_hh_kernel<1>, hh_smem<1>());
    else run(screen_i8_hh_kernel<2>, hh_smem<2>());
}

}  // namespace

void screen_i8(const ScreenInput& g, const EmitBuffers& eb, cudaStream_t st) {
    if (g.ncls != 1 || g.njoins != 1) fail(-7, "the int8-limb screen runs one join at a time");
    const Side& R = *g.R[0];
    const Side& S = *g.S[0];
    if (R.screen != kScreenInt8Limb || S.screen != kScreenInt8Limb) fail(-1, "screen_i8 needs int8-limb sides");
    CUtensorMap tmA, tmB;
    make_tmap_2d(&tmA, R.op8.p, R.rows_pad, 2 * (long long)R.kpad, 1, 128, CU_TENSOR_MAP_DATA_TYPE_UINT8, 128);
    make_tmap_2d(&tmB, S.op8.p, S.rows_pad, 2 * (long long)S.kpad, 1, kI8N, CU_TENSOR_MAP_DATA_TYPE_UINT8, 128);
    if (i8_high_limb_screen(g)) {
        screen_i8_hh(g, eb, tmA, tmB, st);
        return;
    }
    I8Args a;
    a.chunks = g.cand->chunks.p;
    a.nchunks = g.cand->dev_counts.p + 1;
    a.jlist = g.cand->jlist.p;
    a.r_row0 = g.tR[0]->row0.p;
    a.r_nvalid = g.tR[0]->nvalid.p;
    a.r_perm = R.emit;
    a.r_norm = R.inorm.p;
    a.r_hn = R.zn.p;   // the int8-limb preparation stores |h| and |l| upper bounds in zn / zl
    a.r_ln = R.zl.p;
    const TileSet& tS = *g.tS[0];
    DBuf<ColMetaI8> smeta((size_t)std::max(tS.ntiles, 1), st);
    if (tS.ntiles > 0)
        launch(build_col_meta_i8, tS.ntiles, kI8N, 0, st, tS.row0.p, tS.nvalid.p, S.emit, S.inorm.p, tS.maxZ.p,
               tS.maxZl.p, smeta.p);
    a.s_row0 = tS.row0.p;
    a.s_meta = smeta.p;
    a.kblocks = R.kpad / 128;
    a.kpad = R.kpad;
    a.idesc = make_idesc(2u, 1u, 128, kI8N);
    a.T = g.T_int;
    a.jp = g.jp0;
    a.acc = eb.acc;
    a.acc_cap = eb.acc_cap;
    a.ctr = eb.ctr;
    a.wait_ns = pipeline_wait_ns();
    TJ_CUDA(cudaFuncSetAttribute(screen_i8_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kI8Smem));
    launch(screen_i8_kernel, num_sms(), kI8Threads, kI8Smem, st, tmA, tmB, a);
}

bool i8_high_limb_screen(const ScreenInput& g) {
    return !g.i8_four_products && g.R[0]->kpad <= kI8HighLimbPad;
}

}  // namespace tj
