// Stages 2 and 3: residue-bitset intersection and exact 128-bit later filters, over one or many
// windows ("segments") in one launch sequence.
//
// Layout.  The sorted u lists of all segments are concatenated, each starting on a 2048-entry
// boundary, and cut into blocks of K words (32 u per word); a block therefore belongs to exactly
// one segment.  The v lists are concatenated unpadded.  A work item is one u block and a run of
// consecutive v rows (of the block's segment) whose exact u interval meets the block.  The CTA
// that owns an item builds, in shared memory, the residue rows of the first NB residual filters
// of the segment's filter family for its block (row r of filter q, bit i <=> allowed_q[(u_i B -
// r A) mod q]) and then streams its v rows: one lane per (v row, block) piece reads the K-word
// rows selected by v mod q with 128-bit loads, ANDs them, counts the group survivors by
// popcount, and queues the bits that survive every bitset filter.  Queued survivors are tested
// by a warp against the next few filters from residues of u and v (the cheap tier); the rest go
// to a per-CTA slice that k_deep finishes in exact 128-bit arithmetic.
//
// Rows are stored unswizzled, K/4 16-byte units per row; lane l reads unit (l + p) mod (K/4) at
// step p, so the 32 lanes of a warp spread evenly over the bank groups whatever rows they read.
#include "common.cuh"
#include "shares.cuh"
#include <algorithm>
#include <chrono>
#include <cstring>
#include <cstdio>

struct FiltConst {
    ModQ m;
    uint32_t tab_off;   // word offset of the packed allowed bitmap
    uint32_t pad;
};

// Compact filter constants: fast remainder constant, modulus, bitmap offset and 2^(16k) mod q for
// k = 1..5 (x < 2^96).
struct FiltC {
    uint64_t c;
    uint32_t q, tab_off;
    uint16_t r16[5];
    uint16_t pad[3];
};

struct pc_filters {
    uint64_t A = 0, B = 0;
    uint32_t nres = 0, ng = 0;
    std::vector<uint32_t> primes;
    FiltConst *d_fc = nullptr;
    FiltC *d_fcs = nullptr;
    uint32_t *d_bits = nullptr;
    uint32_t *d_pat = nullptr;       // rotation patterns of the first filters (PATW words each)
    uint64_t fc_bytes = 0, fcs_bytes = 0, bits_bytes = 0, pat_bytes = 0;
    uint32_t nbmax = 0;              // filters usable as bitset rows
    uint32_t ainvb[PC_MAX_BITSET] = {};
    uint32_t rows_sum[PC_MAX_BITSET + 1] = {};   // prefix sums of q over the first filters
    std::vector<FiltC> fcs;
};

namespace {

constexpr int PATW = 136;            // pattern words per bitset filter (q <= 2047)
constexpr int TMAX_DEFAULT = 64;     // subtile counter slots per CTA
constexpr uint64_t SEG_ALIGN = 2048; // u entries: every segment's u list starts on a block boundary

struct __align__(16) VRec {
    uint32_t left, right;            // exact u interval as indices into the concatenated u list
    uint64_t v;
    uint16_t row[8];                 // row index (row0 + v mod q) of each bitset filter
};

// One window: its focus moduli, interval, subtile geometry and slices of the concatenated lists.
struct SegDev {
    uint64_t A, B;
    u128 lo, hi;
    uint64_t v_first, width, v_end;
    uint32_t u_off, nu, v_off, nv;
    uint32_t tile_base, ntiles, fam, pad;
};

// One residual filter family (the filter list of one (p, A, B)) as the launch uses it: bitset
// filters 0..NB-1, cheap-tier filters NB..NB+nch-1, the rest in k_deep.
struct FamDev {
    uint32_t nres, ng, total_rows, c2_live;   // c2_live: group 2 ends at the last bitset filter
    uint32_t q[PC_MAX_BITSET], row0[PC_MAX_BITSET];
    uint32_t cq[PC_MAX_CHEAP], cbits_off[PC_MAX_CHEAP];
    uint4 umod[PC_MAX_BITSET + PC_MAX_CHEAP];   // pack_mod of the bitset filters with B A^-1 mod q, of the cheap tier with B mod q
    uint8_t bgroup[16];              // group ended by filter idx (0 = none), idx < NB + nch
    uint32_t cqg[PC_MAX_CHEAP];      // cheap-tier filter t: q | the group it ends (bgroup[NB + t]) << 16
    const uint32_t *pat;
    const uint32_t *bits;
    const FiltC *fcs;
};

struct MatchArgs {
    const uint64_t *us;
    const VRec *rec;
    const uint64_t *cres;            // per v: cheap-tier residues v*A mod q, 16 bits each
    const SegDev *seg;
    const FamDev *fam;
    const uint32_t *blk_seg;         // per u block: its segment
    uint32_t nch, tmax, stride;      // stride: counters per subtile (largest ng + 3)
    uint32_t total_rows;             // largest over the families
    uint64_t *counts;                // ntiles x stride
    const uint4 *bv;                 // per u block: v rows meeting it, v rows covering it
    const uint64_t *prefix;          // work of the blocks before each block; then all work; then its division (Shares)
    uint64_t nblocks;
    uint32_t block_cost, v_chunk;    // a block's fixed work in v rows; most rows per work item
    uint4 *deep;                     // (v lo, v hi, u index, subtile) records
    uint32_t deep_cap;               // records per CTA slice
    uint32_t *deep_count;            // per CTA (may exceed deep_cap: the caller retries larger)
    unsigned long long *share_next;  // shares claimed beyond each CTA's first (zeroed before the launch)
};

struct DeepArgs {
    const uint64_t *us;
    const uint4 *deep;
    const uint32_t *deep_count;
    uint32_t deep_cap, first, stride;        // filters first .. nres-1 remain
    uint64_t ntiles;
    const SegDev *seg;
    const FamDev *fam;
    const uint32_t *tile_seg;
    uint64_t *counts;
    uint64_t *out;
    uint64_t out_cap;
    unsigned long long *n_out;
};

// first j with us[j] * B > key
__device__ __forceinline__ uint64_t count_le(const uint64_t *__restrict__ us, uint64_t n, uint64_t B, u128 key) {
    uint64_t lo = 0, hi = n;
    while (lo < hi) {
        uint64_t mid = lo + (hi - lo) / 2;
        if (less128(key, mul_wide(__ldg(us + mid), B))) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}

// Subtile of v inside a segment, floor((v - v_first) / width), or ntiles when v lies outside.
// The double estimate is within one of the quotient (quotients are below 2^31), and the host
// guarantees ntiles * width < 2^64.
__device__ __forceinline__ uint64_t local_tile(uint64_t v, uint64_t v_first, uint64_t width, uint64_t ntiles) {
    if (v < v_first) return ntiles;
    const uint64_t d = v - v_first;
    uint64_t t = (uint64_t)((double)d / (double)width);
    if (t > ntiles) return ntiles;
    if (t && t * width > d) --t;
    if (t < ntiles && (t + 1) * width <= d) ++t;
    return t;
}

// Last segment whose list starts at or before index j (an empty segment shares its start with the
// next one, so the search lands on the segment that holds j).
__device__ __forceinline__ uint32_t seg_of_v(const SegDev *__restrict__ seg, uint32_t nseg, uint64_t j) {
    uint32_t lo = 0, hi = nseg;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (seg[mid].v_off <= j) lo = mid;
        else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ uint32_t seg_of_u(const SegDev *__restrict__ seg, uint32_t nseg, uint64_t j) {
    uint32_t lo = 0, hi = nseg;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (seg[mid].u_off <= j) lo = mid;
        else hi = mid;
    }
    return lo;
}

// What k_vprep needs of a segment and of a family, beside SegDev.
struct SegPrep {
    uint64_t ia, fa, am;             // A / B: whole part and 64 fraction bits; A mod B
    uint64_t ilo, ihi;               // floor(lo / B), floor(hi / B)
    uint64_t wr;                     // floor(2^64 / subtile width) (2^64 - 1 for width 1)
    uint64_t fast;                   // B < 2^62 and every bound fits 64 bits
};

struct FamPrep {
    uint4 f[PC_MAX_BITSET + PC_MAX_CHEAP];   // pack_mod of the bitset filters with row0, of the cheap tier with A mod q
};

struct PrepArgs {
    const uint64_t *us;
    const uint64_t *vs;
    uint64_t nv;
    const SegDev *seg;
    const SegPrep *segp;
    uint32_t nseg;
    const FamPrep *fam;
    uint32_t nb, stride;
    VRec *rec;
    uint64_t *cres;                  // per v: v*A mod q of the cheap-tier filters, 16 bits each
    uint32_t nch;
    uint64_t *counts;
    unsigned long long *bad;
};

constexpr uint32_t PREP_T = 256;       // threads per CTA; a CTA takes PREP_T x ROWS consecutive v rows

// x mod q for x < 2^32, m = floor(2^32 / q): the quotient estimate is at most one too small.
__device__ __forceinline__ uint32_t mod_short(uint32_t x, uint32_t m, uint32_t q) {
    const uint32_t r = x - __umulhi(x, m) * q;
    return __viaddmin_u32(r, 0u - q, r);
}

// v mod q for a pack_mod entry: 2^16 | 2^32 << 16, 2^48 | q << 16 (all mod q), floor(2^32 / q), a factor.
__device__ __forceinline__ uint32_t residue(const uint4 f, uint64_t v) {
    const uint32_t lo = (uint32_t)v, hi = (uint32_t)(v >> 32);
    return mod_short((lo & 0xffffu) + (lo >> 16) * (f.x & 0xffffu) + (hi & 0xffffu) * (f.x >> 16) + (hi >> 16) * (f.y & 0xffffu),
                     f.z, f.y >> 16);
}

// U = floor((v A + lo) / B) or, for the upper bound, floor((v A + hi) / B), and its remainder: the number of
// u with u B <= v A + lo is the number of u <= U.  The fixed-point estimate is at most two too small, and the
// remainder that corrects it stays below 3 B < 2^64, so 64-bit arithmetic is exact.
__device__ __forceinline__ uint64_t u_bound(const SegDev &g, const SegPrep &p, uint64_t v, bool upper, uint64_t &rem) {
    uint64_t u = v * p.ia + __umul64hi(v, p.fa) + (upper ? p.ihi : p.ilo);
    rem = v * g.A + (upper ? g.hi.lo : g.lo.lo) - u * g.B;
#pragma unroll
    for (int k = 0; k < 2; ++k)
        if (rem >= g.B) ++u, rem -= g.B;
    return u;
}

// The subtile of v, or UINT64_MAX outside the segment's subtiles: the quotient by the fixed-point reciprocal is
// at most one too small.
__device__ __forceinline__ uint64_t tile_of(const SegDev &g, const SegPrep &p, uint64_t v) {
    const uint64_t d = v - g.v_first;
    uint64_t t = __umul64hi(d, p.wr);
    if (d - t * g.width >= g.width) ++t;
    return v >= g.v_first && t < g.ntiles ? g.tile_base + t : UINT64_MAX;
}

// entries of the sorted list a[0, n) that are <= x
__device__ __forceinline__ uint64_t count_le64(const uint64_t *__restrict__ a, uint64_t n, uint64_t x) {
    uint64_t lo = 0, hi = n;
    while (lo < hi) {
        const uint64_t mid = lo + (hi - lo) / 2;
        if (__ldg(a + mid) <= x) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// The same by 2^LOG lanes of a warp (all 32 lanes call it, each group with its own list and x): 32 probes a step
// need five dependent loads for ten million entries.
template <int LOG>
__device__ __forceinline__ uint64_t group_count_le64(const uint64_t *__restrict__ a, uint64_t n, uint64_t x, uint32_t lane) {
    constexpr uint32_t L = 1u << LOG;
    const uint32_t part = lane & (L - 1), group = lane >> LOG << LOG;
    uint64_t lo = 0, len = n;                             // the answer is in [lo, lo + len]
    while (__any_sync(0xffffffffu, len != 0)) {
        const uint64_t step = (len + L - 1) >> LOG, at = lo + umin64((part + 1) * step, len) - 1;   // last entry of the part
        const uint32_t votes = __ballot_sync(0xffffffffu, part * step < len && __ldg(a + at) <= x);
        const uint32_t below = __popc(LOG == 5 ? votes : votes >> group & ((1u << (L & 31)) - 1));
        const uint64_t done = umin64(below * step, len);
        lo += done;
        len = len ? umin64(step - 1, len - done) : 0;
    }
    return lo;
}

// entries <= x of a sorted shared list padded with 0xffffffff to 2 top - 1 entries (top: a power of two <= 2048)
__device__ __forceinline__ uint32_t stage_count_le(const uint32_t *a, uint32_t top, uint32_t x) {
    uint32_t pos = 0;
#define PC_STEP(S) case S: if (a[pos + S - 1] <= x) pos += S; [[fallthrough]];
    switch (top) {
        PC_STEP(2048) PC_STEP(1024) PC_STEP(512) PC_STEP(256) PC_STEP(128) PC_STEP(64) PC_STEP(32) PC_STEP(16) PC_STEP(8) PC_STEP(4) PC_STEP(2)
        case 1: if (a[pos] <= x) pos += 1;
    }
#undef PC_STEP
    return pos;
}

// Per v row: exact u interval as list indices (batch_experiment.py:209-215), bitset row indices, the
// residues v*A mod q of the cheap-tier filters, and the focused-position count of its subtile.
//
// A CTA's rows lie in one segment except at a segment's ends.  Its first row's bounds U, their remainders and the
// residues are computed once; a row then adds what its distance d < 2^32 from the first row adds, in 32-bit
// arithmetic but for two 64-bit remainders.  Four warps find the list index of both bounds of the first and last row;
// the u entries between them (about 0.65 per row) are staged in shared memory as 32-bit offsets, and each row's
// bounds are two searches there (or, where they are too many to stage, in that part of the list).  In a CTA that
// spans segments each warp does the same for its own 32 rows in the list, and a row on its own where even these
// span segments or the moduli are too large for 64-bit bounds.
//
// Bound: the latency of its dependent loads and instruction issue (0.5 per cycle).  A lease's 1.6e7 rows: 0.41 ms at 48
// registers, for 40 warps per SM (at more 0.46; 40 registers spill and are slower for fewer rows).  Against sixteen rows per
// thread whose bounds advance through the list in global memory, waiting on L2: a lease 0.85 -> 0.41 ms, a batch's
// 6e4 rows 50 -> 7 us.
template <int ROWS>
__global__ void __launch_bounds__(PREP_T, 5) k_vprep(const PrepArgs a) {
    constexpr uint32_t PREP_STAGE = ROWS > 4 ? 2048 : 1024;      // u entries staged per bound
    __shared__ uint32_t stage_s[2][2 * PREP_STAGE];
    __shared__ uint64_t end_s[4], u_s[4], rem_s[2];              // per bound: first and last row's index and U; remainders
    __shared__ uint4 res_s[PC_MAX_BITSET + PC_MAX_CHEAP];        // q, floor(2^32 / q), first row's v mod q, row0 or A mod q
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t j0 = blockIdx.x * (uint64_t)(PREP_T * ROWS), j1 = umin64(a.nv, j0 + PREP_T * ROWS);
    const uint32_t s0 = seg_of_v(a.seg, a.nseg, j0);
    const SegDev &g0 = a.seg[s0];
    const SegPrep &p0 = a.segp[s0];
    bool near = j1 <= (uint64_t)g0.v_off + g0.nv && p0.fast;      // rows as distances from the first; CTA-uniform
    bool staged = false;
    uint64_t v_first = 0, first[2] = {}, count[2] = {};
    uint32_t ahead[2] = {}, top[2] = {};                  // first staged entry minus the first row's U
    if (near) {
        const uint64_t *us = a.us + g0.u_off;
        v_first = a.vs[j0];
        const uint64_t v_last = a.vs[j1 - 1];
        if (warp < 4) {                                   // warp: bound * 2 + (first, last row)
            uint64_t rem;
            const uint64_t u = u_bound(g0, p0, warp & 1 ? v_last : v_first, warp >= 2, rem);
            const uint64_t n = group_count_le64<5>(us, g0.nu, u, lane);
            if (lane == 0) {
                end_s[warp] = n;
                u_s[warp] = u;
                if (!(warp & 1)) rem_s[warp >> 1] = rem;
            }
        } else if (warp == 4 && lane < PC_MAX_BITSET + PC_MAX_CHEAP) {
            const uint4 f = a.fam[g0.fam].f[lane];
            res_s[lane] = make_uint4(f.y >> 16, f.z, residue(f, v_first), f.w);
        }
        __syncthreads();
        // distances stay below 2^32, also with a residue added
        near = v_last - v_first < 0xffff0000u && u_s[1] - u_s[0] < 0xffff0000u && u_s[3] - u_s[2] < 0xffff0000u;
        staged = near;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            first[k] = end_s[2 * k];
            count[k] = end_s[2 * k + 1] - first[k];
            const bool some = count[k] && first[k] < g0.nu;       // (an unsorted v list leaves count meaningless)
            ahead[k] = some ? (uint32_t)(us[first[k]] - u_s[2 * k]) : 0xffffffffu;
            staged = staged && count[k] <= PREP_STAGE;
            top[k] = some ? 1u << (31 - __clz((uint32_t)umin64(count[k], PREP_STAGE))) : 0u;
        }
        if (staged)
#pragma unroll
            for (int k = 0; k < 2; ++k)
                for (uint32_t i = threadIdx.x; i < 2 * top[k]; i += PREP_T)
                    stage_s[k][i] = i < count[k] ? (uint32_t)(us[first[k] + i] - u_s[2 * k]) - ahead[k] : 0xffffffffu;
        __syncthreads();
    }
    uint64_t tile = UINT64_MAX, pop = 0;                  // warp-uniform: the subtile being summed
#pragma unroll 1
    for (int m = 0; m < ROWS; ++m) {
        const uint64_t j = j0 + m * PREP_T + threadIdx.x;
        const bool active = j < j1;
        uint64_t mine = UINT64_MAX, v = 0, cr = 0;        // the row's subtile
        uint32_t left = 0, right = 0, row[PC_MAX_BITSET] = {};
        if (near) {
            if (active) {
                v = a.vs[j];
                const uint32_t d = (uint32_t)(v - v_first);
                // U grows by d (A / B): floor by the 64 fraction bits, the rest by the remainders (below 3 B)
                const uint32_t e = (uint32_t)__umul64hi(d, p0.fa);
                const uint64_t t = d * p0.am - e * g0.B, B2 = 2 * g0.B;
                uint32_t at[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const uint64_t r = rem_s[k] + t;
                    const uint32_t grown = d * (uint32_t)p0.ia + e + (r >= g0.B) + (r >= B2);
                    uint64_t n = 0;
                    if (grown >= ahead[k]) {
                        if (staged) n = stage_count_le(stage_s[k], top[k], grown - ahead[k]);
                        else n = count_le64(a.us + g0.u_off + first[k], umin64(count[k], g0.nu - first[k]), u_s[2 * k] + grown);
                    }
                    at[k] = g0.u_off + (uint32_t)(first[k] + n);
                }
                left = at[0];
                right = max(at[0], at[1]);
#pragma unroll
                for (int f = 0; f < PC_MAX_BITSET; ++f)
                    if (f < (int)a.nb) {
                        const uint4 c = res_s[f];
                        row[f] = c.w + mod_short(d + c.z, c.y, c.x);
                    }
#pragma unroll
                for (int f = 0; f < PC_MAX_CHEAP; ++f)
                    if (f < (int)a.nch) {
                        const uint4 c = res_s[PC_MAX_BITSET + f];
                        cr |= (uint64_t)mod_short(mod_short(d + c.z, c.y, c.x) * c.w, c.y, c.x) << (16 * f);
                    }
                mine = tile_of(g0, p0, v);
            }
        } else {
            const uint32_t s = active ? seg_of_v(a.seg, a.nseg, j) : s0;
            const SegDev &g = a.seg[s];
            const SegPrep &p = a.segp[s];
            const uint32_t rows = __ballot_sync(0xffffffffu, active);
            // the warp's rows in one segment with 64-bit bounds: eight lanes for each bound of its first and last row
            const uint32_t lead = __shfl_sync(0xffffffffu, s, 0);
            const bool together = rows && __all_sync(0xffffffffu, !active || (s == lead && p.fast));
            const uint64_t *us = a.us + g.u_off;
            uint64_t rem, lo[2] = {0, 0}, n[2] = {g.nu, g.nu};
            if (active) v = a.vs[j];
            if (together) {
                const uint64_t v_end = __shfl_sync(0xffffffffu, v, lane & 8 ? 31 - __clz(rows) : 0);
                const SegDev &gw = a.seg[lead];
                const uint64_t u = u_bound(gw, a.segp[lead], v_end, lane >= 16, rem);
                const uint64_t at = group_count_le64<3>(a.us + gw.u_off, gw.nu, u, lane);
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    lo[k] = __shfl_sync(0xffffffffu, at, 16 * k);
                    const uint64_t end = __shfl_sync(0xffffffffu, at, 16 * k + 8);
                    n[k] = end > lo[k] ? end - lo[k] : 0;
                }
            }
            if (active) {
                uint64_t at[2];
                if (p.fast) {
#pragma unroll
                    for (int k = 0; k < 2; ++k) at[k] = lo[k] + count_le64(us + lo[k], n[k], u_bound(g, p, v, k, rem));
                } else {
                    const u128 shift = mul_wide(v, g.A);
                    at[0] = count_le(us, g.nu, g.B, add128(shift, g.lo));
                    at[1] = count_le(us, g.nu, g.B, add128(shift, g.hi));
                }
                left = g.u_off + (uint32_t)at[0];
                right = g.u_off + (uint32_t)umax64(at[0], at[1]);
                const FamPrep &F = a.fam[g.fam];
#pragma unroll
                for (int f = 0; f < PC_MAX_BITSET; ++f)
                    if (f < (int)a.nb) {
                        const uint4 c = F.f[f];
                        row[f] = c.w + residue(c, v);
                    }
#pragma unroll
                for (int f = 0; f < PC_MAX_CHEAP; ++f)
                    if (f < (int)a.nch) {
                        const uint4 c = F.f[PC_MAX_BITSET + f];
                        cr |= (uint64_t)mod_short(residue(c, v) * c.w, c.z, c.y >> 16) << (16 * f);
                    }
                mine = tile_of(g, p, v);
            }
        }
        if (active) {
            if (mine == UINT64_MAX) atomicAdd(a.bad, 1ull);
            uint4 *out = (uint4 *)(a.rec + j);
            out[0] = make_uint4(left, right, (uint32_t)v, (uint32_t)(v >> 32));
            out[1] = make_uint4(row[0] | row[1] << 16, row[2] | row[3] << 16, row[4] | row[5] << 16, row[6] | row[7] << 16);
            a.cres[j] = cr;
        }
        // a warp's rows mostly share one subtile, which is summed over the warp's rounds
        const uint32_t width = right - left;
        const uint64_t common = __shfl_sync(0xffffffffu, mine, 0);
        if (__all_sync(0xffffffffu, mine == common)) {
            if (common != tile) {
                if (lane == 0 && tile != UINT64_MAX && pop) atomicAdd((unsigned long long *)&a.counts[tile * a.stride], (unsigned long long)pop);
                tile = common;
                pop = 0;
            }
            pop += __reduce_add_sync(0xffffffffu, width & 0xffffu) + ((uint64_t)__reduce_add_sync(0xffffffffu, width >> 16) << 16);
        } else if (mine != UINT64_MAX && width) {
            atomicAdd((unsigned long long *)&a.counts[mine * a.stride], (unsigned long long)width);
        }
    }
    if (lane == 0 && tile != UINT64_MAX && pop) atomicAdd((unsigned long long *)&a.counts[tile * a.stride], (unsigned long long)pop);
}

// Per subtile: u count and v count of its envelope (searchsorted bounds of
// batch_experiment.py:37-43, as list-independent differences).  A warp per subtile, eight lanes per bound.  Bound:
// the latency of the searches' dependent loads (against a thread per subtile with four searches in turn: a batch
// 13 -> 5 us, a lease's 16,384 subtiles 37 us either way).
__global__ void __launch_bounds__(256) k_geometry(const uint64_t *__restrict__ us, const uint64_t *__restrict__ vs,
                                                  const SegDev *__restrict__ seg, const uint32_t *__restrict__ tile_seg,
                                                  uint64_t ntiles, uint64_t *__restrict__ geometry) {
    const uint32_t lane = threadIdx.x & 31, which = lane >> 3;
    const uint64_t t = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    if (t >= ntiles) return;                              // warp-uniform
    const SegDev &g = seg[tile_seg[t]];
    const uint64_t first = g.v_first + (t - g.tile_base) * g.width;
    const uint64_t end = umin64(first + g.width, g.v_end);
    const uint64_t *su = us + g.u_off, *sv = vs + g.v_off;
    // groups 0 and 1: u B <= first A + lo, (end - 1) A + hi; groups 2 and 3: v < first, end
    const u128 key = which == 0 ? add128(mul_wide(first, g.A), g.lo) : add128(mul_wide(end - 1, g.A), g.hi);
    const uint64_t vkey = which == 2 ? first : end;
    const uint64_t n = group_prefix(which < 2 ? g.nu : g.nv, lane, [&](uint64_t i) {
        return which < 2 ? !less128(key, mul_wide(__ldg(su + i), g.B)) : __ldg(sv + i) < vkey;
    });
    const uint64_t ua = __shfl_sync(0xffffffffu, n, 0), ub = __shfl_sync(0xffffffffu, n, 8);
    const uint64_t va = __shfl_sync(0xffffffffu, n, 16), vb = __shfl_sync(0xffffffffu, n, 24);
    if (lane == 0) {
        geometry[2 * t] = ub > ua ? ub - ua : 0;
        geometry[2 * t + 1] = vb - va;
    }
}

// Per u block of UB entries: [va, vb) of v rows whose [left, right) meets the block, and the
// sub-range [f0, f1) of rows covering the whole block (left <= start and right >= stop); left and
// right are monotone in the row index within a segment, so all four are searches: a warp per block, eight lanes
// each (against a thread per block with four searches in turn: a batch 24 -> 5 us, a lease 57 -> 18).
__global__ void __launch_bounds__(256) k_blocks(const VRec *__restrict__ rec, const SegDev *__restrict__ seg, uint32_t nseg,
                                                uint32_t UB, uint64_t nblocks, uint4 *__restrict__ bv,
                                                uint32_t *__restrict__ blk_seg) {
    const uint32_t lane = threadIdx.x & 31, which = lane >> 3;
    const uint64_t b = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    if (b < nblocks) {                                    // warp-uniform
        const uint64_t start = b * UB;
        const uint32_t s = seg_of_u(seg, nseg, start);
        const SegDev &g = seg[s];
        const uint64_t u_end = (uint64_t)g.u_off + g.nu;
        uint4 range = make_uint4(0, 0, 0, 0);             // also for the padding between segments
        if (start < u_end) {
            const uint64_t stop = umin64(u_end, start + UB);
            // groups: va (right > start), vb (left >= stop), f0 (right >= stop), f1 (left > start)
            const uint64_t x = which == 0 || which == 3 ? start + 1 : stop;
            const uint32_t n = (uint32_t)group_prefix(g.nv, lane, [&](uint64_t i) {
                const VRec &r = rec[g.v_off + i];
                return (which & 1 ? r.left : r.right) < x;
            });
            const uint32_t va = __shfl_sync(0xffffffffu, n, 0), vb = max(va, __shfl_sync(0xffffffffu, n, 8));
            const uint32_t f0 = min(max(__shfl_sync(0xffffffffu, n, 16), va), vb), f1 = min(__shfl_sync(0xffffffffu, n, 24), vb);
            range = make_uint4(g.v_off + va, g.v_off + vb, g.v_off + f0, g.v_off + max(f0, f1));
        }
        if (lane == 0) {
            bv[b] = range;
            blk_seg[b] = s;
        }
    }
}

// Work of the blocks before each block: its v rows and, where it has any, the fixed cost of a block in rows.  Then all
// work, and its division among `grid` CTAs.  One CTA: a lease has 1e4 blocks, two turns of 8,192.
constexpr uint32_t PIECES_T = 1024, PIECES_PER = 8;

__global__ void __launch_bounds__(PIECES_T) k_pieces(const uint4 *__restrict__ bv, uint64_t nblocks, uint32_t block_cost,
                                                     uint32_t grid, uint64_t *__restrict__ prefix) {
    __shared__ uint64_t warp_s[PIECES_T / 32];
    __shared__ uint32_t most_s[PIECES_T / 32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t before = 0;                                  // work of the blocks of earlier turns
    uint32_t most = 0;                                    // of the thread's largest block
    for (uint64_t base = 0; base < nblocks; base += PIECES_T * PIECES_PER) {
        const uint64_t b0 = base + threadIdx.x * PIECES_PER;
        uint32_t rows[PIECES_PER];
        uint64_t own = 0;
#pragma unroll
        for (uint32_t k = 0; k < PIECES_PER; ++k) {
            const uint4 r = b0 + k < nblocks ? bv[b0 + k] : make_uint4(0, 0, 0, 0);
            own += rows[k] = r.y != r.x ? r.y - r.x + block_cost : 0;
            most = max(most, rows[k]);
        }
        uint64_t incl = own;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint64_t y = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= (uint32_t)d) incl += y;
        }
        __syncthreads();                                  // the previous turn's sums have been read
        if (lane == 31) warp_s[warp] = incl;
        __syncthreads();
        uint64_t at = before + incl - own;
        for (uint32_t w = 0; w < PIECES_T / 32; ++w) {
            if (w < warp) at += warp_s[w];
            before += warp_s[w];
        }
#pragma unroll
        for (uint32_t k = 0; k < PIECES_PER; ++k) {
            if (b0 + k < nblocks) prefix[b0 + k] = at;
            at += rows[k];
        }
    }
    most = __reduce_max_sync(0xffffffffu, most);
    if (lane == 0) most_s[warp] = most;
    __syncthreads();
    if (warp == 0) {
        most = __reduce_max_sync(0xffffffffu, most_s[lane]);
        const Shares shares = divide_work(before, most, nblocks, grid, block_cost);
        if (lane == 0) {
            prefix[nblocks] = before;
            prefix[nblocks + 1] = (uint64_t)shares.pairs << 32 | shares.n;
        }
    }
}

// ------------------------------------------------------------------------------------------
// the fused kernel

template <int K>
struct Geo {
    static constexpr int U = K / 4;                      // 16-byte units per row
    static constexpr int UB = K * 32;                    // u entries per block
    __device__ static __forceinline__ uint32_t unit(uint32_t row, uint32_t c) { return row * U + c; }
};

// Residues of the block's u entries: t = u B A^-1 mod q of the bitset filters (t_s) and u B mod q of the cheap tier
// (ures).  A warp takes 32 entries and every other filter.
template <int NB, int K>
__device__ __forceinline__ void block_residues(const uint64_t *__restrict__ us, const FamDev &F, uint32_t nch,
                                               uint16_t *__restrict__ t_s, uint16_t *__restrict__ ures, uint32_t block_u0,
                                               uint32_t n_valid, uint32_t lane, uint32_t warp, uint32_t nwarps) {
    constexpr uint32_t UB = Geo<K>::UB;
    for (uint32_t task0 = warp; task0 < 2 * K; task0 += 3 * nwarps) {
        uint64_t u[3];                                    // loaded together: 64 tasks are three turns of 28 warps
#pragma unroll
        for (uint32_t i = 0; i < 3; ++i) {
            const uint32_t task = task0 + i * nwarps, k = task / 2 * 32 + lane;
            u[i] = task < 2 * K && k < n_valid ? __ldg(us + block_u0 + k) : 0;
        }
#pragma unroll
        for (uint32_t i = 0; i < 3; ++i) {
            const uint32_t task = task0 + i * nwarps, k = task / 2 * 32 + lane, odd = task & 1;
            if (task >= 2 * K) break;
            auto put = [&](uint32_t f, uint16_t *to) {
                const uint4 m = F.umod[f];
                to[k] = (uint16_t)mod_short(residue(m, u[i]) * m.w, m.z, m.y >> 16);
            };
#pragma unroll
            for (uint32_t h = 0; h < (NB + 1) / 2; ++h) {
                const uint32_t f = 2 * h + odd;
                if (f < NB) put(f, t_s + f * UB);
            }
#pragma unroll
            for (uint32_t h = 0; h < PC_MAX_CHEAP / 2; ++h) {
                const uint32_t c = 2 * h + odd;
                if (c < nch) put(PC_MAX_BITSET + c, ures + c * UB);
            }
        }
    }
}

// Residue rows of the family's first NB filters for one block (entries >= n_valid are zero).  A warp builds 32 rows
// of one filter, four 16-byte units at a time: a lane's column of a word is the filter's
// pattern from offset 32 g + q - t on, one funnel shift, and a warp transpose turns 32 columns into 32 rows' words.
// Before they are stored the lanes rotate their units, so that at each store eight neighbouring lanes, whose rows
// lie a multiple of the banks apart, write four different units.  (Two units per warp and filter, stored from two
// lane halves, meet four bank conflicts a store and ten shuffles per word pair: 15.5 -> 11 us of a block's 16.5.
// Eight units at a time have no conflicts, but their 32 words spill: 13.4.)
template <int NB, int K>
__device__ __forceinline__ void build_rows(const FamDev &F, uint4 *__restrict__ rows, const uint16_t *__restrict__ t_s,
                                           const uint32_t *__restrict__ pat_s, uint32_t n_valid, uint32_t lane, uint32_t warp,
                                           uint32_t nwarps) {
    using G = Geo<K>;
    constexpr uint32_t UN = 4;                            // units at a time
    const TransposePair transpose(lane);
    const uint32_t turn = G::U == 4 ? (lane >> 1) & 3 : lane & 3;
    uint32_t f = 0, g = warp;                             // 32-row group g of filter f
    for (;; g += nwarps) {
        while (f < NB && g >= (F.q[f] + 31) / 32) g -= (F.q[f] + 31) / 32, ++f;
        if (f >= NB) return;
        const uint32_t q = F.q[f], r = 32 * g + lane;
        const uint32_t *p = pat_s + f * PATW;
        const uint16_t *t = t_s + f * G::UB + lane;
#pragma unroll 1
        for (uint32_t u0 = 0; u0 < G::U; u0 += UN) {
            uint32_t w[4 * UN];
#pragma unroll
            for (uint32_t k = 0; k < 4 * UN; ++k) {
                const uint32_t st = 32 * g + q - t[u0 * 128 + k * 32];
                w[k] = __funnelshift_r(p[st >> 5], p[(st >> 5) + 1], st & 31);
            }
            transpose.operator()<UN>(w);
            transpose.operator()<UN>(w + 2 * UN);
            if (n_valid < G::UB) {
#pragma unroll
                for (uint32_t k = 0; k < 4 * UN; ++k) {
                    const uint32_t first = u0 * 128 + k * 32;
                    w[k] &= low_bits(n_valid > first ? min(n_valid - first, 32u) : 0u);
                }
            }
#pragma unroll
            for (uint32_t s = 1; s < UN; s *= 2) {        // unit u becomes unit (u + turn) % UN
                uint32_t x[4 * UN];
#pragma unroll
                for (uint32_t k = 0; k < 4 * UN; ++k) x[k] = turn & s ? w[(k + 4 * s) % (4 * UN)] : w[k];
#pragma unroll
                for (uint32_t k = 0; k < 4 * UN; ++k) w[k] = x[k];
            }
            if (r < q) {
                uint4 *row = rows + G::unit(F.row0[f] + r, u0);
#pragma unroll
                for (uint32_t u = 0; u < UN; ++u)
                    row[(u + turn) & (UN - 1)] = make_uint4(w[4 * u], w[4 * u + 1], w[4 * u + 2], w[4 * u + 3]);
            }
        }
    }
}

// The rows that a few v rows read, instead of all rows of the block: a warp takes one filter's row of one v row, word by
// word: each lane looks up its entry's bit, a vote makes the word, and lane w keeps word w for one coalesced store.
template <int NB, int K>
__device__ __forceinline__ void sparse_rows(const FamDev &F, const VRec *__restrict__ rec, uint32_t nv, uint32_t *__restrict__ rows,
                                            const uint16_t *__restrict__ t_s, const uint32_t *__restrict__ pat_s,
                                            uint32_t n_valid, uint32_t lane, uint32_t warp, uint32_t nwarps) {
    using G = Geo<K>;
    for (uint32_t task = warp; task < nv * NB; task += nwarps) {
        const uint32_t f = task % NB, row = rec[task / NB].row[f], st0 = row - F.row0[f] + F.q[f];
        const uint32_t *p = pat_s + f * PATW;
        const uint16_t *t = t_s + f * G::UB + lane;
        for (uint32_t w0 = 0; w0 < K; w0 += 32) {
            uint32_t mine = 0;
#pragma unroll 8
            for (uint32_t w = 0; w < (K < 32 ? K : 32); ++w) {
                const uint32_t k = (w0 + w) * 32, st = st0 - t[k];
                const uint32_t word = __ballot_sync(0xffffffffu, k + lane < n_valid && (p[st >> 5] >> (st & 31) & 1u));
                if (w == lane) mine = word;
            }
            if (w0 + lane < K) rows[row * K + w0 + lane] = mine;
        }
    }
}

constexpr int CBW = 64;                 // bitmap words per cheap-tier filter (q <= 2047)
constexpr uint32_t ITEM_ROWS = 1u << 20;   // most v rows of a work item (a ring entry holds the row in 20 bits)
// Survivor ring per warp (pending < 64 by construction).  An entry is one word pair: the record's
// index in the work item (< 2^20) | the bit's position in the block (< 2^12) << 20, and the
// survivor's subtile slot; the drain reads the v row's cheap-tier residues by the record index.
constexpr int QCAP = 64;
// Leftover list per warp: a piece's marked units after its first, as the record's index in the
// work item | the unit << 20 | the subtile slot << 24 (255: recomputed from v), recomputed 32 at a
// time so the round loop does not wait on a few lanes.
constexpr int LCAP = 32;

__host__ __device__ constexpr uint32_t round16(uint32_t x) { return (x + 15) & ~15u; }

// Shared-memory layout of k_match (byte offsets); every region starts 16-byte aligned.  The u entries' residues t and
// the residue-row patterns are only read while rows are built, when every survivor ring is empty,
// so they share the rings' space.
struct MatchSmem {
    uint32_t rows, ures, ring, lq, t, pat, cbits, cnt, fam, seg, misc, place, total;
    __host__ __device__ MatchSmem(uint32_t total_rows, uint32_t K, uint32_t nb, uint32_t nch, uint32_t tmax,
                                  uint32_t ng, uint32_t warps) {
        rows = 0;
        ures = rows + total_rows * (K / 4) * 16;
        ring = ures + round16(nch * K * 32 * 2);
        lq = ring + warps * QCAP * 8;
        t = ring;
        pat = t + nb * K * 32 * 2;
        const uint32_t ring_end = lq + warps * LCAP * 4, pat_end = pat + nb * PATW * 4;
        cbits = round16(ring_end > pat_end ? ring_end : pat_end);
        cnt = cbits + nch * CBW * 4;
        fam = cnt + round16(tmax * (ng + 2) * 4);
        seg = fam + round16(sizeof(FamDev));
        misc = seg + round16(sizeof(SegDev));
        place = misc + 32;   // after the deep counter (4 B), the division of the work (8 B at +8), the item's first
                             // subtile and its segment's subtile end (8 B each at +16 and +24)
        total = place + 48;
    }
};

__device__ __forceinline__ uint32_t unit_mask(int32_t lo, int32_t hi) {   // bits [lo, hi) of one 32-bit word
    return low_bits((uint32_t)min(max(hi, 0), 32)) & ~low_bits((uint32_t)min(max(lo, 0), 32));
}

__device__ __forceinline__ uint4 lds128(uint32_t addr) {      // 16-byte shared-memory load
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}

// The unit loop of one (v row, block) piece, from the shared address of each filter's row: AND of
// the NB rows per 16-byte unit, range masks unless the row covers the whole block (FULL), the
// group-1 popcount (first four filters) and, when group 2 ends at the last bitset filter (C2), the
// group-2 popcount.  Returns the mask of units that keep a bit after every bitset filter; save
// receives the bits of the last of them.
template <int NB, int U, bool FULL, bool C2>
__device__ __forceinline__ uint32_t piece_units(const uint32_t (&rb)[NB], uint32_t lane, int32_t s, int32_t e,
                                                uint32_t (&c)[2], uint4 &save) {
    uint32_t pend = 0;
#pragma unroll
    for (uint32_t p = 0; p < U; ++p) {
        const uint32_t u = (lane + p) & (U - 1), uo = u * 16;
        uint4 acc = lds128(rb[0] + uo);
        uint4 acc4;
#pragma unroll
        for (int f = 1; f < NB; ++f) {
            if (f == 4) acc4 = acc;
            const uint4 w = lds128(rb[f] + uo);
            acc.x &= w.x;
            acc.y &= w.y;
            acc.z &= w.z;
            acc.w &= w.w;
        }
        if (NB <= 4) acc4 = acc;
        if (!FULL) {
            const int32_t lo = s - (int32_t)u * 128, hi = e - (int32_t)u * 128;
            const uint32_t m0 = unit_mask(lo, hi), m1 = unit_mask(lo - 32, hi - 32);
            const uint32_t m2 = unit_mask(lo - 64, hi - 64), m3 = unit_mask(lo - 96, hi - 96);
            acc.x &= m0, acc.y &= m1, acc.z &= m2, acc.w &= m3;
            acc4.x &= m0, acc4.y &= m1, acc4.z &= m2, acc4.w &= m3;
        }
        c[0] += __popc(acc4.x) + __popc(acc4.y) + __popc(acc4.z) + __popc(acc4.w);
        if (C2) c[1] += __popc(acc.x) + __popc(acc.y) + __popc(acc.z) + __popc(acc.w);
        const bool live = (acc.x | acc.y | acc.z | acc.w) != 0;
        if (live) save = acc;                         // the last marked unit is not read again
        pend |= (uint32_t)live << p;
    }
    return pend;
}

__device__ __forceinline__ void copy_words(void *dst, const void *src, uint32_t bytes) {
    for (uint32_t i = threadIdx.x; i < bytes / 4; i += blockDim.x) ((uint32_t *)dst)[i] = ((const uint32_t *)src)[i];
}

// One lane owns one (v row, u block) piece: it walks the block's K/4 16-byte units in the order
// (lane + p) mod (K/4), so at every step the 32 lanes of a warp hit each 16-byte bank group
// exactly 32/(K/4) times whatever rows they read.  The group-1 and group-2 counters live in
// registers (c[0..1]) and are reduced per subtile when a lane's subtile changes.  The unit loop
// only marks the units that keep a bit after every bitset filter (and keeps the bits of the last
// one in registers); once the piece is done, each lane queues that unit's bits and puts its other
// marked units on a per-warp leftover list, recomputed 32 at a time, so the warp votes and
// diverges once per piece instead of after every unit, and never waits on a few lanes' units.
template <int NB, int K, int NT>
__global__ void __launch_bounds__(NT, 1) k_match(const MatchArgs a) {
    using G = Geo<K>;
    constexpr uint32_t U = G::U;
    extern __shared__ uint4 smem[];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const uint32_t ngmax = a.stride - 3;
    const MatchSmem L(a.total_rows, K, NB, a.nch, a.tmax, ngmax, nwarps);
    char *base = (char *)smem;
    const uint4 *rows = (const uint4 *)(base + L.rows);
    const uint32_t rows_addr = (uint32_t)__cvta_generic_to_shared(rows);
    uint16_t *ures = (uint16_t *)(base + L.ures);
    uint2 *qv = (uint2 *)(base + L.ring) + warp * QCAP;
    uint32_t *lq = (uint32_t *)(base + L.lq) + warp * LCAP;
    uint32_t *pat_s = (uint32_t *)(base + L.pat);
    uint32_t *cbits = (uint32_t *)(base + L.cbits);
    uint32_t *cnt_s = (uint32_t *)(base + L.cnt);      // tmax x (ngmax+2): groups 1..ng
    FamDev &F = *(FamDev *)(base + L.fam);
    SegDev &S = *(SegDev *)(base + L.seg);
    uint32_t *deep_ctr = (uint32_t *)(base + L.misc);
    volatile uint64_t *item_s = (volatile uint64_t *)(base + L.misc + 16);
    const uint32_t cstride = ngmax + 2;

    const uint32_t lanes_below = (1u << lane) - 1u;
    if (threadIdx.x == 0) *deep_ctr = 0;
    uint4 *deep_slice = a.deep + (size_t)blockIdx.x * a.deep_cap;

    uint64_t cur = UINT64_MAX;
    uint32_t cur_seg = UINT32_MAX, cur_fam = UINT32_MAX;
    const uint32_t nch = a.nch;

    // A CTA works through shares (divide_work); claimed in ascending order, they keep the CTAs on neighbouring blocks, whose
    // per-v records then stay in L2.  The division and the place in the share stay in shared memory (shares, place): no
    // register holds them through the unit loop.
    struct Place {
        uint64_t share, b, b_end, at, at_end;             // next share; next block, end of the share's blocks, its work
        uint32_t row, first;                              // rows of block b that are done; b is the share's first
    };
    volatile Place &place = *(volatile Place *)(base + L.place);
    volatile Shares &shares = *(volatile Shares *)(base + L.misc + 8);
    if (threadIdx.x == 0) {
        place.share = blockIdx.x, place.b = place.b_end = 0;
        const uint64_t division = a.prefix[a.nblocks + 1];
        shares.n = (uint32_t)division, shares.pairs = (uint32_t)(division >> 32);
    }
    __syncthreads();
    for (;;) {
        uint64_t b = place.b;
        uint32_t row = place.row;
        if (b >= place.b_end) {
            const uint64_t share = place.share;
            const uint32_t nshares = shares.n, pairs = shares.pairs;
            if (share >= nshares) break;
            uint64_t b_end, at = 0, at_end = 0;
            if (pairs) {
                b = share < pairs ? 2 * share : pairs + share;
                b_end = b + (share < pairs ? 2 : 1);
            } else {
                const uint64_t work = a.prefix[a.nblocks];
                at = work * share / nshares;
                at_end = work * (share + 1) / nshares;
                b_end = b = group_count_le64<5>(a.prefix, a.nblocks, at, lane) - 1;     // last block that starts at or before it
                if (at != at_end) b_end = group_count_le64<5>(a.prefix, a.nblocks, at_end - 1, lane);
            }
            __syncthreads();                              // every thread has read the place
            if (threadIdx.x == 0) {
                place.b = b, place.b_end = b_end, place.at = at, place.at_end = at_end;
                place.row = 0, place.first = 1;
                place.share = gridDim.x + atomicAdd(a.share_next, 1ull);
            }
            __syncthreads();
            continue;
        }
        const uint4 range = a.bv[b];
        uint32_t rows_end = range.y - range.x;            // rows of the block in this share
        if (!shares.pairs) cut_rows(a.prefix[b] + a.block_cost, place.first ? place.at : 0, place.at_end, row, rows_end);
        const uint64_t va = range.x + row;
        const uint32_t nv_item = min(rows_end - row, a.v_chunk);   // <= 2^20
        __syncthreads();                                  // every thread has read the place
        if (threadIdx.x == 0) {                           // the next item (the item's syncs come before its use)
            const bool done = row + nv_item == rows_end;
            place.b = done ? b + 1 : b;
            place.row = done ? 0 : row + nv_item;
            if (done) place.first = 0;
        }
        if (!nv_item) {
            __syncthreads();
            continue;
        }
        // rows of this item covering the whole block, relative to va
        const uint32_t full_lo = (uint32_t)(range.z > va ? umin64(range.z - va, nv_item) : 0);
        const uint32_t full_hi = (uint32_t)(range.w > va ? umin64(range.w - va, nv_item) : 0);
        const uint32_t block_u0 = (uint32_t)(b * G::UB);
        if (b != cur) {
            const uint32_t sg = a.blk_seg[b];
            if (sg != cur_seg) {
                const uint32_t fm = a.seg[sg].fam;
                copy_words(&S, a.seg + sg, sizeof(SegDev));
                if (fm != cur_fam) copy_words(&F, a.fam + fm, sizeof(FamDev));
                __syncthreads();
                if (fm != cur_fam) {
                    for (uint32_t i = threadIdx.x; i < nch * CBW; i += blockDim.x) {
                        const uint32_t t = i / CBW, w = i % CBW;
                        cbits[i] = w * 32 < F.cq[t] ? F.bits[F.cbits_off[t] + w] : 0u;
                    }
                }
                cur_seg = sg;
                cur_fam = fm;
            }
            const uint32_t u_end = S.u_off + S.nu;
            const uint32_t n_valid = u_end > block_u0 ? min(u_end - block_u0, (uint32_t)G::UB) : 0u;
            for (uint32_t i = threadIdx.x; i < NB * PATW; i += blockDim.x) pat_s[i] = F.pat[i];
            block_residues<NB, K>(a.us, F, nch, (uint16_t *)(base + L.t), ures, block_u0, n_valid, lane, warp, nwarps);
            __syncthreads();
            // a vote makes 32 bits where the transpose makes 1,024 with some thirty times the instructions, so up to a
            // row in 12 NB (18 v rows at p = 619) it is less work to make only the rows that the item reads: 300 windows of
            // 1-2 10^6 positions 1.003 -> 0.851 ms of kernel, of 10^6-1.6 10^7 0.998 -> 0.949, leases the same (no such items)
            if (nv_item * NB * 12 <= F.total_rows) {
                sparse_rows<NB, K>(F, a.rec + va, nv_item, (uint32_t *)(base + L.rows), (const uint16_t *)(base + L.t), pat_s, n_valid,
                                   lane, warp, nwarps);
                cur = UINT64_MAX;                         // the block's other rows are not there
            } else {
                build_rows<NB, K>(F, (uint4 *)rows, (const uint16_t *)(base + L.t), pat_s, n_valid, lane, warp, nwarps);
                cur = b;
            }
        }
        for (uint32_t k = threadIdx.x; k < a.tmax * cstride; k += blockDim.x) cnt_s[k] = 0;
        if (threadIdx.x == 0) {                           // the item's first subtile, once per CTA
            item_s[0] = S.tile_base + local_tile(a.rec[va].v, S.v_first, S.width, S.ntiles);
            item_s[1] = (uint64_t)S.tile_base + S.ntiles;
        }
        __syncthreads();
        // subtile geometry of the segment and of the item stays in shared memory (S, item_s): it is
        // read when a lane's subtile changes, once per round for the survivor slots, and when a
        // queued survivor needs its subtile, so no register holds it through the unit loop
        const bool c2_live = F.c2_live != 0;
        volatile uint64_t &tile_base = item_s[0], &seg_tiles_end = item_s[1];

        uint32_t c[2] = {0, 0};                           // group 1 and (C2) group 2 survivors of the lane
        // this lane's subtile as a slot from the item's first one (NO_SLOT: none), and the end of its
        // v range (a lane's rows rise in v within an item)
        constexpr uint32_t NO_SLOT = 0xFFFFFFFFu;
        uint32_t cslot = NO_SLOT;
        uint64_t t_hi = 0;

        auto flush = [&]() {                              // populations reduced over lanes of a subtile
            const uint32_t key = (c[0] | c[1]) ? cslot : NO_SLOT - 1 - lane;
            const uint32_t same = __match_any_sync(0xffffffffu, key);
            const uint32_t leader = __ffs(same) - 1;
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                const uint32_t sum = __reduce_add_sync(same, c[g]);
                if (key == cslot && lane == leader && sum) {
                    if (cslot < a.tmax) atomicAdd(cnt_s + cslot * cstride + 1 + g, sum);
                    else {
                        const uint64_t tile = tile_base + cslot;
                        if (tile < seg_tiles_end)
                            atomicAdd((unsigned long long *)&a.counts[tile * a.stride + 1 + g], (unsigned long long)sum);
                    }
                }
                c[g] = 0;
            }
        };

        uint32_t qhead = 0, qtail = 0;                    // warp-uniform ring positions

        // Cheap-tier filters on up to 32 queued survivors, one per lane; survivors of all of them
        // go to this CTA's deep slice.
        auto drain = [&](uint32_t n) {
            __syncwarp();
            const bool mine = lane < n;
            uint32_t ent = 0, slot = 0;
            if (mine) {
                const uint2 q = qv[(qhead + lane) & (QCAP - 1)];
                ent = q.x, slot = q.y;
            }
            __syncwarp();
            qhead += n;
            if (!mine) return;
            const uint64_t tile = tile_base + slot;
            if (tile >= seg_tiles_end) return;            // v outside the subtile geometry (reported by k_vprep)
            const uint32_t uidx = ent >> 20;
            const uint64_t cr = __ldcg(a.cres + va + (ent & 0xFFFFFu));
            for (uint32_t t = 0; t < nch; ++t) {
                const uint32_t vr = (uint32_t)(cr >> (16 * t)) & 0xFFFFu, qg = F.cqg[t];
                int32_t m = (int32_t)ures[t * G::UB + uidx] - (int32_t)vr;
                if (m < 0) m += (int32_t)(qg & 0xFFFFu);
                if (!((cbits[t * CBW + (m >> 5)] >> (m & 31)) & 1u)) return;
                const uint32_t g = qg >> 16;
                if (g) {
                    if (slot < a.tmax) atomicAdd(cnt_s + slot * cstride + g, 1u);
                    else atomicAdd((unsigned long long *)&a.counts[tile * a.stride + g], 1ull);
                }
            }
            const uint32_t at = atomicAdd(deep_ctr, 1u);
            if (at < a.deep_cap) {
                const uint64_t v = a.rec[va + (ent & 0xFFFFFu)].v;
                deep_slice[at] = make_uint4((uint32_t)v, (uint32_t)(v >> 32), block_u0 + uidx, (uint32_t)tile);
            }
        };

        // The bits of one unit per lane go to the ring, one bit per lane per step (warp-uniform call).
        auto queue_bits = [&](uint4 acc, uint32_t u, uint32_t rel, uint32_t slot) {
            while (__any_sync(0xffffffffu, (acc.x | acc.y | acc.z | acc.w) != 0)) {
                const bool has = (acc.x | acc.y | acc.z | acc.w) != 0;
                const uint32_t bal = __ballot_sync(0xffffffffu, has);
                if (has) {
                    uint32_t bit;
                    if (acc.x) {
                        bit = __ffs(acc.x) - 1;
                        acc.x &= acc.x - 1;
                    } else if (acc.y) {
                        bit = 32 + __ffs(acc.y) - 1;
                        acc.y &= acc.y - 1;
                    } else if (acc.z) {
                        bit = 64 + __ffs(acc.z) - 1;
                        acc.z &= acc.z - 1;
                    } else {
                        bit = 96 + __ffs(acc.w) - 1;
                        acc.w &= acc.w - 1;
                    }
                    const uint32_t at = (qtail + __popc(bal & lanes_below)) & (QCAP - 1);
                    qv[at] = make_uint2(rel | ((u * 128 + bit) << 20), slot);
                }
                qtail += __popc(bal);
                if (qtail - qhead >= 32) drain(32);
            }
        };

        uint32_t nl = 0;                                  // warp-uniform leftover count
        // Up to 32 leftover units, one per lane: recomputed from the record, bits queued.
        auto leftovers = [&]() {
            __syncwarp();
            const bool mine = lane < nl;
            const uint32_t ent = mine ? lq[lane] : 0u;
            __syncwarp();
            nl = 0;
            uint4 acc = make_uint4(0, 0, 0, 0);
            const uint32_t rel = ent & 0xFFFFFu, u = (ent >> 20) & 0xFu;
            uint32_t slot = ent >> 24;
            if (mine) {
                VRec rr;                                  // from L2, like the round's record
                const uint4 *src = (const uint4 *)(a.rec + va + rel);
                const uint4 h0 = __ldcg(src), h1 = __ldcg(src + 1);
                memcpy(&rr, &h0, 16);
                memcpy((char *)&rr + 16, &h1, 16);
                if (slot == 255u) {
                    const uint64_t lt = local_tile(rr.v, S.v_first, S.width, S.ntiles);
                    slot = lt < S.ntiles ? (uint32_t)(S.tile_base + lt - tile_base) : NO_SLOT;
                }
                acc = lds128(rows_addr + ((uint32_t)rr.row[0] * U + u) * 16);
#pragma unroll
                for (int f = 1; f < NB; ++f) {
                    const uint4 w = lds128(rows_addr + ((uint32_t)rr.row[f] * U + u) * 16);
                    acc.x &= w.x;
                    acc.y &= w.y;
                    acc.z &= w.z;
                    acc.w &= w.w;
                }
                const int32_t s = max((int32_t)(rr.left - block_u0), 0);
                const int32_t e = max(min((int32_t)(rr.right - block_u0), (int32_t)G::UB), s);
                const int32_t lo = s - (int32_t)u * 128, hi = e - (int32_t)u * 128;
                acc.x &= unit_mask(lo, hi), acc.y &= unit_mask(lo - 32, hi - 32);
                acc.z &= unit_mask(lo - 64, hi - 64), acc.w &= unit_mask(lo - 96, hi - 96);
            }
            queue_bits(acc, u, rel, slot);
        };

        // a warp takes consecutive rounds, so its lanes stay in one subtile for many rounds; a round whose rows cover
        // only part of the block (the item's first and last ones) counts 9, a full one 8 (a lease: 10.51 ms, 10.53 at
        // 17 : 16, 10.59 at 1 : 1 and 10.79 with equal runs rounded up)
        const uint32_t nrounds = (nv_item + 31) / 32;
        const uint32_t fr = min((full_lo + 31) / 32, nrounds), lr = max(fr, full_hi / 32);    // the full rounds
        const uint32_t w1 = 9 * fr, w2 = w1 + 8 * (lr - fr), weight = w2 + 9 * (nrounds - lr);
        auto round_at = [&](uint32_t x) {
            return x <= w1 ? (x + 8) / 9 : x <= w2 ? fr + (x - w1 + 7) / 8 : lr + (x - w2 + 8) / 9;
        };
        const uint32_t r_end = round_at((warp + 1) * weight / nwarps);
        for (uint32_t r = round_at(warp * weight / nwarps); r < r_end; ++r) {
            const uint32_t rel = r * 32 + lane;
            const bool active = rel < nv_item;
            VRec rec{};
            if (active) {                                 // read once per block: cached in L2 only
                const uint4 *src = (const uint4 *)(a.rec + va + rel);
                const uint4 h0 = __ldcg(src), h1 = __ldcg(src + 1);
                memcpy(&rec, &h0, 16);
                memcpy((char *)&rec + 16, &h1, 16);
            }
            // warp-uniform: all 32 rows exist and cover the whole block
            const bool full = r * 32 >= full_lo && r * 32 + 32 <= full_hi;
            // piece as bits of the block, needed only where a row of the round covers part of it
            // (an inactive lane's zeroed record gives an empty piece)
            int32_t s = 0, e = (int32_t)G::UB;
            if (!full) {
                s = active ? max((int32_t)(rec.left - block_u0), 0) : 0;
                e = max(min((int32_t)(rec.right - block_u0), (int32_t)G::UB), s);
            }
            const bool moved = active && rec.v >= t_hi;
            if (__any_sync(0xffffffffu, moved)) {
                flush();
                if (moved) {
                    const uint64_t swidth = S.width;
                    if (cslot != NO_SLOT && rec.v - t_hi < 2 * swidth) {
                        // the next subtile or the one after it (the common step between rounds)
                        const bool two = rec.v - t_hi >= swidth;
                        cslot += two ? 2 : 1;
                        t_hi += two ? 2 * swidth : swidth;
                        if ((uint64_t)(tile_base + cslot) >= seg_tiles_end) cslot = NO_SLOT, t_hi = 0;
                    } else {
                        const uint64_t stn = S.ntiles;
                        const uint64_t lt = local_tile(rec.v, S.v_first, swidth, stn);
                        // slots fit 32 bits (an item's v rows lie in fewer than 2^31 subtiles)
                        cslot = lt < stn ? (uint32_t)(S.tile_base + lt - tile_base) : NO_SLOT;
                        const uint64_t t_lo = S.v_first + lt * swidth;
                        t_hi = lt < stn ? t_lo + swidth : t_lo;
                    }
                }
            }
            uint32_t rb[NB];                              // shared address of each filter's row
#pragma unroll
            for (int f = 0; f < NB; ++f) rb[f] = rows_addr + (uint32_t)rec.row[f] * (U * 16);   // row 0 if inactive

            // warp-uniform FULL and block-uniform C2 select the loop body, so the range masks and the
            // group-2 popcounts are not issued (as predicated code) where they cannot apply
            uint32_t pend;                                // units of this piece with survivors
            uint4 save;                                   // bits of the last one
            if (full)
                pend = c2_live ? piece_units<NB, U, true, true>(rb, lane, s, e, c, save)
                               : piece_units<NB, U, true, false>(rb, lane, s, e, c, save);
            else
                pend = c2_live ? piece_units<NB, U, false, true>(rb, lane, s, e, c, save)
                               : piece_units<NB, U, false, false>(rb, lane, s, e, c, save);
            // the last marked unit (its bits kept in registers) is queued now; the piece's other
            // marked units go to the leftover list
            uint4 acc = make_uint4(0, 0, 0, 0);
            uint32_t u = 0;
            if (pend) {
                const uint32_t pl = 31 - __clz(pend);
                u = (lane + pl) & (U - 1);
                acc = save;
                pend &= ~(1u << pl);
            }
            queue_bits(acc, u, rel, cslot);
            while (__any_sync(0xffffffffu, pend != 0)) {
                const bool has = pend != 0;
                const uint32_t bal = __ballot_sync(0xffffffffu, has);
                if (nl + __popc(bal) > LCAP) leftovers();
                if (has) {
                    lq[nl + __popc(bal & lanes_below)] =
                        rel | (((lane + __ffs(pend) - 1) & (U - 1)) << 20) | (min(cslot, 255u) << 24);
                    pend &= pend - 1;
                }
                nl += __popc(bal);
            }
        }
        if (nl) leftovers();
        if (qtail != qhead) drain(qtail - qhead);
        flush();
        __syncthreads();
        for (uint32_t k = threadIdx.x; k < a.tmax * cstride; k += blockDim.x) {
            const uint32_t cv = cnt_s[k];
            if (cv) {
                const uint32_t slot = k / cstride, g = k % cstride;
                const uint64_t tile = tile_base + slot;
                if (tile < seg_tiles_end)
                    atomicAdd((unsigned long long *)&a.counts[tile * a.stride + g], (unsigned long long)cv);
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) a.deep_count[blockIdx.x] = *deep_ctr;
}

// x mod q for x < 2^96 from its six 16-bit limbs h (h[0] + sum h[k] (2^16k mod q), then one
// fast remainder; every partial sum stays below 2^32 because q < 2^13).
__device__ __forceinline__ uint32_t mod_limbs(const uint32_t h[6], const FiltC &f) {
    uint32_t t = h[0] + h[1] * f.r16[0] + h[2] * f.r16[1] + h[3] * f.r16[2] + h[4] * f.r16[3] + h[5] * f.r16[4];
    return fastmod32(t, f.c, f.q);
}

// Exact later filters on every deep record: x = uB - vA in two 64-bit limbs, filters first..nres-1
// of the record's family with group counters, then the output record.  A lane tests the next DEEP_ALONE
// filters on its own record; the few records that pass them (1 in 6,000 where each keeps a third) are then
// tested one by one by the whole warp, a filter per lane, so none waits for eighty dependent table loads (against a
// lane per record to the end, where one record's chain is most of the time: a batch 32 -> 8 us).
constexpr uint32_t DEEP_ALONE = 8;

__global__ void __launch_bounds__(256) k_deep(const DeepArgs a) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t slice = blockIdx.y;
    const uint32_t count = min(a.deep_count[slice], a.deep_cap);
    for (uint32_t base = blockIdx.x * blockDim.x; base < count; base += gridDim.x * blockDim.x) {
        const uint32_t at = base + threadIdx.x;
        const uint64_t i = (uint64_t)slice * a.deep_cap + at;
        bool pass = false;
        u128 x{0, 0};
        uint32_t tile = 0, fam = 0;
        auto limbs = [](const u128 &y, uint32_t (&h)[6]) {
            h[0] = (uint32_t)y.lo & 0xffffu, h[1] = (uint32_t)(y.lo >> 16) & 0xffffu;
            h[2] = (uint32_t)(y.lo >> 32) & 0xffffu, h[3] = (uint32_t)(y.lo >> 48);
            h[4] = (uint32_t)y.hi & 0xffffu, h[5] = (uint32_t)(y.hi >> 16) & 0xffffu;
        };
        auto allowed = [](const FamDev &F, uint32_t idx, const uint32_t (&h)[6]) {
            const FiltC f = F.fcs[idx];
            const uint32_t m = mod_limbs(h, f);
            return (__ldg(F.bits + f.tab_off + (m >> 5)) >> (m & 31)) & 1u;
        };
        if (at < count) {
            const uint4 r = a.deep[i];
            const uint64_t v = (uint64_t)r.y << 32 | r.x;
            tile = r.w;
            if (tile < a.ntiles) {
                const SegDev &g = a.seg[a.tile_seg[tile]];
                fam = g.fam;
                const FamDev &F = a.fam[fam];
                const u128 pos = mul_wide(__ldg(a.us + r.z), g.B), shift = mul_wide(v, g.A);
                if (less128(pos, shift)) {
                    atomicAdd((unsigned long long *)&a.counts[(uint64_t)tile * a.stride + F.ng + 2], 1ull);
                } else {
                    x = sub128(pos, shift);
                    uint32_t h[6];
                    limbs(x, h);
                    pass = true;
                    const uint32_t stop = min(F.nres, a.first + DEEP_ALONE);
                    for (uint32_t idx = a.first; idx < stop; ++idx) {
                        if (!allowed(F, idx, h)) {
                            pass = false;
                            break;
                        }
                        if ((idx & 3) == 3 || idx + 1 == F.nres)
                            atomicAdd((unsigned long long *)&a.counts[(uint64_t)tile * a.stride + idx / 4 + 1], 1ull);
                    }
                }
            }
        }
        for (uint32_t left = __ballot_sync(0xffffffffu, pass); left; left &= left - 1) {
            const uint32_t src = __ffs(left) - 1;
            const u128 y{__shfl_sync(0xffffffffu, x.lo, src), __shfl_sync(0xffffffffu, x.hi, src)};
            const uint64_t t = __shfl_sync(0xffffffffu, tile, src);
            const FamDev &F = a.fam[__shfl_sync(0xffffffffu, fam, src)];
            uint64_t *counts = a.counts + t * a.stride;
            uint32_t h[6];
            limbs(y, h);
            const uint32_t nres = F.nres;
            bool ok = true;
            for (uint32_t idx0 = a.first + DEEP_ALONE; ok && idx0 < nres; idx0 += 32) {
                const uint32_t idx = idx0 + lane;
                const bool fails = idx < nres && !allowed(F, idx, h);
                const uint32_t failed = __ballot_sync(0xffffffffu, fails);
                const uint32_t until = failed ? idx0 + __ffs(failed) - 1 : idx0 + 32;    // filters below it have passed
                if (idx < until && ((idx & 3) == 3 || idx + 1 == nres) && idx < nres)
                    atomicAdd((unsigned long long *)&counts[idx / 4 + 1], 1ull);
                ok = !failed;
            }
            if (ok && lane == 0) {
                atomicAdd((unsigned long long *)&counts[F.ng + 1], 1ull);
                const unsigned long long o = atomicAdd(a.n_out, 1ull);
                if (o < a.out_cap) {
                    a.out[2 * o] = y.lo;
                    a.out[2 * o + 1] = y.hi | (t << 32);
                }
            }
        }
    }
}

// ------------------------------------------------------------------------------------------
// plain per-position matcher (pseudocube/gpu.py:147-182)
//
// A CTA owns PLAIN_U consecutive u entries and a run of v rows.  Each thread keeps the residues
// u*B mod q of the first four filters for its u entries in registers; a v row brings its residues
// v*A mod q and its exact u interval (clipped to the CTA's entries) through shared memory, so a position
// costs one subtraction and one bitmap lookup per filter (x mod q = (uB - vA) mod q).  The 1 in 81
// positions that pass are queued per warp and finished 32 at a time in 128-bit arithmetic, filter by
// filter.  The work is split over u chunks and v runs, so a tile of ten v rows fills the device (against a
// warp per v row, which walks 17,400 u entries: 570 -> 11 us).  It takes 275 instructions of a warp for 128 positions, so
// from 64 v rows on (a tile of 7 10^6 positions) k_plain_rows takes over.

constexpr uint32_t PLAIN_T = 256, PLAIN_PER = 4, PLAIN_U = PLAIN_T * PLAIN_PER;   // threads, u entries per thread, per CTA
constexpr uint32_t PLAIN_V = 64;                  // v rows staged at a time
constexpr uint32_t PLAIN_FIRST = 4;               // filters tested from residues (the first group)
constexpr uint32_t PLAIN_QUEUE = 256;             // queued positions per warp (31 left over and 128 of one row fit)
constexpr uint32_t PLAIN_WORDS = 256;             // bitmap words per filter (q < 8192)
constexpr uint64_t PLAIN_RUN_MAX = UINT64_C(1) << 21;   // v rows per CTA (a queue entry holds the row in 22 bits)

struct PlainArgs {
    const uint64_t *us;
    const uint64_t *vs;
    uint64_t nu, nv, A, B;
    u128 lo, hi;
    uint32_t nres, ng;
    const FiltConst *fc;
    const uint32_t *bits;
    uint64_t *counts;
    uint64_t *out;
    uint64_t out_cap;
    uint64_t run;                                 // v rows per CTA
    bool ordered;                                 // the v rows may be in order: a CTA looks for those it shares positions with
    const uint64_t *disorder;                     // where the device found whether they are: 0 (null: they are)
    uint32_t aq[PLAIN_FIRST], bq[PLAIN_FIRST];    // A mod q, B mod q of the first filters
};

// A position that passed the first nf filters: the others on x = uB - vA in two limbs.
__device__ __forceinline__ void plain_rest(const PlainArgs &a, const u128 x, uint32_t nf, unsigned long long *cnt) {
    for (uint32_t idx = nf; idx < a.nres; ++idx) {
        const FiltConst fc = a.fc[idx];
        const uint32_t m = mod128(x, fc.m);
        if (!((__ldg(a.bits + fc.tab_off + (m >> 5)) >> (m & 31)) & 1u)) return;
        if ((idx & 3) == 3 || idx + 1 == a.nres) atomicAdd(&cnt[idx / 4 + 1], 1ull);
    }
    const unsigned long long slot = atomicAdd((unsigned long long *)&a.counts[a.ng + 1], 1ull);
    if (slot < a.out_cap) {
        a.out[2 * slot] = x.lo;
        a.out[2 * slot + 1] = x.hi;
    }
}

// Sets *disorder when a v row is below the one before it.
__global__ void __launch_bounds__(256) k_order(const uint64_t *__restrict__ vs, uint64_t nv, uint64_t *__restrict__ disorder) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x + 1; i < nv; i += (uint64_t)gridDim.x * blockDim.x)
        if (vs[i] < vs[i - 1]) *disorder = 1;
}

// Narrows the CTA's v rows [j0, j1) to those whose interval meets its entries us[0, n), which are consecutive when the rows
// are in order and no v A + hi or v A + lo wraps.  Without it each CTA looks at every row of its run: 4.3e5 u entries and
// 6.8e5 v rows that meet one entry each, or 87, take 32.8 ms, with it 0.17 and 0.21; 6e4 and 6.7e4, where a row meets a third of
// the entries, 0.92 and 0.52 ms.
constexpr uint64_t PLAIN_ORDERED_MIN = UINT64_C(1) << 28;   // (u, v) pairs: some 0.1 ms where every CTA looks at every row,
                                                            // against 3 us for k_order and the search; a tile has 5 10^7 at most
__device__ __forceinline__ void plain_band(const PlainArgs &a, const uint64_t *us, uint32_t n, uint64_t &j0, uint64_t &j1) {
    __shared__ uint64_t band_s[2];
    if (a.disorder && *a.disorder) return;
    if (threadIdx.x < 32) {                       // eight lanes each: rows that end below the entries, that start below the last
        const uint32_t lane = threadIdx.x, which = lane >> 3 & 1;
        const u128 edge = mul_wide(__ldg(us + (which ? n - 1 : 0)), a.B), bound = which ? a.lo : a.hi;
        const uint64_t rows = group_prefix(j1 - j0, lane, [&](uint64_t i) {
            return less128(add128(mul_wide(__ldg(a.vs + j0 + i), a.A), bound), edge);
        });
        if (lane == 0 || lane == 8) band_s[which] = rows;
    }
    __syncthreads();
    j1 = j0 + band_s[1];
    j0 += band_s[0];
}

template <bool ORDERED>
__global__ void __launch_bounds__(PLAIN_T) k_plain(const PlainArgs a) {
    __shared__ unsigned long long cnt[PC_MAX_RES / 4 + 4];
    __shared__ uint32_t bits_s[PLAIN_FIRST][PLAIN_WORDS];
    __shared__ uint4 row_s[PLAIN_V];              // interval start | end << 16, residues of filters 0-1 and 2-3
    __shared__ uint32_t queue_s[PLAIN_T / 32][PLAIN_QUEUE];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lanes_below = (1u << lane) - 1u;
    const uint32_t nf = min(a.nres, PLAIN_FIRST);
    const uint64_t c0 = blockIdx.x * (uint64_t)PLAIN_U;
    const uint32_t n_here = (uint32_t)umin64(a.nu - c0, PLAIN_U);
    uint64_t j0 = blockIdx.y * a.run, j1 = umin64(a.nv, j0 + a.run);
    const uint64_t *us = a.us + c0;
    if (ORDERED) {
        plain_band(a, us, n_here, j0, j1);
        if (j0 >= j1) return;
    }
    for (uint32_t k = threadIdx.x; k < a.ng + 3; k += PLAIN_T) cnt[k] = 0;
    uint32_t q[PLAIN_FIRST], ru[PLAIN_PER][PLAIN_FIRST];
    // entry (warp, k, lane) of the chunk: a warp owns 128 consecutive entries
    const uint32_t u0 = warp * 32 * PLAIN_PER + lane;
#pragma unroll
    for (uint32_t f = 0; f < PLAIN_FIRST; ++f) {
        q[f] = 1;                                 // a missing filter (nres < 4) passes residue 0
#pragma unroll
        for (uint32_t k = 0; k < PLAIN_PER; ++k) ru[k][f] = 0;
        if (f < nf) {
            const FiltConst fc = a.fc[f];
            q[f] = fc.m.q;
            for (uint32_t w = threadIdx.x; w < (fc.m.q + 31) / 32; w += PLAIN_T) bits_s[f][w] = a.bits[fc.tab_off + w];
#pragma unroll
            for (uint32_t k = 0; k < PLAIN_PER; ++k) {
                const uint64_t u = u0 + 32 * k < n_here ? __ldg(us + u0 + 32 * k) : 0;
                ru[k][f] = fastmod32(mod64(u, fc.m) * a.bq[f], fc.m.c, fc.m.q);
            }
        } else if (threadIdx.x == 0) {
            bits_s[f][0] = 1;
        }
    }
    uint32_t passed = 0, qhead = 0, qtail = 0;    // group-1 positions of the lane; warp-uniform queue positions

    // Up to 32 queued positions, one per lane: the remaining filters on x = uB - vA in two limbs.
    auto drain = [&](uint32_t n) {
        __syncwarp();
        const bool mine = lane < n;
        const uint32_t ent = mine ? queue_s[warp][(qhead + lane) & (PLAIN_QUEUE - 1)] : 0u;
        __syncwarp();
        qhead += n;
        if (!mine) return;
        plain_rest(a, sub128(mul_wide(__ldg(us + (ent & (PLAIN_U - 1))), a.B), mul_wide(__ldg(a.vs + j0 + ent / PLAIN_U), a.A)), nf, cnt);
    };

    for (uint64_t base = j0; base < j1; base += PLAIN_V) {
        const uint32_t rows = (uint32_t)umin64(PLAIN_V, j1 - base);
        __syncthreads();                          // every warp has read the previous rows
        if (threadIdx.x < PLAIN_V) {              // the row's interval inside the chunk
            uint32_t left = 0, right = 0;
            if (threadIdx.x < rows) {
                const u128 shift = mul_wide(a.vs[base + threadIdx.x], a.A), above = add128(shift, a.lo);
                left = (uint32_t)count_le(us, n_here, a.B, above);
                right = max(left, (uint32_t)count_le(us, n_here, a.B, add128(shift, a.hi)));
                if (less128(above, shift)) {      // vA + lo wrapped: positions below vA are flagged, not tested
                    uint32_t first = left;
                    while (first < right && less128(mul_wide(__ldg(us + first), a.B), shift)) ++first;
                    if (first > left) atomicAdd(&cnt[a.ng + 2], (unsigned long long)(first - left));
                    left = first;
                }
                if (right > left) atomicAdd(&cnt[0], (unsigned long long)(right - left));
            }
            row_s[threadIdx.x].x = left | right << 16;
        }
        {                                         // its residues: one (row, filter) pair per thread
            const uint32_t r = threadIdx.x / PLAIN_FIRST, f = threadIdx.x % PLAIN_FIRST;
            uint32_t m = 0;
            if (r < rows && f < nf) {
                const FiltConst fc = a.fc[f];
                m = fastmod32(mod64(a.vs[base + r], fc.m) * a.aq[f], fc.m.c, fc.m.q);
            }
            ((uint16_t *)&row_s[r])[2 + f] = (uint16_t)m;
        }
        __syncthreads();
        for (uint32_t r = 0; r < rows; ++r) {
            const uint4 row = row_s[r];
            const uint32_t left = row.x & 0xffffu, right = row.x >> 16, w0 = warp * 32 * PLAIN_PER;
            if (right <= w0 || left >= w0 + 32 * PLAIN_PER || left == right) continue;    // warp-uniform
            const uint32_t rv[PLAIN_FIRST] = {row.y & 0xffffu, row.y >> 16, row.z & 0xffffu, row.z >> 16};
#pragma unroll
            for (uint32_t k = 0; k < PLAIN_PER; ++k) {
                const uint32_t ul = u0 + 32 * k;
                uint32_t ok = ul >= left && ul < right;
#pragma unroll
                for (uint32_t f = 0; f < PLAIN_FIRST; ++f) {
                    const uint32_t d = ru[k][f] - rv[f], m = __viaddmin_u32(d, q[f], d);   // (ru - rv) mod q
                    ok &= bits_s[f][m >> 5] >> (m & 31);
                }
                const uint32_t won = __ballot_sync(0xffffffffu, ok);
                if (won) {
                    passed += ok;
                    if (ok)
                        queue_s[warp][(qtail + __popc(won & lanes_below)) & (PLAIN_QUEUE - 1)] =
                            ul | (uint32_t)(base - j0 + r) * PLAIN_U;
                    qtail += __popc(won);
                }
            }
            while (qtail - qhead >= 32) drain(32);
        }
    }
    if (qtail != qhead) drain(qtail - qhead);
    passed = __reduce_add_sync(0xffffffffu, passed);
    if (lane == 0 && passed) atomicAdd(&cnt[1], (unsigned long long)passed);
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < a.ng + 3; k += PLAIN_T)
        if (k != a.ng + 1 && cnt[k]) atomicAdd((unsigned long long *)&a.counts[k], cnt[k]);
}

// The same with more v rows.  A CTA owns 128 u entries and a run of v rows and first makes, for every residue r of
// the first four filters, the 128 bits allowed[(uB - r) mod q]: a warp takes one filter's word of 32 entries, a lane
// reads 32 residues of its entry as one word of the filter's pattern, and five exchanges transpose the warp's words.
// Then a v row is four words per filter: a lane loads one word of each of the four rows that vA mod q names, four
// lanes to a v row, and 128 positions take some 8 instructions of a warp where the lookups of k_plain take 275.  The
// rest (interval searches in the entries' products, one v row per lane; the queue of the 1 in 81) is as there.
// Bound: latency, of the prologue, the rows and the 128-bit tail, each a few us long with 16 warps on an SM.
// Times with their events, k_plain -> here, by v rows (17,400 u entries): 55 19.2 -> 20, 91 20.7 -> 20.0, 193 26 -> 21,
// 474 39 -> 23, 997 62 -> 25.6, 1,988 108 -> 34 us.
constexpr uint32_t PR_T = 512, PR_U = 128;        // threads, u entries per CTA
static_assert(PR_T / 32 == 4 * PLAIN_FIRST && PR_U == 4 * 32, "a warp per filter and word");
constexpr uint32_t PR_QUEUE = 64;                 // queued positions per warp (31 left over and 32 fit)
constexpr uint32_t PR_ROWS = 2048;                // most rows of the first four filters (32 KB)
constexpr uint32_t PR_PAT = (2 * PR_ROWS + PLAIN_FIRST * 96) / 32;   // pattern words
constexpr uint64_t PLAIN_ROWS_MIN = 64;           // v rows of a launch and of a run from which the rows are worth making
constexpr uint64_t PR_RUN_MAX = UINT64_C(1) << 25;   // v rows per CTA (a queue entry holds the row in 25 bits)

template <bool ORDERED>
__global__ void __launch_bounds__(PR_T) k_plain_rows(const PlainArgs a) {
    extern __shared__ uint4 rows_s[];             // 128 bits per row
    __shared__ unsigned long long cnt[PC_MAX_RES / 4 + 4];
    __shared__ u128 prod_s[PR_U];                 // uB
    __shared__ FiltConst fc_s[PLAIN_FIRST];
    __shared__ uint32_t pat_s[PR_PAT];
    __shared__ uint32_t queue_s[PR_T / 32][PR_QUEUE];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lanes_below = (1u << lane) - 1u;
    const uint32_t nf = min(a.nres, PLAIN_FIRST);
    const uint64_t c0 = blockIdx.x * (uint64_t)PR_U;
    const uint32_t n_here = (uint32_t)umin64(a.nu - c0, PR_U);
    uint64_t j0 = blockIdx.y * a.run, j1 = umin64(a.nv, j0 + a.run);
    const uint64_t *us = a.us + c0;
    if (ORDERED) {
        plain_band(a, us, n_here, j0, j1);
        if (j0 >= j1) return;
    }
    for (uint32_t k = threadIdx.x; k < a.ng + 3; k += PR_T) cnt[k] = 0;
    if (threadIdx.x < n_here) prod_s[threadIdx.x] = mul_wide(__ldg(us + threadIdx.x), a.B);
    if (warp < nf && lane < sizeof(FiltConst) / 4) ((uint32_t *)(fc_s + warp))[lane] = ((const uint32_t *)(a.fc + warp))[lane];
    __syncthreads();
    uint32_t row0[PLAIN_FIRST], rows = 0, words = 0, my_row0 = 0, my_pat = 0;
#pragma unroll
    for (uint32_t f = 0; f < PLAIN_FIRST; ++f) {
        const uint32_t q = f < nf ? fc_s[f].m.q : 0;
        row0[f] = rows;
        if (f == warp / 4) my_row0 = rows, my_pat = words;
        rows += q, words += (2 * q + 63) / 32 + 1;
    }
    const uint32_t filt = warp / 4, part = warp % 4;   // a filter's pattern and rows are made by four warps
    if (filt < nf) {
        // pattern bit b: residue b - 31 mod q, for a window of 32 that ends at any residue below 2q
        const FiltConst &fc = fc_s[filt];
        const uint32_t q = fc.m.q;
        for (uint32_t w = part; w < (2 * q + 63) / 32; w += 4) {
            const uint32_t m = fastmod32(w * 32 + lane + 31 * (q - 1), fc.m.c, q);
            const uint32_t word = __ballot_sync(0xffffffffu, __ldg(a.bits + fc.tab_off + (m >> 5)) >> (m & 31) & 1u);
            if (lane == 0) pat_s[my_pat + w] = word;
        }
    }
    __syncthreads();
    if (filt < nf) {                              // word `part` of the CTA's entries
        const FiltConst &fc = fc_s[filt];
        const uint32_t q = fc.m.q, i = part * 32 + lane;
        const uint32_t ru = fastmod32(mod64(i < n_here ? __ldg(us + i) : 0, fc.m) * a.bq[filt], fc.m.c, q);
        for (uint32_t r0 = 0; r0 < q; r0 += 32) {
            const uint32_t at = ru + q - r0;      // bits 31 - i of the window: residue ru - r0 - i
            const uint32_t *p = pat_s + my_pat + (at >> 5);
            uint32_t x = __brev(__funnelshift_r(p[0], p[1], at));
#pragma unroll
            for (uint32_t d = 16; d; d >>= 1) {   // lane = entry, bit = row -> lane = row, bit = entry
                const uint32_t keep = d == 16 ? 0x0000ffffu : d == 8 ? 0x00ff00ffu : d == 4 ? 0x0f0f0f0fu : d == 2 ? 0x33333333u : 0x55555555u;
                const uint32_t y = __shfl_xor_sync(0xffffffffu, x, d);
                x = lane & d ? (x & ~keep) | (y >> d & keep) : (x & keep) | (y << d & ~keep);
            }
            if (r0 + lane < q) ((uint32_t *)(rows_s + my_row0 + r0 + lane))[part] = x;
        }
    }
    __syncthreads();
    uint32_t passed = 0, qhead = 0, qtail = 0;    // group-1 positions of the lane; warp-uniform queue positions
    uint32_t tested = 0;                          // at most 128 of each of the lane's 2^16 v rows
    auto drain = [&](uint32_t n) {
        __syncwarp();
        const bool mine = lane < n;
        const uint32_t ent = mine ? queue_s[warp][(qhead + lane) & (PR_QUEUE - 1)] : 0u;
        __syncwarp();
        qhead += n;
        if (mine) plain_rest(a, sub128(prod_s[ent & (PR_U - 1)], mul_wide(__ldg(a.vs + j0 + ent / PR_U), a.A)), nf, cnt);
    };
    auto count = [&](u128 key) {                  // entries with uB <= key
        uint32_t lo = 0, hi = n_here;
        if (less128(key, prod_s[0])) hi = 0;
        else if (!less128(key, prod_s[n_here - 1])) lo = n_here;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) / 2;
            if (less128(key, prod_s[mid])) hi = mid;
            else lo = mid + 1;
        }
        return lo;
    };
    for (uint64_t base = j0 + warp * 32; base < j1; base += PR_T) {
        uint32_t span = 0, at01 = 0, at23 = 0;    // the lane's v row: interval start | end << 16, its rows
        if (base + lane < j1) {
            const uint64_t v = __ldg(a.vs + base + lane);
            const u128 shift = mul_wide(v, a.A), above = add128(shift, a.lo);
            uint32_t left = count(above);
            const uint32_t right = max(left, count(add128(shift, a.hi)));
            if (less128(above, shift)) {          // vA + lo wrapped: positions below vA are flagged, not tested
                uint32_t first = left;
                while (first < right && less128(prod_s[first], shift)) ++first;
                if (first > left) atomicAdd(&cnt[a.ng + 2], (unsigned long long)(first - left));
                left = first;
            }
            tested += right - left;
            span = left | right << 16;
            uint32_t row[PLAIN_FIRST];
#pragma unroll
            for (uint32_t f = 0; f < PLAIN_FIRST; ++f)
                row[f] = f < nf ? row0[f] + fastmod32(mod64(v, fc_s[f].m) * a.aq[f], fc_s[f].m.c, fc_s[f].m.q) : 0;
            at01 = row[0] | row[1] << 16, at23 = row[2] | row[3] << 16;
        }
        for (uint32_t k = 0; k < 32 && base + k < j1; k += 8) {     // eight v rows, four lanes each
            const uint32_t src = k + (lane >> 2), w = lane & 3;
            const uint32_t sp = __shfl_sync(0xffffffffu, span, src);
            const uint32_t r01 = __shfl_sync(0xffffffffu, at01, src), r23 = __shfl_sync(0xffffffffu, at23, src);
            uint32_t x = unit_mask((int32_t)(sp & 0xffffu) - 32 * (int32_t)w, (int32_t)(sp >> 16) - 32 * (int32_t)w);
            const uint32_t *rw = (const uint32_t *)rows_s + w;
            if (x) {
                x &= rw[4 * (r01 & 0xffffu)];
                if (nf > 1) x &= rw[4 * (r01 >> 16)];
                if (nf > 2) x &= rw[4 * (r23 & 0xffffu)];
                if (nf > 3) x &= rw[4 * (r23 >> 16)];
            }
            passed += __popc(x);
            for (uint32_t won; (won = __ballot_sync(0xffffffffu, x != 0)) != 0;) {
                if (x) {
                    queue_s[warp][(qtail + __popc(won & lanes_below)) & (PR_QUEUE - 1)] =
                        (w * 32 + __ffs(x) - 1) | (uint32_t)(base - j0 + src) * PR_U;
                    x &= x - 1;
                }
                qtail += __popc(won);
                if (qtail - qhead >= 32) drain(32);
            }
        }
    }
    if (qtail != qhead) drain(qtail - qhead);
    passed = __reduce_add_sync(0xffffffffu, passed);
    if (lane == 0 && passed) atomicAdd(&cnt[1], (unsigned long long)passed);
    tested = __reduce_add_sync(0xffffffffu, tested);
    if (lane == 0 && tested) atomicAdd(&cnt[0], (unsigned long long)tested);
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < a.ng + 3; k += PR_T)
        if (k != a.ng + 1 && cnt[k]) atomicAdd((unsigned long long *)&a.counts[k], cnt[k]);
}

// A plain launch: every u chunk, times as many v runs as fill the device.  k_plain: one wave of four CTAs per SM
// (64 registers); more, shorter runs only repeat the staging of rows and leave fuller last waves.  k_plain_rows from
// PLAIN_ROWS_MIN v rows on, two CTAs per SM with at least that many rows each, unless the first filters' rows are too many.
void plain_launch(PlainArgs &a, const uint32_t *primes, int sm_count, cudaStream_t st) {
    uint32_t rows = 0;
    for (uint32_t k = 0; k < std::min(a.nres, PLAIN_FIRST); ++k) {
        a.aq[k] = (uint32_t)(a.A % primes[k]);
        a.bq[k] = (uint32_t)(a.B % primes[k]);
        rows += primes[k];
    }
    const bool by_rows = a.nv >= PLAIN_ROWS_MIN && rows <= PR_ROWS;
    const uint64_t per = by_rows ? PR_U : PLAIN_U, chunks = (a.nu + per - 1) / per, want = (uint64_t)sm_count * (by_rows ? 2 : 4);
    const uint64_t most = by_rows ? PR_RUN_MAX : PLAIN_RUN_MAX, least = by_rows ? a.nv / PLAIN_ROWS_MIN : a.nv;
    const uint64_t runs = std::max(std::min(least, std::max<uint64_t>(1, want / chunks)), (a.nv + most - 1) / most);
    a.run = (a.nv + runs - 1) / runs;
    const dim3 grid((unsigned)chunks, (unsigned)((a.nv + a.run - 1) / a.run));
    if (by_rows) (a.ordered ? k_plain_rows<true> : k_plain_rows<false>)<<<grid, PR_T, rows * 16, st>>>(a);
    else (a.ordered ? k_plain<true> : k_plain<false>)<<<grid, PLAIN_T, 0, st>>>(a);
}

// Whether the CTAs of a launch may look for their v rows, should these be in order (u entries always are).
bool plain_ordered(const PlainArgs &a) {
    return (unsigned __int128)a.nu * a.nv >= PLAIN_ORDERED_MIN && a.lo.hi <= UINT64_MAX - a.A && a.hi.hi <= UINT64_MAX - a.A;
}

template <int NB, int K, int NT>
int launch_match_t(pc_ctx *ctx, const MatchArgs &a, size_t smem, int grid, int mode) {
    auto kern = k_match<NB, K, NT>;
    if (mode != 1) {       // 0: attribute and launch, 1: launch only (inside a capture), 2: attribute only
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return pc_cuda_fail(ctx, e, "match smem attribute");
        if (mode == 2) return PC_OK;
    }
    kern<<<grid, NT, smem, ctx->stream>>>(a);
    PC_LAUNCHED(ctx, "match");
    return PC_OK;
}

template <int K, int NT>
int launch_match_k(pc_ctx *ctx, const MatchArgs &a, uint32_t nb, size_t smem, int grid, int mode) {
    switch (nb) {
        case 1: return launch_match_t<1, K, NT>(ctx, a, smem, grid, mode);
        case 2: return launch_match_t<2, K, NT>(ctx, a, smem, grid, mode);
        case 3: return launch_match_t<3, K, NT>(ctx, a, smem, grid, mode);
        case 4: return launch_match_t<4, K, NT>(ctx, a, smem, grid, mode);
        case 5: return launch_match_t<5, K, NT>(ctx, a, smem, grid, mode);
        case 6: return launch_match_t<6, K, NT>(ctx, a, smem, grid, mode);
        case 7: return launch_match_t<7, K, NT>(ctx, a, smem, grid, mode);
        case 8: return launch_match_t<8, K, NT>(ctx, a, smem, grid, mode);
    }
    return pc_fail(ctx, PC_INVALID, "unsupported bitset filter count");
}

template <int NT>
int launch_match_n(pc_ctx *ctx, const MatchArgs &a, uint32_t nb, uint32_t K, size_t smem, int grid, int mode) {
    if (K == 16) return launch_match_k<16, NT>(ctx, a, nb, smem, grid, mode);
    if (K == 32) return launch_match_k<32, NT>(ctx, a, nb, smem, grid, mode);
    return launch_match_k<64, NT>(ctx, a, nb, smem, grid, mode);
}

uint32_t inv_mod(uint32_t a, uint32_t q) {
    int64_t t = 0, nt = 1, r = q, nr = a % q;
    while (nr) {
        int64_t quo = r / nr, tmp;
        tmp = t - quo * nt; t = nt; nt = tmp;
        tmp = r - quo * nr; r = nr; nr = tmp;
    }
    if (r != 1) return 0;
    return (uint32_t)(t < 0 ? t + q : t);
}

double elapsed_ms(cudaEvent_t a, cudaEvent_t b) {
    float ms = 0;
    if (cudaEventElapsedTime(&ms, a, b) != cudaSuccess) cudaGetLastError();   // recorded anew by another thread's call
    return ms;
}

}  // namespace

extern "C" int pc_filters_create(pc_ctx *ctx, uint64_t A, uint64_t B, const uint32_t *primes, uint32_t nres,
                                 const uint8_t *allowed, pc_filters **out) {
    *out = nullptr;
    if (nres == 0) return pc_fail(ctx, PC_INVALID, "bitset experiment requires at least one residual filter");
    if (nres > PC_MAX_RES || A == 0 || B == 0) return pc_fail(ctx, PC_INVALID, "invalid residual filters");
    pc_filters *f = new pc_filters();
    f->A = A;
    f->B = B;
    f->nres = nres;
    f->ng = (nres + 3) / 4;
    f->primes.assign(primes, primes + nres);
    std::vector<FiltConst> fc(nres);
    std::vector<uint32_t> bits;
    uint64_t off = 0;
    for (uint32_t i = 0; i < nres; ++i) {
        uint32_t q = primes[i];
        if (q < 2 || q >= 8192 || A % q == 0 || B % q == 0) {
            delete f;
            return pc_fail(ctx, PC_INVALID, "residual modulus must be in [2, 8192) and coprime to A and B");
        }
        fc[i].m = make_modq(q);
        fc[i].tab_off = (uint32_t)bits.size();
        FiltC c{};
        c.c = fc[i].m.c;
        c.q = q;
        c.tab_off = fc[i].tab_off;
        for (int k = 0; k < 5; ++k) c.r16[k] = (uint16_t)fc[i].m.r16[k];
        f->fcs.push_back(c);
        std::vector<uint32_t> w((q + 31) / 32, 0);
        for (uint32_t r = 0; r < q; ++r)
            if (allowed[off + r]) w[r / 32] |= 1u << (r % 32);
        bits.insert(bits.end(), w.begin(), w.end());
        off += q;
    }
    // patterns of the first filters: RR[j] = S'[(-j) mod q] with S'[k] = allowed[(A k) mod q]
    f->nbmax = std::min<uint32_t>(nres, PC_MAX_BITSET);
    std::vector<uint32_t> pat((size_t)PC_MAX_BITSET * PATW, 0);
    uint64_t aoff = 0;
    for (uint32_t i = 0; i < f->nbmax; ++i) {
        uint32_t q = primes[i];
        if (q > 2047) {
            f->nbmax = i;
            break;
        }
        uint32_t a = (uint32_t)(A % q), b = (uint32_t)(B % q);
        f->ainvb[i] = (uint32_t)((uint64_t)b * inv_mod(a, q) % q);
        for (uint32_t j = 0; j < 2 * q + 64; ++j) {
            uint32_t k = (q - j % q) % q;
            uint32_t m = (uint32_t)((uint64_t)a * k % q);
            if (allowed[aoff + m]) pat[(size_t)i * PATW + j / 32] |= 1u << (j % 32);
        }
        aoff += q;
        f->rows_sum[i + 1] = f->rows_sum[i] + q;
    }
    if (f->nbmax < std::min<uint32_t>(nres, 4)) {
        delete f;
        return pc_fail(ctx, PC_INVALID, "first residual filters too large for bitset rows");
    }
    f->fc_bytes = nres * sizeof(FiltConst);
    f->fcs_bytes = nres * sizeof(FiltC);
    f->bits_bytes = bits.size() * 4;
    f->pat_bytes = pat.size() * 4;
    int rc = pc_alloc(ctx, (void **)&f->d_fc, f->fc_bytes);
    if (!rc) rc = pc_alloc(ctx, (void **)&f->d_fcs, f->fcs_bytes);
    if (!rc) rc = pc_alloc(ctx, (void **)&f->d_bits, f->bits_bytes);
    if (!rc) rc = pc_alloc(ctx, (void **)&f->d_pat, f->pat_bytes);
    if (rc) {
        pc_filters_free(ctx, f);
        return rc;
    }
    pc_copy(ctx, f->d_fc, fc.data(), f->fc_bytes, cudaMemcpyHostToDevice);
    pc_copy(ctx, f->d_fcs, f->fcs.data(), f->fcs_bytes, cudaMemcpyHostToDevice);
    pc_copy(ctx, f->d_bits, bits.data(), f->bits_bytes, cudaMemcpyHostToDevice);
    pc_copy(ctx, f->d_pat, pat.data(), f->pat_bytes, cudaMemcpyHostToDevice);
    cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) {
        pc_filters_free(ctx, f);
        return pc_cuda_fail(ctx, e, "filters upload");
    }
    *out = f;
    return PC_OK;
}

extern "C" int pc_filters_free(pc_ctx *ctx, pc_filters *f) {
    if (!f) return PC_OK;
    pc_release(ctx, f->d_fc, f->fc_bytes);
    pc_release(ctx, f->d_fcs, f->fcs_bytes);
    pc_release(ctx, f->d_bits, f->bits_bytes);
    pc_release(ctx, f->d_pat, f->pat_bytes);
    delete f;
    return PC_OK;
}


namespace {

struct Tuned {
    uint32_t nb, K, threads, nch;
    uint64_t v_chunk;
};

// Residual filters after the bitset tier that the cheap tier can test (bitmap of <= 64 words).
uint32_t cheap_count(const pc_filters *f, uint32_t nb) {
    uint32_t n = 0;
    while (n < PC_MAX_CHEAP && nb + n < f->nres && f->primes[nb + n] <= 2047) ++n;
    return n;
}

// One launch shape for every family of a launch: NB inside every family's bitset range, the cheap
// tier as deep as the shallowest family allows, shared memory sized by the largest rows and
// counters.  Defaults: seven bitset filters, 32-word blocks, 896 threads, stepping down (threads,
// then block words, then bitset filters) until the layout fits the opt-in shared memory.
int resolve_tuning(pc_ctx *ctx, const std::vector<const pc_filters *> &fams, const pc_tuning *t, Tuned &r,
                   size_t &smem, uint32_t &tmax) {
    uint32_t nb_lo = 1, nb_hi = PC_MAX_BITSET, ngmax = 0;
    for (const pc_filters *f : fams) {
        nb_lo = std::max(nb_lo, std::min<uint32_t>(f->nres, 4));
        nb_hi = std::min(nb_hi, f->nbmax);
        ngmax = std::max(ngmax, f->ng);
    }
    if (nb_lo > nb_hi) return pc_fail(ctx, PC_INVALID, "filter families cannot share one bitset launch");
    r = Tuned{};
    r.nb = t && t->bitset_filters ? t->bitset_filters : std::min<uint32_t>(nb_hi, 7);
    r.nb = std::max(nb_lo, std::min(r.nb, nb_hi));
    r.K = t && t->block_words ? t->block_words : 32;
    if (r.K != 16 && r.K != 32 && r.K != 64) r.K = 32;
    const bool fixed_threads = t && t->threads;
    r.threads = fixed_threads ? t->threads : 896;
    if (r.threads != 512 && r.threads != 768 && r.threads != 896 && r.threads != 1024) r.threads = 512;
    r.v_chunk = t ? t->v_chunk : 0;
    int optin = 0;
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device);
    if (optin <= 0) optin = 227 * 1024;
    for (;;) {
        r.nch = PC_MAX_CHEAP;
        uint32_t rows = 0;
        for (const pc_filters *f : fams) {
            r.nch = std::min(r.nch, cheap_count(f, r.nb));
            rows = std::max(rows, f->rows_sum[r.nb]);
        }
        for (uint32_t tm = TMAX_DEFAULT; tm >= 4; tm /= 2) {
            MatchSmem L(rows, r.K, r.nb, r.nch, tm, ngmax, r.threads / 32);
            if (L.total <= (uint32_t)optin) {
                tmax = tm;
                smem = L.total;
                return PC_OK;
            }
        }
        if (!fixed_threads && r.threads > 512) r.threads = r.threads > 896 ? 896 : r.threads == 896 ? 768 : 512;
        else if (r.K > 16) r.K /= 2;
        else if (r.nb > nb_lo) r.nb--;
        else return pc_fail(ctx, PC_INVALID, "residual rows do not fit shared memory");
    }
}

// q < 2^11 and a factor below q as residue() and mod_short() use them.
uint4 pack_mod(uint32_t q, uint32_t factor) {
    const ModQ m = make_modq(q);
    return make_uint4(m.r16[0] | m.r16[1] << 16, m.r16[2] | q << 16, (uint32_t)(m.c >> 32), factor);
}

FamDev fam_dev(const pc_filters *f, uint32_t nb, uint32_t nch) {
    FamDev d{};
    d.nres = f->nres;
    d.ng = f->ng;
    d.total_rows = f->rows_sum[nb];
    d.c2_live = nb == 8 || (nb > 4 && nb == f->nres);
    for (uint32_t i = 0; i < nb; ++i) {
        d.q[i] = f->primes[i];
        d.row0[i] = f->rows_sum[i];
        d.umod[i] = pack_mod(f->primes[i], f->ainvb[i]);
    }
    for (uint32_t t = 0; t < nch; ++t) {
        const uint32_t q = f->primes[nb + t];
        d.cq[t] = q;
        d.umod[PC_MAX_BITSET + t] = pack_mod(q, (uint32_t)(f->B % q));
        d.cbits_off[t] = f->fcs[nb + t].tab_off;
    }
    for (uint32_t idx = 0; idx < 16; ++idx)
        d.bgroup[idx] = (uint8_t)(idx < f->nres && ((idx & 3) == 3 || idx + 1 == f->nres) ? idx / 4 + 1 : 0);
    for (uint32_t t = 0; t < nch; ++t) d.cqg[t] = d.cq[t] | (uint32_t)d.bgroup[nb + t] << 16;
    d.pat = f->d_pat;
    d.bits = f->d_bits;
    d.fcs = f->d_fcs;
    return d;
}

FamPrep fam_prep(const pc_filters *f, const FamDev &d, uint32_t nb, uint32_t nch) {
    FamPrep p{};
    for (uint32_t t = 0; t < nb; ++t) p.f[t] = pack_mod(d.q[t], d.row0[t]);
    for (uint32_t t = 0; t < nch; ++t) p.f[PC_MAX_BITSET + t] = pack_mod(d.cq[t], (uint32_t)(f->A % d.cq[t]));
    return p;
}

// Fixed-point A / B and the whole parts of the interval's ends over B.  64-bit bounds need lo <= hi: `fast` is decided by
// hi alone, and floor(lo / B) of a larger lo need not fit 64 bits.
SegPrep seg_prep(const SegDev &g) {
    typedef unsigned __int128 w128;
    const w128 lo = (w128)g.lo.hi << 64 | g.lo.lo, hi = (w128)g.hi.hi << 64 | g.hi.lo, last = (w128)(g.v_end ? g.v_end - 1 : 0) * g.A;
    SegPrep p{};
    p.ia = g.A / g.B;
    p.am = g.A % g.B;
    p.fa = (uint64_t)(((w128)p.am << 64) / g.B);
    p.ilo = (uint64_t)(lo / g.B);
    p.ihi = (uint64_t)(hi / g.B);
    p.wr = g.width > 1 ? (uint64_t)(((w128)1 << 64) / g.width) : UINT64_MAX;
    p.fast = g.B < (UINT64_C(1) << 62) && lo <= hi && hi + last >= last && !((hi + last) / g.B >> 64);
    return p;
}

// The device half of stages 2 and 3 over a set of segments whose u and v lists are already on
// the device.  Every buffer is sized once by engine_prepare, so the launch sequence (front + back)
// can be recorded into a CUDA graph and replayed.
struct Engine {
    pc_ctx *ctx = nullptr;
    const uint64_t *us = nullptr, *vs = nullptr;
    uint64_t nu = 0, nv = 0;
    std::vector<SegDev> segs;
    std::vector<const pc_filters *> fams;
    std::vector<FamDev> famdev;
    std::vector<uint32_t> tile_seg;
    uint64_t ntiles = 0, out_cap = 0;
    Tuned tn{};
    size_t smem = 0;
    uint32_t tmax = 0, stride = 0, ngmax = 0;
    uint64_t nblocks = 0;
    int grid = 0;
    uint32_t deep_cap = 1u << 15, deep_max = 0;
    SegDev *d_seg = nullptr;
    FamDev *d_fam = nullptr;
    SegPrep *d_segp = nullptr;
    FamPrep *d_famp = nullptr;
    std::vector<SegPrep> segprep;
    std::vector<FamPrep> famprep;
    std::vector<unsigned char> upload;                    // the descriptors as copied to the device
    uint32_t *d_tile_seg = nullptr, *d_blk_seg = nullptr;
    VRec *d_rec = nullptr;
    uint64_t *d_cres = nullptr;
    uint4 *d_bv = nullptr;
    uint64_t *d_prefix = nullptr;
    // Everything a run reports lies together, in this order, so that one fill resets it and one copy fetches it:
    // scalars, deep survivors per CTA, counters, envelopes, output records.
    enum { STUCK, NOUT, BAD, SHARE_NEXT, SCALARS };    // STUCK: the window pass gave up
    bool windows = false;                                 // the window pass is the owner's: STUCK is not reset
    uint64_t *d_report = nullptr;
    uint64_t o_deep = 0, o_counts = 0, o_geo = 0, o_out = 0;   // word offsets
    unsigned long long *scalar(int k) const { return (unsigned long long *)d_report + k; }
    uint32_t *d_deep_count() const { return (uint32_t *)(d_report + o_deep); }
    uint64_t *d_counts() const { return d_report + o_counts; }
    uint64_t *d_geo() const { return d_report + o_geo; }
    uint64_t *d_out() const { return d_report + o_out; }
    uint64_t fetch_words() const { return o_out + 2 * std::min<uint64_t>(out_cap, FETCH_RECORDS); }
    static constexpr uint64_t FETCH_RECORDS = 256;        // output records fetched with the counters
    uint4 *d_deep = nullptr;
    uint64_t deep_bytes = 0;
    ~Engine() {
        if (ctx && d_deep) pc_release(ctx, d_deep, deep_bytes);
    }
};

// Slices of `cap` records; of none when they cannot be had, so that a later run of the same engine stores nothing, finds
// them outgrown and asks again.
int engine_deep_alloc(Engine &E, uint32_t cap) {
    if (E.d_deep) pc_release(E.ctx, E.d_deep, E.deep_bytes);
    E.d_deep = nullptr;
    E.deep_cap = 0;
    E.deep_bytes = (uint64_t)E.grid * cap * sizeof(uint4);
    const int rc = pc_alloc(E.ctx, (void **)&E.d_deep, E.deep_bytes);
    if (!rc) E.deep_cap = cap;
    return rc;
}

int engine_prepare(Engine &E, const pc_tuning *tuning, Scratch &hold) {
    pc_ctx *ctx = E.ctx;
    if (E.nu >= (UINT64_C(1) << 31) || E.nv >= (UINT64_C(1) << 32)) return pc_fail(ctx, PC_INVALID, "focus list too long");
    if (E.segs.empty() || E.fams.empty()) return pc_fail(ctx, PC_INVALID, "no segments");
    for (const SegDev &g : E.segs)
        if (g.hi.hi >= (UINT64_C(1) << 32)) return pc_fail(ctx, PC_INVALID, "interval bound must be below 2^96");
    int rc = resolve_tuning(ctx, E.fams, tuning, E.tn, E.smem, E.tmax);
    if (rc) return rc;
    E.ngmax = 0;
    for (const pc_filters *f : E.fams) E.ngmax = std::max(E.ngmax, f->ng);
    E.stride = E.ngmax + 3;
    E.famdev.clear();
    E.famprep.clear();
    E.segprep.clear();
    for (const pc_filters *f : E.fams) {
        E.famdev.push_back(fam_dev(f, E.tn.nb, E.tn.nch));
        E.famprep.push_back(fam_prep(f, E.famdev.back(), E.tn.nb, E.tn.nch));
    }
    for (const SegDev &g : E.segs) E.segprep.push_back(seg_prep(g));
    E.grid = ctx->sm_count;
    if (tuning && tuning->deep_records) E.deep_cap = tuning->deep_records;
    const uint32_t UB = E.tn.K * 32;
    E.nblocks = (E.nu + UB - 1) / UB;
    const uint64_t nb1 = std::max<uint64_t>(1, E.nblocks);
    E.o_deep = Engine::SCALARS;
    E.o_counts = E.o_deep + (E.grid + 1) / 2;
    E.o_geo = E.o_counts + E.ntiles * E.stride;
    E.o_out = E.o_geo + 2 * E.ntiles;
    // one allocation for the descriptors (one upload) and one for the scratch
    Carve in, work;
    in.add(&E.d_seg, E.segs.size());
    in.add(&E.d_fam, E.famdev.size());
    in.add(&E.d_segp, E.segs.size());
    in.add(&E.d_famp, E.famdev.size());
    in.add(&E.d_tile_seg, std::max<uint64_t>(1, E.ntiles));
    work.add(&E.d_report, E.o_out + 2 * std::max<uint64_t>(1, E.out_cap));
    work.add(&E.d_rec, std::max<uint64_t>(1, E.nv));
    work.add(&E.d_cres, std::max<uint64_t>(1, E.nv));
    work.add(&E.d_bv, nb1);
    work.add(&E.d_blk_seg, nb1);
    work.add(&E.d_prefix, E.nblocks + 2);
    rc = in.get(hold);
    if (!rc) rc = work.get(hold);
    if (!rc) rc = engine_deep_alloc(E, E.deep_cap);
    if (rc) return rc;
    E.upload.resize(in.bytes);
    auto put = [&](const void *dev, const void *src, uint64_t bytes) {
        memcpy(E.upload.data() + ((const unsigned char *)dev - (const unsigned char *)E.d_seg), src, bytes);
    };
    put(E.d_seg, E.segs.data(), E.segs.size() * sizeof(SegDev));
    put(E.d_fam, E.famdev.data(), E.famdev.size() * sizeof(FamDev));
    put(E.d_segp, E.segprep.data(), E.segprep.size() * sizeof(SegPrep));
    put(E.d_famp, E.famprep.data(), E.famprep.size() * sizeof(FamPrep));
    put(E.d_tile_seg, E.tile_seg.data(), E.ntiles * 4);
    PC_CHECK(ctx, pc_copy(ctx, E.d_seg, E.upload.data(), in.bytes, cudaMemcpyHostToDevice));
    return PC_OK;
}

// What a block counts beyond its v rows, in rows: 25 sum(q) / NB, 26 us at p = 619 (sum(q) = 1567), where 215 v rows of seven
// filters take a microsecond.  That is more than building its rows takes (16.5 us), as a share that starts inside a block
// builds it again and is charged nothing for it: with 16 sum(q) / NB a batch's k_match and k_deep take 101 us instead of 94, 24 batches
// 1.10 ms instead of 1.04, 48 windows 0.458 instead of 0.388; 200 windows and 512 the same.
uint32_t block_cost(const Engine &E) {
    uint32_t rows = 0;
    for (const FamDev &d : E.famdev) rows = std::max(rows, d.total_rows);
    return rows * 25 / E.tn.nb;
}

// mode 0: set the shared-memory attribute and launch; 1: launch only (inside a capture);
// 2: set the attribute only.
int engine_match(Engine &E, int mode) {
    MatchArgs ma{};
    ma.us = E.us;
    ma.rec = E.d_rec;
    ma.cres = E.d_cres;
    ma.seg = E.d_seg;
    ma.fam = E.d_fam;
    ma.blk_seg = E.d_blk_seg;
    ma.nch = E.tn.nch;
    ma.tmax = E.tmax;
    ma.stride = E.stride;
    ma.total_rows = 0;
    for (const FamDev &d : E.famdev) ma.total_rows = std::max(ma.total_rows, d.total_rows);
    ma.counts = E.d_counts();
    ma.bv = E.d_bv;
    ma.prefix = E.d_prefix;
    ma.nblocks = E.nblocks;
    ma.block_cost = block_cost(E);
    ma.v_chunk = (uint32_t)std::min<uint64_t>(E.tn.v_chunk ? E.tn.v_chunk : ITEM_ROWS, ITEM_ROWS);
    ma.deep = E.d_deep;
    ma.deep_cap = E.deep_cap;
    ma.deep_count = E.d_deep_count();
    ma.share_next = E.scalar(Engine::SHARE_NEXT);
    if (E.tn.threads == 1024) return launch_match_n<1024>(E.ctx, ma, E.tn.nb, E.tn.K, E.smem, E.grid, mode);
    if (E.tn.threads == 896) return launch_match_n<896>(E.ctx, ma, E.tn.nb, E.tn.K, E.smem, E.grid, mode);
    if (E.tn.threads == 768) return launch_match_n<768>(E.ctx, ma, E.tn.nb, E.tn.K, E.smem, E.grid, mode);
    return launch_match_n<512>(E.ctx, ma, E.tn.nb, E.tn.K, E.smem, E.grid, mode);
}

// Counters reset, per-v bounds, subtile envelopes, block ranges, work items, the fused match and the exact
// later filters on its deep survivors (as many as the slices hold).  Nothing waits for the device.
int engine_launch(Engine &E, bool events, bool capturing, int *launches) {
    pc_ctx *ctx = E.ctx;
    cudaStream_t st = ctx->stream;
    const uint64_t from = E.windows ? Engine::NOUT : Engine::STUCK;
    PC_CHECK(ctx, cudaMemsetAsync(E.d_report + from, 0, (E.o_geo - from) * 8, st));
    if (events) PC_CHECK(ctx, cudaEventRecord(ctx->ev[0], st));
    if (E.nv) {
        PrepArgs pa{};
        pa.us = E.us;
        pa.vs = E.vs;
        pa.nv = E.nv;
        pa.seg = E.d_seg;
        pa.nseg = (uint32_t)E.segs.size();
        pa.segp = E.d_segp;
        pa.fam = E.d_famp;
        pa.nb = E.tn.nb;
        pa.stride = E.stride;
        pa.rec = E.d_rec;
        pa.cres = E.d_cres;
        pa.nch = E.tn.nch;
        pa.counts = E.d_counts();
        pa.bad = E.scalar(Engine::BAD);
        // 8 or 4 rows per thread share a CTA's end searches where that still leaves every SM that many CTAs and
        // most CTAs lie in one segment; else one (a lease's 1.6e7 rows: 0.41 ms at 8, 0.44 at 4; 24 batches'
        // 1.5e6 rows: 54 us at 8, 47 at 4)
        uint32_t rows = 1;
        for (uint32_t r : {8u, 4u}) {
            const uint64_t ctas = E.nv / (r * PREP_T);
            if (rows == 1 && ctas >= (uint64_t)E.grid * r && ctas >= 4 * E.segs.size()) rows = r;
        }
        auto kern = rows == 8 ? k_vprep<8> : rows == 4 ? k_vprep<4> : k_vprep<1>;
        kern<<<(unsigned)((E.nv + rows * PREP_T - 1) / (rows * PREP_T)), PREP_T, 0, st>>>(pa);
        PC_LAUNCHED(ctx, "vprep");
        ++*launches;
    }
    if (E.ntiles) {
        k_geometry<<<(unsigned)((E.ntiles + 7) / 8), 256, 0, st>>>(E.us, E.vs, E.d_seg, E.d_tile_seg, E.ntiles, E.d_geo());
        PC_LAUNCHED(ctx, "geometry");
        ++*launches;
    }
    if (events) PC_CHECK(ctx, cudaEventRecord(ctx->ev[1], st));
    if (E.nu && E.nv) {
        k_blocks<<<(unsigned)((E.nblocks + 7) / 8), 256, 0, st>>>(E.d_rec, E.d_seg, (uint32_t)E.segs.size(), E.tn.K * 32,
                                                                E.nblocks, E.d_bv, E.d_blk_seg);
        PC_LAUNCHED(ctx, "blocks");
        k_pieces<<<1, PIECES_T, 0, st>>>(E.d_bv, E.nblocks, block_cost(E), (uint32_t)E.grid, E.d_prefix);
        PC_LAUNCHED(ctx, "pieces");
        if (events) PC_CHECK(ctx, cudaEventRecord(ctx->ev[2], st));
        const int rc = engine_match(E, capturing ? 1 : 0);
        if (rc) return rc;
        DeepArgs da{};
        da.us = E.us;
        da.deep = E.d_deep;
        da.deep_count = E.d_deep_count();
        da.deep_cap = E.deep_cap;
        da.first = E.tn.nb + E.tn.nch;
        da.stride = E.stride;
        da.ntiles = E.ntiles;
        da.seg = E.d_seg;
        da.fam = E.d_fam;
        da.tile_seg = E.d_tile_seg;
        da.counts = E.d_counts();
        da.out = E.d_out();
        da.out_cap = E.out_cap;
        da.n_out = E.scalar(Engine::NOUT);
        k_deep<<<dim3(std::max(1u, std::min<uint32_t>((E.deep_cap + 255) / 256, 8)), (unsigned)E.grid), 256, 0, st>>>(da);
        PC_LAUNCHED(ctx, "deep");
        *launches += 4;
    }
    if (events) PC_CHECK(ctx, cudaEventRecord(ctx->ev[3], st));
    return PC_OK;
}

// A finished run's report, already on the host (head: its scalars and deep counts): whether a window pass gave up (its
// lists then mean nothing), whether the deep slices held every survivor, rows outside the subtile geometry, outputs that did not fit
// and underflows.
int engine_check(Engine &E, const uint64_t *head, const uint64_t *counts, bool &outgrown) {
    const uint32_t *deep = (const uint32_t *)(head + E.o_deep);
    E.deep_max = 0;
    if (E.nu && E.nv)
        for (int b = 0; b < E.grid; ++b) E.deep_max = std::max(E.deep_max, deep[b]);
    outgrown = false;
    if (head[Engine::STUCK]) return pc_fail(E.ctx, PC_ARITHMETIC, "window pass did not finish");
    outgrown = E.deep_max > E.deep_cap;
    if (outgrown) return PC_OK;
    if (head[Engine::BAD]) return pc_fail(E.ctx, PC_INVALID, "v row outside the subtile geometry");
    if (head[Engine::NOUT] > E.out_cap) return pc_fail(E.ctx, PC_OVERFLOW, "output overflow; attempt cannot commit");
    for (uint64_t t = 0; t < E.ntiles; ++t) {
        const uint32_t ng = E.fams[E.segs[E.tile_seg[t]].fam]->ng;
        if (counts[t * E.stride + ng + 2]) return pc_fail(E.ctx, PC_ARITHMETIC, "unsigned underflow flagged");
    }
    return PC_OK;
}

constexpr uint64_t SMALL_REPORT = 1 << 14;                // words

// The report of the run just launched: in one copy through the context's page-locked stage where it fits that
// (a copy to pageable memory costs the host 12 us and a wait each), else straight to the caller's arrays.
// got: the first records, which the copy brought along; they lie in the stage, which `loan` holds.
int engine_fetch(Engine &E, uint64_t *counts, uint64_t *geometry, std::vector<uint64_t> &head, StageLoan &loan,
                 const uint64_t *&records, uint64_t &got) {
    pc_ctx *ctx = E.ctx;
    const uint64_t words = E.fetch_words();
    head.resize(E.o_counts);
    got = 0;
    // a large report goes straight to page-locked arrays, where the caller has them: no second copy on the host
    cudaPointerAttributes at{};
    const bool direct = words > SMALL_REPORT && cudaPointerGetAttributes(&at, counts) == cudaSuccess && at.type == cudaMemoryTypeHost;
    if (words > SMALL_REPORT) cudaGetLastError();
    if (!direct) loan = pc_stage(ctx, words * 8);
    if (uint64_t *stage = loan.get()) {
        PC_CHECK(ctx, pc_copy(ctx, stage, E.d_report, words * 8, cudaMemcpyDeviceToHost));
        PC_CHECK(ctx, cudaStreamSynchronize(ctx->stream));
        memcpy(head.data(), stage, E.o_counts * 8);
        if (E.ntiles) {
            memcpy(counts, stage + E.o_counts, E.ntiles * E.stride * 8);
            memcpy(geometry, stage + E.o_geo, 2 * E.ntiles * 8);
        }
        records = stage + E.o_out;
        got = (words - E.o_out) / 2;
        return PC_OK;
    }
    PC_CHECK(ctx, pc_copy(ctx, head.data(), E.d_report, E.o_counts * 8, cudaMemcpyDeviceToHost));
    PC_CHECK(ctx, pc_copy(ctx, counts, E.d_counts(), E.ntiles * E.stride * 8, cudaMemcpyDeviceToHost));
    PC_CHECK(ctx, pc_copy(ctx, geometry, E.d_geo(), 2 * E.ntiles * 8, cudaMemcpyDeviceToHost));
    PC_CHECK(ctx, cudaStreamSynchronize(ctx->stream));
    return PC_OK;
}

// Output records 0..n-1 to out, the first `got` of them from host memory.
int engine_records(Engine &E, const uint64_t *records, uint64_t got, uint64_t n, uint64_t *out) {
    got = std::min(got, n);
    if (got) memcpy(out, records, 16 * got);
    if (n > got) {
        PC_CHECK(E.ctx, pc_copy(E.ctx, out + 2 * got, E.d_out() + 2 * got, 16 * (n - got), cudaMemcpyDeviceToHost));
        PC_CHECK(E.ctx, cudaStreamSynchronize(E.ctx->stream));
    }
    return PC_OK;
}

// Eager run with its results on the host; once more, with room for every deep survivor, when a slice overflowed.
// `place` gives the array for the output records once their number is known.
template <class F>
int engine_run(Engine &E, uint64_t *counts, uint64_t *geometry, uint64_t *n_out, int *launches, F place) {
    for (int attempt = 0;; ++attempt) {
        int rc = engine_launch(E, true, false, launches);
        std::vector<uint64_t> head;
        StageLoan loan;
        const uint64_t *records = nullptr;
        uint64_t got = 0;
        if (!rc) rc = engine_fetch(E, counts, geometry, head, loan, records, got);
        if (rc) return rc;
        bool outgrown = false;
        rc = engine_check(E, head.data(), counts, outgrown);
        if (outgrown) {
            if (attempt) return pc_fail(E.ctx, PC_ARITHMETIC, "deep survivor count changed between attempts");
            rc = engine_deep_alloc(E, E.deep_max + 1024);
            if (rc) return rc;
            continue;
        }
        *n_out = head[Engine::NOUT];
        if (rc) return rc;
        return engine_records(E, records, got, *n_out, place(*n_out));
    }
}

void engine_stats(Engine &E, pc_stats *stats, int launches, uint64_t n_out) {
    if (!stats) return;
    pc_ctx *ctx = E.ctx;
    const bool matched = E.nu && E.nv;
    stats->bounds_ms = elapsed_ms(ctx->ev[0], ctx->ev[1]);
    stats->kernel_ms = matched ? elapsed_ms(ctx->ev[2], ctx->ev[3]) : 0.0;
    stats->outputs = n_out;
    stats->launches = launches;
    stats->work_items = E.deep_max;
    stats->reserved[0] = E.tn.nb;
    stats->reserved[1] = E.tn.K;
    stats->reserved[2] = E.tn.threads;
    stats->reserved[3] = E.tn.nch;
}

// True when ntiles subtiles of width v fit below 2^64 and match the [first, end) span.
bool tiles_fit(uint64_t first, uint64_t end, uint64_t width, uint64_t ntiles) {
    typedef unsigned __int128 w128;
    if (!width || end <= first) return false;
    if (((w128)ntiles * width) >> 64) return false;
    return (end - first + width - 1) / width == ntiles;
}

SegDev one_segment(const pc_filters *f, uint64_t nu, uint64_t nv, u128 lo, u128 hi, uint64_t v_first,
                   uint64_t width, uint64_t v_end, uint32_t ntiles) {
    SegDev g{};
    g.A = f->A;
    g.B = f->B;
    g.lo = lo;
    g.hi = hi;
    g.v_first = v_first;
    g.width = width;
    g.v_end = v_end;
    g.u_off = 0;
    g.nu = (uint32_t)nu;
    g.v_off = 0;
    g.nv = (uint32_t)nv;
    g.tile_base = 0;
    g.ntiles = ntiles;
    g.fam = 0;
    return g;
}

}  // namespace

extern "C" int pc_run_batch(pc_ctx *ctx, const pc_filters *f, const pc_tuning *tuning, const pc_buf *us, uint64_t u_off,
                            uint64_t nu, const pc_buf *vs, uint64_t v_off, uint64_t nv, uint64_t lo0, uint64_t lo1,
                            uint64_t hi0, uint64_t hi1, uint64_t v_first, uint64_t width, uint32_t ntiles,
                            uint64_t v_end, uint64_t *counts, uint64_t *geometry, uint64_t *out, uint64_t out_cap,
                            uint64_t *n_out, pc_stats *stats) {
    if (!f || !us || !vs || width == 0 || ntiles == 0) return pc_fail(ctx, PC_INVALID, "invalid batch arguments");
    if (u_off > us->n || nu > us->n - u_off || v_off > vs->n || nv > vs->n - v_off)
        return pc_fail(ctx, PC_INVALID, "focus list slice out of range");
    if (!tiles_fit(v_first, v_end, width, ntiles) || ntiles >= (UINT32_C(1) << 31))
        return pc_fail(ctx, PC_INVALID, "inconsistent subtile geometry");
    if (stats) memset(stats, 0, sizeof(*stats));
    *n_out = 0;
    auto t0 = std::chrono::steady_clock::now();
    const uint64_t h2d0 = ctx->h2d, d2h0 = ctx->d2h;
    Engine E;
    E.ctx = ctx;
    E.us = us->d + u_off;
    E.vs = vs->d + v_off;
    E.nu = nu;
    E.nv = nv;
    if (nu >= (UINT64_C(1) << 31) || nv >= (UINT64_C(1) << 32)) return pc_fail(ctx, PC_INVALID, "focus list too long");
    E.segs.push_back(one_segment(f, nu, nv, u128{lo0, lo1}, u128{hi0, hi1}, v_first, width, v_end, ntiles));
    E.fams.push_back(f);
    E.tile_seg.assign(ntiles, 0);
    E.ntiles = ntiles;
    E.out_cap = out_cap;
    Scratch hold(ctx);
    int launches = 0;
    int rc = engine_prepare(E, tuning, hold);
    if (!rc) rc = engine_run(E, counts, geometry, n_out, &launches, [&](uint64_t) { return out; });
    if (!rc || rc == PC_OVERFLOW || rc == PC_ARITHMETIC) engine_stats(E, stats, launches, *n_out);
    if (stats) {
        stats->total_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
        stats->h2d_bytes = ctx->h2d - h2d0;
        stats->d2h_bytes = ctx->d2h - d2h0;
    }
    return rc;
}

extern "C" int pc_run_lease(pc_ctx *ctx, const pc_focus *fa, const pc_focus *fb, const pc_filters *f,
                            const pc_tuning *tuning, uint64_t first, uint64_t end, uint64_t width, uint64_t lo0,
                            uint64_t lo1, uint64_t hi0, uint64_t hi1, uint64_t *counts, uint64_t *geometry,
                            uint64_t *out, uint64_t out_cap, uint64_t *n_out, pc_stats *stats) {
    if (!fa || !fb || !f || width == 0 || end <= first) return pc_fail(ctx, PC_INVALID, "invalid lease arguments");
    if (stats) memset(stats, 0, sizeof(*stats));
    *n_out = 0;
    auto t0 = std::chrono::steady_clock::now();
    const uint64_t h2d0 = ctx->h2d, d2h0 = ctx->d2h;
    typedef unsigned __int128 w128;
    const w128 lo = (w128)lo1 << 64 | lo0, hi = (w128)hi1 << 64 | hi0;
    const w128 ulo = (lo + (w128)first * f->A) / f->B + 1, uhi = (hi + (w128)(end - 1) * f->A) / f->B + 1;
    if (uhi >> 64) return pc_fail(ctx, PC_INVALID, "u window exceeds 64 bits");
    const uint64_t ntiles64 = (end - first + width - 1) / width;
    if (ntiles64 >= (UINT64_C(1) << 31) || !tiles_fit(first, end, width, ntiles64))
        return pc_fail(ctx, PC_INVALID, "too many subtiles");
    int launches = 0;
    Scratch hold(ctx);
    PC_CHECK(ctx, cudaEventRecord(ctx->ev[4], ctx->stream));
    const pc_focus *foc[2] = {fa, fb};
    const uint64_t lows[2] = {(uint64_t)ulo, first}, highs[2] = {(uint64_t)uhi, end};
    WinBatch wb;
    uint64_t *d_lists = nullptr, list_bytes = 0;
    int rc = winbatch_run(ctx, hold, foc, lows, highs, 2, UINT64_C(1) << 33, wb, &d_lists, &list_bytes, &launches);
    if (d_lists) hold.items.emplace_back(d_lists, list_bytes);
    if (rc) return rc;
    for (uint64_t n : wb.total)
        if (n > (UINT64_C(1) << 32) - 1) return pc_fail(ctx, PC_OVERFLOW, "focus buffer overflow; tile invalid");
    PC_CHECK(ctx, cudaEventRecord(ctx->ev[5], ctx->stream));
    Engine E;
    E.ctx = ctx;
    E.us = d_lists + wb.base[0];
    E.nu = wb.total[0];
    E.vs = d_lists + wb.base[1];
    E.nv = wb.total[1];
    E.segs.push_back(one_segment(f, E.nu, E.nv, u128{lo0, lo1}, u128{hi0, hi1}, first, width, end, (uint32_t)ntiles64));
    E.fams.push_back(f);
    E.tile_seg.assign(ntiles64, 0);
    E.ntiles = ntiles64;
    E.out_cap = out_cap;
    rc = engine_prepare(E, tuning, hold);
    if (!rc) rc = engine_run(E, counts, geometry, n_out, &launches, [&](uint64_t) { return out; });
    if (!rc || rc == PC_OVERFLOW || rc == PC_ARITHMETIC) {
        engine_stats(E, stats, launches, *n_out);
        if (stats) stats->window_ms = elapsed_ms(ctx->ev[4], ctx->ev[5]);
    }
    if (stats) {
        stats->total_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
        stats->h2d_bytes = ctx->h2d - h2d0;
        stats->d2h_bytes = ctx->d2h - d2h0;
    }
    return rc;
}

// Leases one after another on the calling thread, so a host runtime that holds a lock while it
// builds receipts (an interpreter) never sits between two device calls.  status[i] becomes
// 1 + the return code of lease i once its outputs are on the host (release order), so another
// thread can consume lease i while later leases run; the loop stops at the first failing lease.
extern "C" int pc_run_leases(pc_ctx *ctx, const pc_focus *fa, const pc_focus *fb, const pc_filters *f,
                             const pc_tuning *tuning, uint32_t n, const uint64_t *first, const uint64_t *end,
                             uint64_t width, uint64_t lo0, uint64_t lo1, uint64_t hi0, uint64_t hi1,
                             uint64_t *const *counts, uint64_t *const *geometry, uint64_t *const *out, uint64_t out_cap,
                             uint64_t *n_out, pc_stats *stats, int32_t *status) {
    if (!ctx || (n && (!first || !end || !counts || !geometry || !out || !n_out || !status)))
        return pc_fail(ctx, PC_INVALID, "invalid lease list");
    for (uint32_t i = 0; i < n; ++i) {
        const int rc = pc_run_lease(ctx, fa, fb, f, tuning, first[i], end[i], width, lo0, lo1, hi0, hi1, counts[i],
                                    geometry[i], out[i], out_cap, n_out + i, stats ? stats + i : nullptr);
        __atomic_store_n(status + i, rc + 1, __ATOMIC_RELEASE);
        if (rc) return rc;
    }
    return PC_OK;
}

extern "C" int pc_run_plain(pc_ctx *ctx, const pc_filters *f, const pc_buf *us, uint64_t u_off, uint64_t nu,
                            const pc_buf *vs, uint64_t v_off, uint64_t nv, uint64_t lo0, uint64_t lo1, uint64_t hi0,
                            uint64_t hi1, uint64_t *counts, uint64_t *out, uint64_t out_cap, pc_stats *stats) {
    if (!f || !us || !vs) return pc_fail(ctx, PC_INVALID, "invalid plain arguments");
    if (u_off > us->n || nu > us->n - u_off || v_off > vs->n || nv > vs->n - v_off)
        return pc_fail(ctx, PC_INVALID, "focus list slice out of range");
    if (stats) memset(stats, 0, sizeof(*stats));
    const uint32_t ng = f->ng;
    Scratch s(ctx);
    uint64_t *d_counts;                                   // then the output records
    int rc = s.get(&d_counts, ng + 3 + 2 * std::max<uint64_t>(1, out_cap));
    if (rc) return rc;
    uint64_t *d_out = d_counts + ng + 3;
    cudaStream_t st = ctx->stream;
    int launches = 0;
    PC_CHECK(ctx, cudaMemsetAsync(d_counts, 0, (ng + 3) * 8, st));
    PC_CHECK(ctx, cudaEventRecord(ctx->ev[6], st));
    if (nu && nv) {
        PlainArgs a{};
        a.us = us->d + u_off;
        a.vs = vs->d + v_off;
        a.nu = nu;
        a.nv = nv;
        a.A = f->A;
        a.B = f->B;
        a.lo = u128{lo0, lo1};
        a.hi = u128{hi0, hi1};
        a.nres = f->nres;
        a.ng = ng;
        a.fc = f->d_fc;
        a.bits = f->d_bits;
        a.counts = d_counts;
        a.out = d_out;
        a.out_cap = out_cap;
        uint64_t *d_disorder = nullptr;
        if (plain_ordered(a) && s.get(&d_disorder, 1) == PC_OK) {   // without it, should it not fit, rows count as unordered
            PC_CHECK(ctx, cudaMemsetAsync(d_disorder, 0, 8, st));
            k_order<<<(unsigned)std::min<uint64_t>((nv + 1023) / 1024, (uint64_t)ctx->sm_count * 4), 256, 0, st>>>(a.vs, nv, d_disorder);
            PC_LAUNCHED(ctx, "plain order");
            a.ordered = true;
            a.disorder = d_disorder;
            ++launches;
        }
        plain_launch(a, f->primes.data(), ctx->sm_count, st);
        PC_LAUNCHED(ctx, "plain match");
        ++launches;
    }
    PC_CHECK(ctx, cudaEventRecord(ctx->ev[7], st));
    // the counters and the first records in one copy
    const uint64_t first = std::min<uint64_t>(out_cap, Engine::FETCH_RECORDS), words = ng + 3 + 2 * first;
    const StageLoan loan = pc_stage(ctx, words * 8);
    uint64_t *stage = loan.get();
    PC_CHECK(ctx, pc_copy(ctx, stage ? stage : counts, d_counts, (stage ? words : ng + 3) * 8, cudaMemcpyDeviceToHost));
    PC_CHECK(ctx, cudaStreamSynchronize(st));
    if (stage) memcpy(counts, stage, (ng + 3) * 8);
    uint64_t n = counts[ng + 1];
    if (stats) {
        stats->kernel_ms = elapsed_ms(ctx->ev[6], ctx->ev[7]);
        stats->outputs = n;
        stats->launches = launches;
    }
    const uint64_t copy = std::min(n, out_cap), got = stage ? std::min(copy, first) : 0;
    if (got) memcpy(out, stage + ng + 3, 16 * got);
    if (copy > got) {
        PC_CHECK(ctx, pc_copy(ctx, out + 2 * got, d_out + 2 * got, 16 * (copy - got), cudaMemcpyDeviceToHost));
        PC_CHECK(ctx, cudaStreamSynchronize(st));
    }
    return PC_OK;
}

// ------------------------------------------------------------------------------------------
// Many windows in one launch sequence (pc_multi_*).
//
// Every window carries its own interval, v range, subtile width, focus pair and filter family.
// Creation plans all u windows (on each window's A focus) and v windows (on its B focus), sizes
// every buffer and keeps them; a run regenerates the windows on the device and runs stages 2 and
// 3 over all of them as segments of one launch sequence.  With PC_RUN_GRAPH the sequence after
// the first eager run is recorded once into a CUDA graph and replayed.

struct pc_multi {
    pc_ctx *ctx;
    Scratch hold;                        // device buffers kept for the object's lifetime
    WinBatch wb;
    uint64_t *d_lists = nullptr;         // u windows (each on a 2048-entry boundary), then v windows
    Engine E;
    uint32_t nwin = 0;
    std::vector<uint32_t> tile_base;     // nwin + 1
    std::vector<uint64_t> sizes;         // per window: u count, v count
    std::vector<uint64_t> counts, geometry, out;
    uint64_t n_out = 0;
    int launches = 0;
    uint64_t graph_d2h = 0;          // bytes the recorded graph copies to the host per replay
    bool ran = false;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    uint64_t *h_report = nullptr;                     // the engine's report, page-locked, written by the graph
    const uint64_t *from = nullptr, *geo_from = nullptr;   // counters and envelopes of the last run
    explicit pc_multi(pc_ctx *c) : ctx(c), hold(c) { E.ctx = c; }
    ~pc_multi() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        if (h_report) cudaFreeHost(h_report);
    }
};

extern "C" int pc_multi_create(pc_ctx *ctx, const pc_focus *const *foci, uint32_t nfoci,
                               const pc_filters *const *families, uint32_t nfam, const pc_window *windows,
                               uint32_t nwin, const pc_tuning *tuning, uint64_t out_cap, pc_multi **out) {
    *out = nullptr;
    if (!foci || !families || !windows || nwin == 0) return pc_fail(ctx, PC_INVALID, "invalid window batch arguments");
    typedef unsigned __int128 w128;
    std::vector<const pc_focus *> focs(2 * (size_t)nwin);
    std::vector<uint64_t> lows(2 * (size_t)nwin), highs(2 * (size_t)nwin), pads(2 * (size_t)nwin);
    std::vector<uint32_t> fam_map(nfam, UINT32_MAX), tile_base(nwin + 1, 0);
    std::vector<const pc_filters *> used;
    uint64_t ntiles = 0;
    for (uint32_t i = 0; i < nwin; ++i) {
        const pc_window &w = windows[i];
        if (w.focus_a >= nfoci || w.focus_b >= nfoci || w.family >= nfam)
            return pc_fail(ctx, PC_INVALID, "window refers to a missing focus or filter family");
        const pc_filters *f = families[w.family];
        const pc_focus *fa = foci[w.focus_a], *fb = foci[w.focus_b];
        if (!f || !fa || !fb) return pc_fail(ctx, PC_INVALID, "null focus or filter family");
        if (pc_focus_modulus(fa) != f->A || pc_focus_modulus(fb) != f->B)
            return pc_fail(ctx, PC_INVALID, "focus moduli differ from the filter family's A and B");
        const w128 lo = (w128)w.lo1 << 64 | w.lo0, hi = (w128)w.hi1 << 64 | w.hi0;
        if (hi <= lo || (hi >> 96)) return pc_fail(ctx, PC_INVALID, "invalid window interval");
        if (w.width == 0 || w.end <= w.first) return pc_fail(ctx, PC_INVALID, "invalid window v range");
        const w128 ulo = (lo + (w128)w.first * f->A) / f->B + 1, uhi = (hi + (w128)(w.end - 1) * f->A) / f->B + 1;
        if (uhi >> 64) return pc_fail(ctx, PC_INVALID, "u window exceeds 64 bits");
        const uint64_t nt = (w.end - w.first + w.width - 1) / w.width;
        if (!tiles_fit(w.first, w.end, w.width, nt)) return pc_fail(ctx, PC_INVALID, "inconsistent subtile geometry");
        tile_base[i] = (uint32_t)ntiles;
        ntiles += nt;
        if (ntiles >= (UINT64_C(1) << 31)) return pc_fail(ctx, PC_INVALID, "too many subtiles");
        focs[i] = fa;
        lows[i] = (uint64_t)ulo;
        highs[i] = (uint64_t)uhi;
        pads[i] = SEG_ALIGN;
        focs[nwin + i] = fb;
        lows[nwin + i] = w.first;
        highs[nwin + i] = w.end;
        pads[nwin + i] = 1;
        if (fam_map[w.family] == UINT32_MAX) {
            fam_map[w.family] = (uint32_t)used.size();
            used.push_back(f);
        }
    }
    tile_base[nwin] = (uint32_t)ntiles;
    pc_multi *m = new pc_multi(ctx);
    m->nwin = nwin;
    m->tile_base = tile_base;
    int rc = winbatch_plan(ctx, m->hold, focs.data(), lows.data(), highs.data(), pads.data(), 2 * nwin,
                           (UINT64_C(1) << 32) - 1, m->wb);
    if (!rc) rc = m->hold.get(&m->d_lists, std::max<uint64_t>(1, m->wb.out_len));
    if (rc) {
        delete m;
        return rc;
    }
    const uint64_t vstart = m->wb.base[nwin];
    Engine &E = m->E;
    E.us = m->d_lists;
    E.nu = vstart;
    E.vs = m->d_lists + vstart;
    E.nv = m->wb.out_len - vstart;
    E.fams = used;
    E.ntiles = ntiles;
    E.out_cap = out_cap;
    E.tile_seg.resize(ntiles);
    m->sizes.resize(2 * (size_t)nwin);
    for (uint32_t i = 0; i < nwin; ++i) {
        const pc_window &w = windows[i];
        const pc_filters *f = families[w.family];
        SegDev g{};
        g.A = f->A;
        g.B = f->B;
        g.lo = u128{w.lo0, w.lo1};
        g.hi = u128{w.hi0, w.hi1};
        g.v_first = w.first;
        g.width = w.width;
        g.v_end = w.end;
        g.u_off = (uint32_t)m->wb.base[i];
        g.nu = (uint32_t)m->wb.total[i];
        g.v_off = (uint32_t)(m->wb.base[nwin + i] - vstart);
        g.nv = (uint32_t)m->wb.total[nwin + i];
        g.tile_base = tile_base[i];
        g.ntiles = tile_base[i + 1] - tile_base[i];
        g.fam = fam_map[w.family];
        E.segs.push_back(g);
        for (uint32_t t = tile_base[i]; t < tile_base[i + 1]; ++t) E.tile_seg[t] = i;
        m->sizes[2 * i] = g.nu;
        m->sizes[2 * i + 1] = g.nv;
    }
    E.windows = true;
    rc = engine_prepare(E, tuning, m->hold);
    // zeroed once: a pass that gave up makes this and every later result of the object an error
    if (!rc) rc = pc_cuda_status(ctx, cudaMemsetAsync(E.d_report, 0, 8, ctx->stream), "window flag");
    m->wb.d_stuck = E.d_report + Engine::STUCK;
    if (!rc) rc = pc_cuda_status(ctx, cudaStreamSynchronize(ctx->stream), "window batch set-up");
    if (rc) {
        delete m;
        return rc;
    }
    *out = m;
    return PC_OK;
}

namespace {

int multi_eager(pc_ctx *ctx, pc_multi *m, pc_stats *stats) {
    Engine &E = m->E;
    int launches = 0;
    PC_CHECK(ctx, cudaEventRecord(ctx->ev[4], ctx->stream));
    int rc = winbatch_emit(ctx, m->wb, m->d_lists, m->wb.out_len);
    if (rc) return rc;
    launches += 1;
    PC_CHECK(ctx, cudaEventRecord(ctx->ev[5], ctx->stream));
    m->counts.resize(E.ntiles * E.stride);
    m->geometry.resize(2 * E.ntiles);
    const uint32_t deep_cap = E.deep_cap;
    rc = engine_run(E, m->counts.data(), m->geometry.data(), &m->n_out, &launches, [&](uint64_t n) {
        m->out.resize(2 * n);
        return m->out.data();
    });
    if (E.deep_cap != deep_cap && m->exec) {              // the recorded graph writes to the slices that were
        cudaGraphExecDestroy(m->exec);
        cudaGraphDestroy(m->graph);
        m->exec = nullptr;
        m->graph = nullptr;
    }
    m->from = m->counts.data();
    m->geo_from = m->geometry.data();
    m->launches = launches;
    if (!rc || rc == PC_OVERFLOW || rc == PC_ARITHMETIC) {
        engine_stats(E, stats, launches, m->n_out);
        if (stats) stats->window_ms = elapsed_ms(ctx->ev[4], ctx->ev[5]);
    }
    return rc;
}

// Records the whole run (windows, stages 2 and 3, and the copies of the counters) into a graph.
// The deep tier's grid and slice capacity come from the eager run that precedes the capture.
int multi_capture(pc_ctx *ctx, pc_multi *m) {
    Engine &E = m->E;
    cudaStream_t st = ctx->stream;
    const uint64_t bytes = E.fetch_words() * 8;
    if (!m->h_report) PC_CHECK(ctx, cudaMallocHost((void **)&m->h_report, bytes));
    int rc = engine_match(E, 2);
    if (rc) return rc;
    PC_CHECK(ctx, cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    int launches = 0;
    rc = winbatch_emit(ctx, m->wb, m->d_lists, m->wb.out_len);
    if (!rc) rc = engine_launch(E, false, true, &launches);
    if (!rc) rc = pc_cuda_status(ctx, pc_copy(ctx, m->h_report, E.d_report, bytes, cudaMemcpyDeviceToHost), "capture copy");
    cudaGraph_t g = nullptr;
    const cudaError_t e = cudaStreamEndCapture(st, &g);       // always leave capture mode
    if (!rc && e != cudaSuccess) rc = pc_cuda_fail(ctx, e, "end capture");
    if (rc) {
        if (g) cudaGraphDestroy(g);
        cudaGetLastError();
        return rc;
    }
    m->graph = g;
    PC_CHECK(ctx, cudaGraphInstantiate(&m->exec, g, 0));
    m->launches = launches + 1;
    // the copies recorded into the graph run at every replay, not at capture
    m->graph_d2h = bytes;
    ctx->d2h -= m->graph_d2h;
    return PC_OK;
}

int multi_replay(pc_ctx *ctx, pc_multi *m, pc_stats *stats) {
    Engine &E = m->E;
    cudaStream_t st = ctx->stream;
    int rc = engine_match(E, 2);                          // another object may have lowered the limit
    if (rc) return rc;
    PC_CHECK(ctx, cudaEventRecord(ctx->ev[0], st));
    PC_CHECK(ctx, cudaGraphLaunch(m->exec, st));
    ctx->d2h += m->graph_d2h;
    PC_CHECK(ctx, cudaEventRecord(ctx->ev[1], st));
    PC_CHECK(ctx, cudaStreamSynchronize(st));
    const uint64_t *counts = m->h_report + E.o_counts;
    bool outgrown = false;
    rc = engine_check(E, m->h_report, counts, outgrown);
    if (outgrown) return pc_fail(ctx, PC_ARITHMETIC, "deep survivor count changed between runs");
    m->from = counts;
    m->geo_from = m->h_report + E.o_geo;
    m->n_out = m->h_report[Engine::NOUT];
    if (!rc) {
        m->out.resize(2 * m->n_out);
        rc = engine_records(E, m->h_report + E.o_out, (E.fetch_words() - E.o_out) / 2, m->n_out, m->out.data());
    }
    if (stats) {
        stats->kernel_ms = elapsed_ms(ctx->ev[0], ctx->ev[1]);
        stats->outputs = m->n_out;
        stats->launches = m->launches;
        stats->work_items = E.deep_max;
        stats->reserved[0] = E.tn.nb;
        stats->reserved[1] = E.tn.K;
        stats->reserved[2] = E.tn.threads;
        stats->reserved[3] = E.tn.nch;
        stats->reserved[4] = 1;
    }
    return rc;
}

}  // namespace

extern "C" int pc_multi_run(pc_ctx *ctx, pc_multi *m, uint32_t flags, pc_stats *stats) {
    if (!m) return pc_fail(ctx, PC_INVALID, "no window batch");
    if (stats) memset(stats, 0, sizeof(*stats));
    auto t0 = std::chrono::steady_clock::now();
    const uint64_t h2d0 = ctx->h2d, d2h0 = ctx->d2h;
    int rc = PC_OK;
    if (!(flags & PC_RUN_GRAPH) || !m->ran) {
        rc = multi_eager(ctx, m, stats);
        if (!rc) m->ran = true;
    }
    if (!rc && (flags & PC_RUN_GRAPH)) {
        if (!m->exec) rc = multi_capture(ctx, m);
        if (!rc) rc = multi_replay(ctx, m, stats);
    }
    // a failed run leaves no results, and the next one runs eagerly (and sizes its slices) before it replays a graph
    if (rc) m->ran = false;
    if (stats) {
        stats->total_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
        stats->h2d_bytes = ctx->h2d - h2d0;
        stats->d2h_bytes = ctx->d2h - d2h0;
    }
    return rc;
}

extern "C" int pc_multi_layout(const pc_multi *m, uint32_t *tile_base, uint64_t *sizes, uint64_t *info) {
    if (!m) return PC_INVALID;
    const Engine &E = m->E;
    if (tile_base) std::copy(m->tile_base.begin(), m->tile_base.end(), tile_base);
    if (sizes) std::copy(m->sizes.begin(), m->sizes.end(), sizes);
    if (info) {
        info[0] = E.ntiles;
        info[1] = E.stride;
        info[2] = E.nu;
        info[3] = E.nv;
        info[4] = E.deep_cap;
        info[5] = E.tn.nb;
        info[6] = E.tn.K;
        info[7] = E.tn.threads;
    }
    return PC_OK;
}

extern "C" int pc_multi_results(pc_ctx *ctx, const pc_multi *m, uint64_t *counts, uint64_t *geometry, uint64_t *out,
                                uint64_t out_cap, uint64_t *n_out) {
    if (!m || !m->ran) return pc_fail(ctx, PC_INVALID, "window batch has not run");
    if (counts) std::copy(m->from, m->from + m->E.ntiles * m->E.stride, counts);
    if (geometry) std::copy(m->geo_from, m->geo_from + 2 * m->E.ntiles, geometry);
    *n_out = m->n_out;
    if (out) std::copy(m->out.begin(), m->out.begin() + 2 * std::min(m->n_out, out_cap), out);
    return PC_OK;
}

extern "C" int pc_multi_free(pc_ctx *ctx, pc_multi *m) {
    if (!m) return PC_OK;
    cudaStreamSynchronize(ctx->stream);
    delete m;
    return PC_OK;
}

// ------------------------------------------------------------------------------------------
// Plain per-tile matcher with no device allocation (pc_run_plain_static).
//
// Its scratch is this file-scope device array, reserved when the library loads and held by every
// GPU that loads it until the process exits.  Host code must not pass the array's name to a
// kernel (on the host the name is only a stand-in, not a device address): the device address is
// looked up once per device with cudaGetSymbolAddress and cached.  Every call reuses the same
// bytes, so calls that overlap on one GPU race with each other.

constexpr uint64_t STATIC_SCRATCH_BYTES = UINT64_C(16) << 20;   // 16 MiB
static __device__ __align__(256) unsigned char g_static_scratch[STATIC_SCRATCH_BYTES];

namespace {
constexpr int STATIC_MAX_DEVICES = 64;
unsigned char *g_static_ptr[STATIC_MAX_DEVICES] = {};

inline uint64_t align256(uint64_t x) { return (x + 255) & ~UINT64_C(255); }

int static_fail(char *err, int err_len, int code, const char *msg) {
    if (err && err_len > 0) {
        strncpy(err, msg, (size_t)err_len - 1);
        err[err_len - 1] = 0;
    }
    return code;
}

int static_cuda(char *err, int err_len, cudaError_t e, const char *what) {
    char buf[256];
    snprintf(buf, sizeof(buf), "%s: %s", what, cudaGetErrorString(e));
    return static_fail(err, err_len, PC_CUDA, buf);
}
}  // namespace

// The body of pc_run_plain_static once its device is current.
static int plain_static_on(int device, const uint64_t *us, uint64_t nu, const uint64_t *vs, uint64_t nv, uint64_t A,
                    uint64_t B, uint64_t lo0, uint64_t lo1, uint64_t hi0, uint64_t hi1, const uint32_t *primes,
                    uint32_t nres, const uint8_t *allowed, uint32_t ng, uint64_t o_counts, uint64_t o_fc,
                    uint64_t o_bits, uint64_t o_us, uint64_t o_vs, uint64_t o_out, uint64_t *counts, uint64_t *out,
                    uint64_t out_cap, char *err, int err_len);

extern "C" int pc_run_plain_static(int device, const uint64_t *us, uint64_t nu, const uint64_t *vs, uint64_t nv,
                                   uint64_t A, uint64_t B, uint64_t lo0, uint64_t lo1, uint64_t hi0, uint64_t hi1,
                                   const uint32_t *primes, uint32_t nres, const uint8_t *allowed, uint64_t *counts,
                                   uint64_t *out, uint64_t out_cap, char *err, int err_len) {
    if (device < 0 || device >= STATIC_MAX_DEVICES) return static_fail(err, err_len, PC_INVALID, "device index out of range");
    if (nres == 0 || nres > PC_MAX_RES || A == 0 || B == 0 || !counts || !primes || !allowed || (nu && !us) ||
        (nv && !vs) || (out_cap && !out))
        return static_fail(err, err_len, PC_INVALID, "invalid plain tile arguments");
    // every size is bounded by the scratch before any offset is formed, so no product below wraps
    constexpr uint64_t too_big = STATIC_SCRATCH_BYTES;
    if (nu > too_big / 8 || nv > too_big / 8 || out_cap > too_big / 16)
        return static_fail(err, err_len, PC_INVALID, "tile exceeds the 16 MiB static scratch of pc_run_plain_static");
    uint64_t words = 0;
    for (uint32_t i = 0; i < nres; ++i) {
        const uint32_t q = primes[i];
        if (q < 2 || q >= 8192 || A % q == 0 || B % q == 0)
            return static_fail(err, err_len, PC_INVALID, "residual modulus must be in [2, 8192) and coprime to A and B");
        words += (q + 31) / 32;
    }
    const uint32_t ng = (nres + 3) / 4;
    // layout of the static scratch: counters | filter constants | bitmaps | us | vs | outputs
    const uint64_t o_counts = 0, o_fc = align256(o_counts + (ng + 3) * 8), o_bits = align256(o_fc + nres * sizeof(FiltConst));
    const uint64_t o_us = align256(o_bits + words * 4), o_vs = align256(o_us + nu * 8), o_out = align256(o_vs + nv * 8);
    const uint64_t need = o_out + 2 * (out_cap ? out_cap : 1) * 8;
    if (need > STATIC_SCRATCH_BYTES)
        return static_fail(err, err_len, PC_INVALID, "tile exceeds the 16 MiB static scratch of pc_run_plain_static");

    // the caller's current device is put back on every return
    int previous = -1;
    cudaError_t e = cudaGetDevice(&previous);
    if (e != cudaSuccess) return static_cuda(err, err_len, e, "cudaGetDevice");
    if (previous != device) {
        e = cudaSetDevice(device);
        if (e != cudaSuccess) return static_cuda(err, err_len, e, "cudaSetDevice");
    }
    const int rc = plain_static_on(device, us, nu, vs, nv, A, B, lo0, lo1, hi0, hi1, primes, nres, allowed, ng,
                                   o_counts, o_fc, o_bits, o_us, o_vs, o_out, counts, out, out_cap, err, err_len);
    if (previous != device) {
        e = cudaSetDevice(previous);
        if (e != cudaSuccess && rc == PC_OK) return static_cuda(err, err_len, e, "cudaSetDevice (restore)");
    }
    return rc;
}

static int plain_static_on(int device, const uint64_t *us, uint64_t nu, const uint64_t *vs, uint64_t nv, uint64_t A,
                    uint64_t B, uint64_t lo0, uint64_t lo1, uint64_t hi0, uint64_t hi1, const uint32_t *primes,
                    uint32_t nres, const uint8_t *allowed, uint32_t ng, uint64_t o_counts, uint64_t o_fc,
                    uint64_t o_bits, uint64_t o_us, uint64_t o_vs, uint64_t o_out, uint64_t *counts, uint64_t *out,
                    uint64_t out_cap, char *err, int err_len) {
    cudaError_t e = cudaSuccess;
    // Set-up, once per device, with that device current.  The cached address belongs to the
    // device's primary context; a process that resets the device (cudaDeviceReset) must not call
    // this entry point on it again.
    if (!g_static_ptr[device]) {
        void *ptr = nullptr;
        e = cudaGetSymbolAddress(&ptr, g_static_scratch);
        if (e != cudaSuccess) return static_cuda(err, err_len, e, "cudaGetSymbolAddress");
        g_static_ptr[device] = (unsigned char *)ptr;
    }
    unsigned char *base = g_static_ptr[device];
    cudaStream_t st = 0;
    // filter constants and packed bitmaps, staged through fixed host buffers
    {
        FiltConst fc[32];
        uint32_t bits[1024];
        uint64_t word_at = 0, nbits = 0, off = 0;
        uint32_t nfc = 0, fc_at = 0;
        for (uint32_t i = 0; i < nres; ++i) {
            const uint32_t q = primes[i];
            FiltConst &c = fc[nfc++];
            c.m = make_modq(q);
            c.tab_off = (uint32_t)(word_at + nbits);
            c.pad = 0;
            for (uint32_t w = 0; w < (q + 31) / 32; ++w) {
                uint32_t v = 0;
                for (uint32_t r = w * 32; r < q && r < w * 32 + 32; ++r)
                    if (allowed[off + r]) v |= 1u << (r - w * 32);
                bits[nbits++] = v;
                if (nbits == 1024) {
                    e = cudaMemcpyAsync(base + o_bits + word_at * 4, bits, nbits * 4, cudaMemcpyHostToDevice, st);
                    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
                    if (e != cudaSuccess) return static_cuda(err, err_len, e, "bitmap upload");
                    word_at += nbits;
                    nbits = 0;
                }
            }
            off += q;
            if (nfc == 32 || i + 1 == nres) {
                e = cudaMemcpyAsync(base + o_fc + (uint64_t)fc_at * sizeof(FiltConst), fc, nfc * sizeof(FiltConst),
                                    cudaMemcpyHostToDevice, st);
                if (e == cudaSuccess) e = cudaStreamSynchronize(st);
                if (e != cudaSuccess) return static_cuda(err, err_len, e, "filter upload");
                fc_at += nfc;
                nfc = 0;
            }
        }
        if (nbits) {
            e = cudaMemcpyAsync(base + o_bits + word_at * 4, bits, nbits * 4, cudaMemcpyHostToDevice, st);
            if (e == cudaSuccess) e = cudaStreamSynchronize(st);
            if (e != cudaSuccess) return static_cuda(err, err_len, e, "bitmap upload");
        }
    }
    e = cudaMemsetAsync(base + o_counts, 0, (ng + 3) * 8, st);   // the array keeps the previous call's counts
    if (e == cudaSuccess && nu) e = cudaMemcpyAsync(base + o_us, us, nu * 8, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess && nv) e = cudaMemcpyAsync(base + o_vs, vs, nv * 8, cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return static_cuda(err, err_len, e, "input upload");
    if (nu && nv) {
        int sm = 0;
        cudaDeviceGetAttribute(&sm, cudaDevAttrMultiProcessorCount, device);
        PlainArgs a{};
        a.us = (const uint64_t *)(base + o_us);
        a.vs = (const uint64_t *)(base + o_vs);
        a.nu = nu;
        a.nv = nv;
        a.A = A;
        a.B = B;
        a.lo = u128{lo0, lo1};
        a.hi = u128{hi0, hi1};
        a.nres = nres;
        a.ng = ng;
        a.fc = (const FiltConst *)(base + o_fc);
        a.bits = (const uint32_t *)(base + o_bits);
        a.counts = (uint64_t *)(base + o_counts);
        a.out = (uint64_t *)(base + o_out);
        a.out_cap = out_cap;
        a.ordered = plain_ordered(a) && std::is_sorted(vs, vs + nv);
        plain_launch(a, primes, std::max(sm, 1), st);
        e = cudaGetLastError();
        if (e != cudaSuccess) return static_cuda(err, err_len, e, "plain match launch");
    }
    e = cudaMemcpyAsync(counts, base + o_counts, (ng + 3) * 8, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return static_cuda(err, err_len, e, "counter download");
    const uint64_t copy = std::min(counts[ng + 1], out_cap);
    if (copy && out) {
        e = cudaMemcpyAsync(out, base + o_out, 2 * copy * 8, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return static_cuda(err, err_len, e, "output download");
    }
    return PC_OK;
}
