// Stage 1: CRT focus-wheel tables and sorted focus windows.
//
// A focus of modulus M is the set of y >= 0 whose residue mod every ring modulus q | M lies in
// the ring's (coefficient-adjusted) allowed set R_q.  Split the rings into S (small moduli) and
// T (the largest few).  With M1 = prod(S), the sorted wheel W1 = {w in [0, M1): w mod q in R_q
// for q in S} is built once, from the wheel of its smallest rings up (below).  Every y = K*M1 + w (w in W1)
// satisfies the S rings; it is in the focus iff (K*M1 + w) mod q in R_q for the T rings.  For
// each T ring and each s in [0, q), a bitset row over W1's index space marks the w with
// (s + w) mod q in R_q; the window for period K is the AND of the rows s = K*M1 mod q.
//
// A window [low, high) is therefore walked in (period, wheel index) order, which is ascending
// value order: one pass that finds its output positions as it goes (a decoupled look-back over the
// tiles before it) produces the sorted values with no sort and no residue set materialised.  Tables
// are p-independent for p above the largest focus prime.
#include "common.cuh"
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <memory>
#include <numeric>

struct pc_focus {
    uint64_t M = 0, M1 = 1, count1 = 0, words1 = 0;
    uint64_t stride = 0;         // words from one row to the next: words1 rounded up to 16 bytes
    uint32_t nT = 0;
    uint32_t tq[PC_MAX_WHEEL_T] = {};
    uint32_t t_m1mod[PC_MAX_WHEEL_T] = {};
    uint32_t t_row0[PC_MAX_WHEEL_T] = {};
    uint32_t total_rows = 0;
    uint64_t *W1 = nullptr;      // device, sorted wheel
    uint32_t *rows = nullptr;    // device, total_rows x stride
    uint64_t W1_bytes = 0, rows_bytes = 0;
    std::vector<uint64_t> sample; // host: every SAMPLE-th wheel entry (window ends are refined on the device)
    uint64_t count_lo = 0, count_hi = 0;
    double build_ms = 0;
    double density = 0;          // focus values per coordinate
};

namespace {

constexpr int WT = 256;          // threads per CTA of the window kernels
constexpr uint64_t SAMPLE = 128;      // wheel entries per host sample: the 128 entries of a lane's four words
constexpr uint64_t BASE_STEPS = 1 << 16;   // candidates of one ring's step of the host's base wheel
constexpr int WIN_WORDS = 128;   // wheel words per window unit: four per lane, one 16-byte load per row
constexpr int WIN_WARPS = WT / 32;
constexpr uint32_t WIN_ROUNDS = 8;    // most units per warp
constexpr uint32_t WIN_FEW = 2;                         // windows whose descriptors are launch parameters
constexpr uint32_t WIN_STAGE = 512;   // values of one warp staged in shared memory (a denser warp writes unit by unit)

// Rings whose rows one launch of k_wheel_rows builds.
struct RowRings {
    uint32_t q[PC_MAX_WHEEL_T], off[PC_MAX_WHEEL_T], row0[PC_MAX_WHEEL_T];   // off: first word of the ring's pattern
    ModQ mq[PC_MAX_WHEEL_T];
};

// rows[row0 + s][w] bit l = R[(s + W1[32w + l] mod q) mod q], via the rotation of the pattern
// RR (R repeated) by m = W1 mod q and a warp transpose.  A warp builds four consecutive words of every
// row of one ring (blockIdx.y), so a row's four words are one 16-byte store.
__global__ void k_wheel_rows(const uint64_t *__restrict__ W1, uint64_t count1, const uint32_t *__restrict__ patterns,
                             const RowRings rings, uint32_t *__restrict__ rows, uint64_t stride) {
    const uint32_t lane = threadIdx.x & 31, ring = blockIdx.y, q = rings.q[ring];
    const uint64_t w = ((blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5) * 4;
    if (w >= stride) return;                            // the words that pad a row are zero
    const uint32_t *pattern = patterns + rings.off[ring];
    uint32_t m[4];
    bool valid[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint64_t j = (w + k) * 32 + lane;
        valid[k] = j < count1;
        m[k] = valid[k] ? mod64(W1[j], rings.mq[ring]) : 0;
    }
    uint32_t sh[5], keep[5];
    transpose_consts(lane, sh, keep);
    for (uint32_t g = 0; g * 32 < q; ++g) {
        uint32_t v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t st = 32 * g + m[k];
            const uint32_t col = __funnelshift_r(pattern[st >> 5], pattern[(st >> 5) + 1], st & 31);
            v[k] = transpose32c(valid[k] ? col : 0u, sh, keep);
        }
        const uint32_t s = 32 * g + lane;
        if (s < q) *(uint4 *)(rows + (uint64_t)(rings.row0[ring] + s) * stride + w) = make_uint4(v[0], v[1], v[2], v[3]);
    }
}

__global__ void k_sample(const uint64_t *__restrict__ W1, uint64_t n, uint64_t *__restrict__ out) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i < n) out[i] = W1[i * SAMPLE];
}

struct WindowPlan {
    uint64_t K0, K1, j_lo, j_hi;       // wheel range: j_lo and j_hi are the ends of the 128-entry blocks
    uint64_t rem_lo, rem_hi;           // that hold the first entry >= rem_lo and the last < rem_hi
    uint64_t wa0, wb0, wa1, wb1;       // word ranges of the first and last period
    uint64_t units_first, units_mid, units_last, units;
    uint64_t chunks;                   // 32-word chunks, the measure of the refusal of too long windows
};

// Device view of one focus: the sorted wheel and the bitset rows of its T rings.
struct FocusDev {
    const uint64_t *W1;
    const uint32_t *rows;
    uint64_t M1, count1, words1, stride;
    uint32_t nT, pad;
    uint32_t t_m1mod[PC_MAX_WHEEL_T];
    uint32_t t_row0[PC_MAX_WHEEL_T];
    ModQ tmq[PC_MAX_WHEEL_T];
};

// Bits [a, e) of one 32-bit word.
__device__ __forceinline__ uint32_t span_bits(int32_t a, int32_t e) {
    return low_bits((uint32_t)min(max(e, 0), 32)) & ~low_bits((uint32_t)min(max(a, 0), 32));
}

// One window of a batch: its plan, its first unit in the batch-wide unit numbering and its focus.
struct WinDesc {
    WindowPlan plan;
    uint64_t unit_base;
    uint32_t focus, pad;
};

// The descriptors of one or two windows (a focus window, the window pair of a lease) travel with the launch: no
// device copy of them is allocated and filled first.
struct WinFew {
    WinDesc desc[WIN_FEW];
    FocusDev foci[WIN_FEW];
};
static_assert(sizeof(WinFew) <= 2048, "kernel parameters");

__device__ __forceinline__ void unit_of(const WindowPlan &p, uint64_t words1, uint64_t u, uint64_t &K,
                                        uint64_t &wa, uint64_t &wb) {
    if (u < p.units_first) {
        K = p.K0;
        wa = p.wa0 + u * WIN_WORDS;
        wb = min(p.wb0, wa + WIN_WORDS);
        return;
    }
    u -= p.units_first;
    uint64_t mid_periods = p.K1 > p.K0 + 1 ? p.K1 - p.K0 - 1 : 0;
    if (u < mid_periods * p.units_mid) {
        const uint32_t um = (uint32_t)p.units_mid, uu = (uint32_t)u;     // unit counts < 2^32
        const uint32_t period = uu / um;
        K = p.K0 + 1 + period;
        wa = (uint64_t)(uu - period * um) * WIN_WORDS;
        wb = min(words1, wa + WIN_WORDS);
        return;
    }
    u -= mid_periods * p.units_mid;
    K = p.K1;
    wa = p.wa1 + u * WIN_WORDS;
    wb = min(p.wb1, wa + WIN_WORDS);
}

// Device buffers of one emitting pass.
struct WinOut {
    unsigned long long *ticket;        // next tile; the words after it are the tile states, all zeroed before the launch
    unsigned long long *state;         // per tile: values << 2 | 1 (its own) or 2 (its own and all before it)
    uint64_t *starts;                  // per window: values of the windows before it; the last entry, the total
    const uint64_t *delta;             // per window: added to its output positions (modulo 2^64), or null
    uint64_t *out;
    uint64_t cap;                      // entries of out
    uint64_t *stuck;                   // set when a look-back wait ran out
    uint64_t ntiles;
    uint32_t polls;                    // most of one such wait
};

// Walks a warp's consecutive units.  The first is found by a binary search over the windows' first units
// and a division; each next one is 128 words on, in the next period or in the next window.  The rows of a
// period are located by one lane per T ring when the period changes.
struct UnitWalk {
    const WinDesc *desc;
    const FocusDev *foci, *f;
    uint32_t lane, win, nT;
    uint32_t row[PC_MAX_WHEEL_T];                       // the period's rows, in 16-byte steps from the table's start
    uint64_t K, K0, K1, wa, wb;                         // the unit's period and first word, the period's word end

    __device__ __forceinline__ UnitWalk(const WinDesc *d, uint32_t ndesc, const FocusDev *fs, uint64_t u0, uint32_t l)
        : desc(d), foci(fs), lane(l), win(0) {
        uint32_t hi = ndesc;                            // last window with unit_base <= u0
        while (hi - win > 1) {
            const uint32_t mid = (win + hi) / 2;
            if (desc[mid].unit_base <= u0) win = mid;
            else hi = mid;
        }
        open();
        unit_of(desc[win].plan, f->words1, u0 - desc[win].unit_base, K, wa, wb);
        wb = K == K0 ? desc[win].plan.wb0 : K == K1 ? desc[win].plan.wb1 : f->words1;
        locate();
    }

    __device__ __forceinline__ void open() {            // the first period of window `win`
        const WindowPlan &p = desc[win].plan;
        f = foci + desc[win].focus;
        nT = f->nT;
        K0 = K = p.K0, K1 = p.K1, wa = p.wa0, wb = p.wb0;
    }

    __device__ __forceinline__ void locate() {
        uint32_t mine = 0;
        if (lane < nT) {
            const ModQ &m = f->tmq[lane];
            const uint32_t s = fastmod32(mod64(K, m) * f->t_m1mod[lane], m.c, m.q);   // < q^2 < 2^32
            mine = (uint32_t)((uint64_t)(f->t_row0[lane] + s) * (f->stride / 4));
        }
#pragma unroll
        for (uint32_t k = 0; k < PC_MAX_WHEEL_T; ++k) row[k] = __shfl_sync(0xffffffffu, mine, k);
    }

    __device__ __forceinline__ void step() {            // only while another unit follows
        wa += WIN_WORDS;
        if (wa < wb) return;
        while (wa >= wb) {
            if (K < K1) {
                ++K;
                wa = 0;
                wb = K == K1 ? desc[win].plan.wb1 : f->words1;
            } else {
                ++win;
                open();
            }
        }
        locate();
    }

    // Entries below x among the 128 wheel entries from j on (the whole warp, for one block).
    __device__ __forceinline__ uint32_t below(uint64_t j, uint64_t x) const {
        uint32_t n = 0;
#pragma unroll
        for (uint32_t k = 0; k < SAMPLE; k += 32)
            n += __popc(__ballot_sync(0xffffffffu, j + k + lane < f->count1 && __ldg(f->W1 + j + k + lane) < x));
        return n;
    }

    // The lane's four words of the unit; w: the first of them.
    __device__ __forceinline__ uint4 words(uint32_t &w) const {
        w = (uint32_t)wa + 4 * lane;
        const uint4 ones = make_uint4(0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu);
        uint4 t[PC_MAX_WHEEL_T];
        const bool in = w < wb;
        const uint4 *rows = (const uint4 *)f->rows + (w >> 2);
#pragma unroll
        for (uint32_t k = 0; k < PC_MAX_WHEEL_T; ++k) { // all row loads in flight before the first use
            t[k] = ones;
            if (k < nT && in) t[k] = __ldg(rows + row[k]);
        }
        uint4 b = in ? ones : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (uint32_t k = 0; k < PC_MAX_WHEEL_T; ++k)
            if (k < nT) b.x &= t[k].x, b.y &= t[k].y, b.z &= t[k].z, b.w &= t[k].w;
        if (K == K0 || K == K1 || !nT) {                // entries of [jmin, jmax) only (rows end in zero bits)
            const WindowPlan &p = desc[win].plan;
            uint64_t jmin = 0, jmax = f->count1;
            const uint64_t j = (uint64_t)w * 32, first = wa * 32;
            if (K == K0) jmin = first <= p.j_lo && p.j_lo < first + 32 * WIN_WORDS ? p.j_lo + below(p.j_lo, p.rem_lo) : p.j_lo;
            if (K == K1) {
                const uint64_t block = p.j_hi ? (p.j_hi - 1) & ~(SAMPLE - 1) : 0;
                jmax = first <= block && block < first + 32 * WIN_WORDS ? block + below(block, p.rem_hi) : p.j_hi;
            }
            const int32_t a = j < jmin ? (int32_t)umin64(jmin - j, 128) : 0;
            const int32_t e = j < jmax ? (int32_t)umin64(jmax - j, 128) : 0;
            b.x &= span_bits(a, e), b.y &= span_bits(a - 32, e - 32);
            b.z &= span_bits(a - 64, e - 64), b.w &= span_bits(a - 96, e - 96);
        }
        return b;
    }
};

__device__ __forceinline__ uint32_t popc128(uint4 b) { return __popc(b.x) + __popc(b.y) + __popc(b.z) + __popc(b.w); }

// The windows' values, in order.  A unit is 128 wheel words: a lane takes four, so each row of the
// period is one 16-byte load per lane and 512 coalesced bytes per warp, and the unit's address
// arithmetic, warp scan and window lookup are paid once for 4,096 wheel entries.  A warp takes `rounds`
// consecutive units.  Without EMIT only the windows' totals are counted.  With EMIT the warp stages
// its values in shared memory (the wheel indices first, so that the wheel loads are one value per
// lane) while warp 0 finds the tile's output position by look-back, and then stores them
// coalesced.  A warp whose units hold more than WIN_STAGE values (a focus without T rings keeps every wheel
// entry) writes them word by word after the look-back instead, one bit per lane.
//
// Bound: L2 (per lease 1.07 GB of row words, one 32-byte sector of W1 for each of 26M values, 0.2 GB of
// stores) and the look-back's latency.  Against a count pass, a scan and an emit pass with one wheel word per lane: the
// two windows of a lease 1.15 -> 0.46 ms, 512 uneven windows 0.86 -> 0.35 ms.
template <bool EMIT, bool FEW>
__global__ void __launch_bounds__(WT, 4) k_windows(const WinDesc *__restrict__ many, uint32_t ndesc,
                                                const FocusDev *__restrict__ many_foci, uint64_t units, uint32_t rounds,
                                                unsigned long long *__restrict__ totals, const WinOut o,
                                                const __grid_constant__ WinFew few) {
    const WinDesc *__restrict__ desc = FEW ? few.desc : many;
    const FocusDev *__restrict__ foci = FEW ? few.foci : many_foci;
    __shared__ uint64_t tile_s, before_s;
    __shared__ uint32_t sum_s[WIN_WARPS];
    __shared__ uint64_t value_s[EMIT ? WIN_WARPS : 1][EMIT ? WIN_STAGE : 1];
    __shared__ uint16_t index_s[EMIT ? WIN_WARPS : 1][EMIT ? WIN_STAGE : 1];   // round << 12 | entry of the unit
    __shared__ struct {
        uint64_t kbase, delta;                          // K * M1; output position minus values before the window
        const uint64_t *wheel;                          // the unit's first entry
        uint32_t before, win;                           // values of the warp's earlier units
    } unit_s[EMIT ? WIN_WARPS : 1][EMIT ? WIN_ROUNDS : 1];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t tile = blockIdx.x;
    if (EMIT) {
        if (threadIdx.x == 0) tile_s = atomicAdd(o.ticket, 1ull);
        __syncthreads();
        tile = tile_s;
    }
    const uint64_t u0 = (tile * WIN_WARPS + warp) * rounds;
    const uint32_t mine = u0 < units ? (uint32_t)umin64(units - u0, rounds) : 0;      // warp-uniform
    uint32_t own = 0;                                   // EMIT: values of the warp; else of the lane
    if (mine) {
        UnitWalk walk(desc, ndesc, foci, u0, lane);
        uint32_t counted = walk.win;
        for (uint32_t r = 0; r < mine; ++r) {
            if (r) walk.step();
            if (!EMIT && walk.win != counted) {
                const uint32_t sum = __reduce_add_sync(0xffffffffu, own);
                if (lane == 0 && sum) atomicAdd(totals + counted, (unsigned long long)sum);
                own = 0;
                counted = walk.win;
            }
            uint32_t w;
            const uint4 b = walk.words(w);
            const uint32_t n = popc128(b);
            if (!EMIT) {
                own += n;
                continue;
            }
            if (lane == 0) {
                auto &u = unit_s[warp][r];
                u.kbase = walk.K * walk.f->M1;
                u.delta = o.delta ? o.delta[walk.win] : 0;
                u.wheel = walk.f->W1 + (uint64_t)w * 32;
                u.before = own;
                u.win = walk.win;
            }
            uint32_t incl = n;
#pragma unroll
            for (int s = 1; s < 32; s <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, s);
                if (lane >= (uint32_t)s) incl += y;
            }
            const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
            if (own + total <= WIN_STAGE) {
                uint16_t *at = index_s[warp] + own + incl - n;
                const uint32_t e = r << 12 | lane * 128;
                for (uint64_t x = (uint64_t)b.y << 32 | b.x; x; x &= x - 1) *at++ = (uint16_t)(e + __ffsll(x) - 1);
                for (uint64_t x = (uint64_t)b.w << 32 | b.z; x; x &= x - 1) *at++ = (uint16_t)(e + 64 + __ffsll(x) - 1);
            }
            own += total;
        }
        if (!EMIT) {
            const uint32_t sum = __reduce_add_sync(0xffffffffu, own);
            if (lane == 0 && sum) atomicAdd(totals + counted, (unsigned long long)sum);
        }
    }
    if (!EMIT) return;
    if (lane == 0) sum_s[warp] = own;
    __syncthreads();
    if (warp == 0) {
        const uint32_t all = __reduce_add_sync(0xffffffffu, lane < WIN_WARPS ? sum_s[lane] : 0u);
        const uint64_t before = look_back(o.state, o.stuck, o.polls, tile, all, lane);
        if (lane == 0) {
            before_s = before;
            if (tile + 1 == o.ntiles) o.starts[ndesc] = before + all;
        }
    }
    const bool staged = own <= WIN_STAGE;
    if (staged)
        for (uint32_t i = lane; i < own; i += 32) {     // the wheel loads overlap the look-back
            const uint32_t e = index_s[warp][i];
            const auto &u = unit_s[warp][e >> 12];
            value_s[warp][i] = u.kbase + __ldg(u.wheel + (e & 0xfffu));
        }
    __syncthreads();
    uint64_t at = before_s;                             // values before the warp's
    for (uint32_t k = 0; k < warp; ++k) at += sum_s[k];
    if (lane < mine) {
        const auto &u = unit_s[warp][lane];
        if (u0 + lane == desc[u.win].unit_base) o.starts[u.win] = at + u.before;
    }
    if (staged) {
        for (uint32_t i = lane; i < own; i += 32) {
            const uint64_t pos = at + i + unit_s[warp][index_s[warp][i] >> 12].delta;
            if (pos < o.cap) o.out[pos] = value_s[warp][i];
        }
    } else if (mine) {
        UnitWalk walk(desc, ndesc, foci, u0, lane);
        for (uint32_t r = 0; r < mine; ++r) {
            if (r) walk.step();
            uint32_t w;
            const uint4 b = walk.words(w);
            const auto &u = unit_s[warp][r];
            uint64_t pos = at + u.before + u.delta;
            for (uint32_t k = 0; k < 128; ++k) {        // word k of the unit: lane k / 4, component k % 4
                const uint32_t own_word = (k & 2) ? (k & 1) ? b.w : b.z : (k & 1) ? b.y : b.x;
                const uint32_t word = __shfl_sync(0xffffffffu, own_word, k >> 2);
                if (word >> lane & 1) {
                    const uint64_t slot = pos + __popc(word & ((1u << lane) - 1));
                    if (slot < o.cap) o.out[slot] = u.kbase + __ldg(u.wheel + k * 32 + lane);
                }
                pos += __popc(word);
            }
        }
    }
}

// 128-bit product of 64-bit counts, host side.
void mul_acc(uint64_t &lo, uint64_t &hi, uint64_t f) {
    unsigned __int128 v = ((unsigned __int128)hi << 64 | lo) * f;
    lo = (uint64_t)v;
    hi = (uint64_t)(v >> 64);
}

uint64_t gcd64(uint64_t a, uint64_t b) {
    while (b) {
        uint64_t t = a % b;
        a = b;
        b = t;
    }
    return a;
}

struct Ring {
    uint32_t q, n;
    std::vector<uint32_t> res;
};

int focus_tables(pc_ctx *ctx, pc_focus *f, const std::vector<Ring> &rings, uint32_t nS, uint64_t base_steps);

}  // namespace

extern "C" int pc_focus_create(pc_ctx *ctx, uint64_t M, uint32_t nrings, const uint32_t *q, const uint32_t *counts,
                               const uint32_t *residues, uint64_t table_budget, pc_focus **out) {
    *out = nullptr;
    if (M == 0 || M >= (UINT64_C(1) << 63) || nrings > 16) return pc_fail(ctx, PC_INVALID, "invalid focus modulus");
    auto t_start = std::chrono::steady_clock::now();
    if (!table_budget) table_budget = UINT64_C(256) << 20;
    std::vector<Ring> rings;
    uint64_t prodq = 1, off = 0;
    for (uint32_t k = 0; k < nrings; ++k) {
        Ring r{q[k], counts[k], std::vector<uint32_t>(residues + off, residues + off + counts[k])};
        off += counts[k];
        if (r.q < 2 || r.q > 65535 || r.n == 0 || r.n > r.q) return pc_fail(ctx, PC_INVALID, "invalid ring");
        for (uint32_t a : r.res)
            if (a >= r.q) return pc_fail(ctx, PC_INVALID, "ring residue out of range");
        if (M % r.q || gcd64(M / r.q, r.q) != 1) return pc_fail(ctx, PC_INVALID, "ring moduli must be coprime factors of M");
        prodq *= r.q;
        rings.push_back(std::move(r));
    }
    if (prodq != M) return pc_fail(ctx, PC_INVALID, "ring moduli do not multiply to M");
    std::sort(rings.begin(), rings.end(), [](const Ring &a, const Ring &b) { return a.q < b.q; });

    pc_focus *f = new pc_focus();
    f->M = M;
    f->count_lo = 1;
    for (auto &r : rings) mul_acc(f->count_lo, f->count_hi, r.n);
    f->density = 1;
    for (auto &r : rings) f->density *= (double)r.n / r.q;
    // Choose the T rings: the fewest largest rings whose removal makes the sieve over M1 and
    // the tables fit; among the feasible, the smallest table budget use wins ties.
    uint32_t chosen = UINT32_MAX;
    uint64_t tables_bytes = 0;
    for (uint32_t nT = 0; nT <= std::min<uint32_t>(PC_MAX_WHEEL_T, nrings); ++nT) {
        uint64_t M1 = M, count1_lo = f->count_lo, count1_hi = f->count_hi, rowsum = 0;
        for (uint32_t k = nrings - nT; k < nrings; ++k) {
            M1 /= rings[k].q;
            rowsum += rings[k].q;
            unsigned __int128 c = ((unsigned __int128)count1_hi << 64 | count1_lo) / rings[k].n;
            count1_lo = (uint64_t)c;
            count1_hi = (uint64_t)(c >> 64);
        }
        if (count1_hi || M1 > (UINT64_C(1) << 36)) continue;
        uint64_t words1 = (count1_lo + 31) / 32;
        uint64_t bytes = count1_lo * 8 + rowsum * words1 * 4;
        if (bytes <= table_budget) {
            chosen = nT;
            tables_bytes = bytes;
            break;
        }
    }
    if (chosen == UINT32_MAX) {
        delete f;
        return pc_fail(ctx, PC_INVALID, "focus wheel does not fit the table budget");
    }
    f->nT = chosen;
    const uint32_t nS = nrings - chosen;
    int rc = focus_tables(ctx, f, rings, nS, BASE_STEPS);
    // tables that fit the memory cap, but not with the scratch of their making: the whole wheel comes from the host
    for (bool again = rc == PC_NOMEM; rc; again = false) {
        pc_release(ctx, f->W1, f->W1_bytes);
        pc_release(ctx, f->rows, f->rows_bytes);
        f->W1 = nullptr;
        f->rows = nullptr;
        if (!again || ctx->in_use + tables_bytes > ctx->cap) {
            delete f;
            return rc;
        }
        rc = focus_tables(ctx, f, rings, nS, UINT64_MAX);
    }
    f->build_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_start).count();
    *out = f;
    return PC_OK;
}

uint64_t pc_focus_modulus(const pc_focus *f) { return f->M; }

extern "C" int pc_focus_free(pc_ctx *ctx, pc_focus *f) {
    if (!f) return PC_OK;
    pc_release(ctx, f->W1, f->W1_bytes);
    pc_release(ctx, f->rows, f->rows_bytes);
    delete f;
    return PC_OK;
}

extern "C" int pc_focus_info(const pc_focus *f, uint64_t *info) {
    info[0] = f->M;
    info[1] = f->M1;
    info[2] = f->count1;
    info[3] = f->nT;
    info[4] = f->W1_bytes + f->rows_bytes;
    info[5] = f->count_lo;
    info[6] = f->count_hi;
    info[7] = (uint64_t)f->build_ms;
    return PC_OK;
}

namespace {

// Host plan of the window [low, high) of focus f: period and wheel-index range, units per part.
int plan_window(pc_ctx *ctx, const pc_focus *f, uint64_t low, uint64_t high, WindowPlan &p) {
    p = WindowPlan{};
    if (high < low) return pc_fail(ctx, PC_INVALID, "invalid bounded focus window");
    if (high == low) return PC_OK;
    if ((high - 1) / f->M - low / f->M + 1 > 4096) return pc_fail(ctx, PC_OVERFLOW, "focus window exceeds bounded period count");
    p.K0 = low / f->M1;
    p.K1 = (high - 1) / f->M1;
    // samples below x: the first entry >= x lies in the block of the last of them, or is its end
    auto samples_below = [&](uint64_t x) -> uint64_t {
        if (x == 0 || x >= f->M1) return x ? (f->count1 + SAMPLE - 1) / SAMPLE : 0;
        return std::lower_bound(f->sample.begin(), f->sample.end(), x) - f->sample.begin();
    };
    p.rem_lo = low - p.K0 * f->M1;
    p.rem_hi = high - p.K1 * f->M1;
    const uint64_t below_lo = samples_below(p.rem_lo);
    p.j_lo = below_lo ? (below_lo - 1) * SAMPLE : 0;
    p.j_hi = std::min(samples_below(p.rem_hi) * SAMPLE, f->count1);
    if (p.K0 == p.K1) {
        p.wa0 = p.j_lo / 32;
        p.wb0 = std::max(p.wa0, (p.j_hi + 31) / 32);
        p.wa1 = p.wb1 = 0;
    } else {
        p.wa0 = p.j_lo / 32;
        p.wb0 = f->words1;
        p.wa1 = 0;
        p.wb1 = (p.j_hi + 31) / 32;
    }
    const uint64_t mid_periods = p.K1 > p.K0 + 1 ? p.K1 - p.K0 - 1 : 0;
    auto units = [&](uint64_t words) {
        p.units_first = (p.wb0 - p.wa0 + words - 1) / words;
        p.units_mid = (f->words1 + words - 1) / words;
        p.units_last = p.K1 > p.K0 ? (p.wb1 - p.wa1 + words - 1) / words : 0;
        return p.units_first + mid_periods * p.units_mid + p.units_last;
    };
    p.chunks = units(32);
    if (p.chunks >= (UINT64_C(1) << 31)) return pc_fail(ctx, PC_OVERFLOW, "focus window too long");
    p.wa0 &= ~UINT64_C(3);             // a unit starts on a 16-byte boundary of the rows
    p.units = units(WIN_WORDS);
    return PC_OK;
}

FocusDev focus_dev(const pc_focus *f) {
    FocusDev d{};
    d.W1 = f->W1;
    d.rows = f->rows;
    d.M1 = f->M1;
    d.count1 = f->count1;
    d.words1 = f->words1;
    d.stride = f->stride;
    d.nT = f->nT;
    for (uint32_t t = 0; t < f->nT; ++t) {
        d.t_m1mod[t] = f->t_m1mod[t];
        d.t_row0[t] = f->t_row0[t];
        d.tmq[t] = make_modq(f->tq[t]);
    }
    return d;
}

}  // namespace

namespace {

// Units per warp: enough tiles for four CTAs per SM, then as many units as keep a warp's values well inside
// its stage (per_unit: expected values of the densest focus's unit), so that there are few tiles to look
// back over and a window's lookup and a period's rows serve several units.
uint32_t win_rounds(const pc_ctx *ctx, uint64_t units, double per_unit) {
    const double most = std::min<double>(WIN_ROUNDS, 0.75 * WIN_STAGE / std::max(per_unit, 1.0));
    return (uint32_t)std::max(1.0, std::min(most, (double)(units / ((uint64_t)ctx->sm_count * 4 * WIN_WARPS))));
}

uint64_t win_tiles(const WinBatch &wb) {
    const uint64_t per = (uint64_t)WIN_WARPS * wb.rounds;
    return (wb.units + per - 1) / per;
}

// Plans of n windows, their descriptors and the foci on the device.
int winbatch_describe(pc_ctx *ctx, Scratch &hold, const pc_focus *const *focus, const uint64_t *low, const uint64_t *high,
                      uint32_t n, WinBatch &wb) {
    wb = WinBatch{};
    wb.n = n;
    std::vector<WinDesc> desc(n);
    std::vector<FocusDev> foci;
    std::vector<const pc_focus *> seen;
    uint64_t chunks = 0;
    double per_unit = 0;
    wb.has.resize(n);
    for (uint32_t i = 0; i < n; ++i) {
        int rc = plan_window(ctx, focus[i], low[i], high[i], desc[i].plan);
        if (rc) return rc;
        desc[i].unit_base = wb.units;
        wb.has[i] = desc[i].plan.units != 0;
        wb.units += desc[i].plan.units;
        chunks += desc[i].plan.chunks;
        uint32_t k = 0;
        while (k < seen.size() && seen[k] != focus[i]) ++k;
        if (k == seen.size()) {
            seen.push_back(focus[i]);
            foci.push_back(focus_dev(focus[i]));
            per_unit = std::max(per_unit, focus[i]->density * (double)focus[i]->M1 / (double)focus[i]->count1 * 32 * WIN_WORDS);
        }
        desc[i].focus = k;
    }
    if (chunks >= (UINT64_C(1) << 34)) return pc_fail(ctx, PC_OVERFLOW, "focus windows too long");
    wb.rounds = win_rounds(ctx, wb.units, per_unit);
    // the descriptors, then the foci: parameters of the launch, or one upload
    const uint64_t at = (n * sizeof(WinDesc) + 15) & ~UINT64_C(15), bytes = at + foci.size() * sizeof(FocusDev);
    wb.staged.resize(bytes);
    memcpy(wb.staged.data(), desc.data(), n * sizeof(WinDesc));
    memcpy(wb.staged.data() + at, foci.data(), foci.size() * sizeof(FocusDev));
    // ticket, tile states, starts (one per window and the total), the stuck flag
    int rc = hold.get(&wb.d_scan, 1 + win_tiles(wb) + n + 2);
    if (rc) return rc;
    wb.d_starts = wb.d_scan + 1 + win_tiles(wb);
    wb.d_stuck = wb.d_starts + n + 1;
    if (n <= WIN_FEW) return PC_OK;
    unsigned char *d = nullptr;
    rc = hold.get(&d, bytes);
    if (rc) return rc;
    wb.d_desc = d;
    wb.d_foci = d + at;
    PC_CHECK(ctx, pc_copy(ctx, d, wb.staged.data(), bytes, cudaMemcpyHostToDevice));
    return PC_OK;
}

// The pass over all windows' units; a few windows' descriptors go with it.
template <bool EMIT>
int windows_launch(pc_ctx *ctx, const WinBatch &wb, uint64_t *totals, const WinOut &o) {
    WinFew few{};
    if (wb.n <= WIN_FEW) {
        const uint64_t at = (wb.n * sizeof(WinDesc) + 15) & ~UINT64_C(15);
        memcpy(few.desc, wb.staged.data(), wb.n * sizeof(WinDesc));
        memcpy(few.foci, wb.staged.data() + at, wb.staged.size() - at);
    }
    (wb.n <= WIN_FEW ? k_windows<EMIT, true> : k_windows<EMIT, false>)<<<(unsigned)win_tiles(wb), WT, 0, ctx->stream>>>(
        (const WinDesc *)wb.d_desc, wb.n, (const FocusDev *)wb.d_foci, wb.units, wb.rounds, (unsigned long long *)totals, o, few);
    PC_LAUNCHED(ctx, "windows");
    return PC_OK;
}

}  // namespace

// Emits every window's values (out_cap entries of out).  Nothing is allocated and nothing waits for the
// device, so the pass can be recorded into a CUDA graph.
int winbatch_emit(pc_ctx *ctx, const WinBatch &wb, uint64_t *out, uint64_t out_cap) {
    if (!wb.units) return PC_OK;
    const uint64_t tiles = win_tiles(wb);
    PC_CHECK(ctx, cudaMemsetAsync(wb.d_scan, 0, (1 + tiles + wb.n + 2) * 8, ctx->stream));
    WinOut o{};
    o.ticket = (unsigned long long *)wb.d_scan;
    o.state = o.ticket + 1;
    o.starts = wb.d_starts;
    o.stuck = wb.d_stuck;
    o.delta = wb.d_delta;
    o.out = out;
    o.cap = out_cap;
    o.ntiles = tiles;
    o.polls = ctx->polls;
    return windows_launch<true>(ctx, wb, nullptr, o);
}

namespace {

// Bitset rows of `rings` over the wheel f->W1 (count1 entries), into f->rows: total_rows x stride words.
int wheel_rows(pc_ctx *ctx, pc_focus *f, const Ring *rings, uint32_t n, const uint32_t *d_pat, const uint32_t *off) {
    RowRings rr{};
    for (uint32_t t = 0; t < n; ++t) {
        rr.q[t] = rings[t].q;
        rr.off[t] = off[t];
        rr.row0[t] = f->t_row0[t];
        rr.mq[t] = make_modq(rings[t].q);
    }
    const uint64_t threads = f->stride / 4 * 32;
    k_wheel_rows<<<dim3((unsigned)((threads + WT - 1) / WT), n), WT, 0, ctx->stream>>>(f->W1, f->count1, d_pat, rr, f->rows,
                                                                                     f->stride);
    PC_LAUNCHED(ctx, "wheel rows");
    return PC_OK;
}

// The T rings of f are rings[0..n): moduli, periods mod each, row places.
void set_rings(pc_focus *f, const Ring *rings, uint32_t n) {
    f->nT = n;
    f->total_rows = 0;
    for (uint32_t t = 0; t < n; ++t) {
        f->tq[t] = rings[t].q;
        f->t_m1mod[t] = (uint32_t)(f->M1 % f->tq[t]);
        f->t_row0[t] = f->total_rows;
        f->total_rows += f->tq[t];
    }
    f->words1 = (f->count1 + 31) / 32;
    f->stride = (f->words1 + 3) & ~UINT64_C(3);
    f->rows_bytes = std::max<uint64_t>(16, (uint64_t)f->total_rows * f->stride * 4);
}

// The wheel W1 over the rings [0, nS) and the bitset rows of the rest.  The wheel of the smallest rings is
// enumerated on the host (period by period, so in order; a few thousand entries).  Then up to six rings
// at a time: the sorted values of one whole period of the larger modulus are a window of the smaller wheel
// with those rings as bitset rows, written by k_windows like any other.  That tests 32 candidates of the
// smaller wheel per word and ring, where a bit sieve walks all M1 positions of [0, M1) (the two foci of a (7, 6)
// split: 0.33 and 0.48 ms a pass, two passes -> 26 and 24 us).  The host keeps one wheel entry in 128 for planning, not
// the whole wheel (0.27 and 0.82 ms of copies).  `base_steps`: most candidates of a ring's step on the host.
int focus_tables(pc_ctx *ctx, pc_focus *f, const std::vector<Ring> &rings, uint32_t nS, uint64_t base_steps) {
    Scratch hold(ctx);
    std::vector<std::vector<char>> ok(rings.size());
    for (size_t k = 0; k < rings.size(); ++k) {
        ok[k].assign(rings[k].q, 0);
        for (uint32_t a : rings[k].res) ok[k][a] = 1;
    }
    std::vector<uint64_t> base(1, 0), next;
    uint64_t M = 1, expect = 1;
    uint32_t k = 0;
    for (; k < nS && base.size() * rings[k].q <= base_steps; ++k) {
        const uint32_t q = rings[k].q;
        next.clear();
        for (uint32_t period = 0; period < q; ++period)
            for (uint64_t w : base)
                if (ok[k][(period * M + w) % q]) next.push_back(period * M + w);
        base.swap(next);
        M *= q;
        expect *= rings[k].n;
    }
    if (base.size() != expect) return pc_fail(ctx, PC_ARITHMETIC, "wheel size disagrees with the ring counts");
    // patterns of the remaining rings: R repeated, so that any 32 bits from an offset below q are one funnel shift
    std::vector<uint32_t> pat, off(rings.size(), 0);
    for (size_t r = k; r < rings.size(); ++r) {
        off[r] = (uint32_t)pat.size();
        const uint32_t nbits = 2 * rings[r].q + 64;
        std::vector<uint32_t> words((nbits + 31) / 32 + 1, 0);
        for (uint32_t b = 0; b < nbits; ++b)
            if (ok[r][b % rings[r].q]) words[b / 32] |= 1u << (b % 32);
        pat.insert(pat.end(), words.begin(), words.end());
    }
    uint32_t *d_pat = nullptr;
    int rc = hold.get(&d_pat, pat.size() + 1);
    if (rc) return rc;
    if (!pat.empty()) PC_CHECK(ctx, pc_copy(ctx, d_pat, pat.data(), pat.size() * 4, cudaMemcpyHostToDevice));

    struct Level {                                      // kept until the stream has run it
        pc_focus wheel;
        WinBatch wb;
        uint64_t got[3];                                // start, total, stuck flag
    };
    std::vector<std::unique_ptr<Level>> levels;
    pc_focus small;                                     // the wheel so far
    small.M1 = M;
    small.count1 = base.size();
    uint64_t *d_base = nullptr;
    auto wheel_buffer = [&](uint64_t entries, bool last) {
        if (!last) return hold.get(&d_base, entries);
        f->W1_bytes = std::max<uint64_t>(16, entries * 8);
        const int rc2 = pc_alloc(ctx, (void **)&f->W1, f->W1_bytes);
        d_base = f->W1;
        return rc2;
    };
    rc = wheel_buffer(base.size(), k == nS);
    if (rc) return rc;
    PC_CHECK(ctx, pc_copy(ctx, d_base, base.data(), base.size() * 8, cudaMemcpyHostToDevice));
    small.W1 = d_base;
    while (k < nS) {
        const uint32_t n = std::min<uint32_t>(PC_MAX_WHEEL_T, nS - k);
        levels.emplace_back(new Level());
        Level &l = *levels.back();
        l.wheel = small;
        set_rings(&l.wheel, rings.data() + k, n);
        uint64_t period = small.M1, entries = small.count1;
        double density = (double)small.count1 / (double)small.M1;
        for (uint32_t t = 0; t < n; ++t) {
            period *= rings[k + t].q;
            entries *= rings[k + t].n;
            density *= (double)rings[k + t].n / rings[k + t].q;
        }
        l.wheel.M = period;
        l.wheel.density = density;
        rc = hold.get(&l.wheel.rows, l.wheel.rows_bytes / 4);
        if (!rc) rc = wheel_rows(ctx, &l.wheel, rings.data() + k, n, d_pat, off.data() + k);
        const pc_focus *wheel = &l.wheel;
        const uint64_t low = 0, high = period;
        if (!rc) rc = winbatch_describe(ctx, hold, &wheel, &low, &high, 1, l.wb);
        if (!rc) rc = wheel_buffer(entries, k + n == nS);
        if (!rc) rc = winbatch_emit(ctx, l.wb, d_base, entries);
        if (rc) return rc;
        small.M1 = period;
        small.count1 = entries;
        small.W1 = d_base;
        k += n;
    }
    f->M1 = small.M1;
    f->count1 = small.count1;
    set_rings(f, rings.data() + nS, (uint32_t)rings.size() - nS);
    rc = pc_alloc(ctx, (void **)&f->rows, f->rows_bytes);
    if (!rc && f->nT) rc = wheel_rows(ctx, f, rings.data() + nS, f->nT, d_pat, off.data() + nS);
    if (rc) return rc;
    const uint64_t samples = (f->count1 + SAMPLE - 1) / SAMPLE;
    f->sample.resize(samples);
    if (levels.empty()) {
        for (uint64_t i = 0; i < samples; ++i) f->sample[i] = base[i * SAMPLE];
    } else {
        uint64_t *d_sample = nullptr;
        rc = hold.get(&d_sample, samples);
        if (rc) return rc;
        k_sample<<<(unsigned)((samples + WT - 1) / WT), WT, 0, ctx->stream>>>(f->W1, samples, d_sample);
        PC_LAUNCHED(ctx, "wheel samples");
        PC_CHECK(ctx, pc_copy(ctx, f->sample.data(), d_sample, samples * 8, cudaMemcpyDeviceToHost));
    }
    for (const auto &l : levels)
        PC_CHECK(ctx, pc_copy(ctx, l->got, l->wb.d_scan + 1 + win_tiles(l->wb), sizeof(l->got), cudaMemcpyDeviceToHost));
    PC_CHECK(ctx, cudaStreamSynchronize(ctx->stream));
    for (const auto &l : levels) {
        if (l->got[2]) return pc_fail(ctx, PC_ARITHMETIC, "window pass did not finish");
        uint64_t entries = l->wheel.count1;
        for (uint32_t t = 0; t < l->wheel.nT; ++t)
            for (const Ring &r : rings)
                if (r.q == l->wheel.tq[t]) entries *= r.n;
        if (l->got[1] != entries) return pc_fail(ctx, PC_ARITHMETIC, "wheel size disagrees with the ring counts");
    }
    return PC_OK;
}

}  // namespace

namespace {

// The windows' sizes by a counting pass (d_total: a word per window), into wb.total.
int windows_count(pc_ctx *ctx, WinBatch &wb, uint64_t *d_total) {
    if (!wb.units) return PC_OK;
    PC_CHECK(ctx, cudaMemsetAsync(d_total, 0, wb.n * 8, ctx->stream));
    const int rc = windows_launch<false>(ctx, wb, d_total, WinOut{});
    if (rc) return rc;
    PC_CHECK(ctx, pc_copy(ctx, wb.total.data(), d_total, wb.n * 8, cudaMemcpyDeviceToHost));
    PC_CHECK(ctx, cudaStreamSynchronize(ctx->stream));
    return PC_OK;
}

}  // namespace

// Windows one after another (unpadded) into one buffer allocated here: sized from the foci's densities
// and filled in one pass; a pass whose values outgrow it reruns once with room for all.  Where the memory cap has no
// room for the estimate (1 % and some 1,000 entries above the need), the values are counted first and given exactly their
// room.  A total above `cap` is an overflow (with no buffer, if it was counted), and no more than `cap` entries are allocated.
int winbatch_run(pc_ctx *ctx, Scratch &hold, const pc_focus *const *focus, const uint64_t *low, const uint64_t *high,
                 uint32_t n, uint64_t cap, WinBatch &wb, uint64_t **out, uint64_t *out_bytes, int *launches) {
    *out = nullptr;
    *out_bytes = 0;
    int rc = winbatch_describe(ctx, hold, focus, low, high, n, wb);
    if (rc) return rc;
    wb.total.assign(n, 0);
    wb.base.assign(n, 0);
    double expect = 0;
    uint64_t most = 0;
    for (uint32_t i = 0; i < n; ++i) {
        expect += (double)(high[i] - low[i]) * focus[i]->density;
        most += high[i] - low[i];
    }
    uint64_t room = (uint64_t)(expect * 1.01 + 8 * std::sqrt(expect)) + 1024;
    room = std::min(std::min(room, most), cap);
    // A few words: the kernel writes them to the page-locked stage itself.  With the descriptors as parameters
    // that saves an allocation, an upload and a copy a call.
    std::vector<uint64_t> pageable;
    const StageLoan stage = pc_stage(ctx, (n + 2) * 8);
    uint64_t *got = stage.get();
    const bool direct = got && n <= WIN_FEW;
    if (direct) {
        wb.d_starts = got;
        wb.d_stuck = got + n + 1;
    }
    if (!got) {
        pageable.resize(n + 2);
        got = pageable.data();
    }
    for (int attempt = 0;; ++attempt) {
        *out_bytes = std::max<uint64_t>(16, room * 8);
        rc = pc_alloc(ctx, (void **)out, *out_bytes);
        if (rc == PC_NOMEM && wb.units && !attempt) {
            *out = nullptr;
            rc = windows_count(ctx, wb, wb.d_scan + 1 + win_tiles(wb));    // the words the emitting pass resets
            if (rc) return rc;
            wb.out_len = std::accumulate(wb.total.begin(), wb.total.end(), UINT64_C(0));
            if (wb.out_len > cap) return PC_OK;
            room = wb.out_len;
            continue;
        }
        if (rc) return rc;
        if (!wb.units) return PC_OK;
        if (direct) {
            got[n + 1] = 0;
            ctx->d2h += (n + 2) * 8;
        }
        rc = winbatch_emit(ctx, wb, *out, room);
        if (launches) ++*launches;
        if (!rc && !direct)
            rc = pc_cuda_status(ctx, pc_copy(ctx, got, wb.d_scan + 1 + win_tiles(wb), (n + 2) * 8, cudaMemcpyDeviceToHost),
                                "window totals");
        if (!rc) rc = pc_cuda_status(ctx, cudaStreamSynchronize(ctx->stream), "window totals");
        if (!rc && got[n + 1]) rc = pc_fail(ctx, PC_ARITHMETIC, "window pass did not finish");
        const uint64_t total = got[n];
        if (!rc && (total <= room || total > cap)) {
            uint64_t next = total;
            for (uint32_t i = n; i-- > 0;) {           // a window without units starts where the next one does
                wb.base[i] = wb.has[i] ? got[i] : next;
                wb.total[i] = next - wb.base[i];
                next = wb.base[i];
            }
            wb.out_len = total;
            return PC_OK;
        }
        if (!rc && attempt) rc = pc_fail(ctx, PC_ARITHMETIC, "window size changed between attempts");
        pc_release(ctx, *out, *out_bytes);
        *out = nullptr;
        if (rc) return rc;
        room = total;
    }
}

// The windows' sizes by a counting pass, and their places in a shared output: window i starts on a
// multiple of pad[i].  The emitting passes follow with winbatch_emit.
int winbatch_plan(pc_ctx *ctx, Scratch &hold, const pc_focus *const *focus, const uint64_t *low, const uint64_t *high,
                  const uint64_t *pad, uint32_t n, uint64_t cap, WinBatch &wb) {
    int rc = winbatch_describe(ctx, hold, focus, low, high, n, wb);
    uint64_t *d_total = nullptr;
    if (!rc) rc = hold.get(&d_total, n);
    if (!rc) rc = hold.get(&wb.d_delta, n);
    if (rc) return rc;
    wb.total.assign(n, 0);
    wb.base.assign(n, 0);
    rc = windows_count(ctx, wb, d_total);
    if (rc) return rc;
    wb.delta.assign(n, 0);
    uint64_t before = 0;
    for (uint32_t i = 0; i < n; ++i) {
        if (wb.total[i] > cap) return pc_fail(ctx, PC_OVERFLOW, "focus buffer overflow; tile invalid");
        const uint64_t pd = pad[i] ? pad[i] : 1;
        wb.base[i] = (wb.out_len + pd - 1) / pd * pd;
        wb.out_len = wb.base[i] + wb.total[i];
        wb.delta[i] = wb.base[i] - before;
        before += wb.total[i];
    }
    PC_CHECK(ctx, pc_copy(ctx, wb.d_delta, wb.delta.data(), n * 8, cudaMemcpyHostToDevice));
    return PC_OK;
}

extern "C" int pc_focus_window(pc_ctx *ctx, const pc_focus *f, uint64_t low, uint64_t high, uint64_t cap,
                               pc_buf **out, uint64_t *count) {
    *out = nullptr;
    *count = 0;
    if (high < low) return pc_fail(ctx, PC_INVALID, "invalid bounded focus window");
    Scratch hold(ctx);
    WinBatch wb;
    uint64_t *d = nullptr, bytes = 0;
    int rc = winbatch_run(ctx, hold, &f, &low, &high, 1, cap, wb, &d, &bytes, nullptr);
    if (!rc) *count = wb.out_len;
    if (!rc && wb.out_len > cap) rc = pc_fail(ctx, PC_OVERFLOW, "focus buffer overflow; tile invalid");
    if (rc) {
        pc_release(ctx, d, bytes);
        return rc;
    }
    pc_buf *b = new pc_buf();
    b->d = d;
    b->n = wb.out_len;
    b->bytes = bytes;
    *out = b;
    return PC_OK;
}
