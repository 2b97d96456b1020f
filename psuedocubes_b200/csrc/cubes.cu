// Genuine-cube control: the integers a in [first, last] coprime to every prime <= p.
//
// Every such a gives a cube a^3 that is a pseudocube candidate of bound p (it is +-1 mod 9 when
// 3 does not divide a, and a cubic residue and a unit modulo every other prime <= p), so the
// count over the cube roots of (lo, hi] is the number of genuine cubes a correct sieve of (lo, hi]
// must emit.  The reference counts them on the host with a byte-segment sieve
// (review/cube_count.c:12-37) and an odd-only bit sieve (review/cube_count_independent.c:9-34)
// over inclusive root bounds 1 <= first <= last < 2^32, 2 <= p <= 2000.
//
// Device form: a = W k + r with W the product of the primes 2, 3, 5 that are <= p and r one of the residues
// coprime to W, so only 8 of 30 numbers are sieved, one bitmap over k per residue class.  The other
// primes are packed into groups whose product P stays <= 2^16; q | W k + r exactly when
// q | k + r W^-1 (mod q), so one bit pattern per group (bit z set when z shares a factor with P) serves
// every class from the offset (k + r W^-1) mod P.  Patterns are stored past P, so that consecutive words
// starting at any offset below P are read without a wrap; each CTA marks them in its shared memory from
// the primes (a few thousand bits), so only the table of groups (a few KB) comes from the host.
#include "common.cuh"
#include <algorithm>
#include <cstring>
#include <vector>

namespace {

constexpr uint32_t ROOT_GROUP_MAX = 1u << 16;   // largest product of one prime group
constexpr uint32_t ROOT_GROUPS = 304, ROOT_CLASSES = 8;   // 303 primes below 2000
constexpr int ROOT_THREADS = 1024, LIST_THREADS = 512;
constexpr uint32_t LIST_K = LIST_THREADS * 2 / ROOT_CLASSES;   // words of every class in a tile of k_root_list: a thread, two classes
constexpr uint32_t LIST_STAGE = 32 * 32 * ROOT_CLASSES;         // a warp's candidates, 16 bits each while staged

struct __align__(16) RootGroup {
    uint64_t c;                      // fastmod constant of P
    uint32_t P, inv;                 // period; W^-1 mod P
    uint32_t off, words;             // first word of the pattern, its words
    uint32_t pad[2];
};

struct RootPrime {
    uint32_t q, off, bits;           // the prime; its group's pattern: first word, bits
    uint32_t every;                  // bit i set when q | i, i < 32
};

// A prime that k_roots strikes out multiple by multiple.
struct __align__(16) RootStrike {
    uint64_t c;                      // fastmod constant of q
    uint32_t q, inv;                 // the prime; W^-1 mod q
};

// The table in shared memory and its source: groups, primes, then strikes.
struct RootParams {
    uint32_t ngroups, nprimes, nstrikes, W, nclass, table_words;
    uint64_t first, last, k0, nk;    // numbers; k of the first number, k values
    uint32_t cls[ROOT_CLASSES];      // residues coprime to W, ascending
    const uint4 *table;
    __host__ __device__ uint32_t table_bytes() const {
        return ngroups * sizeof(RootGroup) + nprimes * sizeof(RootPrime) + nstrikes * sizeof(RootStrike);
    }
};

// W^-1 mod P = (1 + m P) / W for the m that makes it whole
uint32_t inverse_w(uint64_t P, uint64_t W) {
    uint64_t m = 0;
    while ((1 + m * P) % W) ++m;
    return (uint32_t)((1 + m * P) / W % P);
}

// The groups and their patterns' places; `run` consecutive words are read from any offset below P.  Primes above
// `strike` have no pattern but a RootStrike.
void root_params(RootParams &p, std::vector<unsigned char> &table, uint64_t first, uint64_t last, uint32_t bound, uint32_t run,
                 uint32_t strike) {
    std::vector<char> composite(bound + 1, 0);
    std::vector<uint32_t> primes;
    p.W = 1;
    for (uint32_t q = 2; q <= bound; ++q) {
        if (composite[q]) continue;
        if (q <= 5) p.W *= q;
        else primes.push_back(q);
        for (uint32_t m = q * q; m <= bound; m += q) composite[m] = 1;
    }
    p.nclass = 0;
    for (uint32_t r = 1; r < p.W; ++r)
        if ((p.W % 2 || r % 2) && (p.W % 3 || r % 3) && (p.W % 5 || r % 5)) p.cls[p.nclass++] = r;
    p.first = first;
    p.last = last;
    p.k0 = first / p.W;
    p.nk = last / p.W - p.k0 + 1;
    p.table_words = 0;
    std::vector<RootGroup> groups;
    std::vector<RootPrime> marks;
    std::vector<RootStrike> strikes;
    for (; !primes.empty() && primes.back() > strike; primes.pop_back())
        strikes.push_back(RootStrike{fastmod_constant(primes.back()), primes.back(), inverse_w(primes.back(), p.W)});
    for (size_t i = 0; i < primes.size();) {
        RootGroup g{};
        g.P = 1;
        const size_t i0 = i;
        while (i < primes.size() && (uint64_t)g.P * primes[i] <= ROOT_GROUP_MAX) g.P *= primes[i++];
        g.c = fastmod_constant(g.P);
        g.inv = inverse_w(g.P, p.W);
        g.off = p.table_words;
        g.words = (g.P - 1) / 32 + run + 1;
        p.table_words += g.words;
        for (size_t k = i0; k < i; ++k) {
            RootPrime m{primes[k], g.off, g.words * 32, 0};
            for (uint32_t b = 0; b < 32; b += m.q) m.every |= 1u << b;
            marks.push_back(m);
        }
        groups.push_back(g);
    }
    p.table_words = (p.table_words + 3) & ~3u;
    p.ngroups = (uint32_t)groups.size();
    p.nprimes = (uint32_t)marks.size();
    p.nstrikes = (uint32_t)strikes.size();
    table.resize(p.table_bytes());
    std::copy((const unsigned char *)groups.data(), (const unsigned char *)(groups.data() + groups.size()), table.begin());
    std::copy((const unsigned char *)marks.data(), (const unsigned char *)(marks.data() + marks.size()),
              table.begin() + groups.size() * sizeof(RootGroup));
    std::copy((const unsigned char *)strikes.data(), (const unsigned char *)(strikes.data() + strikes.size()),
              table.end() - strikes.size() * sizeof(RootStrike));
}

// The CTA's table and patterns.  A prime below 32 gives each of its group's words whole (32 lanes
// marking it bit by bit would meet in the same words); larger ones are marked bit by bit.
__device__ const RootGroup *mark_patterns(const RootParams &p, uint4 *smem, uint32_t *&pattern) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5, tw = p.table_bytes() / 16;
    uint4 *zero = smem + tw;
    pattern = (uint32_t *)zero;
    for (uint32_t i = threadIdx.x; i < tw; i += blockDim.x) smem[i] = p.table[i];
    for (uint32_t i = threadIdx.x; i < p.table_words / 4; i += blockDim.x) zero[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    const RootGroup *groups = (const RootGroup *)smem;
    const RootPrime *primes = (const RootPrime *)(groups + p.ngroups);
    for (uint32_t i = warp; i < p.nprimes; i += warps) {
        const RootPrime m = primes[i];
        uint32_t *w = pattern + m.off;
        if (m.q < 32) {
            for (uint32_t z = lane; z < m.bits / 32; z += 32) {
                const uint32_t r = 32 * z % m.q;
                atomicOr(w + z, m.every << (r ? m.q - r : 0));
            }
        } else {
            for (uint32_t z = m.q * lane; z < m.bits; z += 32 * m.q) atomicOr(w + (z >> 5), 1u << (z & 31));
        }
    }
    __syncthreads();
    return groups;
}

// Bits of the 32 k values from k (relative to k0) on that give numbers of [first, last] in class r.
__device__ __forceinline__ uint32_t class_bits(const RootParams &p, uint64_t k, uint32_t r) {
    const uint64_t lo = p.k0 * p.W + r < p.first;                                    // the first k value is too small
    const uint64_t end = p.nk - ((p.k0 + p.nk - 1) * p.W + r > p.last);              // the last one too large
    if (k >= end) return 0;
    uint32_t bits = end - k >= 32 ? 0xffffffffu : low_bits((uint32_t)(end - k));
    if (k < lo) bits &= ~1u;
    return bits;
}

// Counting: a warp owns 32 x RUN consecutive words of one class's bitmap, RUN per lane.  The patterns
// reach 32 x RUN words past P, so the whole warp reads one window without a wrap: its offset and shift are
// warp-uniform, a lane's window for one word shares a pattern word with the next (one shared load, one
// funnel shift and half a three-input OR per group and word), and RUN is odd, so the lanes' loads always
// fall in 32 different banks.  A prime above STRIKE hits a word in eight at most and would have a pattern to
// itself: it is struck out instead, multiple by multiple in the warp's bitmap in shared memory, a lane per prime
// (about one shared OR of a warp per prime where the pattern takes RUN + 1 loads and 1.5 RUN operations).
// Bound: marking the patterns and the first task (19 us for a range of one task per SM), then those loads and ORs, one per
// clock and SM.  4e8 numbers with p = 619: 39 us (all 30 residues and patterns that wrap per lane 201, a pattern for every prime 61,
// primes above 128 struck out 41); all below 2^32 with p = 1999, whose patterns would leave room for 3 words: 2,052 -> 359.
constexpr uint32_t STRIKE = 256;   // the square root of ROOT_GROUP_MAX: no two larger primes share a pattern
template <int RUN>
__global__ void __launch_bounds__(ROOT_THREADS) k_roots(const RootParams p, unsigned long long *__restrict__ total) {
    extern __shared__ uint4 smem[];
    __shared__ uint32_t cls_s[ROOT_CLASSES];
#pragma unroll
    for (uint32_t i = 0; i < ROOT_CLASSES; ++i)
        if (threadIdx.x == i) cls_s[i] = p.cls[i];
    uint32_t *pattern;
    const RootGroup *groups = mark_patterns(p, smem, pattern);
    const RootStrike *strikes = (const RootStrike *)((const RootPrime *)(groups + p.ngroups) + p.nprimes);
    const uint32_t lane = threadIdx.x & 31, warps = ROOT_THREADS / 32;
    uint32_t *struck = pattern + p.table_words + (threadIdx.x >> 5) * (32 * RUN);   // the warp's bitmap
#pragma unroll
    for (int w = 0; w < RUN; ++w) struck[lane * RUN + w] = 0;
    constexpr uint32_t K = 32 * 32 * RUN;                  // k values of one warp task
    const uint64_t tasks = (p.nk + K - 1) / K * p.nclass;
    uint32_t count = 0;
    for (uint64_t task = (threadIdx.x >> 5) * (uint64_t)gridDim.x + blockIdx.x; task < tasks;
         task += (uint64_t)gridDim.x * warps) {            // warp-uniform; consecutive tasks on different SMs
        const uint32_t r = cls_s[task % p.nclass];
        const uint64_t k0 = task / p.nclass * K, k = k0 + lane * (32 * RUN);
        const uint32_t x = (uint32_t)(p.k0 + k0);          // with any group W = 30, so this is below 2^28
        __syncwarp();
        for (uint32_t i = lane; i < p.nstrikes; i += 32) {
            const RootStrike S = strikes[i];
            const uint32_t at = fastmod32(x + r * S.inv, S.c, S.q);   // x + r inv < 2^28 + 30 2^11
            for (uint32_t z = at ? S.q - at : 0; z < K; z += S.q) atomicOr(struck + (z >> 5), 1u << (z & 31));
        }
        uint32_t acc[RUN];
#pragma unroll
        for (int w = 0; w < RUN; ++w) acc[w] = 0;
        const uint32_t *lane_pattern = pattern + lane * RUN;
        for (uint32_t g0 = 0; g0 < p.ngroups; g0 += 32) {  // lane i finds the window of group g0 + i
            const uint32_t n = min(p.ngroups - g0, 32u);
            uint32_t place = 0;                            // pattern word << 5 | shift
            if (lane < n) {
                const RootGroup G = groups[g0 + lane];
                place = G.off * 32 + fastmod32(x + r * G.inv, G.c, G.P);   // x + r inv < 2^28 + 30 2^16
            }
            uint32_t i = 0;
            for (; i + 1 < n; i += 2) {
                const uint32_t sa = __shfl_sync(0xffffffffu, place, i), sb = __shfl_sync(0xffffffffu, place, i + 1);
                const uint32_t *pa = lane_pattern + (sa >> 5), *pb = lane_pattern + (sb >> 5);
                uint32_t la = pa[0], lb = pb[0];
#pragma unroll
                for (int w = 0; w < RUN; ++w) {
                    const uint32_t ha = pa[w + 1], hb = pb[w + 1];
                    acc[w] |= __funnelshift_r(la, ha, sa) | __funnelshift_r(lb, hb, sb);   // by the low five bits
                    la = ha, lb = hb;
                }
            }
            if (i < n) {
                const uint32_t sa = __shfl_sync(0xffffffffu, place, i);
                const uint32_t *pa = lane_pattern + (sa >> 5);
                uint32_t la = pa[0];
#pragma unroll
                for (int w = 0; w < RUN; ++w) {
                    const uint32_t ha = pa[w + 1];
                    acc[w] |= __funnelshift_r(la, ha, sa);
                    la = ha;
                }
            }
        }
        __syncwarp();
#pragma unroll
        for (int w = 0; w < RUN; ++w) {
            acc[w] |= struck[lane * RUN + w];
            struck[lane * RUN + w] = 0;
            count += __popc(~acc[w] & class_bits(p, k + 32 * w, r));
        }
    }
    count = __reduce_add_sync(0xffffffffu, count);
    if (lane == 0 && count) atomicAdd(total, (unsigned long long)count);
}

// Listing (and counting short ranges, which would leave k_roots a few long warps): a tile is LIST_K words of 32
// consecutive k values in every class, a thread sieves one word of two classes.  Then one thread per word takes all
// its classes, so number order is lane order, then k, then class.  The tile's place in
// the list comes from a look-back over the tiles before it (out may be null: count only).  A warp's roots
// are staged in the patterns' space, which nothing reads any more, and stored coalesced.  Bound: latency, of marking the
// patterns and of a thread's way through all groups.  Against a thread per word, 128 of them, sieving all eight classes: a
// list over 1e6 numbers 33 -> 29.5 us (p = 1999: 59.5 -> 52; 2e7 numbers, where every SM has work: 41.5 -> 43.5).
__global__ void __launch_bounds__(LIST_THREADS) k_root_list(const RootParams p,
                                                            unsigned long long *__restrict__ ticket, uint64_t ntiles,
                                                            uint64_t *__restrict__ stuck, uint32_t polls, uint64_t *__restrict__ total,
                                                            uint32_t *__restrict__ out, uint64_t cap) {
    extern __shared__ uint4 smem[];
    __shared__ uint64_t tile_s, before_s;
    __shared__ uint32_t sum_s[LIST_K / 32];
    __shared__ uint32_t acc_s[ROOT_CLASSES][LIST_K];
    __shared__ uint32_t shift_s[ROOT_GROUPS][ROOT_CLASSES / 2];    // r W^-1 mod P of every class, 16 bits each
    __shared__ uint32_t cls_s[ROOT_CLASSES];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) tile_s = atomicAdd(ticket, 1ull);
#pragma unroll
    for (uint32_t i = 0; i < ROOT_CLASSES; ++i)
        if (threadIdx.x == i) cls_s[i] = p.cls[i];
    uint32_t *pattern;
    const RootGroup *groups = mark_patterns(p, smem, pattern);
    for (uint32_t i = threadIdx.x; i < p.ngroups * ROOT_CLASSES; i += LIST_THREADS) {
        const RootGroup &g = groups[i / ROOT_CLASSES];
        ((uint16_t *)shift_s)[i] = (uint16_t)fastmod32(cls_s[i % ROOT_CLASSES] * g.inv, g.c, g.P);
    }
    __syncthreads();
    const uint32_t word = threadIdx.x % LIST_K, two = threadIdx.x / LIST_K;   // `two` is warp-uniform
    const uint64_t tile = tile_s, k = (tile * LIST_K + word) * 32;
    uint32_t both[2] = {};
#pragma unroll 2
    for (uint32_t g = 0; g < p.ngroups; ++g) {                     // with any group there are eight classes
        const RootGroup G = groups[g];
        const uint32_t P = G.P, s0 = fastmod32((uint32_t)(p.k0 + k), G.c, P), shift = shift_s[g][two];
        const uint32_t *pat = pattern + G.off;
#pragma unroll
        for (uint32_t i = 0; i < 2; ++i) {
            uint32_t s = s0 + (shift >> (16 * i) & 0xffffu);
            s -= s >= P ? P : 0;
            both[i] |= __funnelshift_r(pat[s >> 5], pat[(s >> 5) + 1], s & 31);
        }
    }
#pragma unroll
    for (uint32_t i = 0; i < 2; ++i) {
        const uint32_t c = 2 * two + i;
        acc_s[c][word] = c < p.nclass ? ~both[i] & class_bits(p, k, cls_s[c]) : 0u;
    }
    __syncthreads();
    const bool mine = threadIdx.x < LIST_K;                        // warp-uniform
    uint32_t acc[ROOT_CLASSES], n = 0;
#pragma unroll
    for (uint32_t i = 0; i < ROOT_CLASSES; ++i) {
        acc[i] = mine ? acc_s[i][word] : 0u;
        n += __popc(acc[i]);
    }
    uint32_t incl = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= (uint32_t)d) incl += y;
    }
    if (lane == 31 && mine) sum_s[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const uint32_t all = __reduce_add_sync(0xffffffffu, lane < LIST_K / 32 ? sum_s[lane] : 0u);
        const uint64_t before = look_back(ticket + 1, stuck, polls, tile, all, lane);
        if (lane == 0) {
            before_s = before;
            if (tile + 1 == ntiles) *total = before + all;
        }
    }
    if (!out) return;
    uint16_t *stage = (uint16_t *)pattern + warp * LIST_STAGE;
    uint32_t any = 0, slot = incl - n;
#pragma unroll
    for (uint32_t i = 0; i < ROOT_CLASSES; ++i) any |= acc[i];
    for (; any; any &= any - 1) {                                  // k values with a root, ascending
        const uint32_t b = __ffs(any) - 1;
#pragma unroll
        for (uint32_t i = 0; i < ROOT_CLASSES; ++i)
            if (acc[i] >> b & 1) stage[slot++] = (uint16_t)((lane * 32 + b) * ROOT_CLASSES + i);
    }
    __syncthreads();
    if (!mine) return;
    uint64_t at = before_s;
    for (uint32_t w = 0; w < warp; ++w) at += sum_s[w];
    const uint64_t k_warp = p.k0 + k - lane * 32;
    for (uint32_t i = lane; i < sum_s[warp]; i += 32) {
        const uint32_t e = stage[i];
        if (at + i < cap) out[at + i] = (uint32_t)((k_warp + e / ROOT_CLASSES) * p.W) + cls_s[e % ROOT_CLASSES];
    }
}

// The share of all numbers that is coprime to every prime.
double root_density(const RootParams &p, const std::vector<unsigned char> &table) {
    double d = (double)p.nclass / p.W;
    const RootPrime *m = (const RootPrime *)(table.data() + p.ngroups * sizeof(RootGroup));
    for (uint32_t i = 0; i < p.nprimes; ++i) d *= 1.0 - 1.0 / m[i].q;
    return d;
}

// Words per lane of k_roots: patterns and bitmaps take 135 KB of shared memory at p = 619.  Fewer words mean more
// offsets per word; more words, longer tasks that short ranges have too few of (5, 9, 13, 17 words: 4e8 numbers 41.6, 39.5, 38,
// 39.4 us; 6e6 numbers 17, 19, 27, 27 us).
constexpr uint32_t ROOT_RUN = 9;

}  // namespace

extern "C" int pc_cube_roots(pc_ctx *ctx, uint64_t first, uint64_t last, uint32_t p, uint32_t *roots, uint64_t cap,
                             uint64_t *count, double *kernel_ms) {
    if (!ctx || !count) return pc_fail(ctx, PC_INVALID, "null argument");
    if (kernel_ms) *kernel_ms = 0;
    if (first < 1 || last < first || last > UINT32_MAX || p < 2 || p > 2000)
        return pc_fail(ctx, PC_INVALID, "cube roots need 1 <= first <= last < 2^32 and 2 <= p <= 2000");
    const uint64_t n = last - first + 1;
    // counts take k_roots from one warp task per SM on (4e6 numbers): its fixed cost, marking the
    // longer patterns, is then below what the list kernel's three times as many shared loads cost
    const uint64_t W = p < 3 ? 2 : p < 5 ? 6 : 30, classes = p < 3 ? 1 : p < 5 ? 2 : 8, nk = last / W - first / W + 1;
    const bool longer = !roots && (nk + 1024 * ROOT_RUN - 1) / (1024 * ROOT_RUN) * classes >= (uint64_t)ctx->sm_count;
    RootParams rp{};
    std::vector<unsigned char> table;
    root_params(rp, table, first, last, p, longer ? 32 * ROOT_RUN : 1, longer ? STRIKE : UINT32_MAX);
    const uint64_t ntiles = (rp.nk + LIST_K * 32 - 1) / (LIST_K * 32);
    Scratch hold(ctx);
    uint64_t *d_scan = nullptr;                            // total, stuck flag, ticket, tile states
    const uint64_t words = 3 + (longer ? 0 : ntiles);
    uint4 *d_table = nullptr;
    int rc = hold.get(&d_scan, words);
    if (!rc) rc = hold.get(&d_table, std::max<size_t>(1, table.size() / 16));
    if (rc) return rc;
    rp.table = d_table;
    if (!table.empty()) PC_CHECK(ctx, pc_copy(ctx, d_table, table.data(), table.size(), cudaMemcpyHostToDevice));
    auto elapsed = [&](double &ms) {
        float f = 0;
        PC_CHECK(ctx, cudaEventElapsedTime(&f, ctx->ev[0], ctx->ev[1]));
        ms += f;
        return (int)PC_OK;
    };
    // a listing pass is sized by the density; a list that outgrows it (never seen) is written again.  Where the memory cap
    // has no room for the estimate, the first pass only counts.
    uint64_t room = roots ? std::min(std::min(n, cap), (uint64_t)(root_density(rp, table) * n * 1.02) + 4096) : 0;
    double ms = 0;
    uint64_t got[2] = {0, 0};
    for (int attempt = 0;; ++attempt) {
        Scratch list(ctx);
        uint32_t *d_out = nullptr;
        if (roots) rc = list.get(&d_out, std::max<uint64_t>(1, room));
        const bool counting = rc == PC_NOMEM && !attempt;
        if (counting) rc = PC_OK, room = 0;
        if (rc) return rc;
        PC_CHECK(ctx, cudaMemsetAsync(d_scan, 0, words * 8, ctx->stream));
        if (kernel_ms) PC_CHECK(ctx, cudaEventRecord(ctx->ev[0], ctx->stream));
        if (longer) {
            const uint32_t smem = rp.table_bytes() + rp.table_words * 4 + (ROOT_THREADS / 32) * (32 * ROOT_RUN) * 4;
            PC_CHECK(ctx, cudaFuncSetAttribute(k_roots<ROOT_RUN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            k_roots<ROOT_RUN><<<ctx->sm_count, ROOT_THREADS, smem, ctx->stream>>>(rp, (unsigned long long *)d_scan);
            PC_LAUNCHED(ctx, "cube roots count");
        } else {
            const size_t smem = rp.table_bytes() + std::max(rp.table_words * 4, LIST_K / 32 * LIST_STAGE * 2);
            PC_CHECK(ctx, cudaFuncSetAttribute(k_root_list, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            k_root_list<<<(unsigned)ntiles, LIST_THREADS, smem, ctx->stream>>>(
                rp, (unsigned long long *)d_scan + 2, ntiles, d_scan + 1, ctx->polls, d_scan, d_out, room);
            PC_LAUNCHED(ctx, "cube root list");
        }
        if (kernel_ms) PC_CHECK(ctx, cudaEventRecord(ctx->ev[1], ctx->stream));
        // the sums, and a list with them, through the page-locked stage: one wait, and no copy in pieces to pageable
        // memory
        const StageLoan loan = pc_stage(ctx, sizeof(got) + room * 4);
        uint64_t *stage = loan.get();
        PC_CHECK(ctx, pc_copy(ctx, stage ? stage : got, d_scan, sizeof(got), cudaMemcpyDeviceToHost));
        if (stage && room) PC_CHECK(ctx, pc_copy(ctx, stage + 2, d_out, room * 4, cudaMemcpyDeviceToHost));
        PC_CHECK(ctx, cudaStreamSynchronize(ctx->stream));
        if (stage) memcpy(got, stage, sizeof(got));
        if (kernel_ms) {
            if ((rc = elapsed(ms))) return rc;
            *kernel_ms = ms;
        }
        if (got[1]) return pc_fail(ctx, PC_ARITHMETIC, "cube root pass did not finish");
        *count = got[0];
        if (!roots) return PC_OK;
        if (got[0] > cap) return pc_fail(ctx, PC_OVERFLOW, "more cube roots than the output capacity");
        if (got[0] <= room) {
            if (!got[0]) return PC_OK;
            if (stage) {
                memcpy(roots, stage + 2, got[0] * 4);
                return PC_OK;
            }
            PC_CHECK(ctx, pc_copy(ctx, roots, d_out, got[0] * 4, cudaMemcpyDeviceToHost));
            PC_CHECK(ctx, cudaStreamSynchronize(ctx->stream));
            return PC_OK;
        }
        if (attempt) return pc_fail(ctx, PC_ARITHMETIC, "cube root count changed between attempts");   // counted or written before
        room = got[0];
    }
}
