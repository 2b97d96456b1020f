// Shared device/host definitions of libpcube (sm_100a).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <string>
#include <vector>
#include "../../include/pcube.h"
#include "stage.cuh"

#define PC_MAX_BITSET 8        // residual filters intersected as bitsets
#define PC_MAX_RES 1024        // residual filters per (p, A, B)
#define PC_MAX_WHEEL_T 6       // focus rings handled as wheel bitset rows
#define PC_MAX_CHEAP 4         // residual filters tested per survivor from u and v residues

// ------------------------------------------------------------------------------------------
// context, errors, memory accounting

struct pc_ctx {
    int device = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev[8] = {};
    cudaEvent_t marks[8] = {};
    uint64_t cap = 0, in_use = 0, peak = 0;
    uint64_t h2d = 0, d2h = 0;       // bytes the library has copied to and from the host
    int sm_count = 0, cc_major = 0, cc_minor = 0;
    uint32_t polls = 1u << 22;       // of one wait between the tiles of a pass before it gives up
    StageBuffer stage;               // PC_STAGE_BYTES of page-locked memory for results
    char name[256] = {};
    std::string err;
};

struct pc_buf {
    uint64_t *d = nullptr;
    uint64_t n = 0;
    uint64_t bytes = 0;
};

int pc_fail(pc_ctx *ctx, int code, const std::string &msg);
int pc_cuda_fail(pc_ctx *ctx, cudaError_t e, const char *what);
constexpr uint64_t PC_STAGE_BYTES = UINT64_C(4) << 20;   // a lease's counters and envelopes: 3.8 MB
// The context's page-locked stage for as long as the loan lasts; none when `bytes` do not fit it, it cannot be had or
// another call has it.  A loan ends after the stream has finished all that writes to the stage.
StageLoan pc_stage(pc_ctx *ctx, uint64_t bytes);
int pc_alloc(pc_ctx *ctx, void **ptr, uint64_t bytes);
void pc_release(pc_ctx *ctx, void *ptr, uint64_t bytes);

#define PC_CHECK(ctx, call)                                                   \
    do {                                                                      \
        cudaError_t e_ = (call);                                              \
        if (e_ != cudaSuccess) return pc_cuda_fail((ctx), e_, #call);         \
    } while (0)

// An asynchronous copy on the context's stream, counted in ctx->h2d / ctx->d2h.
inline cudaError_t pc_copy(pc_ctx *ctx, void *dst, const void *src, size_t bytes, cudaMemcpyKind kind) {
    if (kind == cudaMemcpyHostToDevice) ctx->h2d += bytes;
    else if (kind == cudaMemcpyDeviceToHost) ctx->d2h += bytes;
    return cudaMemcpyAsync(dst, src, bytes, kind, ctx->stream);
}

inline int pc_cuda_status(pc_ctx *ctx, cudaError_t e, const char *what) {
    return e == cudaSuccess ? PC_OK : pc_cuda_fail(ctx, e, what);
}

#define PC_LAUNCHED(ctx, what)                                                \
    do {                                                                      \
        cudaError_t e_ = cudaGetLastError();                                  \
        if (e_ != cudaSuccess) return pc_cuda_fail((ctx), e_, what);          \
    } while (0)

// RAII holder for device scratch owned by one call.
struct Scratch {
    pc_ctx *ctx;
    std::vector<std::pair<void *, uint64_t>> items;
    explicit Scratch(pc_ctx *c) : ctx(c) {}
    ~Scratch() {
        for (auto &it : items) pc_release(ctx, it.first, it.second);
    }
    template <class T>
    int get(T **p, uint64_t count) {
        uint64_t bytes = count * sizeof(T);
        if (bytes == 0) bytes = 16;
        void *q = nullptr;
        int rc = pc_alloc(ctx, &q, bytes);
        if (rc) return rc;
        items.emplace_back(q, bytes);
        *p = (T *)q;
        return PC_OK;
    }
};

// Several device arrays in one allocation, each 256-byte aligned, in the order added.
struct Carve {
    std::vector<std::pair<void **, uint64_t>> parts;     // pointer to set, byte offset
    uint64_t bytes = 0;
    template <class T>
    void add(T **p, uint64_t count) {
        parts.emplace_back((void **)p, bytes);
        bytes = (bytes + count * sizeof(T) + 255) & ~UINT64_C(255);
    }
    int get(Scratch &s) {
        unsigned char *base = nullptr;
        const int rc = s.get(&base, bytes);
        if (!rc)
            for (auto &p : parts) *p.first = base + p.second;
        return rc;
    }
};

__host__ __device__ __forceinline__ uint64_t umin64(uint64_t a, uint64_t b) { return a < b ? a : b; }
__host__ __device__ __forceinline__ uint64_t umax64(uint64_t a, uint64_t b) { return a > b ? a : b; }
__host__ __device__ __forceinline__ int64_t imin64(int64_t a, int64_t b) { return a < b ? a : b; }
__host__ __device__ __forceinline__ int64_t imax64(int64_t a, int64_t b) { return a > b ? a : b; }

// ------------------------------------------------------------------------------------------
// 128-bit unsigned arithmetic in two 64-bit limbs (add.cc/addc and sub.cc/subc carry chains)

struct u128 {
    uint64_t lo, hi;
};

__device__ __forceinline__ u128 mul_wide(uint64_t a, uint64_t b) {
    u128 r;
    r.lo = a * b;
    r.hi = __umul64hi(a, b);
    return r;
}

__device__ __forceinline__ u128 add128(u128 a, u128 b) {
    u128 r;
    asm("add.cc.u64 %0, %2, %4;\n\taddc.u64 %1, %3, %5;"
        : "=l"(r.lo), "=l"(r.hi)
        : "l"(a.lo), "l"(a.hi), "l"(b.lo), "l"(b.hi));
    return r;
}

__device__ __forceinline__ u128 sub128(u128 a, u128 b) {
    u128 r;
    asm("sub.cc.u64 %0, %2, %4;\n\tsubc.u64 %1, %3, %5;"
        : "=l"(r.lo), "=l"(r.hi)
        : "l"(a.lo), "l"(a.hi), "l"(b.lo), "l"(b.hi));
    return r;
}

__device__ __forceinline__ bool less128(u128 a, u128 b) {
    return a.hi < b.hi || (a.hi == b.hi && a.lo < b.lo);
}

// ------------------------------------------------------------------------------------------
// Remainders by small odd or even moduli q < 2^16 without a hardware divide.
//
// fastmod32: Lemire, Kaser and Kurz, "Faster Remainder by Direct Computation" (2019): with
// c = floor((2^64 - 1) / q) + 1, x mod q = floor(((c * x) mod 2^64) * q / 2^64) for every 32-bit x.
//
// A 128-bit value is folded first: with 16-bit limbs h_k and r_k = 2^(16k) mod q,
// sum h_k r_k < 8 * 2^16 * 2^16 = 2^35 when q < 2^16; limbs are folded in two halves so each
// partial sum stays below 2^32 for q < 2^13 (residual primes are far smaller).

struct ModQ {
    uint32_t q;
    uint32_t r16[7];   // 2^(16k) mod q, k = 1..7
    uint64_t c;        // fastmod constant
};

__host__ __device__ __forceinline__ uint64_t fastmod_constant(uint32_t q) {
    return UINT64_C(0xFFFFFFFFFFFFFFFF) / q + 1;
}

__device__ __forceinline__ uint32_t fastmod32(uint32_t x, uint64_t c, uint32_t q) {
    uint64_t low = c * x;
    return (uint32_t)__umul64hi(low, q);
}

// x mod q for 64-bit x, q < 2^13 (r16 from a ModQ).
__device__ __forceinline__ uint32_t mod64(uint64_t x, const ModQ &m) {
    uint32_t w0 = (uint32_t)x, w1 = (uint32_t)(x >> 32);
    uint32_t t = (w0 & 0xffffu) + (w0 >> 16) * m.r16[0] + (w1 & 0xffffu) * m.r16[1] + (w1 >> 16) * m.r16[2];
    return fastmod32(t, m.c, m.q);
}

// x mod q for 128-bit x, q < 2^13.
__device__ __forceinline__ uint32_t mod128(u128 x, const ModQ &m) {
    uint32_t w0 = (uint32_t)x.lo, w1 = (uint32_t)(x.lo >> 32), w2 = (uint32_t)x.hi, w3 = (uint32_t)(x.hi >> 32);
    uint32_t t0 = (w0 & 0xffffu) + (w0 >> 16) * m.r16[0] + (w1 & 0xffffu) * m.r16[1] + (w1 >> 16) * m.r16[2];
    uint32_t t1 = (w2 & 0xffffu) * m.r16[3] + (w2 >> 16) * m.r16[4] + (w3 & 0xffffu) * m.r16[5] + (w3 >> 16) * m.r16[6];
    return fastmod32(fastmod32(t0, m.c, m.q) + fastmod32(t1, m.c, m.q), m.c, m.q);
}

inline ModQ make_modq(uint32_t q) {
    ModQ m{};
    m.q = q;
    uint64_t r = 1;
    for (int k = 0; k < 7; ++k) {
        r = (r << 16) % q;
        m.r16[k] = (uint32_t)r;
    }
    m.c = fastmod_constant(q);
    return m;
}

// Bits [n, 32) cleared for n in [0, 32]; PTX shl clamps shift counts >= 32 to a zero result.
__device__ __forceinline__ uint32_t low_bits(uint32_t n) {
    uint32_t r;
    asm("shl.b32 %0, %1, %2;" : "=r"(r) : "r"(0xffffffffu), "r"(n));
    return ~r;
}

// ------------------------------------------------------------------------------------------
// 32x32 bit-matrix transpose across a warp: lane l holds row l (bit i = column i) on entry and
// column l on exit.  Five exchange rounds of the off-diagonal blocks, with per-lane constants
// computed once: in exchange round r (block size j = 16 >> r) a lane rotates its partner's word by sh[r]
// (left by j for the lower lane of a pair, right by j for the upper one) and keeps its own bits where
// keep[r] is set, one funnel shift and one bit-select per round.
__device__ __forceinline__ void transpose_consts(uint32_t lane, uint32_t (&sh)[5], uint32_t (&keep)[5]) {
#pragma unroll
    for (int r = 0; r < 5; ++r) {
        const uint32_t j = 16u >> r;
        const uint32_t hm = r == 0 ? 0xffff0000u : r == 1 ? 0xff00ff00u : r == 2 ? 0xf0f0f0f0u
                          : r == 3 ? 0xccccccccu : 0xaaaaaaaau;
        const bool upper = lane & j;
        sh[r] = upper ? 32u - j : j;
        keep[r] = upper ? hm : ~hm;
    }
}

__device__ __forceinline__ uint32_t transpose32c(uint32_t x, const uint32_t (&sh)[5], const uint32_t (&keep)[5]) {
#pragma unroll
    for (int r = 0; r < 5; ++r) {
        const uint32_t p = __shfl_xor_sync(0xffffffffu, x, 16u >> r);
        const uint32_t moved = __funnelshift_l(p, p, sh[r]);
        x = (x & keep[r]) | (moved & ~keep[r]);
    }
    return x;
}

// The same for two matrices at once.  Every exchange moves half of each word, so one shuffle carries the halves
// of both: five shuffles instead of ten, which share the load/store pipe with everything around them.
struct TransposePair {
    uint32_t send[2], a[2], b[2];                        // byte selectors of the rounds of 16 and 8
    uint32_t up[3], keep[3];                             // shift and kept bits of the rounds of 4, 2 and 1
    __device__ __forceinline__ explicit TransposePair(uint32_t lane) {
        const bool u16 = lane & 16, u8 = lane & 8;
        send[0] = u16 ? 0x5410u : 0x7632u, a[0] = u16 ? 0x3254u : 0x5410u, b[0] = u16 ? 0x3276u : 0x7610u;
        send[1] = u8 ? 0x6420u : 0x7531u, a[1] = u8 ? 0x3514u : 0x5240u, b[1] = u8 ? 0x3716u : 0x7260u;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            up[r] = ~lane & (4u >> r);                   // j for the lower lane of a pair, 0 for the upper
            keep[r] = up[r] ? ~half(r) : half(r);
        }
    }
    __device__ static __forceinline__ constexpr uint32_t half(int r) {
        return r == 0 ? 0xf0f0f0f0u : r == 1 ? 0xccccccccu : 0xaaaaaaaau;
    }
    // N pairs v[0], v[1]; v[2], v[3]; ... round by round, so that their shuffles overlap.
    template <int N>
    __device__ __forceinline__ void operator()(uint32_t *v) const {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            uint32_t p[N];
#pragma unroll
            for (int i = 0; i < N; ++i) p[i] = __shfl_xor_sync(0xffffffffu, __byte_perm(v[2 * i], v[2 * i + 1], send[r]), 16u >> r);
#pragma unroll
            for (int i = 0; i < N; ++i) {
                v[2 * i] = __byte_perm(v[2 * i], p[i], a[r]);
                v[2 * i + 1] = __byte_perm(v[2 * i + 1], p[i], b[r]);
            }
        }
#pragma unroll
        for (int r = 0; r < 3; ++r) {                    // the upper lane sends its lower half, the lower lane its upper
            const uint32_t h = half(r), j = 4u >> r, u = up[r], d = j - u;
            uint32_t p[N];
#pragma unroll
            for (int i = 0; i < N; ++i)
                p[i] = __shfl_xor_sync(0xffffffffu, ((v[2 * i] >> u) & ~h) | ((v[2 * i + 1] << d) & h), j);
#pragma unroll
            for (int i = 0; i < N; ++i) {
                v[2 * i] = (v[2 * i] & keep[r]) | ((p[i] << u) & ~keep[r]);
                v[2 * i + 1] = (v[2 * i + 1] & keep[r]) | ((p[i] >> d) & ~keep[r]);
            }
        }
    }
};

// Entries of a sorted range of n for which `below(index)` holds (a prefix of it), by each group of eight lanes of a
// warp for its own range: three bits a step, where a thread alone takes one dependent load per bit.
template <class F>
__device__ __forceinline__ uint64_t group_prefix(uint64_t n, uint32_t lane, F below) {
    const uint32_t part = lane & 7, group = lane & 24;
    uint64_t lo = 0, len = n;                             // the answer is in [lo, lo + len]
    while (__any_sync(0xffffffffu, len != 0)) {
        const uint64_t step = (len + 7) / 8, at = lo + umin64((part + 1) * step, len) - 1;   // last entry of the part
        bool hit = false;
        if (part * step < len) hit = below(at);
        const uint32_t parts = __popc(__ballot_sync(0xffffffffu, hit) >> group & 0xffu);
        const uint64_t done = umin64(parts * step, len);
        lo += done;
        len = len ? umin64(step - 1, len - done) : 0;
    }
    return lo;
}

// ------------------------------------------------------------------------------------------
// Exclusive prefix over the tiles of one launch (decoupled look-back).  A tile's state is one word:
// value << 2 | 1 (its own sum) or 2 (its own and all before it), zeroed before the launch.
// Values of the tiles before `tile`, by warp 0: it publishes the tile's own sum, then adds the states of
// the 32 tiles before it, and of the 32 before those, until one already holds its whole prefix.  Tiles take
// ascending tickets, so every tile waited for is running or done; a wait that does not end in `polls`
// polls sets *stuck and goes on, and the host refuses the result.
__device__ __forceinline__ uint64_t look_back(volatile unsigned long long *state, uint64_t *stuck, uint32_t polls,
                                              uint64_t tile, uint64_t own, uint32_t lane) {
    if (tile == 0) {
        if (lane == 0) state[0] = own << 2 | 2;
        return 0;
    }
    if (lane == 0) state[tile] = own << 2 | 1;
    uint64_t before = 0;
    for (int64_t at = (int64_t)tile - 1 - lane;; at -= 32) {
        unsigned long long s = at < 0 ? 2 : state[at];
        for (uint32_t spin = 0; __any_sync(0xffffffffu, (s & 3) == 0); ++spin) {
            if (spin == polls) {
                if (lane == 0) *stuck = 1;
                s |= 2;
            } else if ((s & 3) == 0) {
                s = state[at];
            }
        }
        const uint32_t whole = __ballot_sync(0xffffffffu, (s & 3) == 2);
        const uint32_t last = whole ? __ffs(whole) - 1 : 31;
        uint64_t v = lane <= last ? s >> 2 : 0;
#pragma unroll
        for (int d = 16; d; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
        before += v;
        if (whole) break;
    }
    if (lane == 0) state[tile] = (before + own) << 2 | 2;
    return before;
}

// ------------------------------------------------------------------------------------------
// internal host helpers shared across translation units

// Many sorted focus windows generated together by one launch.  winbatch_run writes them one after another
// into a buffer it sizes; winbatch_plan counts them first and gives window i a place that starts on a
// multiple of pad[i] (so a u list can start on a block boundary of the matcher), for winbatch_emit.
struct WinBatch {
    uint32_t n = 0, rounds = 1;
    uint64_t units = 0;
    void *d_desc = nullptr, *d_foci = nullptr;   // null for a few windows: launch parameters
    uint64_t *d_scan = nullptr;      // ticket, tile states, window starts and total, stuck flag
    uint64_t *d_starts = nullptr;    // window starts and total (in d_scan, or where the owner reads them)
    uint64_t *d_stuck = nullptr;     // set by an emitting pass that gave up (in d_scan, or where the owner reads it)
    uint64_t *d_delta = nullptr;     // per window: output position minus values before it (null: 0)
    std::vector<uint64_t> total, base, delta;
    std::vector<char> has;           // windows with any unit
    std::vector<unsigned char> staged;   // descriptors and foci, as uploaded or passed (kept until the copy has run)
    uint64_t out_len = 0;
};
struct pc_focus;
uint64_t pc_focus_modulus(const pc_focus *f);
int winbatch_plan(pc_ctx *ctx, Scratch &hold, const pc_focus *const *focus, const uint64_t *low, const uint64_t *high,
                  const uint64_t *pad, uint32_t n, uint64_t cap, WinBatch &wb);
int winbatch_emit(pc_ctx *ctx, const WinBatch &wb, uint64_t *out, uint64_t out_cap);
int winbatch_run(pc_ctx *ctx, Scratch &hold, const pc_focus *const *focus, const uint64_t *low, const uint64_t *high,
                 uint32_t n, uint64_t cap, WinBatch &wb, uint64_t **out, uint64_t *out_bytes, int *launches);
