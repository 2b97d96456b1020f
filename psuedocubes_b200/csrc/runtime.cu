// Context, memory accounting, device buffers, the page-locked stage, sorted searches and the limb self-test.
#include "common.cuh"
#include <algorithm>
#include <cstring>

int pc_fail(pc_ctx *ctx, int code, const std::string &msg) {
    if (ctx) ctx->err = msg;
    return code;
}

int pc_cuda_fail(pc_ctx *ctx, cudaError_t e, const char *what) {
    if (ctx) ctx->err = std::string(what) + ": " + cudaGetErrorString(e);
    return PC_CUDA;
}

int pc_alloc(pc_ctx *ctx, void **ptr, uint64_t bytes) {
    bytes = (bytes + 255) & ~UINT64_C(255);
    if (ctx->in_use + bytes > ctx->cap)
        return pc_fail(ctx, PC_NOMEM, "device memory cap exceeded");
    cudaError_t e = cudaMallocAsync(ptr, bytes, ctx->stream);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return pc_fail(ctx, PC_NOMEM, std::string("device allocation failed: ") + cudaGetErrorString(e));
    }
    ctx->in_use += bytes;
    ctx->peak = std::max(ctx->peak, ctx->in_use);
    return PC_OK;
}

void pc_release(pc_ctx *ctx, void *ptr, uint64_t bytes) {
    if (!ptr) return;
    bytes = (bytes + 255) & ~UINT64_C(255);
    cudaFreeAsync(ptr, ctx->stream);
    ctx->in_use -= std::min(ctx->in_use, bytes);
}

StageLoan pc_stage(pc_ctx *ctx, uint64_t bytes) {
    if (bytes > PC_STAGE_BYTES) return {};
    return StageLoan(ctx->stage, [] {
        void *words = nullptr;
        if (cudaHostAlloc(&words, PC_STAGE_BYTES, cudaHostAllocDefault) != cudaSuccess) {
            cudaGetLastError();
            words = nullptr;
        }
        return (uint64_t *)words;
    });
}

extern "C" int pc_version(void) { return 1; }

extern "C" int pc_device_count(int *count) {
    cudaError_t e = cudaGetDeviceCount(count);
    if (e != cudaSuccess) {
        cudaGetLastError();
        *count = 0;
    }
    return PC_OK;
}

extern "C" const char *pc_last_error(const pc_ctx *ctx) { return ctx ? ctx->err.c_str() : "no context"; }

extern "C" int pc_init(int device, uint64_t mem_cap, double fraction, pc_ctx **out) {
    *out = nullptr;
    if (fraction <= 0.0 || fraction > 1.0) return PC_INVALID;
    pc_ctx *ctx = new pc_ctx();
    ctx->device = device;
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) {
        cudaGetLastError();
        delete ctx;
        return PC_CUDA;
    }
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess || cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking) != cudaSuccess) {
        cudaGetLastError();
        delete ctx;
        return PC_CUDA;
    }
    for (auto &ev : ctx->ev) cudaEventCreate(&ev);
    for (auto &ev : ctx->marks) cudaEventCreate(&ev);
    int64_t by_free = (int64_t)free_b - (int64_t)256 * 1024 * 1024;
    int64_t cap = std::min<int64_t>((int64_t)mem_cap, std::min<int64_t>((int64_t)(total_b * fraction), by_free));
    if (cap <= 0) {
        pc_free(ctx);
        return PC_NOMEM;
    }
    ctx->cap = (uint64_t)cap;
    cudaDeviceProp prop;
    cudaGetDeviceProperties(&prop, device);
    ctx->sm_count = prop.multiProcessorCount;
    ctx->cc_major = prop.major;
    ctx->cc_minor = prop.minor;
    strncpy(ctx->name, prop.name, sizeof(ctx->name) - 1);
    // Keep freed stream-ordered allocations cached in the pool between calls.
    cudaMemPool_t pool;
    if (cudaDeviceGetDefaultMemPool(&pool, device) == cudaSuccess) {
        uint64_t threshold = UINT64_MAX;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &threshold);
    }
    cudaGetLastError();
    *out = ctx;
    return PC_OK;
}

extern "C" int pc_host_alloc(uint64_t bytes, void **out) {
    if (!out) return PC_INVALID;
    *out = nullptr;
    if (cudaHostAlloc(out, std::max<uint64_t>(bytes, 16), cudaHostAllocDefault) != cudaSuccess) {
        cudaGetLastError();
        *out = nullptr;
        return PC_NOMEM;
    }
    return PC_OK;
}

extern "C" int pc_host_free(void *p) {
    if (p && cudaFreeHost(p) != cudaSuccess) {
        cudaGetLastError();
        return PC_CUDA;
    }
    return PC_OK;
}

extern "C" int pc_free(pc_ctx *ctx) {
    if (!ctx) return PC_OK;
    if (ctx->stream) cudaStreamSynchronize(ctx->stream);
    for (auto &ev : ctx->ev)
        if (ev) cudaEventDestroy(ev);
    for (auto &ev : ctx->marks)
        if (ev) cudaEventDestroy(ev);
    if (ctx->stream) cudaStreamDestroy(ctx->stream);
    if (ctx->stage.words) cudaFreeHost(ctx->stage.words);
    delete ctx;
    return PC_OK;
}

extern "C" int pc_mem_info(const pc_ctx *ctx, uint64_t *in_use, uint64_t *peak, uint64_t *cap) {
    *in_use = ctx->in_use;
    *peak = ctx->peak;
    *cap = ctx->cap;
    return PC_OK;
}

extern "C" int pc_copy_info(const pc_ctx *ctx, uint64_t *h2d, uint64_t *d2h) {
    if (!ctx || !h2d || !d2h) return PC_INVALID;
    *h2d = ctx->h2d;
    *d2h = ctx->d2h;
    return PC_OK;
}

extern "C" int pc_device_info(const pc_ctx *ctx, int *sm_count, int *cc_major, int *cc_minor, char *name, int name_len) {
    *sm_count = ctx->sm_count;
    *cc_major = ctx->cc_major;
    *cc_minor = ctx->cc_minor;
    if (name && name_len > 0) {
        strncpy(name, ctx->name, name_len - 1);
        name[name_len - 1] = 0;
    }
    return PC_OK;
}

extern "C" int pc_sync(pc_ctx *ctx) {
    PC_CHECK(ctx, cudaStreamSynchronize(ctx->stream));
    return PC_OK;
}

extern "C" int pc_wait_limit(pc_ctx *ctx, uint32_t polls) {
    if (!ctx) return PC_INVALID;
    ctx->polls = polls;
    return PC_OK;
}

extern "C" int pc_mark(pc_ctx *ctx, int slot) {
    if (slot < 0 || slot >= 8) return pc_fail(ctx, PC_INVALID, "timer slot out of range");
    PC_CHECK(ctx, cudaEventRecord(ctx->marks[slot], ctx->stream));
    return PC_OK;
}

extern "C" int pc_elapsed(pc_ctx *ctx, int a, int b, double *ms) {
    if (a < 0 || a >= 8 || b < 0 || b >= 8) return pc_fail(ctx, PC_INVALID, "timer slot out of range");
    PC_CHECK(ctx, cudaEventSynchronize(ctx->marks[b]));
    float f = 0;
    PC_CHECK(ctx, cudaEventElapsedTime(&f, ctx->marks[a], ctx->marks[b]));
    *ms = f;
    return PC_OK;
}

// ------------------------------------------------------------------------------------------
// buffers

extern "C" int pc_buf_upload(pc_ctx *ctx, const uint64_t *host, uint64_t n, pc_buf **out) {
    *out = nullptr;
    pc_buf *b = new pc_buf();
    b->n = n;
    b->bytes = std::max<uint64_t>(n * 8, 16);
    int rc = pc_alloc(ctx, (void **)&b->d, b->bytes);
    if (rc) {
        delete b;
        return rc;
    }
    if (n) {
        cudaError_t e = pc_copy(ctx, b->d, host, n * 8, cudaMemcpyHostToDevice);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) {
            pc_release(ctx, b->d, b->bytes);
            delete b;
            return pc_cuda_fail(ctx, e, "upload");
        }
    }
    *out = b;
    return PC_OK;
}

extern "C" int pc_buf_download(pc_ctx *ctx, const pc_buf *buf, uint64_t offset, uint64_t n, uint64_t *host) {
    if (offset > buf->n || n > buf->n - offset) return pc_fail(ctx, PC_INVALID, "download out of range");
    if (!n) return PC_OK;
    PC_CHECK(ctx, pc_copy(ctx, host, buf->d + offset, n * 8, cudaMemcpyDeviceToHost));
    PC_CHECK(ctx, cudaStreamSynchronize(ctx->stream));
    return PC_OK;
}

extern "C" int pc_buf_size(const pc_buf *buf, uint64_t *n) {
    *n = buf ? buf->n : 0;
    return PC_OK;
}

extern "C" int pc_buf_free(pc_ctx *ctx, pc_buf *buf) {
    if (!buf) return PC_OK;
    pc_release(ctx, buf->d, buf->bytes);
    delete buf;
    return PC_OK;
}

// Up to SEARCH_FEW queries (the subtile bounds of a batch of 64 and less) travel with the launch, and their answers are
// written to the page-locked stage by the kernel: one launch instead of an upload, a launch and a copy.
constexpr uint32_t SEARCH_FEW = 256;
constexpr uint64_t SEARCH_MANY = 1 << 17;
struct SearchFew {
    uint64_t q[SEARCH_FEW];
};

// Eight lanes per query (group_prefix): a dependent load for every three bits of the list's length.  From SEARCH_MANY queries
// on, which fill the device anyway, a lane per query needs fewer loads (MANY), and the answers go straight to the caller: through
// the stage they would be copied twice (131,072 queries 197 -> 172 us, 524,288 641 -> 496, 4,194,304 3,830 -> 3,300).
template <bool MANY>
__global__ void __launch_bounds__(256) k_searchsorted(const uint64_t *__restrict__ a, uint64_t n, const uint64_t *__restrict__ q,
                                                      uint64_t nq, uint64_t *__restrict__ out, const __grid_constant__ SearchFew few) {
    const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (MANY) {
        if (t >= nq) return;
        const uint64_t key = q[t];
        uint64_t lo = 0, hi = n;
        while (lo < hi) {
            const uint64_t mid = lo + (hi - lo) / 2;
            if (__ldg(a + mid) < key) lo = mid + 1;
            else hi = mid;
        }
        out[t] = lo;
        return;
    }
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t i = t / 8;
    const uint64_t key = i < nq ? q ? q[i] : few.q[i] : 0;
    const uint64_t at = group_prefix(i < nq ? n : 0, lane, [&](uint64_t j) { return __ldg(a + j) < key; });
    if (i < nq && (lane & 7) == 0) out[i] = at;
}

extern "C" int pc_buf_searchsorted(pc_ctx *ctx, const pc_buf *buf, const uint64_t *queries, uint64_t n, uint64_t *positions) {
    if (!n) return PC_OK;
    const bool many = n >= SEARCH_MANY;
    const unsigned blocks = (unsigned)(many ? (n + 255) / 256 : (n + 31) / 32);
    SearchFew few;
    const StageLoan loan = many ? StageLoan() : pc_stage(ctx, n * 8);
    uint64_t *stage = loan.get();
    if (stage && n <= SEARCH_FEW) {
        memcpy(few.q, queries, n * 8);
        k_searchsorted<false><<<blocks, 256, 0, ctx->stream>>>(buf->d, buf->n, nullptr, n, stage, few);
        PC_LAUNCHED(ctx, "searchsorted");
        ctx->d2h += n * 8;
        PC_CHECK(ctx, cudaStreamSynchronize(ctx->stream));
        memcpy(positions, stage, n * 8);
        return PC_OK;
    }
    Scratch s(ctx);
    uint64_t *dq, *dp;
    Carve both;
    both.add(&dq, n);
    both.add(&dp, n);
    const int rc = both.get(s);
    if (rc) return rc;
    PC_CHECK(ctx, pc_copy(ctx, dq, queries, n * 8, cudaMemcpyHostToDevice));
    (many ? k_searchsorted<true> : k_searchsorted<false>)<<<blocks, 256, 0, ctx->stream>>>(buf->d, buf->n, dq, n, dp, few);
    PC_LAUNCHED(ctx, "searchsorted");
    PC_CHECK(ctx, pc_copy(ctx, stage ? stage : positions, dp, n * 8, cudaMemcpyDeviceToHost));
    PC_CHECK(ctx, cudaStreamSynchronize(ctx->stream));
    if (stage) memcpy(positions, stage, n * 8);
    return PC_OK;
}

// ------------------------------------------------------------------------------------------
// limb self-test (kernels/pseudocube.cuh:7-11 semantics)

__global__ void k_wide(const uint64_t *__restrict__ in4, uint64_t *__restrict__ out3, uint64_t n) {
    uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    u128 l = mul_wide(in4[4 * i], in4[4 * i + 1]), r = mul_wide(in4[4 * i + 2], in4[4 * i + 3]);
    u128 d = sub128(l, r);
    out3[3 * i] = d.lo;
    out3[3 * i + 1] = d.hi;
    out3[3 * i + 2] = less128(l, r);
}

extern "C" int pc_selftest_wide(pc_ctx *ctx, const uint64_t *in4, uint64_t *out3, uint64_t n) {
    if (!n) return PC_OK;
    Scratch s(ctx);
    uint64_t *din, *dout;
    int rc = s.get(&din, 4 * n);
    if (!rc) rc = s.get(&dout, 3 * n);
    if (rc) return rc;
    PC_CHECK(ctx, pc_copy(ctx, din, in4, 32 * n, cudaMemcpyHostToDevice));
    k_wide<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(din, dout, n);
    PC_LAUNCHED(ctx, "wide self-test");
    PC_CHECK(ctx, pc_copy(ctx, out3, dout, 24 * n, cudaMemcpyDeviceToHost));
    PC_CHECK(ctx, cudaStreamSynchronize(ctx->stream));
    return PC_OK;
}
