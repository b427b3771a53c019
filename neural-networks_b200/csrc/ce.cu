// Softmax cross-entropy, forward and backward in one pass over the logits.
//
// One CTA (wide rows) or one warp (narrow rows) owns a row: it streams the logits once
// from HBM while keeping them in shared memory / registers, reduces max and sum-exp, then
// writes dlogits = (softmax - onehot) * inv from the on-chip copy: 8*C bytes per row. A CTA adds up
// its own rows' losses and a second launch adds the CTAs' sums in a fixed order into *loss_accum,
// so no host read-back sits on the step's critical path.
//
// Math: src/nn2/loss.rs:10-53 (p_t floored at 1e-30); masked form: src/gpu/cuda/
// mlstm_ops.cu:332-370. Kernels replaced: src/gpu/cuda/common.cu:270-289.
#include "common.cuh"
#include "tc.cuh"

namespace xl {

int* tc_status_ptr();

// Soft-cap cap*tanh(x/cap) of the flat LM's head (src/nn2/ops.rs:25-42), fused into the loss kernels when
// CAP: the input is then the pre-cap logit, and the gradient is taken through the cap,
// d/dx = (p - onehot) * inv * (1 - tanh^2).
template <bool CAP>
__device__ __forceinline__ float capped(float x, float cap, float icap) {
    if (!CAP) return x;
    return cap * (1.f - __fdividef(2.f, 1.f + __expf(2.f * x * icap)));
}
template <bool CAP>
__device__ __forceinline__ float through_cap(float g, float t, float icap) {
    if (!CAP) return g;
    const float u = t * icap;
    return g * (1.f - u * u);
}

// ---- wide rows: one CTA per row, row cached in shared memory ---------------------------------
// SPLIT: the gradient leaves as two bf16 terms, hi = bf16(g) and mid = bf16(g - hi), the operands of the head's three-product GEMMs, instead of as
// fp32 for a pass that splits it: 8 rather than 16 bytes of traffic per element behind the loss (4096 x 50304: 445 + 315 -> 466 us).
__device__ __forceinline__ void put_split(bf16* hi, bf16* mid, float g) {
    const bf16 h = __float2bfloat16_rn(g);
    *hi = h;
    *mid = __float2bfloat16_rn(g - __bfloat162float(h));
}
template <bool CACHE, bool CAP, bool SPLIT = false>
__global__ void __launch_bounds__(1024) ce_row_cta(const float* __restrict__ logits, const uint32_t* __restrict__ targets,
                                                   const uint32_t* __restrict__ mask, float* __restrict__ dlogits,
                                                   float* __restrict__ cta_loss, int rows, int C, float inv, float cap, bf16* __restrict__ hi,
                                                   bf16* __restrict__ mid) {
    const float icap = CAP ? 1.f / cap : 0.f;
    extern __shared__ __align__(16) float srow[];  // [C + 4] when CACHE
    __shared__ float red[32];
    float loss = 0.f;
    for (int r = blockIdx.x; r < rows; r += gridDim.x) {
        const float* z = logits + (size_t)r * C;
        float* d = SPLIT ? nullptr : dlogits + (size_t)r * C;
        bf16 *dh = SPLIT ? hi + (size_t)r * C : nullptr, *dm = SPLIT ? mid + (size_t)r * C : nullptr;
        if (mask && !mask[r]) {
            for (int j = threadIdx.x; j < C; j += blockDim.x) {
                if (SPLIT) put_split(dh + j, dm + j, 0.f);
                else d[j] = 0.f;
            }
            continue;
        }
        // pass 1: load + running max / sum-exp per thread (online softmax). The row is taken from its first 16-byte boundary on in
        // 16-byte pieces, the up to three elements on either side one by one; the shared copy starts at the same offset in a piece.
        float mx = -INFINITY, sum = 0.f;
        const int off = (int)(((uintptr_t)z & 15) >> 2);
        const bool v4 = (SPLIT || (((uintptr_t)z ^ (uintptr_t)d) & 15) == 0) && C >= 8;  // SPLIT: hi and mid 16-byte aligned as `logits` is
        const int head = v4 ? (4 - off) & 3 : 0, n4 = v4 ? (C - head) / 4 : 0, tail = head + 4 * n4;
        float* sr = srow + (v4 ? off : 0);
        auto take = [&](int j) {
            const float t = capped<CAP>(z[j], cap, icap);
            if (CACHE) sr[j] = t;
            if (t > mx) { sum *= __expf(mx - t); mx = t; }
            sum += __expf(t - mx);
        };
        if (v4) {
            const float4* z4 = reinterpret_cast<const float4*>(z + head);
            const int stride = blockDim.x;
            // four independent 16-byte loads in flight per thread before any of them is consumed
            for (int j0 = threadIdx.x; j0 < n4; j0 += 4 * stride) {
                float4 t[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int j = j0 + u * stride;
                    t[u] = (j < n4) ? __ldcs(z4 + j) : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int j = j0 + u * stride;
                    if (j < n4) {
                        if (CAP) {
                            t[u].x = capped<CAP>(t[u].x, cap, icap); t[u].y = capped<CAP>(t[u].y, cap, icap);
                            t[u].z = capped<CAP>(t[u].z, cap, icap); t[u].w = capped<CAP>(t[u].w, cap, icap);
                        }
                        if (CACHE) *reinterpret_cast<float4*>(sr + head + 4 * j) = t[u];
                        float m4 = fmaxf(fmaxf(t[u].x, t[u].y), fmaxf(t[u].z, t[u].w));
                        if (m4 > mx) { sum *= __expf(mx - m4); mx = m4; }
                        sum += __expf(t[u].x - mx) + __expf(t[u].y - mx) + __expf(t[u].z - mx) + __expf(t[u].w - mx);
                    }
                }
            }
            if ((int)threadIdx.x < head) take(threadIdx.x);
            else if ((int)threadIdx.x >= 4 && tail + (int)threadIdx.x - 4 < C) take(tail + threadIdx.x - 4);
        } else {
            for (int j = threadIdx.x; j < C; j += blockDim.x) take(j);
        }
        if (CACHE && r + (int)gridDim.x < rows) {
            // pull this CTA's next row into L2 while this row is reduced and its gradient written, so that DRAM
            // keeps reading through those phases and the next pass 1 starts from L2
            const char* nz = reinterpret_cast<const char*>(logits + (size_t)(r + gridDim.x) * C);
            for (size_t o = (size_t)threadIdx.x * 128; o < (size_t)C * sizeof(float); o += (size_t)blockDim.x * 128)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(nz + o));
        }
        float gmx = block_max(mx, red);
        sum = (mx == -INFINITY) ? 0.f : sum * expf(mx - gmx);
        float gsum = block_sum(sum, red);
        const float is = 1.f / gsum;
        const uint32_t tg = targets[r];
        if (threadIdx.x == 0) {
            float pt = 0.f;  // a target that is no symbol has none
            if (tg < (uint32_t)C) pt = expf((CACHE ? sr[tg] : capped<CAP>(z[tg], cap, icap)) - gmx) * is;
            loss -= logf(fmaxf(pt, 1e-30f));
        }
        if (!CACHE) __syncthreads();  // dlogits may alias logits: read z[target] before anyone overwrites it
        // pass 2: gradient from the on-chip copy
        auto grad = [&](float t, int j) {
            float o = __expf(t - gmx) * is;
            if ((uint32_t)j == tg) o -= 1.f;
            return through_cap<CAP>(o * inv, t, icap);
        };
        auto put = [&](int j) {
            const float g = grad(CACHE ? sr[j] : capped<CAP>(z[j], cap, icap), j);
            if (SPLIT) put_split(dh + j, dm + j, g);
            else d[j] = g;
        };
        if (v4) {
            float4* d4 = SPLIT ? nullptr : reinterpret_cast<float4*>(d + head);
            for (int j = threadIdx.x; j < n4; j += blockDim.x) {
                float4 t = CACHE ? *reinterpret_cast<float4*>(sr + head + 4 * j) : reinterpret_cast<const float4*>(z + head)[j];
                if (CAP && !CACHE) {
                    t.x = capped<CAP>(t.x, cap, icap); t.y = capped<CAP>(t.y, cap, icap);
                    t.z = capped<CAP>(t.z, cap, icap); t.w = capped<CAP>(t.w, cap, icap);
                }
                const int base = head + 4 * j;
                const float4 g = make_float4(grad(t.x, base), grad(t.y, base + 1), grad(t.z, base + 2), grad(t.w, base + 3));
                if (SPLIT) {
                    union { bf16 b[4]; uint2 u; } h, m;
                    put_split(&h.b[0], &m.b[0], g.x);
                    put_split(&h.b[1], &m.b[1], g.y);
                    put_split(&h.b[2], &m.b[2], g.z);
                    put_split(&h.b[3], &m.b[3], g.w);
                    __stcs(reinterpret_cast<uint2*>(dh + base), h.u);
                    __stcs(reinterpret_cast<uint2*>(dm + base), m.u);
                } else {
                    __stcs(d4 + j, g);
                }
            }
            if ((int)threadIdx.x < head) put(threadIdx.x);
            else if ((int)threadIdx.x >= 4 && tail + (int)threadIdx.x - 4 < C) put(tail + threadIdx.x - 4);
        } else {
            for (int j = threadIdx.x; j < C; j += blockDim.x) put(j);
        }
        __syncthreads();  // srow is reused by the next row
    }
    if (threadIdx.x == 0) cta_loss[blockIdx.x] = loss;
}

// ---- narrow rows (C <= 1024): a warp per row, the row in registers ------------------------------------------------------------
// The rows' losses as one number per CTA: lanes, then warps, in a fixed order.
__device__ __forceinline__ void put_cta_loss(float loss, float* cta_loss) {
    __shared__ float wl[8];
    loss = warp_sum(loss);
    if ((threadIdx.x & 31) == 0) wl[threadIdx.x >> 5] = loss;
    __syncthreads();
    if (threadIdx.x == 0) {
        float s = 0.f;
        for (int i = 0; i < 8; ++i) s += wl[i];
        cta_loss[blockIdx.x] = s;
    }
}

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// One row: z -> gradient into d (they may be the same memory). Returns the loss in lane 0. FULL: pieces of 32 that are whole for
// every C this variant serves. Instructions weigh most (31 a warp for 32 elements, three of them on the special-function unit: at 147312 x 257
// the issue slots are 58 % busy and that unit 38 %, the bytes would take 46 of the kernel's 63 us): with CAP the row is kept as tanh(z / cap),
// whose exponent and cap factor are one multiply-add, and the target's element is patched afterwards.
template <int VPL, int FULL, bool CAP>
__device__ __forceinline__ float narrow_row(const float* z, float* d, bool live, uint32_t tg, int C, float inv, float cap, float icap, int lane) {
    if (!live) {
        for (int j = lane; j < C; j += 32) d[j] = 0.f;
        return 0.f;
    }
    const float k1 = 2.f * icap * 1.4426950408889634f, k2 = (CAP ? cap : 1.f) * 1.4426950408889634f;
    auto squash = [&](float x) { return CAP ? 1.f - __fdividef(2.f, 1.f + ex2(x * k1)) : x; };
    float v[VPL], e[VPL], mx = -INFINITY, sum = 0.f;
    const bool any = tg < (uint32_t)C;  // a target that is no symbol: its probability is 0, nothing is patched
    const float zt = squash(z[any ? tg : 0u]);
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
        const int j = i * 32 + lane;
        v[i] = i < FULL || j < C ? z[j] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
        v[i] = squash(v[i]);
        if (i < FULL || i * 32 + lane < C) mx = fmaxf(mx, v[i]);
    }
    mx = warp_max(mx);
    const float mk = mx * k2;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
        e[i] = i < FULL || i * 32 + lane < C ? ex2(fmaf(v[i], k2, -mk)) : 0.f;
        sum += e[i];
    }
    const float is = 1.f / warp_sum(sum), gs = is * inv;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
        const int j = i * 32 + lane;
        if (i < FULL || j < C) d[j] = e[i] * gs * (CAP ? fmaf(-v[i], v[i], 1.f) : 1.f);
    }
    __syncwarp();
    const float pt = any ? ex2(fmaf(zt, k2, -mk)) * is : 0.f;
    if (any && lane == 0) d[tg] = (pt - 1.f) * inv * (CAP ? fmaf(-zt, zt, 1.f) : 1.f);
    return lane == 0 ? -logf(fmaxf(pt, 1e-30f)) : 0.f;
}

// Rows straight from global memory: for arrays that do not start on 16 bytes, which bulk copies need.
template <int VPL, int FULL, bool CAP>
__global__ void __launch_bounds__(256) ce_row_warp(const float* __restrict__ logits, const uint32_t* __restrict__ targets,
                                                   const uint32_t* __restrict__ mask, float* __restrict__ dlogits,
                                                   float* __restrict__ cta_loss, int rows, int C, float inv, float cap) {
    const int lane = threadIdx.x & 31;
    float loss = 0.f;
    for (int r = blockIdx.x * 8 + (threadIdx.x >> 5); r < rows; r += gridDim.x * 8)
        loss += narrow_row<VPL, FULL, CAP>(logits + (size_t)r * C, dlogits + (size_t)r * C, !(mask && !mask[r]), targets[r], C, inv, cap,
                                     CAP ? 1.f / cap : 0.f, lane);
    put_cta_loss(loss, cta_loss);
}

// Tiles of RT rows (a multiple of eight: RT * C floats start and end on 16 bytes whatever C is) move whole between global and shared
// memory by bulk copies, three stages deep in a persistent CTA: while one tile is computed the next is loading and the one before
// leaves. A 257-symbol row has no 16-byte boundary a warp could use, and 4-byte accesses with one row in flight per warp ran at 1.5 TB/s
// (147312 x 257: 200 us, and 57 us for one CTA to add 147312 row losses; now 63 and 3).
static constexpr int kCeStages = 3;
template <int VPL, int FULL, bool CAP>
__global__ void __launch_bounds__(256) ce_tile(const float* logits, const uint32_t* __restrict__ targets, const uint32_t* __restrict__ mask,
                                               float* dlogits, float* __restrict__ cta_loss, int rows, int C, int RT, float inv, float cap, int* status) {
    extern __shared__ __align__(128) float tiles[];  // [kCeStages][RT * C]
    __shared__ uint64_t full[kCeStages];
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, ntiles = (rows + RT - 1) / RT;
    const float icap = CAP ? 1.f / cap : 0.f;
    const size_t stage = (size_t)RT * C;
    auto load = [&](int t, int s) {  // whole 16-byte pieces; the last tile's rest (at most three floats) follows in the loop
        const int n = min(RT, rows - t * RT) * C;
        const uint32_t bytes = (uint32_t)(n / 4) * 16;
        tc::mbar_expect_tx(full + s, bytes);
        if (bytes)
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                         ::"r"(tc::smem_u32(tiles + s * stage)), "l"(logits + (size_t)t * stage), "r"(bytes), "r"(tc::smem_u32(full + s)) : "memory");
    };
    if (tid == 0) {
        for (int s = 0; s < kCeStages; ++s) tc::mbar_init(full + s, 1);
        tc::fence_mbar_init();
        for (int k = 0; k < kCeStages - 1; ++k)
            if ((int)(blockIdx.x + k * gridDim.x) < ntiles) load(blockIdx.x + k * gridDim.x, k);
    }
    __syncthreads();
    float loss = 0.f;
    int k = 0;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++k) {
        const int s = k % kCeStages, r0 = t * RT, nr = min(RT, rows - r0), n = nr * C, whole = n / 4 * 4;
        float* tile = tiles + s * stage;
        const bool ok = tc::mbar_wait(full + s, (k / kCeStages) & 1);
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                atomicCAS(status, 0, 401);
                if (t + (int)gridDim.x < ntiles) (void)tc::mbar_wait(full + (k + 1) % kCeStages, ((k + 1) / kCeStages) & 1);  // the next tile's load is on its way
            }
            break;
        }
        if (n != whole) {
            if (tid < n - whole) tile[whole + tid] = logits[(size_t)t * stage + whole + tid];
            __syncthreads();
        }
        for (int r = w; r < nr; r += 8)
            loss += narrow_row<VPL, FULL, CAP>(tile + r * C, tile + r * C, !(mask && !mask[r0 + r]), targets[r0 + r], C, inv, cap, icap, lane);
        tc::fence_async_smem();
        __syncthreads();
        if (tid < n - whole) dlogits[(size_t)t * stage + whole + tid] = tile[whole + tid];
        if (tid == 0) {
            if (whole)
                asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                             ::"l"(dlogits + (size_t)t * stage), "r"(tc::smem_u32(tile)), "r"((uint32_t)whole * 4) : "memory");
            tc::tma_store_commit();
            const int t2 = t + (kCeStages - 1) * gridDim.x;
            if (t2 < ntiles) {
                asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");  // the tile before this one has left its stage
                load(t2, (k + kCeStages - 1) % kCeStages);
            }
        }
    }
    if (tid == 0) tc::tma_store_wait_all();
    put_cta_loss(loss, cta_loss);
}

// *loss_accum += inv * sum of the CTAs' losses, in a fixed order.
__global__ void __launch_bounds__(1024) ce_loss_reduce(const float* __restrict__ cta_loss, float* loss_accum, int n, float inv) {
    __shared__ float red[32];
    float s = 0.f;
    for (int r = threadIdx.x; r < n; r += blockDim.x) s += cta_loss[r];
    s = block_sum(s, red);
    if (threadIdx.x == 0) *loss_accum += s * inv;
}

}  // namespace xl

using namespace xl;

extern "C" size_t xlstm_ce_workspace_bytes(int rows) { return rows > 0 ? (size_t)rows * sizeof(float) : 0; }

template <bool CAP>
static int ce_run(void* stream, const float* logits, const uint32_t* targets, const uint32_t* mask, float* dlogits,
                  float* loss_accum, int rows, int C, float inv, float cap, void* workspace, size_t workspace_bytes) {
    XL_CHECK_ARG(logits && targets && dlogits && loss_accum, "ce_fw_bw: null pointer");
    XL_CHECK_ARG(rows >= 0 && C > 0, "ce_fw_bw: bad shape rows=%d C=%d", rows, C);
    if (rows == 0) return XLSTM_OK;
    if (!workspace || workspace_bytes < xlstm_ce_workspace_bytes(rows)) {
        set_error("ce_fw_bw: workspace of %zu B is smaller than the %zu B required", workspace_bytes,
                  xlstm_ce_workspace_bytes(rows));
        return XLSTM_ERR_WORKSPACE;
    }
    cudaStream_t st = (cudaStream_t)stream;
    float* cta_loss = (float*)workspace;  // one sum per CTA, never more CTAs than rows
    int grid;
    if (C <= 1024 && !(((uintptr_t)logits | (uintptr_t)dlogits) & 15)) {
        // tiles of at most 24 KB in whole groups of eight rows (257 columns: 16 rows, 16 KB), fewer rows where that leaves SMs without one;
        // an SM's shared memory holds three CTAs of three such stages at 24 KB, four at 257 columns
        int RT = (24 * 1024 / (4 * C)) / 8 * 8;
        const int fair = (rows / sm_count() + 7) / 8 * 8;
        if (RT > fair) RT = fair;
        if (RT < 8) RT = 8;
        if (RT > 64) RT = 64;
        const size_t smem = (size_t)kCeStages * RT * C * sizeof(float);
        int per_sm = (int)(224 * 1024 / (smem + 1200));
        if (per_sm > 8) per_sm = 8;
        const int ntiles = (rows + RT - 1) / RT, maxb = sm_count() * per_sm;
        grid = ntiles < maxb ? ntiles : maxb;
        int* status = tc_status_ptr();
        if (!status) return XLSTM_ERR_CUDA;
#define RUN(V, F)                                                                                                                     \
    do {                                                                                                                              \
        XL_CUDA(cudaFuncSetAttribute(ce_tile<V, F, CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024));                   \
        ce_tile<V, F, CAP><<<grid, 256, smem, st>>>(logits, targets, mask, dlogits, cta_loss, rows, C, RT, inv, cap, status);        \
    } while (0)
        if (C <= 64) RUN(2, 0);
        else if (C <= 128) RUN(4, 2);
        else if (C <= 256) RUN(8, 4);
        else if (C <= 288) RUN(9, 8);
        else if (C <= 512) RUN(16, 9);
        else RUN(32, 16);
#undef RUN
        XL_LAUNCH_OK("ce_tile");
    } else if (C <= 1024) {
        const int nb = (rows + 7) / 8, maxb = sm_count() * 8;
        grid = nb < maxb ? nb : maxb;
#define RUN(V) ce_row_warp<V, 0, CAP><<<grid, 256, 0, st>>>(logits, targets, mask, dlogits, cta_loss, rows, C, inv, cap)
        if (C <= 256) RUN(8);
        else RUN(32);
#undef RUN
        XL_LAUNCH_OK("ce_row_warp");
    } else {
        size_t smem = (size_t)(C + 4) * sizeof(float);
        int threads = C >= 8192 ? 1024 : 256;
        if (smem <= 200 * 1024) {
            XL_CUDA(cudaFuncSetAttribute(ce_row_cta<true, CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            int per_sm = (int)((220 * 1024) / (smem + 1024));
            if (per_sm < 1) per_sm = 1;
            if (per_sm > 2048 / threads) per_sm = 2048 / threads;
            int maxb = sm_count() * per_sm;
            grid = rows < maxb ? rows : maxb;
            ce_row_cta<true, CAP><<<grid, threads, smem, st>>>(logits, targets, mask, dlogits, cta_loss, rows, C, inv, cap, nullptr, nullptr);
        } else {
            int maxb = sm_count() * 2;
            grid = rows < maxb ? rows : maxb;
            ce_row_cta<false, CAP><<<grid, 1024, 0, st>>>(logits, targets, mask, dlogits, cta_loss, rows, C, inv, cap, nullptr, nullptr);
        }
        XL_LAUNCH_OK("ce_row_cta");
    }
    ce_loss_reduce<<<1, 1024, 0, st>>>(cta_loss, loss_accum, grid, inv);
    XL_LAUNCH_OK("ce_loss_reduce");
    return XLSTM_OK;
}

extern "C" int xlstm_ce_fw_bw(void* stream, const float* logits, const uint32_t* targets, const uint32_t* mask,
                              float* dlogits, float* loss_accum, int rows, int C, float inv, void* workspace,
                              size_t workspace_bytes) {
    return ce_run<false>(stream, logits, targets, mask, dlogits, loss_accum, rows, C, inv, 0.f, workspace, workspace_bytes);
}

extern "C" int xlstm_softcap_ce_fw_bw(void* stream, const float* pre_logits, const uint32_t* targets, const uint32_t* mask,
                                      float* d_pre, float* loss_accum, int rows, int C, float inv, float cap, void* workspace,
                                      size_t workspace_bytes) {
    XL_CHECK_ARG(cap > 0.f, "softcap_ce_fw_bw: cap must be positive (got %g)", (double)cap);
    return ce_run<true>(stream, pre_logits, targets, mask, d_pre, loss_accum, rows, C, inv, cap, workspace, workspace_bytes);
}

extern "C" int xlstm_softcap_ce_split_fw_bw(void* stream, const float* pre_logits, const uint32_t* targets, const uint32_t* mask, void* d_hi,
                                            void* d_mid, float* loss_accum, int rows, int C, float inv, float cap, void* workspace,
                                            size_t workspace_bytes) {
    XL_CHECK_ARG(pre_logits && targets && d_hi && d_mid && loss_accum, "softcap_ce_split: null pointer");
    XL_CHECK_ARG(rows >= 0 && C > 0 && cap > 0.f, "softcap_ce_split: bad shape rows=%d C=%d or cap %g", rows, C, (double)cap);
    const size_t smem = (size_t)(C + 4) * sizeof(float);
    if (C <= 1024 || smem > 200 * 1024 || (((uintptr_t)pre_logits | (uintptr_t)d_hi | (uintptr_t)d_mid) & 15)) {
        set_error("softcap_ce_split: rows of 1025 to 51196 logits, 16-byte aligned (got %d)", C);
        return XLSTM_DECLINED;
    }
    if (rows == 0) return XLSTM_OK;
    if (!workspace || workspace_bytes < xlstm_ce_workspace_bytes(rows)) {
        set_error("softcap_ce_split: workspace of %zu B is smaller than the %zu B required", workspace_bytes, xlstm_ce_workspace_bytes(rows));
        return XLSTM_ERR_WORKSPACE;
    }
    cudaStream_t st = (cudaStream_t)stream;
    const int threads = C >= 8192 ? 1024 : 256;
    int per_sm = (int)((220 * 1024) / (smem + 1024));
    if (per_sm < 1) per_sm = 1;
    if (per_sm > 2048 / threads) per_sm = 2048 / threads;
    const int maxb = sm_count() * per_sm, grid = rows < maxb ? rows : maxb;
    float* cta_loss = (float*)workspace;
    XL_CUDA(cudaFuncSetAttribute(ce_row_cta<true, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    ce_row_cta<true, true, true><<<grid, threads, smem, st>>>(pre_logits, targets, mask, nullptr, cta_loss, rows, C, inv, cap, (bf16*)d_hi, (bf16*)d_mid);
    XL_LAUNCH_OK("ce_row_cta");
    ce_loss_reduce<<<1, 1024, 0, st>>>(cta_loss, loss_accum, grid, inv);
    XL_LAUNCH_OK("ce_loss_reduce");
    return XLSTM_OK;
}

// ---- the same op for callers that cannot allocate device memory --------------------------------
//
// xlstm_ce_fw_bw needs one float of scratch per row and asks the caller for it. Some hosts have no
// way to supply that: the reference's own runtime hands every byte of device memory to its buffer
// pool up front, and a step loop that must never touch the CUDA allocator (because cudaMalloc and
// cudaFree can synchronise the whole device, or because the surrounding code runs where allocation
// calls are not allowed) has the same problem. For them the scratch lives inside the library, in a
// fixed array that every GPU loading the library keeps resident until the process exits.
//
// Limits and sharing rules, because the array is one per device and is never cleared:
//   - at most XLSTM_CE_NOALLOC_MAX_ROWS rows per call (256 KiB of scratch); more is refused;
//   - every element a call reads is written earlier in the same call, so stale contents from the
//     previous call are harmless and nothing needs zeroing;
//   - two calls whose kernels may overlap on the same device (different streams) race on the
//     array; serialise them on one stream.
// The first call on each device looks up the array's device address (cudaGetSymbolAddress, which
// is not an allocation); make that first call before starting any stream capture.
static constexpr int kCeNoAllocMaxRows = 65536;
static __device__ __align__(256) float g_ce_noalloc_scratch[kCeNoAllocMaxRows];

static float* ce_noalloc_scratch_ptr(int* rc) {
    // In host code the array's name is only a handle; the kernels need its device address.
    static std::atomic<float*> cached[64];
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= 64) {
        set_error("ce_fw_bw_noalloc: cudaGetDevice failed or device index out of range: %s", cudaGetErrorString(e));
        *rc = XLSTM_ERR_CUDA;
        return nullptr;
    }
    float* p = cached[dev].load(std::memory_order_acquire);
    if (!p) {
        void* addr = nullptr;
        e = cudaGetSymbolAddress(&addr, g_ce_noalloc_scratch);
        if (e != cudaSuccess || !addr) {
            set_error("ce_fw_bw_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
            *rc = XLSTM_ERR_CUDA;
            return nullptr;
        }
        p = (float*)addr;
        cached[dev].store(p, std::memory_order_release);
    }
    *rc = XLSTM_OK;
    return p;
}

extern "C" int xlstm_ce_fw_bw_noalloc(void* stream, const float* logits, const uint32_t* targets, const uint32_t* mask,
                                      float* dlogits, float* loss_accum, int rows, int C, float inv) {
    if (rows > kCeNoAllocMaxRows) {
        set_error("ce_fw_bw_noalloc: %d rows exceed the built-in scratch of %d rows; split the call or use xlstm_ce_fw_bw "
                  "with a caller-owned workspace", rows, kCeNoAllocMaxRows);
        return XLSTM_ERR_ARG;
    }
    int rc = XLSTM_OK;
    float* scratch = ce_noalloc_scratch_ptr(&rc);
    if (!scratch) return rc;
    return xlstm_ce_fw_bw(stream, logits, targets, mask, dlogits, loss_accum, rows, C, inv, scratch,
                          (size_t)kCeNoAllocMaxRows * sizeof(float));
}
