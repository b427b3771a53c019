// Chunk-parallel mLSTM, part 1: gate vectors and the state recurrence.
//
// The one-CTA-per-head kernels walk a head's chunks with everything (scores, outputs, epilogues) on the sequential path: 1 us a
// chunk forward and 2.6 us backward at a few percent of the tensor pipe, eight CTAs for eight heads, and four sub-head passes with
// fp32 partial planes for 256-wide heads. Only the state is sequential. Here one kernel walks C alone and records it at
// 128-position borders (backward: dC), and everything else is independent per chunk and runs on all SMs
// (mlstm_par_out.cu, mlstm_par_grad.cu).
#include "mlstm_par.cuh"

namespace xl {
namespace par {

// ---- gate vectors: one CTA per head, a warp per chunk, four consecutive positions per lane --------------------------------------
// fc = cumulative log sigmoid(f) inside the chunk; m_t = fc_t + max(m_prev, max_{j<=t}(i_j - fc_j)); the chain of m_prev over the
// chunks is NC dependent steps of one thread. FROM_M: m is given (backward), nothing is chained.
// A call that takes or leaves a state as a result (F = double) sums the gates and chains m in 64 bits: fc grows to tens over a chunk, and its rounding at
// 32, added up along the chain, made m and n, then results of the call, two to four times less exact than the kernels with chunks of 64
// positions (8 heads, 4069 positions: m 1.0e-7 there and 3.6e-7 here, now 0.4e-7; n 1.8e-7, 7.0e-7, 0.9e-7). Pairs of floats are as exact and
// take longer, in the chain above all. Within a training step (no state, or XLSTM_SWEEP) m and n only weigh bf16 products, 1e-3 off themselves,
// and floats do.
struct GateArgs {
    const float *ig, *fg, *m_in;
    float *m, *m_last;
    Vecs v;
    int B, H, T, NC;
};
static constexpr int kMaxChunks = 2048;
__device__ __forceinline__ float larger(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ double larger(double a, double b) { return fmax(a, b); }
template <typename F>
struct Local { F fc[4], um[4], u[4]; };
template <typename F>
__device__ __forceinline__ Local<F> chunk_local(const GateArgs& p, int b, int h, int ck, int lane) {
    Local<F> r;
    F s = 0, mx = -INFINITY;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int t = ck * LC + lane * 4 + e;
        float f = INFINITY, i = -INFINITY;  // past T: log sigmoid 0, no input
        if (t < p.T) {
            const size_t gi = ((size_t)b * p.T + t) * p.H + h;
            f = p.fg[gi];
            i = p.ig[gi];
        }
        s += (F)log_sigmoid(f);
        r.fc[e] = s;
        r.u[e] = i;
    }
    F pre = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const F y = __shfl_up_sync(0xffffffffu, pre, o);
        if (lane >= o) pre += y;
    }
    const F before = __shfl_up_sync(0xffffffffu, pre, 1);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        if (lane) r.fc[e] += before;
        r.u[e] -= r.fc[e];
        mx = larger(mx, r.u[e]);
        r.um[e] = mx;
    }
    F pm = mx;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const F y = __shfl_up_sync(0xffffffffu, pm, o);
        if (lane >= o) pm = larger(pm, y);
    }
    const F mb = __shfl_up_sync(0xffffffffu, pm, 1);
    if (lane)
#pragma unroll
        for (int e = 0; e < 4; ++e) r.um[e] = larger(r.um[e], mb);
    return r;
}
template <bool FROM_M, typename F>
__global__ void __launch_bounds__(1024) par_gates(const GateArgs p) {
    __shared__ F s_fc[FROM_M ? 1 : kMaxChunks], s_um[FROM_M ? 1 : kMaxChunks];
    const int bh = blockIdx.x, b = bh / p.H, h = bh % p.H, w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const bool again = FROM_M || p.NC > nw;  // else a warp has one chunk, and keeps it
    Local<F> l;
    if (!FROM_M) {
        for (int ck = w; ck < p.NC; ck += nw) {
            l = chunk_local<F>(p, b, h, ck, lane);
            if (lane == 31) { s_fc[ck] = l.fc[3]; s_um[ck] = l.um[3]; }
        }
        __syncthreads();
        if (threadIdx.x == 0) {  // s_um becomes the m each chunk enters with
            F m = p.m_in ? p.m_in[bh] : 0.f;
            for (int ck = 0; ck < p.NC; ++ck) {
                const F next = s_fc[ck] + larger(m, s_um[ck]);
                s_um[ck] = m;
                m = next;
            }
        }
        __syncthreads();
    }
    for (int ck = w; ck < p.NC; ck += nw) {
        if (again) l = chunk_local<F>(p, b, h, ck, lane);
        const int t0 = ck * LC;
        float m_in, m[4];  // as they are stored: what the entering state is scaled by, and what the backward will read
        if (FROM_M) {
            m_in = ck ? p.m[(size_t)bh * p.T + t0 - 1] : p.m_in ? p.m_in[bh] : 0.f;
#pragma unroll
            for (int e = 0; e < 4; ++e) m[e] = p.m[(size_t)bh * p.T + min(t0 + lane * 4 + e, p.T - 1)];
        } else {
            const F m_prev = s_um[ck];
            m_in = (float)m_prev;
#pragma unroll
            for (int e = 0; e < 4; ++e) m[e] = (float)(l.fc[e] + larger(m_prev, l.um[e]));
        }
        // m of the last position in the sequence (the scan's tree rounds the positions behind it differently)
        const int tl = min(p.T - 1 - t0, LC - 1);
        const F fcL = __shfl_sync(0xffffffffu, l.fc[3], 31);
        const float mL = __shfl_sync(0xffffffffu, (tl & 3) == 0 ? m[0] : (tl & 3) == 1 ? m[1] : (tl & 3) == 2 ? m[2] : m[3], tl >> 2);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int t = t0 + lane * 4 + e;
            const size_t o = (size_t)bh * p.v.Tp + t;
            const bool in = t < p.T;
            if (!FROM_M && in) {
                p.m[(size_t)bh * p.T + t] = m[e];
                if (t == p.T - 1 && p.m_last) p.m_last[bh] = m[e];
            }
            p.v.rowt[o] = in ? (float)(l.fc[e] - m[e]) : -INFINITY;  // past T the decay mask is 0 whatever colt is
            p.v.colt[o] = (float)l.u[e];
            p.v.a[o] = in ? expf((float)(fcL + l.u[e] - mL)) : 0.f;
            p.v.b[o] = in ? expf((float)(l.fc[e] + m_in - m[e])) : 0.f;
        }
        if (lane == 0) p.v.g[(size_t)bh * p.NC + ck] = expf((float)(fcL + m_in - mL));
    }
}
int gates_launch(cudaStream_t st, const float* ig, const float* fg, const float* m_in, float* m, float* m_last, const Vecs& v,
                 int B, int H, int T, int NC, bool from_m, bool exact) {
    GateArgs p = {ig, fg, m_in, m, m_last, v, B, H, T, NC};
    const int threads = NC >= 32 ? 1024 : 32 * NC;
    if (from_m && exact) par_gates<true, double><<<B * H, threads, 0, st>>>(p);
    else if (from_m) par_gates<true, float><<<B * H, threads, 0, st>>>(p);
    else if (exact) par_gates<false, double><<<B * H, threads, 0, st>>>(p);
    else par_gates<false, float><<<B * H, threads, 0, st>>>(p);
    XL_LAUNCH_OK("par_gates");
    return XLSTM_OK;
}

// ---- the state recurrence --------------------------------------------------------------------------------------------------------
// A CTA owns a [128 v] x [NT qk] block of one head's state, fp32 in tensor memory for the whole walk. Per chunk: the state pass reads
// it, leaves the bf16 record entry (TMA store from shared memory) and scales it by the chunk's decay; the MMA warp then adds
// (w.X)^T Y, 64 positions at a time. Loads and the scaling of X by w run ahead in a ring of 64-position stages, so the period is the
// state pass plus the products' latency. n (fp32, CUDA cores) is taken by the CTAs of the first v rows.
struct ScanP {
    CUtensorMap tx, ty, trec;
    const float *w, *g, *c0, *n0;
    float *recn, *oC, *on;
    int H, T, D, NC, Tp, entries, nv, nt;
    int* status;
};
static constexpr int kStateThreads = 256, kAuxThreads = 256;
static constexpr int kScanThreads = kStateThreads + kAuxThreads + 64;
template <int NT>
struct ScanS {
    static constexpr int kStages = NT == 256 ? 3 : 4;
    static constexpr uint32_t kX = 16384, kY = NT * 128, kStage = kX + kY;
    static constexpr uint32_t rec = kStages * kStage;                // bf16 [128][NT] as boxes of 64 columns
    static constexpr uint32_t w = rec + 128 * NT * 2;                // [kStages][64]
    static constexpr uint32_t red = w + kStages * 256;               // n partial sums [512 / (NT / 2) / ...][NT]: 8 * 64 .. floats
    static constexpr uint32_t g = red + 512 * 4;
    static constexpr uint32_t total = g + kMaxChunks * 4 + 256;
};
#define PAR_WAIT(bar, par) do { if (!mbar_wait(bar, par)) { fail = true; } } while (0)

template <int NT, bool BWD>
__global__ void __launch_bounds__(kScanThreads, 1) par_scan(const __grid_constant__ ScanP p) {
    typedef ScanS<NT> S;
    extern __shared__ unsigned char raw[];
    unsigned char* sm = (unsigned char*)(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
    float* sw = (float*)(sm + S::w);
    float* red = (float*)(sm + S::red);
    float* sg = (float*)(sm + S::g);
    uint64_t* bars = (uint64_t*)(sm + S::g + kMaxChunks * 4);
    uint64_t *full = bars, *scaled = bars + S::kStages, *empty = bars + 2 * S::kStages, *sready = bars + 3 * S::kStages, *cdone = sready + 1;
    uint32_t* slot = (uint32_t*)(cdone + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int qi = blockIdx.x % p.nt, vi = (blockIdx.x / p.nt) % p.nv, bh = blockIdx.x / (p.nt * p.nv), b = bh / p.H, h = bh % p.H;
    const bool do_n = vi == 0;
    bool fail = false;
    if (tid == 0) {
        for (int i = 0; i < S::kStages; ++i) { mbar_init(full + i, 1); mbar_init(scaled + i, 8); mbar_init(empty + i, 9); }
        mbar_init(sready, 8);
        mbar_init(cdone, 1);
        fence_mbar_init();
    }
    for (int i = tid; i < p.NC; i += kScanThreads) sg[i] = p.g[(size_t)bh * p.NC + i];
    if (warp == 17) tmem_alloc(slot, NT < 32 ? 32 : NT);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tC = *slot;
    const int halves = 2 * p.NC;
    auto chunk = [&](int i) { return BWD ? p.NC - 1 - i : i; };

    if (warp == 16) {
        // ---- loads ----
        if (lane == 0) {
            int i = 0;
            for (; i < halves && !fail; ++i) {
                const int st = i % S::kStages, ck = chunk(i >> 1), t0 = ck * LC + (i & 1) * 64;
                if (i >= S::kStages) PAR_WAIT(empty + st, ((i / S::kStages) - 1) & 1);
                if (fail) break;
                unsigned char* d = sm + st * S::kStage;
                mbar_expect_tx(full + st, S::kStage + 256);
                tma_load_4d(smem_u32(d), &p.tx, smem_u32(full + st), 0, t0, (h * p.D + vi * 128) >> 6, b);
                tma_load_4d(smem_u32(d + S::kX), &p.ty, smem_u32(full + st), 0, t0, (h * p.D + qi * NT) >> 6, b);
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], 256, [%2];"
                             ::"r"(smem_u32(sw + st * 64)), "l"(p.w + (size_t)bh * p.Tp + t0), "r"(smem_u32(full + st)) : "memory");
            }
            if (fail) ring_landed<S::kStages>(full, i);
        }
        __syncwarp();
    } else if (warp == 17) {
        // ---- products ----
        const uint64_t dM = smem_desc(0, 8192, 1024);
        constexpr uint32_t id = instr_desc(128, NT, 1, 1);
        for (int i = 0; i < halves && !fail; ++i) {
            const int st = i % S::kStages;
            if (!(i & 1)) PAR_WAIT(sready, (i >> 1) & 1);
            PAR_WAIT(BWD ? full + st : scaled + st, (i / S::kStages) & 1);
            if (fail) break;
            tc_fence_after();
            const uint32_t ax = smem_u32(sm + st * S::kStage);
            const uint64_t xd = desc_at(dM, ax), yd = desc_at(dM, ax + S::kX);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) mma_ss_w(tC, xd + ks * 128, yd + ks * 128, id, 1);
            mma_commit_w(empty + st);
            if (i & 1) mma_commit_w(cdone);
        }
    } else if (warp >= 8) {
        // ---- scaling of X, and n: thread = column pair cp of NT / 2, row group rg ----
        const int at = tid - kStateThreads;
        constexpr int CP = NT / 2, RG = kAuxThreads / CP, RPG = 64 / RG;  // row groups and rows of a stage per group
        const int cp = at % CP, rg = at / CP;
        float n0 = 0.f, n1 = 0.f, nn = 0.f;  // partial sums of this chunk; thread at < NT owns n of column at
        if (do_n && at < NT && p.n0) nn = p.n0[(size_t)bh * p.D + qi * NT + at];
        for (int i = 0; i < halves; ++i) {
            const int st = i % S::kStages, ck = chunk(i >> 1);
            if (fail && !do_n) break;
            PAR_WAIT(full + st, (i / S::kStages) & 1);
            if (fail && !(do_n && (i & 1))) continue;  // the warps leave together, at the barrier below (no barriers without n)
            unsigned char* X = sm + st * S::kStage;
            const float* wv = sw + st * 64;
            if (!BWD) {
                // 64 rows x 16 pieces of 8 values, four per thread: row = piece / 16
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int e = at + q * kAuxThreads, row = e >> 4, pc = e & 15;
                    uint4* a = reinterpret_cast<uint4*>(X + (pc >> 3) * 8192 + swz(row, pc & 7));
                    uint4 v = *a;
                    const float s = wv[row];
                    uint32_t* u = &v.x;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float2 f = unpack_bf16(u[j]);
                        u[j] = pack_bf16(f.x * s, f.y * s);
                    }
                    *a = v;
                }
                fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(scaled + st);
            }
            if (do_n) {
                const unsigned char* Y = X + S::kX + (cp >> 5) * 8192 + (cp & 3) * 4;
#pragma unroll 8
                for (int r = 0; r < RPG; ++r) {
                    const int row = rg * RPG + r;
                    const float2 f = unpack_bf16(*reinterpret_cast<const uint32_t*>(Y + swz(row, (cp & 31) >> 2)));
                    n0 = fmaf(wv[row], f.x, n0);
                    n1 = fmaf(wv[row], f.y, n1);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty + st);
            if (do_n && (i & 1)) {
                red[rg * NT + 2 * cp] = n0;
                red[rg * NT + 2 * cp + 1] = n1;
                n0 = n1 = 0.f;
                fail = named_barrier_or(2, kAuxThreads, fail);
                if (fail) break;
                if (at < NT) {
                    p.recn[((size_t)bh * p.entries + ck) * p.D + qi * NT + at] = nn;
                    float s = 0.f;
#pragma unroll
                    for (int r = 0; r < RG; ++r) s += red[r * NT + at];
                    nn = sg[ck] * nn + s;
                }
                named_barrier(2, kAuxThreads);
            }
        }
        if (do_n && at < NT && !fail) {
            if (!BWD) p.recn[((size_t)bh * p.entries + p.NC) * p.D + qi * NT + at] = nn;
            if (p.on) p.on[(size_t)bh * p.D + qi * NT + at] = nn;
        }
    } else {
        // ---- state pass: thread = row v of the block, half of its columns ----
        const int qd = warp & 3, half = warp >> 2, row = 32 * qd + lane;
        constexpr int HC = NT / 2, PC = HC / 32;
        const uint32_t t0 = tC + ((uint32_t)(32 * qd) << 16) + half * HC;
        const size_t crow = ((size_t)bh * p.D + vi * 128 + row) * p.D + qi * NT + half * HC;
        const bool c0_whole = p.c0 && ((uintptr_t)p.c0 & 15) == 0;
        for (int i = 0; i <= p.NC && !fail; ++i) {
            const bool last = i == p.NC;
            const int ck = last ? 0 : chunk(i);
            if (i) PAR_WAIT(cdone, (i - 1) & 1);
            tc_fence_after();
            const float g = last ? 1.f : sg[ck];
            const bool rec = !last || !BWD;
            if (rec && tid == 0) tma_store_wait_read();
            fail = named_barrier_or(1, kStateThreads, fail);  // the previous entry has left the staging buffer; all warps leave together
            if (fail) break;
#pragma unroll
            for (int c = 0; c < PC; ++c) {
                float v[32];
                if (i == 0) {
#pragma unroll
                    for (int j = 0; j < 32; j += 4) {  // a caller's state may start at any float
                        const float* src = p.c0 + crow + c * 32 + j;
                        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (c0_whole) x = *reinterpret_cast<const float4*>(src);
                        else if (p.c0) x = make_float4(src[0], src[1], src[2], src[3]);
                        v[j] = x.x; v[j + 1] = x.y; v[j + 2] = x.z; v[j + 3] = x.w;
                    }
                } else {
                    tmem_ld32(t0 + c * 32, v);
                    tmem_ld_wait();
                }
                if (rec) {
                    const int col = half * HC + c * 32;
                    unsigned char* box = sm + S::rec + (col >> 6) * kBox;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        uint4 k;
                        k.x = pack_bf16(v[8 * q], v[8 * q + 1]); k.y = pack_bf16(v[8 * q + 2], v[8 * q + 3]);
                        k.z = pack_bf16(v[8 * q + 4], v[8 * q + 5]); k.w = pack_bf16(v[8 * q + 6], v[8 * q + 7]);
                        *reinterpret_cast<uint4*>(box + swz(row, ((col & 63) >> 3) + q)) = k;
                    }
                }
                if (last) {
                    if (p.oC)
#pragma unroll
                        for (int j = 0; j < 32; j += 4) *reinterpret_cast<float4*>(p.oC + crow + c * 32 + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                } else {
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] *= g;
                    tmem_st32(t0 + c * 32, v);
                }
            }
            if (!last) tmem_st_wait();
            if (rec) {
                fence_async_smem();
                named_barrier(1, kStateThreads);
                if (tid == 0) {
                    const int y = (bh * p.entries + (last ? p.NC : ck)) * p.D + vi * 128;
                    tma_store_4d(&p.trec, sm + S::rec, 0, y, qi * NT >> 6, 0);
                    tma_store_commit();
                }
            }
            if (!last) {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(sready);
            }
        }
        if (tid == 0) tma_store_wait_all();
    }
    if (fail && lane == 0) atomicCAS(p.status, 0, 501);
    tc_fence_before();
    __syncthreads();
    if (warp == 17) {
        tc_fence_after();
        tmem_dealloc(tC, NT < 32 ? 32 : NT);
    }
}

template <int NT, bool BWD>
static int scan_run(cudaStream_t st, const ScanP& p, int ctas) {
    static std::atomic<uint64_t> done{0};
    int dev = 0;
    XL_CUDA(cudaGetDevice(&dev));
    const size_t smem = ScanS<NT>::total + 1024;
    if (!(done.load(std::memory_order_acquire) >> (dev & 63) & 1)) {
        XL_CUDA(cudaFuncSetAttribute(par_scan<NT, BWD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        done.fetch_or(1ull << (dev & 63), std::memory_order_release);
    }
    par_scan<NT, BWD><<<ctas, kScanThreads, smem, st>>>(p);
    XL_LAUNCH_OK("par_scan");
    return XLSTM_OK;
}

int scan_launch(cudaStream_t st, const ScanArgs& a) {
    ScanP p = {};
    if (a.NC > kMaxChunks) { set_error("mlstm: %d chunks exceed the state kernel's %d", a.NC, kMaxChunks); return XLSTM_DECLINED; }
    p.status = tc_status_ptr();
    if (!p.status) return XLSTM_ERR_CUDA;
    p.w = a.w; p.g = a.g; p.c0 = a.c0; p.n0 = a.n0; p.recn = a.recn; p.oC = a.oC; p.on = a.on;
    p.H = a.H; p.T = a.T; p.D = a.D; p.NC = a.NC; p.Tp = a.NC * LC; p.entries = a.entries;
    p.nv = a.D / 128;
    // columns per CTA: the narrowest block whose launch is still one wave (a narrow block's state pass and products are shorter, but
    // every block reads all of X), else the widest
    int nt = 64;
    while (nt < a.D && a.B * a.H * p.nv * (a.D / nt) > sm_count()) nt *= 2;
    p.nt = a.D / nt;
    if (!tc_make_map4(&p.tx, a.x, 2, a.B, a.T, a.H * a.D, 64, 2) || !tc_make_map4(&p.ty, a.y, 2, a.B, a.T, a.H * a.D, 64, nt / 64) ||
        !tc_make_map4(&p.trec, a.recC, 2, 1, (uint64_t)a.B * a.H * a.entries * a.D, a.D, 128, nt / 64)) {
        set_error("mlstm: cuTensorMapEncodeTiled failed");
        return XLSTM_ERR_CUDA;
    }
    const int ctas = a.B * a.H * p.nv * p.nt;
    if (a.bwd) return nt == 64 ? scan_run<64, true>(st, p, ctas) : nt == 128 ? scan_run<128, true>(st, p, ctas) : scan_run<256, true>(st, p, ctas);
    return nt == 64 ? scan_run<64, false>(st, p, ctas) : nt == 128 ? scan_run<128, false>(st, p, ctas) : scan_run<256, false>(st, p, ctas);
}

}  // namespace par
}  // namespace xl
