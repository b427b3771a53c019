// Chunk-parallel mLSTM, part 2: the outputs of every chunk from its entering state.
//
//   S = Q K^T ; P = Dbar . S ; y = (P V + b (Q C^T)) / psi ; psi = max(|rowsum(P) + b q.n|, exp(-m))
//
// A unit is (head, chunk of 128 positions, 128 of the head's v columns); a persistent CTA per SM takes them in turn. Every operand
// is a 128 x 128 pair of tiles streamed by TMA through one ring (the loads of the next unit run while this one is in its
// epilogues); accumulators are position-major (lane = position), so row sums stay inside a thread. q.n comes out of the tensor core
// too: n is split into three bf16 terms (its full 24 bits) as rows of one more operand. HBM traffic is what bounds it: q, k, v, the
// record entry and y once each.
#include "mlstm_par.cuh"

namespace xl {
namespace par {

#define PAR_WAIT(bar, par) do { if (!mbar_wait(bar, par)) { fail = true; } } while (0)

struct OutP {
    CUtensorMap tq, tk, tv, tc, ty;
    Vecs v;
    const float *recn, *m;
    float *psiv, *qnv;
    int H, T, NC, units;
    int* status;
};
struct OutS {
    static constexpr int R = 4;                       // pairs
    static constexpr uint32_t P = R * kPair;           // 2 boxes
    static constexpr uint32_t Y = P + 2 * kBox;       // 2 boxes
    static constexpr uint32_t nt = Y + 2 * kBox;      // up to 4 x 2 KB: n as rows 0..2 of [16][64]
    static constexpr uint32_t colt = nt + 8192;       // [2][128]: units in turn
    static constexpr uint32_t rsum = colt + 1024;     // row sums [4][128]
    static constexpr uint32_t bars = rsum + 2048;
    static constexpr uint32_t total = bars + 256;
};

static constexpr int kOutEpi = 512, kOutThreads = kOutEpi + 64;

template <int NS>
__global__ void __launch_bounds__(kOutThreads, 1) par_out(const __grid_constant__ OutP p) {
    constexpr int D = NS * 128;
    extern __shared__ unsigned char raw[];
    unsigned char* sm = (unsigned char*)(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
    float* colt = (float*)(sm + OutS::colt);
    float* rsum = (float*)(sm + OutS::rsum);
    uint64_t* full = (uint64_t*)(sm + OutS::bars);
    uint64_t *empty = full + OutS::R, *nready = empty + OutS::R, *she = nready + 1, *pready = she + 1, *hi = pready + 1, *hfree = hi + 1;
    uint32_t* slot = (uint32_t*)(hfree + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    bool fail = false;
    if (tid == 0) {
        for (int i = 0; i < OutS::R; ++i) { mbar_init(full + i, 1); mbar_init(empty + i, 1); }
        mbar_init(nready, 16); mbar_init(she, 1); mbar_init(pready, 16); mbar_init(hi, 1); mbar_init(hfree, 16);
        fence_mbar_init();
    }
    for (int i = tid; i < 8192 / 16; i += kOutThreads) reinterpret_cast<uint4*>(sm + OutS::nt)[i] = make_uint4(0, 0, 0, 0);
    if (warp == 17) tmem_alloc(slot, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tS = *slot, tHe = tS + 128, tHi = tS + 256, tN = tS + 384;

    if (warp == 16) {
        if (lane == 0) {
            const uint32_t ring = smem_u32(sm), fb = smem_u32(full);
            int n = 0;
            auto pair = [&](const CUtensorMap* m, int y, int x, int z) {
                const int s = n & 3;
                if (n >= OutS::R && !fail) PAR_WAIT(empty + s, ((n >> 2) - 1) & 1);
                if (fail) return;
                mbar_expect_tx(full + s, kPair);
                tma_load_4d(ring + s * kPair, m, fb + 8 * s, 0, y, x, z);
                ++n;
            };
            for (int u = blockIdx.x; u < p.units && !fail; u += gridDim.x) {
                int bh, ck, f;
                unit_of(u, NS, p.NC, bh, ck, f);
                const int b = bh / p.H, x = (bh - b * p.H) * (D / 64), t0 = ck * LC, crow = (bh * (p.NC + 1) + ck) * D + f * 128;
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    pair(&p.tq, t0, x + 2 * s, b);
                    pair(&p.tk, t0, x + 2 * s, b);
                    pair(&p.tc, crow, 2 * s, 0);
                }
                pair(&p.tv, t0, x + 2 * f, b);
            }
            if (fail) ring_landed<OutS::R>(full, n);
        }
        __syncwarp();
    } else if (warp == 17) {
        const uint32_t ring = smem_u32(sm);
        const uint64_t rK = desc_at(smem_desc(0, 16, 1024), ring), rM = desc_at(smem_desc(0, kBox, 1024), ring);  // ring as K-major / MN-major
        const uint64_t dP = rK + (OutS::P >> 4), dN = rK + (OutS::nt >> 4);
        constexpr uint32_t id_kk = instr_desc(128, 128, 0, 0), id_n = instr_desc(128, 16, 0, 0), id_km = instr_desc(128, 128, 0, 1);
        int n = 0, it = 0;
        auto at = [&](int k) { return (uint64_t)(((n + k) & 3) * (kPair >> 4)); };
        auto ready = [&](int k) { PAR_WAIT(full + ((n + k) & 3), ((n + k) >> 2) & 1); };
        for (int u = blockIdx.x; u < p.units && !fail; u += gridDim.x, ++it) {
            if (it) PAR_WAIT(hfree, (it - 1) & 1);
            PAR_WAIT(nready, it & 1);
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                ready(0); ready(1);
                tc_fence_after();
                if (!fail) {
                    product<8, false, false>(tS, rK + at(0), rK + at(1), id_kk, s == 0);
                    product<4, false, false>(tN, rK + at(0), dN + s * 256, id_n, s == 0);
                    product<4, false, false>(tN, rK + at(0) + (kBox >> 4), dN + s * 256 + 128, id_n, false);
                }
                ready(2);
                if (!fail) product<8, false, false>(tHe, rK + at(0), rK + at(2), id_kk, s == 0);
                for (int k = 0; k < 3; ++k, ++n) mma_commit_w(empty + (n & 3));
            }
            if (fail) break;
            mma_commit_w(she);
            ready(0);
            PAR_WAIT(pready, it & 1);
            if (fail) break;
            tc_fence_after();
            product<8, false, true>(tHi, dP, rM + at(0), id_km, true);
            mma_commit_w(hi);
            mma_commit_w(empty + (n & 3));
            ++n;
        }
    } else {
        // ---- epilogues: thread = position, a quarter of the columns ----
        const int qd = warp & 3, qt = warp >> 2, row = 32 * qd + lane;
        const uint32_t lb = ((uint32_t)(32 * qd) << 16) + 32 * qt;
        constexpr float kLog2e = 1.4426950408889634f;
        auto put = [&](unsigned char* pair, const float* v) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                uint4 k;
                k.x = pack_bf16(v[8 * q], v[8 * q + 1]); k.y = pack_bf16(v[8 * q + 2], v[8 * q + 3]);
                k.z = pack_bf16(v[8 * q + 4], v[8 * q + 5]); k.w = pack_bf16(v[8 * q + 6], v[8 * q + 7]);
                *reinterpret_cast<uint4*>(pair + (qt >> 1) * kBox + swz(row, 4 * (qt & 1) + q)) = k;
            }
        };
        // a unit's vectors, fetched while the unit before it is in its products
        float rt = 0.f, bt = 0.f, mt = 0.f, ct = 0.f, nx = 0.f;
        auto fetch = [&](int u) {
            int bh, ck, f;
            unit_of(u, NS, p.NC, bh, ck, f);
            const int t = ck * LC + row;
            const size_t vo = (size_t)bh * p.v.Tp + t;
            rt = p.v.rowt[vo] * kLog2e;
            bt = p.v.b[vo];
            mt = p.m[(size_t)bh * p.T + min(t, p.T - 1)];
            if (tid < LC) ct = p.v.colt[(size_t)bh * p.v.Tp + ck * LC + tid] * kLog2e;
            if (tid < D) nx = p.recn[((size_t)bh * (p.NC + 1) + ck) * D + tid];
        };
        int it = 0;
        if ((int)blockIdx.x < p.units) fetch(blockIdx.x);
        for (int u = blockIdx.x; u < p.units; u += gridDim.x, ++it) {
            int bh, ck, f;
            unit_of(u, NS, p.NC, bh, ck, f);
            const int t = ck * LC + row;
            float* ctv = colt + (it & 1) * 128;
            const float rt_ = rt, bt_ = bt, mt_ = mt;
            if (tid < LC) ctv[tid] = ct;
            if (tid < D) {
                const bf16 h0 = __float2bfloat16_rn(nx);
                const float r1 = nx - __bfloat162float(h0);
                const bf16 h1 = __float2bfloat16_rn(r1), h2 = __float2bfloat16_rn(r1 - __bfloat162float(h1));
                unsigned char* d = sm + OutS::nt + (tid >> 6) * 2048 + (tid & 7) * 2;
                *reinterpret_cast<bf16*>(d + swz(0, (tid & 63) >> 3)) = h0;
                *reinterpret_cast<bf16*>(d + swz(1, (tid & 63) >> 3)) = h1;
                *reinterpret_cast<bf16*>(d + swz(2, (tid & 63) >> 3)) = h2;
            }
            fence_async_smem();
            fail = named_barrier_or(1, kOutEpi, fail);  // the warps of this role leave together
            if (fail) break;
            if (lane == 0) mbar_arrive(nready);
            if (u + (int)gridDim.x < p.units) fetch(u + gridDim.x);
            PAR_WAIT(she, it & 1);
            tc_fence_after();
            float nq[8], s[32], sum = 0.f;
            tmem_ld8(tN + ((uint32_t)(32 * qd) << 16), nq);
            if (qt <= qd) {
                const int j0 = 32 * qt;
                tmem_ld32(tS + lb, s);
                tmem_ld_wait();
#pragma unroll
                for (int i4 = 0; i4 < 8; ++i4) {
                    const float4 c4 = *reinterpret_cast<const float4*>(ctv + j0 + 4 * i4);
                    const float cc[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int i = 4 * i4 + e;
                        float dbar;
                        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(dbar) : "f"(j0 + i <= row ? rt_ + cc[e] : -INFINITY));
                        s[i] *= dbar;
                        sum += s[i];
                    }
                }
            } else {
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 32; ++i) s[i] = 0.f;
            }
            put(sm + OutS::P, s);
            rsum[qt * 128 + row] = sum;
            fence_async_smem();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(pready);
            if (tid == 0) tma_store_wait_read();  // the previous tile has left the staging buffer
            fail = named_barrier_or(1, kOutEpi, fail);
            if (fail) break;
            const float qn = ((rsum[row] + rsum[128 + row]) + (rsum[256 + row] + rsum[384 + row])) + bt_ * ((nq[2] + nq[1]) + nq[0]);
            const float psi = fmaxf(fabsf(qn), expf(-mt_)), ip = 1.f / psi, bp = bt_ * ip;
            if (f == 0 && qt == 0 && t < p.T) {
                p.psiv[(size_t)bh * p.T + t] = psi;
                p.qnv[(size_t)bh * p.T + t] = qn;
            }
            float e[32];
            tmem_ld32(tHe + lb, e);
            PAR_WAIT(hi, it & 1);
            tc_fence_after();
            tmem_ld32(tHi + lb, s);
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(hfree);
#pragma unroll
            for (int i = 0; i < 32; ++i) s[i] = s[i] * ip + bp * e[i];
            put(sm + OutS::Y, s);
            fence_async_smem();
            fail = named_barrier_or(1, kOutEpi, fail);
            if (fail) break;
            if (tid == 0) {
                tma_store_4d(&p.ty, sm + OutS::Y, 0, ck * LC, (bh % p.H) * (D / 64) + 2 * f, bh / p.H);
                tma_store_commit();
            }
        }
        if (tid == 0) tma_store_wait_all();
    }
    if (fail && lane == 0) atomicCAS(p.status, 0, 502);
    tc_fence_before();
    __syncthreads();
    if (warp == 17) {
        tc_fence_after();
        tmem_dealloc(tS, 512);
    }
}

template <int NS>
static int out_run(cudaStream_t st, const OutP& p) {
    static std::atomic<uint64_t> done{0};
    int dev = 0;
    XL_CUDA(cudaGetDevice(&dev));
    const size_t smem = OutS::total + 1024;
    if (!(done.load(std::memory_order_acquire) >> (dev & 63) & 1)) {
        XL_CUDA(cudaFuncSetAttribute(par_out<NS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        done.fetch_or(1ull << (dev & 63), std::memory_order_release);
    }
    par_out<NS><<<p.units < sm_count() ? p.units : sm_count(), kOutThreads, smem, st>>>(p);
    XL_LAUNCH_OK("par_out");
    return XLSTM_OK;
}

}  // namespace par

// ---- the forward through the chunk-parallel kernels ----------------------------------------------------------------------------
using namespace par;

size_t mlstm_par_saved_bytes(int B, int H, int T, int d) {
    const int NC = (T + LC - 1) / LC;
    return record_C_bytes(B * H, NC, d) + record_n_bytes(B * H, NC, d);
}
size_t mlstm_par_fw_workspace_bytes(int B, int H, int T, int d) {  // the record too, for calls that keep none
    return vecs_bytes(B * H, (T + LC - 1) / LC, false) + mlstm_par_saved_bytes(B, H, T, d);
}

int mlstm_par_fw_launch(cudaStream_t st, const MlstmFwArgs& a, void* saved, void* workspace, size_t workspace_bytes) {
    const int NC = (a.T + LC - 1) / LC, BH = a.B * a.H, d = a.dqk;
    const size_t vb = vecs_bytes(BH, NC, false), need = vb + (saved ? 0 : mlstm_par_saved_bytes(a.B, a.H, a.T, d));
    if (!workspace || workspace_bytes < need) {
        set_error("mlstm_fw: workspace of %zu B is smaller than the %zu B required", workspace_bytes, need);
        return XLSTM_ERR_WORKSPACE;
    }
    if (((uintptr_t)a.q | (uintptr_t)a.k | (uintptr_t)a.v | (uintptr_t)a.ytil | (uintptr_t)a.oC | (uintptr_t)saved | (uintptr_t)workspace) & 15) {
        set_error("mlstm_fw (tensor-core path): tensors must be 16-byte aligned");
        return XLSTM_ERR_ARG;
    }
    char* ws = (char*)workspace;
    const Vecs v = vecs_at(ws, BH, NC, false);
    if (!saved) saved = ws + vb;
    int rc = gates_launch(st, a.ig, a.fg, a.cm, a.msv, a.om, v, a.B, a.H, a.T, NC, false, a.exact && (a.cm || a.om));
    if (rc) return rc;
    ScanArgs s = {};
    s.x = a.v; s.y = a.k; s.w = v.a; s.g = v.g; s.c0 = a.cC; s.n0 = a.cn;
    s.recC = saved; s.recn = (float*)((char*)saved + record_C_bytes(BH, NC, d));
    s.oC = a.oC; s.on = a.on; s.B = a.B; s.H = a.H; s.T = a.T; s.D = d; s.NC = NC; s.entries = NC + 1; s.bwd = false;
    rc = scan_launch(st, s);
    if (rc) return rc;
    OutP p = {};
    if (!tc_make_map4(&p.tq, a.q, 2, a.B, a.T, a.H * d, 128, 2) || !tc_make_map4(&p.tk, a.k, 2, a.B, a.T, a.H * d, 128, 2) ||
        !tc_make_map4(&p.tv, a.v, 2, a.B, a.T, a.H * d, 128, 2) || !tc_make_map4(&p.ty, a.ytil, 2, a.B, a.T, a.H * d, 128, 2) ||
        !tc_make_map4(&p.tc, saved, 2, 1, (uint64_t)BH * (NC + 1) * d, d, 128, 2)) {
        set_error("mlstm_fw: cuTensorMapEncodeTiled failed");
        return XLSTM_ERR_CUDA;
    }
    p.v = v; p.recn = s.recn; p.m = a.msv; p.psiv = a.psiv; p.qnv = a.qnv; p.H = a.H; p.T = a.T; p.NC = NC; p.units = BH * NC * (d / 128);
    p.status = tc_status_ptr();
    if (!p.status) return XLSTM_ERR_CUDA;
    return d == 128 ? out_run<1>(st, p) : out_run<2>(st, p);
}

}  // namespace xl
