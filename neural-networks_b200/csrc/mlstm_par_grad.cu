// Chunk-parallel mLSTM, part 3: the backward.
//
//   par_dn         dN = dy / psi, b.dN (bf16), dqn and b dqn per position: one pass over dy and y
//   par_scan       dC right to left with a record at the chunk borders (mlstm_par_scan.cu)
//   par_grad       per chunk: S, dds -> DS, dS -> dQ, dK, dV and the row dots dq.q, dk.k
//   par_gate_grad  suffix sums of dq.q - dk.k over the sequence -> gate gradients
#include "mlstm_par.cuh"

namespace xl {
namespace par {

#define PAR_WAIT(bar, par) do { if (!mbar_wait(bar, par)) { fail = true; } } while (0)

// ---- dN: a warp per (position, head) ---------------------------------------------------------------------------------------------
struct DnArgs {
    const void* dy;
    const bf16* ytil;
    const float *psiv, *qnv, *m;
    Vecs v;
    bf16 *dn, *dnb;
    int B, H, T;
};
template <typename GT, int NS>
__global__ void __launch_bounds__(256) par_dn(const DnArgs p) {
    constexpr int D = NS * 128, V = NS;  // 4-value pieces per lane
    const int lane = threadIdx.x & 31;
    const long long row = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);  // (b * Tp + t) * H + h, Tp padded to whole chunks
    const int h = (int)(row % p.H), t = (int)(row / p.H % p.v.Tp), b = (int)(row / p.H / p.v.Tp);
    if (b >= p.B) return;
    const size_t bh = (size_t)b * p.H + h, vo = bh * p.v.Tp + t;
    if (t >= p.T) {
        if (lane == 0) p.v.dqn[vo] = p.v.bq[vo] = 0.f;
        return;
    }
    const size_t o = (((size_t)b * p.T + t) * p.H + h) * D + lane * 4, so = bh * p.T + t;
    float d[V][4], dot = 0.f;
#pragma unroll
    for (int i = 0; i < V; ++i) {
        if (sizeof(GT) == 4) {
            const float4 x = __ldcs(reinterpret_cast<const float4*>((const float*)p.dy + o + i * 128));
            d[i][0] = x.x; d[i][1] = x.y; d[i][2] = x.z; d[i][3] = x.w;
        } else {
            const uint2 x = __ldcs(reinterpret_cast<const uint2*>((const bf16*)p.dy + o + i * 128));
            const float2 lo = unpack_bf16(x.x), hi = unpack_bf16(x.y);
            d[i][0] = lo.x; d[i][1] = lo.y; d[i][2] = hi.x; d[i][3] = hi.y;
        }
        const uint2 y = __ldcs(reinterpret_cast<const uint2*>(p.ytil + o + i * 128));
        const float2 lo = unpack_bf16(y.x), hi = unpack_bf16(y.y);
        dot += d[i][0] * lo.x + d[i][1] * lo.y + d[i][2] * hi.x + d[i][3] * hi.y;
    }
    const float psi = p.psiv[so], qn = p.qnv[so], mt = p.m[so], bt = p.v.b[vo];
    dot = warp_sum(dot);
    const float ip = 1.f / psi;
#pragma unroll
    for (int i = 0; i < V; ++i) {
        uint2 a, c;
        const float e0 = d[i][0] * ip, e1 = d[i][1] * ip, e2 = d[i][2] * ip, e3 = d[i][3] * ip;
        a.x = pack_bf16(e0, e1); a.y = pack_bf16(e2, e3);
        c.x = pack_bf16(e0 * bt, e1 * bt); c.y = pack_bf16(e2 * bt, e3 * bt);
        *reinterpret_cast<uint2*>(p.dn + o + i * 128) = a;
        *reinterpret_cast<uint2*>(p.dnb + o + i * 128) = c;
    }
    if (lane == 0) {
        // dqn_t = sign(qn) (-dot / psi) where the q.n term, not the floor, set psi
        const float r = fabsf(qn) > expf(-mt) ? (qn > 0.f ? -1.f : 1.f) * dot / psi : 0.f;
        p.v.dqn[vo] = r;
        p.v.bq[vo] = bt * r;
    }
}

// ---- gate gradients: one CTA per head ------------------------------------------------------------------------------------------------
// d(i)_t = dk.k ; d(f)_t = (sum_{r >= t} (dq.q - dk.k)_r + <dC_in, C_end> + dn_in . n_end) (1 - sigmoid(f_t))
struct GgArgs {
    const float *pu, *pw;             // [planes][BH][Tp]: the row dots over 32 columns each
    const float *fg, *cdC, *cdn, *recn;
    const bf16* recC;
    float *dig, *dfg;
    int BH, H, T, Tp, NC, D, planes;
};
__global__ void __launch_bounds__(1024) par_gate_grad(const GgArgs p) {
    __shared__ float red[32], wsum[32];
    const int bh = blockIdx.x, b = bh / p.H, h = bh % p.H, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    float run = 0.f;
    if (p.cdC) {
        const size_t DD = (size_t)p.D * p.D;
        const bf16* Ce = p.recC + ((size_t)bh * (p.NC + 1) + p.NC) * DD;
        float acc = 0.f;
        for (size_t i = (size_t)tid * 4; i < DD; i += 4096) {
            const float* x = p.cdC + bh * DD + i;  // the caller's: aligned to a float and no more
            const uint2 c = *reinterpret_cast<const uint2*>(Ce + i);
            const float2 lo = unpack_bf16(c.x), hi = unpack_bf16(c.y);
            acc += x[0] * lo.x + x[1] * lo.y + x[2] * hi.x + x[3] * hi.y;
        }
        if (tid < p.D) acc += p.cdn[(size_t)bh * p.D + tid] * p.recn[((size_t)bh * (p.NC + 1) + p.NC) * p.D + tid];
        run = block_sum(acc, red);
    }
    // 1024 positions at a time from the right, the suffix sum running on
    for (int base = (p.T - 1) / 1024 * 1024; base >= 0; base -= 1024) {
        const int t = base + tid;
        float u = 0.f, k = 0.f;
        if (t < p.T)
            for (int f = 0; f < p.planes; ++f) {
                u += p.pu[((size_t)f * p.BH + bh) * p.Tp + t];
                k += p.pw[((size_t)f * p.BH + bh) * p.Tp + t];
            }
        float s = u - k;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float y = __shfl_down_sync(0xffffffffu, s, o);
            if (lane + o < 32) s += y;
        }
        __syncthreads();
        if (lane == 0) wsum[w] = s;
        __syncthreads();
        float behind = 0.f, all = 0.f;
        for (int i = 31; i >= 0; --i) {
            if (i == w) behind = all;
            all += wsum[i];
        }
        if (t < p.T) {
            const size_t gi = ((size_t)b * p.T + t) * p.H + h;
            p.dfg[gi] = (run + behind + s) * (1.f - stable_sigmoid(p.fg[gi]));
            p.dig[gi] = k;
        }
        run += all;
    }
}

// ---- gradients of one chunk -----------------------------------------------------------------------------------------------------------
// A unit is (head, chunk of 128 positions, 128 of the head's columns f): dq and dk of the qk columns f, dv of the v columns f. All
// operands are 128 x 128 pairs of tiles streamed through one ring of four (TMA, running ahead of the products and across units); the
// ones needed twice come from L2 again, which leaves room for DS and dS. Both single threads on the path count: issuing a load costs
// some 500 cycles (with 16 KB boxes a unit's 22 loads took 11 k), a tensor-core instruction 60 to 85 whatever its N. 8 x 8 heads of 256, 4096
// positions: 558 us, 2.55 GB through L2 to the SMs (4.6 TB/s), the tensor pipe active 18 %: the chain of a unit's roles bounds it.
// Accumulators (tensor memory, four regions of 128 columns, lane = position):
//   R0: S, then dQ = b.dN C + dS K, then DS^T dN     R1: K dC^T     R2: dds, then dS^T Q     R3: V dC
// Epilogues in the order dQ, dK, dV: the K and Q pairs, from which dk.k and dq.q are taken, leave the ring before the last of them, so
// the next unit's first operands arrive under it.
// At heads of 256 the scores are formed by both halves: a fifth of the products, instead of partial planes in HBM.
struct GradP {
    CUtensorMap tq, tk, tv, tdn, tdnb, tc, tdc, tdq, tdk, tdv;
    Vecs v;
    const float *recn, *recdn;  // n entering [BH][NC+1][D], dn leaving [BH][NC][D]
    float *pu, *pw;
    int BH, H, T, NC, units;
    int* status;
};
// bf16 gradients are staged in DS and dS once their products are done; an fp32 tile (64 KB) takes a buffer of its own beside DS, at the
// price of the ring's fifth pair.
template <typename OT>
struct GradS {
    static constexpr int R = sizeof(OT) == 4 ? 4 : 5;  // pairs
    static constexpr uint32_t DS = R * kPair;
    static constexpr uint32_t ST = DS + kPair;         // fp32: with dS behind it dQ's and dK's tile, with DS before it dV's
    static constexpr uint32_t dS = ST + (sizeof(OT) == 4 ? kPair : 0);
    static constexpr uint32_t vec = dS + kPair;        // colt | n | dn, 128 each
    static constexpr uint32_t bars = vec + 3 * 512;
    static constexpr uint32_t total = bars + 256;
};
// A place in a ring of R slots: slot and the parity of its current use.
template <int R>
struct Place {
    int s = 0, ph = 0;
    __device__ __forceinline__ Place ahead(int k) const { Place q; q.s = s + k >= R ? s + k - R : s + k; q.ph = s + k >= R ? ph ^ 1 : ph; return q; }
    __device__ __forceinline__ void next() { if (++s == R) { s = 0; ph ^= 1; } }
};
static constexpr int kGradEpi = 512, kGradThreads = kGradEpi + 64;

template <int NS, typename OT>
__global__ void __launch_bounds__(kGradThreads, 1) par_grad(const __grid_constant__ GradP p) {
    constexpr int D = NS * 128, NB = 8 * NS + 3, oK = NB - 3;  // pairs per unit; K, Q and dN are the last three
    typedef GradS<OT> Sh;
    constexpr int R = Sh::R;
    extern __shared__ unsigned char raw[];
    unsigned char* sm = (unsigned char*)(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
    float* colt = (float*)(sm + Sh::vec);
    float *sn = colt + 128, *sdn = colt + 256;
    uint64_t* full = (uint64_t*)(sm + Sh::bars);
    uint64_t *empty = full + R, *sdp = empty + R, *dsr = sdp + 1, *vr = sdp + 2, *qr = sdp + 3, *kr = sdp + 4, *vfree = sdp + 5,
             *qfree = sdp + 6, *kfree = sdp + 7, *pdone = sdp + 8;
    uint32_t* slot = (uint32_t*)(sdp + 9);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    bool fail = false;
    if (tid == 0) {
        for (int i = 0; i < R; ++i) { mbar_init(full + i, 1); mbar_init(empty + i, 1); }
        mbar_init(sdp, 1); mbar_init(vr, 1); mbar_init(qr, 1); mbar_init(kr, 1);
        mbar_init(dsr, 16); mbar_init(vfree, 16); mbar_init(qfree, 16); mbar_init(kfree, 16); mbar_init(pdone, 16);
        fence_mbar_init();
    }
    if (warp == 17) tmem_alloc(slot, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t R0 = *slot, R1 = R0 + 128, R2 = R0 + 256, R3 = R0 + 384;

    if (warp == 16) {
        // ---- loads: the order in which the products take the boxes ----
        if (lane == 0) {
            const uint32_t ring = smem_u32(sm), fb = smem_u32(full);
            uint32_t phases = 0;  // parity of the next completion of each slot's empty barrier
            int n = 0, it = 0;
            Place<R> at;
            // pair i of a unit. Its slot was last a pair of the products, or (two pairs of every unit but the first) the K or Q pair
            // of the unit before, which the epilogue gives back.
            auto pair = [&](int i, const CUtensorMap* m, int y, int x, int z) {
                const int s = at.s;
                if (fail) return;
                if ((i == R - 3 || i == R - 2) && it) PAR_WAIT(pdone, (it - 1) & 1);
                else if (n >= R) { PAR_WAIT(empty + s, (phases >> s) & 1); phases ^= 1u << s; }
                if (fail) return;
                mbar_expect_tx(full + s, kPair);
                tma_load_4d(ring + s * kPair, m, fb + 8 * s, 0, y, x, z);
                ++n;
                at.next();
            };
            for (int u = blockIdx.x; u < p.units && !fail; u += gridDim.x, ++it) {
                int bh, ck, f;
                unit_of(u, NS, p.NC, bh, ck, f);
                const int b = bh / p.H, x = (bh - b * p.H) * (D / 64), t0 = ck * LC;
                const int crow = (bh * (p.NC + 1) + ck) * D, drow = (bh * p.NC + ck) * D;
                int i = 0;
#pragma unroll
                for (int s = 0; s < NS; ++s) {  // S, K dC^T
                    pair(i++, &p.tq, t0, x + 2 * s, b);
                    pair(i++, &p.tk, t0, x + 2 * s, b);
                    pair(i++, &p.tdc, drow + f * 128, 2 * s, 0);
                }
#pragma unroll
                for (int v = 0; v < NS; ++v) {  // dds, V dC
                    pair(i++, &p.tdn, t0, x + 2 * v, b);
                    pair(i++, &p.tv, t0, x + 2 * v, b);
                    pair(i++, &p.tdc, drow + v * 128, 2 * f, 0);
                }
#pragma unroll
                for (int v = 0; v < NS; ++v) {  // b.dN C
                    pair(i++, &p.tdnb, t0, x + 2 * v, b);
                    pair(i++, &p.tc, crow + v * 128, 2 * f, 0);
                }
                pair(i++, &p.tk, t0, x + 2 * f, b);   // dS K; kept for dk.k
                pair(i++, &p.tq, t0, x + 2 * f, b);   // dS^T Q; kept for dq.q
                pair(i++, &p.tdn, t0, x + 2 * f, b);  // DS^T dN
            }
            if (fail) ring_landed<R>(full, n);
        }
        __syncwarp();
    } else if (warp == 17) {
        // ---- products ----
        const uint32_t ring = smem_u32(sm);
        const uint64_t rK = desc_at(smem_desc(0, 16, 1024), ring), rM = desc_at(smem_desc(0, kBox, 1024), ring);  // ring as K-major / MN-major
        constexpr uint32_t id_kk = instr_desc(128, 128, 0, 0), id_km = instr_desc(128, 128, 0, 1), id_mm = instr_desc(128, 128, 1, 1);
        constexpr uint32_t oDS = Sh::DS >> 4, odS = Sh::dS >> 4;
        int it = 0;
        Place<R> pl;
        auto at = [&](int k) { return (uint64_t)(pl.ahead(k).s * (kPair >> 4)); };
        auto ready = [&](int k) { const Place<R> q = pl.ahead(k); PAR_WAIT(full + q.s, q.ph); };
        auto release = [&](int k) { for (int i = 0; i < k; ++i) { mma_commit_w(empty + pl.s); pl.next(); } };
        for (int u = blockIdx.x; u < p.units && !fail; u += gridDim.x, ++it) {
            if (it) PAR_WAIT(vfree, (it - 1) & 1);
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                ready(0); ready(1);
                tc_fence_after();
                if (!fail) product<8, false, false>(R0, rK + at(0), rK + at(1), id_kk, s == 0);
                release(1);
                ready(1);
                if (!fail) product<8, false, false>(R1, rK + at(0), rK + at(1), id_kk, s == 0);
                release(2);
            }
            if (it) PAR_WAIT(kfree, (it - 1) & 1);
#pragma unroll
            for (int v = 0; v < NS; ++v) {
                ready(0); ready(1);
                tc_fence_after();
                if (!fail) product<8, false, false>(R2, rK + at(0), rK + at(1), id_kk, v == 0);
                if (v == NS - 1) mma_commit_w(sdp);  // S and dds are complete: their epilogue runs beside V dC
                release(1);
                ready(1);
                if (!fail) product<8, false, true>(R3, rK + at(0), rM + at(1), id_km, v == 0);
                release(2);
            }
            PAR_WAIT(dsr, it & 1);  // DS and dS are in shared memory, R0 and R2 have been read
#pragma unroll
            for (int v = 0; v < NS; ++v) {
                ready(0); ready(1);
                tc_fence_after();
                if (!fail) product<8, false, true>(R0, rK + at(0), rM + at(1), id_km, v == 0);
                release(2);
            }
            ready(0);
            if (fail) break;
            product<8, false, true>(R0, rK + odS, rM + at(0), id_km, false);
            mma_commit_w(qr);
            ready(1);
            if (fail) break;
            product<8, true, true>(R2, rM + odS, rM + at(1), id_mm, true);
            mma_commit_w(kr);
            pl = pl.ahead(2);  // the K and Q pairs are released by the epilogue, which takes the row dots from them
            ready(0);
            PAR_WAIT(qfree, it & 1);
            if (fail) break;
            tc_fence_after();
            product<8, true, true>(R0, rM + oDS, rM + at(0), id_mm, true);
            mma_commit_w(vr);
            release(1);
        }
    } else {
        // ---- epilogues: thread = position, a quarter of the columns ----
        const int qd = warp & 3, qt = warp >> 2, row = 32 * qd + lane;
        const uint32_t lb = ((uint32_t)(32 * qd) << 16) + 32 * qt;
        // A 128 x 128 output tile (32 columns of it in v) through shared memory and TMA: two staged tiles of bf16, four of fp32.
        auto store_tile = [&](const CUtensorMap* m, uint32_t at, int x, int t0, int b, const float* v) {
            if (tid == 0) tma_store_wait_read();  // what was staged before has left
            named_barrier(1, kGradEpi);
            if (sizeof(OT) == 4) {
                unsigned char* box = sm + at + qt * kBox;         // [128 rows][32 fp32]
#pragma unroll
                for (int q = 0; q < 8; ++q) *reinterpret_cast<float4*>(box + swz(row, q)) = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
            } else {
                unsigned char* box = sm + at + (qt >> 1) * kBox;  // [128 rows][64 bf16]
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    uint4 k;
                    k.x = pack_bf16(v[8 * q], v[8 * q + 1]); k.y = pack_bf16(v[8 * q + 2], v[8 * q + 3]);
                    k.z = pack_bf16(v[8 * q + 4], v[8 * q + 5]); k.w = pack_bf16(v[8 * q + 6], v[8 * q + 7]);
                    *reinterpret_cast<uint4*>(box + swz(row, 4 * (qt & 1) + q)) = k;
                }
            }
            fence_async_smem();
            named_barrier(1, kGradEpi);
            if (tid == 0) {
                tma_store_4d(m, sm + at, 0, t0, x, b);
                tma_store_commit();
            }
        };
        // v . (this thread's 32 columns of its row) of pair number n of the ring's sequence
        auto dot_row = [&](int n, const float* v) {
            PAR_WAIT(full + n % R, (n / R) & 1);
            const unsigned char* tile = sm + (n % R) * kPair + (qt >> 1) * kBox;
            float a = 0.f;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint4 x = *reinterpret_cast<const uint4*>(tile + swz(row, 4 * (qt & 1) + q));
                const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 e = unpack_bf16(w[j]);
                    a = fmaf(v[8 * q + 2 * j], e.x, a);
                    a = fmaf(v[8 * q + 2 * j + 1], e.y, a);
                }
            }
            return a;
        };
        auto arrive = [&](uint64_t* bar) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar);
        };
        constexpr float kLog2e = 1.4426950408889634f;
        int it = 0;
        for (int u = blockIdx.x; u < p.units; u += gridDim.x, ++it) {
            int bh, ck, f;
            unit_of(u, NS, p.NC, bh, ck, f);
            const int b = bh / p.H, h = bh % p.H, t0 = ck * LC, t = t0 + row, x = (h * D + f * 128) * (int)sizeof(OT) / 128;
            const size_t vo = (size_t)bh * p.v.Tp + t;
            const float rt = p.v.rowt[vo] * kLog2e, at = p.v.a[vo], dq_t = p.v.dqn[vo], bq_t = p.v.bq[vo];
            if (tid < 128) colt[tid] = p.v.colt[(size_t)bh * p.v.Tp + t0 + tid] * kLog2e;
            else if (tid < 256) sn[tid - 128] = p.recn[((size_t)bh * (p.NC + 1) + ck) * D + f * 128 + tid - 128];
            else if (tid < 384) sdn[tid - 256] = p.recdn[((size_t)bh * p.NC + ck) * D + f * 128 + tid - 256];
            if (tid == 0) tma_store_wait_read();  // the last tile of the unit before has left the dS buffer
            fail = named_barrier_or(1, kGradEpi, fail);  // the warps of this role leave together
            if (fail) break;
            PAR_WAIT(sdp, it & 1);
            tc_fence_after();
            {
                float s[32], dd[32];
                const int j0 = 32 * qt;
                if (qt <= qd) {
                    tmem_ld32(R0 + lb, s);
                    tmem_ld32(R2 + lb, dd);
                    tmem_ld_wait();
#pragma unroll
                    for (int i4 = 0; i4 < 8; ++i4) {
                        const float4 c4 = *reinterpret_cast<const float4*>(colt + j0 + 4 * i4);
                        const float cc[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const int i = 4 * i4 + e;
                            float dbar;
                            asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(dbar) : "f"(j0 + i <= row ? rt + cc[e] : -INFINITY));
                            s[i] *= dbar;
                            dd[i] = dbar * (dd[i] + dq_t);
                        }
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 32; ++i) s[i] = dd[i] = 0.f;
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    uint4 k, l;
                    k.x = pack_bf16(s[8 * q], s[8 * q + 1]); k.y = pack_bf16(s[8 * q + 2], s[8 * q + 3]);
                    k.z = pack_bf16(s[8 * q + 4], s[8 * q + 5]); k.w = pack_bf16(s[8 * q + 6], s[8 * q + 7]);
                    l.x = pack_bf16(dd[8 * q], dd[8 * q + 1]); l.y = pack_bf16(dd[8 * q + 2], dd[8 * q + 3]);
                    l.z = pack_bf16(dd[8 * q + 4], dd[8 * q + 5]); l.w = pack_bf16(dd[8 * q + 6], dd[8 * q + 7]);
                    const uint32_t o = (qt >> 1) * kBox + swz(row, 4 * (qt & 1) + q);
                    *reinterpret_cast<uint4*>(sm + Sh::DS + o) = k;
                    *reinterpret_cast<uint4*>(sm + Sh::dS + o) = l;
                }
            }
            fence_async_smem();
            arrive(dsr);
            float v[32], e[32];
            // dQ = b.dN C + dS K + b dqn n
            PAR_WAIT(qr, it & 1);
            tc_fence_after();
            tmem_ld32(R0 + lb, v);
            tmem_ld_wait();
            arrive(qfree);
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] += bq_t * sn[32 * qt + i];
            const size_t dot_at = ((size_t)(f * 4 + qt) * p.BH + bh) * p.v.Tp + t;
            p.pu[dot_at] = dot_row(it * NB + oK + 1, v);
            PAR_WAIT(kr, it & 1);  // the products are done with dS
            store_tile(&p.tdq, Sh::ST, x, t0, b, v);
            // dK = dS^T Q + a (V dC + dn)
            tc_fence_after();
            tmem_ld32(R2 + lb, v);
            tmem_ld32(R3 + lb, e);
            tmem_ld_wait();
            arrive(kfree);
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] += at * (e[i] + sdn[32 * qt + i]);
            p.pw[dot_at] = dot_row(it * NB + oK, v);
            __syncwarp();
            if (lane == 0) mbar_arrive(pdone);
            store_tile(&p.tdk, Sh::ST, x, t0, b, v);
            // dV = DS^T dN + a K dC^T
            PAR_WAIT(vr, it & 1);
            tc_fence_after();
            tmem_ld32(R0 + lb, v);
            tmem_ld32(R1 + lb, e);
            tmem_ld_wait();
            arrive(vfree);
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] += at * e[i];
            store_tile(&p.tdv, Sh::DS, x, t0, b, v);
        }
        if (tid == 0) tma_store_wait_all();
    }
    if (fail && lane == 0) atomicCAS(p.status, 0, 503);
    tc_fence_before();
    __syncthreads();
    if (warp == 17) {
        tc_fence_after();
        tmem_dealloc(R0, 512);
    }
}

template <int NS, typename OT>
static int grad_run(cudaStream_t st, const GradP& p) {
    static std::atomic<uint64_t> done{0};
    int dev = 0;
    XL_CUDA(cudaGetDevice(&dev));
    const size_t smem = GradS<OT>::total + 1024;
    if (!(done.load(std::memory_order_acquire) >> (dev & 63) & 1)) {
        XL_CUDA(cudaFuncSetAttribute(par_grad<NS, OT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        done.fetch_or(1ull << (dev & 63), std::memory_order_release);
    }
    par_grad<NS, OT><<<p.units < sm_count() ? p.units : sm_count(), kGradThreads, smem, st>>>(p);
    XL_LAUNCH_OK("par_grad");
    return XLSTM_OK;
}
template <typename GT>
static int dn_run(cudaStream_t st, const DnArgs& p, int d) {
    const long long rows = (long long)p.B * p.v.Tp * p.H;
    const unsigned grid = (unsigned)((rows + 7) / 8);
    if (d == 128) par_dn<GT, 1><<<grid, 256, 0, st>>>(p);
    else par_dn<GT, 2><<<grid, 256, 0, st>>>(p);
    XL_LAUNCH_OK("par_dn");
    return XLSTM_OK;
}

namespace {
struct BwWs { size_t vecs, dn, dc, dnn, dots, rec, total; };
BwWs bw_ws(int B, int H, int T, int d, bool recompute) {
    const int NC = (T + LC - 1) / LC, BH = B * H;
    BwWs w;
    w.vecs = vecs_bytes(BH, NC, true);
    w.dn = align_up((size_t)B * T * H * d * 2, 256);
    w.dc = align_up((size_t)BH * NC * d * d * 2, 256);
    w.dnn = align_up((size_t)BH * NC * d * 4, 256);
    w.dots = align_up((size_t)(d / 32) * BH * NC * LC * 4, 256);
    w.rec = recompute ? record_C_bytes(BH, NC, d) + record_n_bytes(BH, NC, d) : 0;
    w.total = w.vecs + 2 * w.dn + w.dc + w.dnn + 2 * w.dots + w.rec;
    return w;
}
}  // namespace
}  // namespace par

using namespace par;

size_t mlstm_par_bw_workspace_bytes(int B, int H, int T, int d, bool recompute) { return bw_ws(B, H, T, d, recompute).total; }

// `carry_C`, `carry_n`: the state the forward entered with, for the recomputation (saved == null)
int mlstm_par_bw_launch(cudaStream_t st, const MlstmBwArgs& a, const float* carry_C, const float* carry_n, const void* saved, int gdtype,
                        void* workspace, size_t workspace_bytes) {
    const int NC = (a.T + LC - 1) / LC, BH = a.B * a.H, d = a.dqk, gb = gdtype == XLSTM_BF16 ? 2 : 4;
    const BwWs w = bw_ws(a.B, a.H, a.T, d, saved == nullptr);
    if (!workspace || workspace_bytes < w.total) {
        set_error("mlstm_bw: workspace of %zu B is smaller than the %zu B required", workspace ? workspace_bytes : 0, w.total);
        return XLSTM_ERR_WORKSPACE;
    }
    if (((uintptr_t)a.q | (uintptr_t)a.k | (uintptr_t)a.v | (uintptr_t)a.ytil | (uintptr_t)a.dytil | (uintptr_t)a.dq | (uintptr_t)a.dk |
         (uintptr_t)a.dv | (uintptr_t)a.odC | (uintptr_t)saved | (uintptr_t)workspace) & 15) {
        set_error("mlstm_bw (tensor-core path): tensors must be 16-byte aligned");
        return XLSTM_ERR_ARG;
    }
    char* ws = (char*)workspace;
    const Vecs v = vecs_at(ws, BH, NC, true);
    ws += w.vecs;
    bf16 *dn = (bf16*)ws, *dnb = (bf16*)(ws + w.dn);
    ws += 2 * w.dn;
    void* dc = ws;
    float* recdn = (float*)(ws + w.dc);
    float* pu = (float*)(ws + w.dc + w.dnn);
    float* pw = (float*)(ws + w.dc + w.dnn + w.dots);
    void* rec = ws + w.dc + w.dnn + 2 * w.dots;
    int rc = gates_launch(st, a.ig, a.fg, a.cm, const_cast<float*>(a.msv), nullptr, v, a.B, a.H, a.T, NC, true, a.exact && a.cm);
    if (rc) return rc;
    ScanArgs s = {};
    s.g = v.g; s.B = a.B; s.H = a.H; s.T = a.T; s.D = d; s.NC = NC;
    if (!saved) {
        s.x = a.v; s.y = a.k; s.w = v.a; s.c0 = carry_C; s.n0 = carry_n; s.recC = rec; s.recn = (float*)((char*)rec + record_C_bytes(BH, NC, d));
        s.entries = NC + 1;
        rc = scan_launch(st, s);
        if (rc) return rc;
        saved = rec;
    }
    const float* recn = (const float*)((const char*)saved + record_C_bytes(BH, NC, d));
    DnArgs x = {a.dytil, (const bf16*)a.ytil, a.psiv, a.qnv, a.msv, v, dn, dnb, a.B, a.H, a.T};
    rc = gb == 2 ? dn_run<bf16>(st, x, d) : dn_run<float>(st, x, d);
    if (rc) return rc;
    s.x = dnb; s.y = a.q; s.w = v.bq; s.c0 = a.cdC; s.n0 = a.cdn; s.recC = dc; s.recn = recdn; s.oC = a.odC; s.on = a.odn; s.entries = NC; s.bwd = true;
    rc = scan_launch(st, s);
    if (rc) return rc;
    GradP p = {};
    const int W = a.H * d;
    auto seq = [&](CUtensorMap* m, const void* x, int eb) { return tc_make_map4(m, x, eb, a.B, a.T, W, 128, eb); };  // 128 columns
    if (!seq(&p.tq, a.q, 2) || !seq(&p.tk, a.k, 2) || !seq(&p.tv, a.v, 2) || !seq(&p.tdn, dn, 2) || !seq(&p.tdnb, dnb, 2) ||
        !seq(&p.tdq, a.dq, gb) || !seq(&p.tdk, a.dk, gb) || !seq(&p.tdv, a.dv, gb) ||
        !tc_make_map4(&p.tc, saved, 2, 1, (uint64_t)BH * (NC + 1) * d, d, 128, 2) ||
        !tc_make_map4(&p.tdc, dc, 2, 1, (uint64_t)BH * NC * d, d, 128, 2)) {
        set_error("mlstm_bw: cuTensorMapEncodeTiled failed");
        return XLSTM_ERR_CUDA;
    }
    p.v = v; p.recn = recn; p.recdn = recdn; p.pu = pu; p.pw = pw;
    p.BH = BH; p.H = a.H; p.T = a.T; p.NC = NC; p.units = BH * NC * (d / 128);
    p.status = tc_status_ptr();
    if (!p.status) return XLSTM_ERR_CUDA;
    if (d == 128) rc = gb == 2 ? grad_run<1, bf16>(st, p) : grad_run<1, float>(st, p);
    else rc = gb == 2 ? grad_run<2, bf16>(st, p) : grad_run<2, float>(st, p);
    if (rc) return rc;
    GgArgs g = {pu, pw, a.fg, a.cdC, a.cdn, recn, (const bf16*)saved, a.dig, a.dfg, BH, a.H, a.T, v.Tp, NC, d, d / 32};
    par_gate_grad<<<BH, 1024, 0, st>>>(g);
    XL_LAUNCH_OK("par_gate_grad");
    return XLSTM_OK;
}

}  // namespace xl
