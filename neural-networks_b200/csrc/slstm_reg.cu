// sLSTM time loops with the recurrent matrix in registers (see slstm_reg.cuh). Math: src/nn2/slstm.rs:286-325, 399-423 with the GPU
// kernels' gate clamps (src/gpu/cuda/slstm_fused.cu:132-142).
#include <stdlib.h>

#include <algorithm>
#include <initializer_list>
#include <mutex>

#include "slstm_reg.cuh"

namespace xl {

int* tc_status_ptr();

namespace sreg {

// ---------------------------------------------------------------------------------------------
// Forward
// ---------------------------------------------------------------------------------------------
// A CTA owns UPC = 16 CG units, that is 64 CG gate columns in the order (unit, gate). A half-warp multiplies a slice of R rows of the head's
// h with 64 columns, a lane the four gates of one unit: wide enough that the staged rows, 16 bytes per lane and load, cost the
// shared-memory pipe half of what the products cost the FMA pipes (with two columns a lane they cost more than the products did). A warp polls
// its own rows, into shared memory of its own, so no barrier stands between the exchange and the product. The slices' sums meet in
// shared memory; then two neighbouring lanes finish a (sequence, unit), two of the gates each. The gate inputs and the records go through
// shared memory: four further warps copy them in two passes ahead and write them out a pass later.
template <int CG, int R, int NB>
__global__ void __launch_bounds__(kThr + kHelp, 1) slstm_reg_fw_k(const Args a, int* status) {
    constexpr int UPC = 16 * CG, NC = 4 * UPC, KS = 2 * kWarps / CG;
    const int G = a.G, dhd = a.dhd, H = a.H, T = a.T;
    const int cr = blockIdx.x % G, team = (blockIdx.x / G) % a.teams, hd = blockIdx.x / (G * a.teams);
    const int b_first = team * a.BT, nb_team = min(a.BT, a.B - b_first);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cg = warp % CG, ks = warp / CG * 2 + (lane >> 4);

    extern __shared__ __align__(16) float smem[];
    float* const xw = smem + warp * (2 * R * NB);        // [2 R][NB]: this warp's rows of h
    const float* const xh = xw + (lane >> 4) * R * NB;   // this half-warp's
    float* const part0 = smem + kWarps * 2 * R * NB;     // two buffers [KS][NB][NC]
    constexpr int part_sz = KS * NB * NC;
    float* const st = part0 + 2 * part_sz;               // c, n, m, h: [4][nsub * NB * UPC]
    const int NS = a.nsub * NB * UPC;
    constexpr int NIT = NB * UPC;                        // items of a pass
    float* const gin = st + 4 * NS;                      // three buffers [4][NIT]: the input's share of the gates
    float* const res = gin + 12 * NIT;                   // two buffers [11][NIT]: what a pass records
    const int npass = T * a.nsub;

    for (int i = tid; i < NS; i += kThr + kHelp) {
        const int b = i / UPC, ul = i % UPC;
        const size_t si = (size_t)(b_first + b) * H + hd * dhd + cr * UPC + ul;
        const bool live = a.carry && b < nb_team;
        st[i] = live ? a.c[si] : 0.f;
        st[NS + i] = live ? a.n[si] : 0.f;
        st[2 * NS + i] = live ? a.m[si] : 0.f;
        st[3 * NS + i] = live ? a.h[si] : 0.f;
    }
    for (int i = tid; i < 12 * NIT; i += kThr + kHelp) gin[i] = 0.f;
    bool ok = true;
    if (warp >= kWarps) {  // the helpers
        helper_registers();
        const int ht = tid - kThr;
        __shared__ float* table[11];
        if (ht < 11)
            table[ht] = ht == 0 ? a.s.c : ht == 1 ? a.s.n : ht == 2 ? a.s.zt : ht == 3 ? a.s.ipr : ht == 4 ? a.s.c_prev : ht == 5 ? a.out
                        : ht == 6 ? a.s.fpr : ht == 7 ? a.s.ot : ht == 8 ? a.s.h_prev : ht == 9 ? a.s.n_prev : a.g + 2 * H;
        __syncthreads();
        const int j0 = hd * dhd + cr * UPC;
        auto fetch = [&](int t, int s0, int buf) {
            if (t < T)
                for (int e = ht; e < NIT; e += kHelp) {  // 4 gates x NIT / 4 pieces
                    const int gate = e / (NIT / 4), it = e % (NIT / 4) * 4, b = s0 + it / UPC;
                    if (b >= nb_team) continue;
                    copy16(gin + buf * 4 * NIT + gate * NIT + it, a.g + (((size_t)(b_first + b) * T + t) * 4 + gate) * H + j0 + it % UPC);
                }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        auto record = [&](int t, int s0, int ph) {
            for (int e = ht; e < 11 * NIT / 4; e += kHelp) {
                const int arr = e / (NIT / 4), it = e % (NIT / 4) * 4, b = s0 + it / UPC;
                if (b >= nb_team) continue;
                const size_t row = ((size_t)(b_first + b) * T + t) * H;
                __stcs(reinterpret_cast<float4*>(table[arr] + (arr == 10 ? 4 * row : row) + j0 + it % UPC),
                       *reinterpret_cast<const float4*>(res + (ph * 11 + arr) * NIT + it));
            }
        };
        int ft = 0, fs = 0, fb = 0;  // the next pass to fetch
        auto fetch_next = [&] {
            fetch(ft, fs * NB, fb);
            if (++fs == a.nsub) { fs = 0; ++ft; }
            fb = fb == 2 ? 0 : fb + 1;
        };
        fetch_next();
        fetch_next();
        int rt = 0, rs = 0;
        for (int pass = 0; pass < npass; ++pass) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            if (__syncthreads_or(0)) { ok = false; break; }
            if (pass > 0) {
                record(rt, rs * NB, (pass - 1) & 1);
                if (++rs == a.nsub) { rs = 0; ++rt; }
            }
            fetch_next();
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (!ok) return;
        __syncthreads();
        record(rt, rs * NB, (npass - 1) & 1);
        return;
    }
    worker_registers();
    float4 w[R];  // rows ks R + r, the four gates of unit cg 16 + lane % 16
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int row = ks * R + r;
        const float* p = a.wh + ((size_t)hd * dhd + row) * 4 * dhd + cr * UPC + cg * 16 + (lane & 15);
        w[r] = row < dhd ? make_float4(p[0], p[dhd], p[2 * dhd], p[3 * dhd]) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    // staging: the warp's 2 R rows, RPL of them and BPL sequences of each to a lane
    constexpr int RPL = R == 32 ? 2 : 1, LR = 2 * R / RPL, BPL = NB * LR >= 32 ? NB * LR / 32 : 1;
    const int srow = lane % LR, sb = lane / LR * BPL, row0 = warp / CG * 2 * R;
    auto slot = [](int r, int b) {  // 16-byte pieces of a row swap places by bit 2 of the row: a quarter-warp's stores meet no bank twice
        return NB == 8 ? r * NB + ((b & 4) ^ (r & 4)) + (b & 3) : r * NB + b;
    };
    for (int i = lane; i < 2 * R * NB; i += 32) xw[i] = 0.f;
    // what this thread finishes: gates (z, i) or (f, o) of NI (sequence, unit) items
    const int pair = tid >> 1, p = tid & 1;
    constexpr int NI = NB * CG > 8 ? NB * CG / 8 : 1;
    constexpr bool whole = NB * UPC >= kThr / 2;  // every pair of lanes has items
    const size_t slab = (size_t)a.NH * a.B * dhd;  // words of one step parity
    uint2* const ll = a.ll + ((size_t)hd * a.B + b_first) * dhd;
    const float2 bias = make_float2(a.bcat[2 * p * H + hd * dhd + cr * UPC + pair % UPC], a.bcat[(2 * p + 1) * H + hd * dhd + cr * UPC + pair % UPC]);
    __syncthreads();

    int phase = 0, gbuf = 0;
    for (int t = 0; t < T && ok; ++t) {
        for (int sg = 0; sg < a.nsub; ++sg, phase ^= 1) {
            const int s0 = sg * NB;
            float* const part = part0 + phase * part_sz;
            if (sb < NB) {
                float v[RPL][BPL];
                const int nlive = min(BPL, nb_team - s0 - sb);
                if (t > 0) {
                    const uint2* src = ll + (size_t)((t - 1) & 1) * slab + (size_t)(s0 + sb) * dhd + row0 + srow;
                    ok = gather<RPL, BPL>(v, src, LR, dhd, [&](int r, int b) { return b < nlive && row0 + srow + r * LR < dhd; }, (unsigned)t, a.abort);
                } else {
#pragma unroll
                    for (int r = 0; r < RPL; ++r)
#pragma unroll
                        for (int i = 0; i < BPL; ++i)
                            v[r][i] = a.carry && i < nlive && row0 + srow + r * LR < dhd
                                ? a.h[(size_t)(b_first + s0 + sb + i) * H + hd * dhd + row0 + srow + r * LR] : 0.f;
                }
#pragma unroll
                for (int r = 0; r < RPL; ++r) {
                    if (BPL >= 4) {
#pragma unroll
                        for (int i = 0; i < BPL / 4; ++i)
                            *reinterpret_cast<float4*>(xw + slot(srow + r * LR, sb + 4 * i)) = make_float4(v[r][4 * i], v[r][4 * i + 1], v[r][4 * i + 2], v[r][4 * i + 3]);
                    } else {
#pragma unroll
                        for (int i = 0; i < BPL; ++i) xw[slot(srow + r * LR, sb + i)] = v[r][i];
                    }
                }
            }
            __syncwarp();
            float cp[NI], np[NI], mp[NI], hp[NI];  // the items' state, read ahead of the product
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                const int it = s0 * UPC + pair + i * kThr / 2;
                if (whole || pair < NB * UPC) {
                    cp[i] = st[it];
                    np[i] = st[NS + it];
                    mp[i] = st[2 * NS + it];
                    hp[i] = st[3 * NS + it];
                }
            }
            float2 acc[4][NB / 2];
#pragma unroll
            for (int i = 0; i < NB / 2; ++i) acc[0][i] = acc[1][i] = acc[2][i] = acc[3][i] = make_float2(0.f, 0.f);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                float2 x[NB / 2];
                if (NB >= 4) {
#pragma unroll
                    for (int i = 0; i < NB / 4; ++i) {
                        const float4 f = *reinterpret_cast<const float4*>(xh + slot(r, 4 * i));
                        x[2 * i] = make_float2(f.x, f.y);
                        x[2 * i + 1] = make_float2(f.z, f.w);
                    }
                } else {
                    x[0] = *reinterpret_cast<const float2*>(xh + slot(r, 0));
                }
#pragma unroll
                for (int i = 0; i < NB / 2; ++i) {
                    acc[0][i] = __ffma2_rn(make_float2(w[r].x, w[r].x), x[i], acc[0][i]);
                    acc[1][i] = __ffma2_rn(make_float2(w[r].y, w[r].y), x[i], acc[1][i]);
                    acc[2][i] = __ffma2_rn(make_float2(w[r].z, w[r].z), x[i], acc[2][i]);
                    acc[3][i] = __ffma2_rn(make_float2(w[r].w, w[r].w), x[i], acc[3][i]);
                }
            }
            float* const pw = part + (size_t)ks * NB * NC + cg * 64 + 4 * (lane & 15);
#pragma unroll
            for (int i = 0; i < NB / 2; ++i) {
                *reinterpret_cast<float4*>(pw + (2 * i) * NC) = make_float4(acc[0][i].x, acc[1][i].x, acc[2][i].x, acc[3][i].x);
                *reinterpret_cast<float4*>(pw + (2 * i + 1) * NC) = make_float4(acc[0][i].y, acc[1][i].y, acc[2][i].y, acc[3][i].y);
            }
            if (__syncthreads_or(!ok)) { ok = false; break; }
            if (!whole && pair >= NB * UPC) continue;  // whole warps
            const float* const gi = gin + (gbuf * 4 + 2 * p) * NIT;
            gbuf = gbuf == 2 ? 0 : gbuf + 1;
            float2 pre[NI];
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                const int it = pair + i * kThr / 2;
                float2 s2[4] = {};
                const float* pp = part + (size_t)(it / UPC) * NC + 4 * (it % UPC) + 2 * p;
#pragma unroll
                for (int k = 0; k < KS; k += 4)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 v = *reinterpret_cast<const float2*>(pp + (size_t)(k + e) * NB * NC);
                        s2[e].x += v.x;
                        s2[e].y += v.y;
                    }
                pre[i].x = gi[it] + ((s2[0].x + s2[1].x) + (s2[2].x + s2[3].x)) + bias.x;
                pre[i].y = gi[NIT + it] + ((s2[0].y + s2[1].y) + (s2[2].y + s2[3].y)) + bias.y;
            }
            float z[NI], og[NI], ip[NI], fp[NI], c[NI], n[NI], m[NI], h[NI];
#pragma unroll
            for (int i = 0; i < NI; ++i) {  // sequences past the batch are computed like the others, so that the items' chains overlap
                // lane 0: tanh(z) and i as it is; lane 1: sigmoid(o) and log sigmoid(f)
                const float d = __fdividef(p ? 1.f : 2.f, 1.f + __expf(p ? -pre[i].y : 2.f * pre[i].x));
                const float act = p ? d : 1.f - d;
                const float gate = p ? fminf(pre[i].x, 0.f) - __logf(1.f + __expf(-fabsf(pre[i].x))) : pre[i].y;
                const float act_x = __shfl_xor_sync(0xffffffffu, act, 1), gate_x = __shfl_xor_sync(0xffffffffu, gate, 1);
                const float i_ = p ? gate_x : gate, fm = (p ? gate : gate_x) + mp[i];
                z[i] = p ? act_x : act;
                og[i] = p ? act : act_x;
                m[i] = np[i] == 0.f ? i_ : fmaxf(fm, i_);
                ip[i] = fminf(1.f, __expf(i_ - m[i]));
                fp[i] = fminf(1.f, __expf(fm - m[i]));
                c[i] = fp[i] * cp[i] + ip[i] * z[i];
                n[i] = fp[i] * np[i] + ip[i];
                h[i] = __fdividef(og[i] * c[i], n[i]);
            }
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                const int it = pair + i * kThr / 2, b = s0 + it / UPC;
                if (p == 0 && b < nb_team) put(ll + (size_t)(t & 1) * slab + (size_t)b * dhd + cr * UPC + it % UPC, h[i], (unsigned)t + 1);
            }
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                const int it = pair + i * kThr / 2;
                float* const sp = st + s0 * UPC + it;
                sp[(p ? 2 : 0) * NS] = p ? m[i] : c[i];
                sp[(p ? 3 : 1) * NS] = p ? h[i] : n[i];
                float* const rp = res + (phase * 11 + 5 * p) * NIT + it;  // c, n, z, i', c_prev; h, f', o, h_prev, n_prev, f
                rp[0] = p ? h[i] : c[i];
                rp[NIT] = p ? fp[i] : n[i];
                rp[2 * NIT] = p ? og[i] : z[i];
                rp[3 * NIT] = p ? hp[i] : ip[i];
                rp[4 * NIT] = p ? np[i] : cp[i];
                if (p) rp[5 * NIT] = pre[i].x;
            }
        }
    }
    if (!ok) {
        if (tid == 0) {
            atomicExch(a.abort, 1u);
            atomicCAS(status, 0, 301);
        }
        return;
    }
    __syncthreads();
    for (int i = tid; i < NS; i += kThr) {
        const int b = i / UPC;
        if (b >= nb_team) continue;
        const size_t si = (size_t)(b_first + b) * H + hd * dhd + cr * UPC + i % UPC;
        a.c[si] = st[i];
        a.n[si] = st[NS + i];
        a.m[si] = st[2 * NS + i];
        a.h[si] = st[3 * NS + i];
    }
}

// ---------------------------------------------------------------------------------------------
// Backward
// ---------------------------------------------------------------------------------------------
// dh_{t-1}[u] = sum_k delta_t[k] Wh[u][k]. A CTA computes the gate deltas of its UPC own units and multiplies them with their columns of
// Wh: a partial dh for every unit of the head. A thread has four output columns (see the forward for why) of one of 2 KH row slices; the two
// half-warps of a warp hold two slices of the same columns and add them by shuffles. The KH sums of every CTA travel through L2. Clusters of four that
// add theirs over distributed shared memory first, and move a quarter of it, were no faster: that exchange took what it saved.
// A (sequence, unit) belongs to LPI neighbouring lanes: they share the words to add up and all hold the cell. Its operands are copied to
// shared memory two passes ahead.
template <int R, int NB>
__global__ void __launch_bounds__(kThr + kHelp, 1) slstm_reg_bw_k(const Args a, int* status) {
    const int G = a.G, UPC = a.UPC, dhd = a.dhd, H = a.H, T = a.T, KH = a.KH, LPI = a.LPI;
    const int cr = blockIdx.x % G, team = (blockIdx.x / G) % a.teams, hd = blockIdx.x / (G * a.teams);
    const int b_first = team * a.BT, nb_team = min(a.BT, a.B - b_first);
    const int tid = threadIdx.x, lane = tid & 31, hf = lane >> 4;
    const int NI = NB * UPC, rows = 2 * KH * R;

    extern __shared__ __align__(16) float smem[];
    float* const xin0 = smem;                           // two buffers [rows][NB]: own deltas, rows in the order (unit, gate)
    float* const op0 = xin0 + 2 * rows * NB;            // two buffers [10][NI]
    constexpr int RS = R == 32 && NB == 8 ? 12 : 0;      // rows whose weights stay in shared memory: 128 in registers left none to work with
    float4* const ws = (float4*)(op0 + 20 * NI);        // [RS][kThr]
    float* const st = op0 + 20 * NI + 4 * RS * kThr;                    // dc, dn: [2][nsub * NI]
    const int NS = a.nsub * NI;

    for (int i = tid; i < NS; i += kThr + kHelp) {
        const int b = i / UPC;
        const size_t si = (size_t)(b_first + b) * H + hd * dhd + cr * UPC + i % UPC;
        const bool live = a.carry && b < nb_team;
        st[i] = live ? a.dc[si] : 0.f;
        st[NS + i] = live ? a.dn[si] : 0.f;
    }
    for (int i = tid; i < 2 * rows * NB; i += kThr + kHelp) xin0[i] = 0.f;
    for (int i = tid; i < 20 * NI; i += kThr + kHelp) op0[i] = 0.f;
    __syncthreads();
    const int npass = T * a.nsub;
    bool ok = true;
    if (tid >= kThr) {  // the helpers
        helper_registers();
        const int ht = tid - kThr, j0 = hd * dhd + cr * UPC;
        __shared__ const float* table[10];
        if (ht < 10)
            table[ht] = ht == 0 ? a.dy : ht == 1 ? a.s.ot : ht == 2 ? a.s.c : ht == 3 ? a.s.n : ht == 4 ? a.s.fpr : ht == 5 ? a.s.ipr
                        : ht == 6 ? a.s.zt : ht == 7 ? a.s.c_prev : ht == 8 ? a.s.n_prev : a.g + 2 * H;
        asm volatile("bar.sync 1, %0;" ::"n"(kHelp) : "memory");
        const int lg_upc = __ffs(UPC) - 1, lg_row = __ffs(NI / 4) - 1;  // powers of two
        auto fetch = [&](int t, int s0, int buf) {
            if (t >= 0)
                for (int e = ht; e < 10 * NI / 4; e += kHelp) {
                    const int arr = e >> lg_row, it = (e & (NI / 4 - 1)) * 4, b = s0 + (it >> lg_upc);
                    if (b >= nb_team) continue;
                    copy16(op0 + buf * 10 * NI + 4 * e, table[arr] + ((size_t)(b_first + b) * T + t) * H * (arr == 9 ? 4 : 1) + j0 + (it & (UPC - 1)));
                }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        int ft = T - 1, fs = 0, fb = 0;  // the next pass to fetch; a buffer is free once the barrier of the pass that read it is behind
        auto fetch_next = [&] {
            fetch(ft, fs * NB, fb);
            if (++fs == a.nsub) { fs = 0; --ft; }
            fb ^= 1;
        };
        fetch_next();
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        fetch_next();
        int rt = T - 1, rs = 0;
        for (int pass = 0; pass < npass; ++pass) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            if (__syncthreads_or(0)) { ok = false; break; }
            const float* xin = xin0 + (pass & 1) * rows * NB;
            for (int e = ht; e < 4 * NI; e += kHelp) {  // the record: consecutive threads, consecutive units
                const int gate = e >> (lg_row + 2), it = e & (NI - 1), b = it >> lg_upc, ul = it & (UPC - 1);
                if (rs * NB + b < nb_team)
                    __stcs(a.g + (((size_t)(b_first + rs * NB + b) * T + rt) * 4 + gate) * H + j0 + ul, xin[(4 * ul + gate) * NB + b]);
            }
            if (++rs == a.nsub) { rs = 0; --rt; }
            fetch_next();
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        return;
    }
    worker_registers();
    const int quad = (tid >> 5) * 16 + (lane & 15), kh = quad / (dhd / 4), u = quad % (dhd / 4) * 4;  // KH * dhd / 4 half-lanes multiply
    const bool mul = kh < KH;
    const int slice = 2 * kh + hf;
    float4 w[R - RS];  // columns u .. u + 3; row r = 4 ul + gate: four units' columns are one 16-byte load
#pragma unroll
    for (int i = 0; i < R / 16 + (R < 16); ++i)
#pragma unroll
        for (int gate = 0; gate < 4; ++gate)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int ul = (slice * R) / 4 + 4 * i;
                float v[4] = {0.f, 0.f, 0.f, 0.f};
                if (mul && ul < UPC) {
                    const float* p = a.wh + ((size_t)hd * dhd + u + c) * 4 * dhd + (size_t)gate * dhd + cr * UPC + ul;
                    if (R >= 16) {
                        const float4 f = *reinterpret_cast<const float4*>(p);
                        v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
                    } else {
                        v[0] = p[0]; v[1] = p[1];
                    }
                }
#pragma unroll
                for (int e = 0; e < (R < 16 ? R / 4 : 4); ++e) {
                    const int r = 16 * i + 4 * e + gate;
                    if (r < R - RS) {
                        float4& d = w[r];
                        (c == 0 ? d.x : c == 1 ? d.y : c == 2 ? d.z : d.w) = v[e];
                    } else {
                        ((float*)(ws + (r - (R - RS)) * kThr + tid))[c] = v[e];
                    }
                }
            }
    __syncthreads();  // the first operands

    const int item = tid / LPI, q = tid % LPI, ib = item / UPC, ul = item % UPC, j = hd * dhd + cr * UPC + ul;
    const int S = G * KH, nw = item < NI ? (S - q + LPI - 1) / LPI : 0;  // senders q, q + LPI, ...
    const size_t sender = (size_t)a.B * dhd;
    const size_t slab = (size_t)a.NH * S * sender;
    uint2* const llh = a.ll + (size_t)hd * S * sender + (size_t)b_first * dhd;
    // the recurrent dh of the own items of the sub-group at s0, from the words of the step before
    auto recurrent = [&](int t, int s0, bool& ok) {
        float v[1][2 * NB], sum = 0.f;
        const bool live = item < NI && s0 + ib < nb_team;
        ok = gather<1, 2 * NB>(v, llh + (size_t)(t & 1) * slab + q * sender + (size_t)(s0 + ib) * dhd + cr * UPC + ul, 0, LPI * sender,
                               [&](int, int i) { return live && i < nw; }, (unsigned)(T - t), a.abort);
#pragma unroll
        for (int i = 0; i < 2 * NB; ++i) sum += v[0][i];
        for (int d = 1; d < LPI; d <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
        return sum;
    };
    int pass = 0;
    for (int t = T - 1; t >= 0 && ok; --t) {
        for (int sg = 0; sg < a.nsub; ++sg, ++pass) {
            const int s0 = sg * NB, b = s0 + ib;
            const bool live = item < NI && b < nb_team;
            float dhr = 0.f;
            if (t < T - 1) {
                if (sg == 0) rest(a.rest);
                dhr = recurrent(t + 1, s0, ok);
            }
            else if (a.carry && live) dhr = a.dh[(size_t)(b_first + b) * H + j];
            float* const xin = xin0 + (pass & 1) * rows * NB;
            const float* op = op0 + (pass & 1) * 10 * NI + item;
            SlstmBwCell r = {};
            __syncwarp();  // the item's first lane wrote the state in the pass before
            if (live) {
                const int it = s0 * UPC + item;
                const float dc = st[it], dn = st[NS + it];
                r = slstm_cell_bw(op[0] + dhr, op[NI], op[2 * NI], op[3 * NI], op[4 * NI], op[5 * NI], op[6 * NI], op[7 * NI], op[8 * NI],
                                  op[9 * NI], dc, dn);
            }
            // gate g is lane g's, or lane g % LPI's where an item has fewer than four
            const float delta[4] = {r.dz, r.di, r.df, r.dob};
#pragma unroll
            for (int g = 0; g < 4; ++g)
                if (item < NI && (g & (LPI - 1)) == q) xin[(4 * ul + g) * NB + ib] = delta[g];
            if (__syncthreads_or(!ok)) { ok = false; break; }
            const float* xp = xin + slice * R * NB;
            float2 acc[4][NB / 2];
#pragma unroll
            for (int i = 0; i < NB / 2; ++i) acc[0][i] = acc[1][i] = acc[2][i] = acc[3][i] = make_float2(0.f, 0.f);
            if (mul) {
#pragma unroll
                for (int k = 0; k < R; ++k) {
                    const float4 wk = k < R - RS ? w[k < R - RS ? k : 0] : ws[(k - (R - RS)) * kThr + tid];
                    float2 x[NB / 2];
                    if (NB >= 4) {
#pragma unroll
                        for (int i = 0; i < NB / 4; ++i) {
                            const float4 f = *reinterpret_cast<const float4*>(xp + k * NB + 4 * i);
                            x[2 * i] = make_float2(f.x, f.y);
                            x[2 * i + 1] = make_float2(f.z, f.w);
                        }
                    } else {
                        x[0] = *reinterpret_cast<const float2*>(xp + k * NB);
                    }
#pragma unroll
                    for (int i = 0; i < NB / 2; ++i) {
                        acc[0][i] = __ffma2_rn(make_float2(wk.x, wk.x), x[i], acc[0][i]);
                        acc[1][i] = __ffma2_rn(make_float2(wk.y, wk.y), x[i], acc[1][i]);
                        acc[2][i] = __ffma2_rn(make_float2(wk.z, wk.z), x[i], acc[2][i]);
                        acc[3][i] = __ffma2_rn(make_float2(wk.w, wk.w), x[i], acc[3][i]);
                    }
                }
            }
            // the two half-warps' slices: each lane keeps two columns and hands over the others, so that the 32 bytes of a sector leave in one
            // store (with half of the sequences each, and half sectors stored, the readers waited 1.5 to 2 k cycles longer)
            uint2* const dst = llh + (t & 1) * slab + (size_t)(cr * KH + kh) * sender + s0 * dhd + u + 2 * hf;
            const unsigned tag = (unsigned)(T - t);
#pragma unroll
            for (int i = 0; i < NB / 2; ++i) {
                const float2 g0 = hf ? acc[0][i] : acc[2][i], g1 = hf ? acc[1][i] : acc[3][i];
                float2 k0 = hf ? acc[2][i] : acc[0][i], k1 = hf ? acc[3][i] : acc[1][i];
                k0.x += __shfl_xor_sync(0xffffffffu, g0.x, 16);
                k1.x += __shfl_xor_sync(0xffffffffu, g1.x, 16);
                k0.y += __shfl_xor_sync(0xffffffffu, g0.y, 16);
                k1.y += __shfl_xor_sync(0xffffffffu, g1.y, 16);
                if (mul && s0 + 2 * i < nb_team) put2(dst + 2 * i * dhd, k0.x, k1.x, tag);
                if (mul && s0 + 2 * i + 1 < nb_team) put2(dst + (2 * i + 1) * dhd, k0.y, k1.y, tag);
            }
            if (live && q == 0) {
                st[s0 * UPC + item] = r.dc;
                st[NS + s0 * UPC + item] = r.dn;
            }
        }
    }
    const int left = ok ? a.nsub : 0;
    for (int sg = 0; sg < left; ++sg) {  // dh that leaves the call: the words of step 0
        bool got;
        const float dhr = recurrent(0, sg * NB, got);
        ok = ok && got;
        if (item < NI && sg * NB + ib < nb_team && q == 0 && ok) a.dh[(size_t)(b_first + sg * NB + ib) * H + j] = dhr;
    }
    const bool bad = workers_or(!ok);
    if (bad && tid == 0) {
        atomicExch(a.abort, 1u);
        atomicCAS(status, 0, 303);
    }
    if (bad) return;
    for (int i = tid; i < NS; i += kThr) {
        const int b = i / UPC;
        if (b >= nb_team) continue;
        const size_t si = (size_t)(b_first + b) * H + hd * dhd + cr * UPC + i % UPC;
        a.dc[si] = st[i];
        a.dn[si] = st[NS + i];
    }
}

// ---------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------
struct Plan {
    int NB, R, CG = 1;
    size_t smem, words;
    double cost = 1e30;
};
static constexpr size_t kSmemCap = 220 * 1024;

// Cycles of a step, the model the geometry is chosen by: every pass over NB sequences costs its FMAs (two warps a scheduler, R rows x NB sequences
// x four columns a lane, two a packed FMA of two cycles) and some 900 cycles around them, and the last pass' exchange is exposed.
static double step_cost(int R, int NB, int nsub) { return nsub * (8.0 * R * NB + 900.0) + 900.0; }

// Batch groups: as many as there are SMs for, each with as few passes as that leaves.
static bool groups_of(int B, int NB, int per_team, Args* a) {
    const int fit = sm_count() / per_team;
    if (fit < 1) return false;
    const int passes = (B + NB - 1) / NB;
    a->teams = std::min(fit, passes);
    a->nsub = (passes + a->teams - 1) / a->teams;
    a->teams = (passes + a->nsub - 1) / a->nsub;
    a->BT = a->nsub * NB;
    return true;
}

static bool plan_fw(Args* out, Plan* best) {
    for (int CG = 1; CG <= 2; CG *= 2)
        for (int NB = 8; NB >= 2; NB /= 2) {
            Args a = *out;
            Plan p;
            p.CG = CG; a.UPC = 16 * CG;
            if (a.dhd % a.UPC || (NB > 2 && NB / 2 >= a.B)) continue;
            a.G = a.dhd / a.UPC;
            const int KS = 2 * kWarps / CG, need = (a.dhd + KS - 1) / KS;
            p.R = need <= 8 ? 8 : need <= 16 ? 16 : 32;
            p.NB = NB;
            if (need > 32 || !groups_of(a.B, NB, a.NH * a.G, &a)) continue;
            p.smem = 4 * ((size_t)kWarps * 2 * p.R * NB + 2 * (size_t)KS * NB * 4 * a.UPC + 4 * (size_t)a.nsub * NB * a.UPC + 34 * (size_t)NB * a.UPC);
            p.words = 2 * (size_t)a.NH * a.B * a.dhd;
            p.cost = step_cost(p.R, NB, a.nsub);
            if (p.smem > kSmemCap || p.cost >= best->cost) continue;
            *out = a;
            *best = p;
        }
    return best->cost < 1e30;
}

static bool plan_bw(Args* out, Plan* best) {
    for (int UPC = 16; UPC <= 64; UPC *= 2)
        for (int NB = 8; NB >= 2; NB /= 2) {
            Args a = *out;
            Plan p;
            a.UPC = UPC;
            if (a.dhd % UPC || (NB > 2 && NB / 2 >= a.B)) continue;
            a.G = a.dhd / UPC;
            a.KH = std::min(2 * kThr / a.dhd, 4 * UPC / 16);
            const int need = (2 * UPC + a.KH - 1) / a.KH;
            p.R = need <= 8 ? 8 : need <= 16 ? 16 : 32;
            p.NB = NB;
            const int senders = a.G * a.KH;
            a.LPI = std::min(32, kThr / (NB * UPC));
            if (need > 32 || a.LPI < 1 || (senders + a.LPI - 1) / a.LPI > 2 * NB || !groups_of(a.B, NB, a.NH * a.G, &a)) continue;
            p.smem = 4 * (4 * (size_t)a.KH * p.R * NB + 20 * (size_t)NB * UPC + 2 * (size_t)a.nsub * NB * UPC + (p.R == 32 && NB == 8 ? 4 * 12 * kThr : 0));
            p.words = 2 * (size_t)a.NH * senders * a.B * a.dhd;
            // Many senders' words for eight sequences come in late enough that polling at once only gets in their way, where a thread has
            // rows enough to multiply. us a step at 24 to 32 senders without a rest and after 600 cycles of it (sequences x heads x units):
            //   32 rows  8 x 4 x 512 4.52 3.96   12 x 2 x 512 4.46 3.95   5 x 4 x 384 3.85 3.61   8 x 4 x 448 4.45 4.44   16 x 2 x 384 4.21 4.23
            //   16 rows  12 x 4 x 256 3.56 3.28  32 x 2 x 256 3.54 3.29   32 x 2 x 192 3.69 3.58
            //    8 rows  32 x 4 x 128 2.62 2.87  12 x 8 x 128 2.62 2.85
            // With two sequences a pass, several passes or fewer senders, the wait is lost (up to 0.3 us); with four it would have to be shorter.
            a.rest = senders >= 24 && NB == 8 && p.R >= 16 && a.nsub == 1 ? 600 : 0;
            p.cost = step_cost(p.R, NB, a.nsub);
            if (p.smem > kSmemCap || p.cost >= best->cost) continue;
            *out = a;
            *best = p;
        }
    return best->cost < 1e30;
}

// Where the device has no memory left to give (a host whose own runtime holds all of it), the call goes to the kernels of slstm.cu, which up to
// 256 units a head need none beyond their arguments.
#define XL_ROOM(expr)                                 \
    do {                                              \
        cudaError_t room__ = (expr);                  \
        if (room__ == cudaErrorMemoryAllocation) {    \
            (void)cudaGetLastError();                 \
            return XLSTM_DECLINED;                    \
        }                                             \
        XL_CUDA(room__);                              \
    } while (0)

// The exchange words come from a memory pool of the library's own, in stream order: launches on several streams or threads each have theirs,
// and the pool gives back what it holds beyond kPoolKeep whenever the device is synchronised.
static constexpr size_t kPoolKeep = 32 << 20;
static int pool_of(int dev, cudaMemPool_t* out) {
    static std::mutex mu;
    static cudaMemPool_t pools[64];
    std::lock_guard<std::mutex> lock(mu);
    if (!pools[dev]) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        XL_ROOM(cudaMemPoolCreate(&pools[dev], &props));
        unsigned long long keep = kPoolKeep;
        XL_CUDA(cudaMemPoolSetAttribute(pools[dev], cudaMemPoolAttrReleaseThreshold, &keep));
    }
    *out = pools[dev];
    return XLSTM_OK;
}

static int start(cudaStream_t st, const void* kern, Args& a, const Plan& p, const char* what) {
    int dev = 0;
    XL_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return XLSTM_DECLINED;
    const int grid = a.NH * a.teams * a.G;
    XL_ROOM(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemCap));  // loads the kernel on its first call
    int* status = tc_status_ptr();
    if (!status) return XLSTM_ERR_CUDA;
    if (getenv("XLSTM_DEBUG"))
        fprintf(stderr, "[xlstm] slstm %s: G=%d UPC=%d NB=%d R=%d groups=%d passes=%d smem=%zu CTAs=%d\n", what, a.G, a.UPC, p.NB, p.R, a.teams,
                a.nsub, p.smem, grid);
    cudaMemPool_t pool;
    const int rc = pool_of(dev, &pool);
    if (rc) return rc;
    void* mem = nullptr;
    const size_t bytes = 256 + p.words * sizeof(uint2);
    XL_ROOM(cudaMallocFromPoolAsync(&mem, bytes, pool, st));
    a.abort = (unsigned*)mem;
    a.ll = (uint2*)((char*)mem + 256);
    void* args[2] = {&a, &status};
    cudaError_t e = cudaMemsetAsync(mem, 0, bytes, st);
    if (e == cudaSuccess) e = cudaLaunchCooperativeKernel(kern, dim3((unsigned)grid), dim3(kThr + kHelp), args, p.smem, st);  // all CTAs resident, or an error
    XL_CUDA(cudaFreeAsync(mem, st));
    XL_CUDA(e);
    count_launch();
    return XLSTM_OK;
}

template <int CG, int NB>
static const void* fw_kernel(int R) {
    return R == 32 ? (const void*)slstm_reg_fw_k<CG, 32, NB> : R == 16 ? (const void*)slstm_reg_fw_k<CG, 16, NB> : (const void*)slstm_reg_fw_k<CG, 8, NB>;
}
template <int CG>
static const void* fw_kernel(const Plan& p) {
    return p.NB == 8 ? fw_kernel<CG, 8>(p.R) : p.NB == 4 ? fw_kernel<CG, 4>(p.R) : fw_kernel<CG, 2>(p.R);
}
template <int NB>
static const void* bw_kernel(int R) {
    return R == 32 ? (const void*)slstm_reg_bw_k<32, NB> : R == 16 ? (const void*)slstm_reg_bw_k<16, NB> : (const void*)slstm_reg_bw_k<8, NB>;
}

// On short sequences the launch (a cooperative one, words to clear, weights to lay out: some 20 us more per direction) outweighs what a step
// saves: 4 steps of one 32-unit head took 51 against 38 us, 6 of 2 x 384 units 82 against 76; 8 of 4 x 256 units, 32 sequences 94 against 140.
// The forward also needs two steps: the second one's exchange is what tells a CTA that the others have read the carried h it will overwrite.
static bool takes(const Args& a) { return a.dhd % 16 == 0 && a.dhd <= 512 && a.T >= (a.dhd >= 256 ? 8 : 14) && a.T < (1 << 30); }

// Large batches: a step takes a pass after the other over as many sequences as fit the SMs, while the cluster kernels take all that are resident
// at once, and past that whole waves. Measured against them, 64 steps, us forward | backward (sequences x heads x units):
//   one pass    32 x 4 x 256 335 -> 215 | 417 -> 262   64 x 2 x 160 246 -> 215 | 288 -> 270   128 x 4 x 64 195 -> 128 | 185 -> 187
//               192 x 4 x 32 178 -> 119 | 140 -> 164   64 x 4 x 96  205 -> 170 | 198 -> 249 (backwards only the 32-unit CTAs of narrow heads lose)
//   several     64 x 4 x 256 858 -> 404 | 991 -> 487   512 x 4 x 256 5033 -> 3076 | 5876 -> 4789   64 x 4 x 224 766 -> 415 | 900 -> 490
//               64 x 4 x 512 2041 -> 1396 | 2584 -> 2024   128 x 4 x 240 1370 -> 1071 | 20 x 4 x 240 324 -> 384, 256 x 4 x 240 2832 -> 2963
//               128 x 4 x 128 341 -> 316 | 402 -> 418  128 x 8 x 64 287 -> 240 | 243 -> 346   64 x 4 x 192 318 -> 403 | 382 -> 532
//               64 x 4 x 160 285 -> 397 | 324 -> 567   256 x 4 x 48 224 -> 280 | 185 -> 379 (rows padded to a power of two)
static bool pays(const Args& a, const Plan& p, bool bwd) {
    const int d = a.dhd;
    if (a.nsub == 1) return !bwd || d >= 128 || a.UPC < 32 || p.NB < 8;
    return d > 256 || (d > 192 && (!bwd || d % 32 == 0)) || (!bwd && (d & (d - 1)) == 0);
}

// Sequences per launch: all, or as few equal slices as keep each one's words in what the pool holds on to (a larger allocation is mapped
// anew, some 0.5 to 3 ms, after every synchronisation).
static int batch_of(const Args& a, bool bwd) {
    Args s = a;
    for (int n = 1; n <= a.B; ++n) {
        Plan p;
        const int B = (a.B + n - 1) / n;
        if (n > 1 && B == s.B) continue;
        s = a;
        s.B = B;
        if (!(bwd ? plan_bw(&s, &p) : plan_fw(&s, &p)) || (n == 1 && !pays(s, p, bwd))) return 0;
        if (256 + p.words * sizeof(uint2) <= kPoolKeep) return B;
    }
    return 0;
}

}  // namespace sreg

static bool aligned(std::initializer_list<const void*> ptrs) {  // read and written 16 bytes at a time
    for (const void* p : ptrs)
        if ((uintptr_t)p & 15) return false;
    return true;
}

int slstm_reg_batch(const sreg::Args& a, bool bwd) {
    const bool ok = bwd ? aligned({a.wh, a.dy, a.g, a.s.ot, a.s.c, a.s.n, a.s.fpr, a.s.ipr, a.s.zt, a.s.c_prev, a.s.n_prev})
                        : aligned({a.g, a.out, a.s.c, a.s.n, a.s.fpr, a.s.ipr, a.s.zt, a.s.ot, a.s.c_prev, a.s.n_prev, a.s.h_prev});
    return ok && sreg::takes(a) ? sreg::batch_of(a, bwd) : 0;
}

int slstm_reg_fw(cudaStream_t st, sreg::Args a) {
    sreg::Plan p;
    if (!sreg::plan_fw(&a, &p)) return XLSTM_DECLINED;
    return sreg::start(st, p.CG == 2 ? sreg::fw_kernel<2>(p) : sreg::fw_kernel<1>(p), a, p, "fw");
}

int slstm_reg_bw(cudaStream_t st, sreg::Args a) {
    sreg::Plan p;
    if (!sreg::plan_bw(&a, &p)) return XLSTM_DECLINED;
    return sreg::start(st, p.NB == 8 ? sreg::bw_kernel<8>(p.R) : p.NB == 4 ? sreg::bw_kernel<4>(p.R) : sreg::bw_kernel<2>(p.R), a, p, "bw");
}

}  // namespace xl
