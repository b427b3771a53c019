// sLSTM time loops with the recurrent matrix in registers and a flagged exchange: shared declarations.
//
// A step of the loop is a mat-vec per (head, sequence) and an exchange of its result among the CTAs that share the head; T steps follow one
// another, so the sum of the latencies in a step is the whole time. What a step cannot do without is its fp32 FMAs (a CTA of 256 threads
// with 128 weights each: 32 k x 8 sequences = 2048 cycles of the FMA pipes) and one trip through L2 (a store and the load that sees it, some
// 1300 cycles). The kernels here are built so that little else is left on that chain:
//   - a team of G CTAs owns one (head, batch group); groups are independent, so a batch is spread over the SMs that one group leaves idle;
//   - a thread keeps its weights in registers for the whole call and multiplies two sequences per packed FMA. The weight is the duplicated
//     operand: one pair of moves serves all sequences of a row (duplicating the state instead cost a pair of moves per FMA, twice the time);
//   - values travel as (value, tag) words of eight bytes that the reader polls: no fence, no counter, no barrier between CTAs;
//   - one __syncthreads per step, everything around it is private to a warp or double-buffered.
#pragma once
#include <atomic>

#include "common.cuh"
#include "slstm_cell.cuh"

namespace xl {
namespace sreg {

static constexpr int kThr = 256, kWarps = 8;  // the threads that multiply
// and the warpgroup that moves operands in and records out: by the multiplying warps themselves the some ten strided copies and as many stores
// of a step were 0.4 to 1.9 k cycles of the chain (a row of every array and sequence, each in a page of its own)
static constexpr int kHelp = 128;
static constexpr unsigned kSpin = 1u << 21;  // about a second of polling

struct Args {
    const float *wh, *bcat, *dy;
    float *g, *c, *n, *m, *h, *out, *dh, *dc, *dn;
    xlstm_slstm_slabs s;
    int B, H, NH, T, carry, dhd;
    int G, UPC;           // CTAs of a team, units of a CTA
    int teams, BT, nsub;  // batch groups; sequences of a group (a multiple of the kernel's NB) and its passes of NB
    int rest;             // backward: cycles between a step's last store and its first poll
    int KH, LPI;          // backward: row slices per column, lanes per (sequence, unit)
    unsigned* abort;      // zeroed with the words
    uint2* ll;            // exchange words, zeroed before the launch: tag t + 1 marks a value of step t
};

__device__ __forceinline__ void put(uint2* p, float v, unsigned tag) {
    asm volatile("st.relaxed.gpu.global.v2.b32 [%0], {%1, %2};" ::"l"(p), "r"(__float_as_uint(v)), "r"(tag) : "memory");
}
// Two neighbouring words, the first 16-byte aligned; each of them is one 64-bit access.
__device__ __forceinline__ void put2(uint2* p, float v0, float v1, unsigned tag) {
    asm volatile("{.reg .b64 a, b; mov.b64 a, {%1, %3}; mov.b64 b, {%2, %3}; st.relaxed.gpu.global.v2.b64 [%0], {a, b};}" ::"l"(p),
                 "r"(__float_as_uint(v0)), "r"(__float_as_uint(v1)), "r"(tag) : "memory");
}
__device__ __forceinline__ uint2 get(const uint2* p) {
    uint2 v;
    asm volatile("ld.relaxed.gpu.global.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ bool aborted(const unsigned* p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v != 0;
}

// 384 threads are launched with 168 registers each; 256 x 216 + 128 x 72 is the same sum.
__device__ __forceinline__ void worker_registers() { asm volatile("setmaxnreg.inc.sync.aligned.u32 216;" ::: "memory"); }
__device__ __forceinline__ void helper_registers() { asm volatile("setmaxnreg.dec.sync.aligned.u32 72;" ::: "memory"); }
__device__ __forceinline__ bool workers_or(bool v) {  // a barrier of the multiplying threads alone
    int r;
    asm volatile("{.reg .pred p, q; setp.ne.u32 p, %1, 0; barrier.cta.red.or.pred q, 2, 256, p; selp.s32 %0, 1, 0, q;}" : "=r"(r) : "r"((int)v) : "memory");
    return r != 0;
}
__device__ __forceinline__ void copy16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

__device__ __forceinline__ void rest(int cycles) {
    const unsigned c0 = (unsigned)clock();
    while ((unsigned)clock() - c0 < (unsigned)cycles) {}
}

// v[r][i] <- the value of the word p + r * rstride + i * stride, where `want(r, i)`, once it carries `tag`, else 0; false when a word did not
// come or another CTA gave up.
template <int M, int N, typename F>
__device__ __forceinline__ bool gather(float (&v)[M][N], const uint2* p, size_t rstride, size_t stride, F want, unsigned tag, const unsigned* abort) {
    uint2 w[M][N];
#pragma unroll
    for (int r = 0; r < M; ++r)
#pragma unroll
        for (int i = 0; i < N; ++i) w[r][i] = want(r, i) ? get(p + r * rstride + i * stride) : make_uint2(0u, tag);
    for (unsigned spins = 0;;) {
        bool all = true;
#pragma unroll
        for (int r = 0; r < M; ++r)
#pragma unroll
            for (int i = 0; i < N; ++i)
                if (w[r][i].y != tag) {
                    all = false;
                    w[r][i] = get(p + r * rstride + i * stride);
                }
        if (all) break;
        if (++spins > kSpin || ((spins & 255u) == 0 && aborted(abort))) return false;
    }
#pragma unroll
    for (int r = 0; r < M; ++r)
#pragma unroll
        for (int i = 0; i < N; ++i) v[r][i] = __uint_as_float(w[r][i].x);
    return true;
}

}  // namespace sreg

// Sequences that these kernels take in a launch (0: they do not take the call), and a launch over that many or fewer of them.
// XLSTM_DECLINED: the device has no memory for the exchange words; nothing was launched.
int slstm_reg_batch(const sreg::Args& a, bool bwd);
int slstm_reg_fw(cudaStream_t st, sreg::Args a);
int slstm_reg_bw(cudaStream_t st, sreg::Args a);

}  // namespace xl
