// Shared pieces of the chunk-parallel mLSTM kernels (mlstm_par_scan.cu, mlstm_par_out.cu, mlstm_par_grad.cu).
#pragma once
#include <cuda.h>

#include "common.cuh"
#include "mlstm.cuh"
#include "tc.cuh"

namespace xl {

int* tc_status_ptr();
bool tc_make_map4(CUtensorMap* m, const void* base, int elem_bytes, int B, uint64_t T, int W, int rows, int groups);

namespace par {

using namespace tc;

static constexpr int LC = 128;               // positions per chunk
static constexpr uint32_t kBox = 128 * 128;  // bytes of a tile: 128 rows x 64 bf16, 128-byte swizzle
static constexpr uint32_t kPair = 2 * kBox;  // 128 x 128 as two tiles

// Per-position and per-chunk vectors of a call, fp32. Positions past T: rowt = colt = -inf, a = b = dqn = bq = 0.
struct Vecs {
    float *rowt, *colt, *a, *b;  // [BH][Tp]: fc - m, i - fc, state weight, inter-chunk factor
    float *dqn, *bq;             // backward: gradient of q.n, b * dqn
    float* g;                    // [BH][NC] decay of a whole chunk
    int Tp;                      // NC * 128
};
inline size_t vecs_bytes(int BH, int NC, bool bwd) {
    return align_up((size_t)(bwd ? 6 : 4) * BH * NC * LC * 4, 256) + align_up((size_t)BH * NC * 4, 256);
}
inline Vecs vecs_at(void* base, int BH, int NC, bool bwd) {
    Vecs v = {};
    const size_t n = (size_t)BH * NC * LC;
    float* f = (float*)base;
    v.rowt = f; v.colt = f + n; v.a = f + 2 * n; v.b = f + 3 * n;
    if (bwd) { v.dqn = f + 4 * n; v.bq = f + 5 * n; }
    v.g = (float*)((char*)base + align_up((size_t)(bwd ? 6 : 4) * n * 4, 256));
    v.Tp = NC * LC;
    return v;
}

// The state record: C entering every chunk and the final one, bf16 [BH][NC+1][D][D], then n, fp32 [BH][NC+1][D].
inline size_t record_C_bytes(int BH, int NC, int D) { return align_up((size_t)BH * (NC + 1) * D * D * 2, 256); }
inline size_t record_n_bytes(int BH, int NC, int D) { return align_up((size_t)BH * (NC + 1) * D * 4, 256); }

struct ScanArgs {           // one state recurrence: forward over (a.V, K) or backward over (b.dN, Q)
    const void *x, *y;      // [B*T, H*D] bf16: rows of the state (v), columns of the state (qk)
    const float* w;         // [BH][Tp]: weights of n's sum; forward: also scales x
    const float* g;         // [BH][NC]
    const float *c0, *n0;   // state the walk starts from, fp32 [BH][D][D], [BH][D], or null = 0
    void* recC;             // bf16 [BH][entries][D][D]; entry k: the state before chunk k's update
    float* recn;
    float *oC, *on;         // state after the walk, or null
    int B, H, T, D, NC, entries;
    bool bwd;
};
int scan_launch(cudaStream_t st, const ScanArgs& a);
int gates_launch(cudaStream_t st, const float* ig, const float* fg, const float* m_in, float* m, float* m_last, const Vecs& v,
                 int B, int H, int T, int NC, bool from_m, bool exact);

// Eight or four k16 steps of a product, issued by a converged warp. Descriptor arithmetic stays out of the loop: a step is a constant
// added to the start address field (K-major: 32 bytes a step, four steps to a tile; MN-major: sixteen 128-byte rows a step).
template <int STEPS, bool A_MN, bool B_MN>
__device__ __forceinline__ void product(uint32_t acc, uint64_t a, uint64_t b, uint32_t id, bool fresh) {
#pragma unroll
    for (int k = 0; k < STEPS; ++k) {
        const uint32_t oa = A_MN ? k * 128 : (k >> 2) * (kBox >> 4) + (k & 3) * 2, ob = B_MN ? k * 128 : (k >> 2) * (kBox >> 4) + (k & 3) * 2;
        mma_ss_w(acc, a + oa, b + ob, id, k > 0 || !fresh);
    }
}

// C-ordered units over a persistent grid: unit -> (bh, chunk, 128-wide half of the head)
__device__ __forceinline__ void unit_of(int u, int NS, int NC, int& bh, int& ck, int& f) {
    f = u % NS;
    ck = (u / NS) % NC;
    bh = u / (NS * NC);
}

}  // namespace par
}  // namespace xl
