// Instructed (delta-rule) plasticity at frame ends, the drop-in for flyzero/batch.py:226-451
// (BatchInstruct, BatchInstructDeep, BatchInstructDeep2):
//
//   traces:   trace[b][k] += a_pre * (c[b][upre_k] * scale_pre - trace[b][k])        (float32)
//             rate[b][k]  += a_rate * (c[b][upost_k] * hz - rate[b][k])
//   update:   for a set of plastic synapses s (sel), per fly f:
//               d_f[s] = sum over slots b of f: coef_b * trace[b][pre_k[s]] * x[b][post_x[s]]
//             every slot b of fly f:  w = sign * clip(sign * (w + d_f[s]), 0, wmax)
//             (coef_b = eta_b / learning slots of its fly for a learning slot, else 0: the onehot
//             average of batch.py:158-172, or the deep_update kernel's coefficient, batch.py:401-404)
//   backprop: delta[b][pre_l[s]] += (pw[b][sel[s]] / w_syn) * x[b][post_x[s]]      (float atomics,
//             like the reference's scatter_add: the summation order is not fixed)
//
// With x = the DN error (target - rate) the update is the DN synapses' delta rule; with x = the
// retrograde error of layer 1 (2) it is the deep update of the layer behind it.
#pragma once
#include "common.cuh"

namespace fb {

// a thread per neuron and TRACE_ROWS instances, their loads in flight together
constexpr int TRACE_ROWS = 4;
__global__ void __launch_bounds__(256) k_trace_rates(const int32_t* counts, int64_t n, int32_t B, const int32_t* upre,
                                                     int32_t n_upre, float* trace, float a_pre, float scale_pre,
                                                     const int32_t* upost, int32_t n_upost, float* rate, float a_rate, float hz)
{
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= (int64_t)n_upre + n_upost) return;
    const bool pre = k < n_upre;
    const int32_t i = pre ? upre[k] : upost[k - n_upre];
    const float a = pre ? a_pre : a_rate, scale = pre ? scale_pre : hz;
    float* t = pre ? trace + k : rate + (k - n_upre);
    const int64_t stride = pre ? n_upre : n_upost;
    for (int32_t b0 = blockIdx.y * TRACE_ROWS; b0 < B; b0 += gridDim.y * TRACE_ROWS) {
        float c[TRACE_ROWS], x[TRACE_ROWS];
#pragma unroll
        for (int u = 0; u < TRACE_ROWS; u++)
            if (b0 + u < B) {
                c[u] = (float)counts[(int64_t)(b0 + u) * n + i];
                x[u] = t[(b0 + u) * stride];
            }
#pragma unroll
        for (int u = 0; u < TRACE_ROWS; u++)
            if (b0 + u < B) t[(b0 + u) * stride] = __fadd_rn(x[u], __fmul_rn(a, __fsub_rn(__fmul_rn(c[u], scale), x[u])));
    }
}

struct DeltaArgs {
    int32_t B, n_flies, n_sel, n_tr, n_x;
    int64_t n_pl;
    const int32_t* sel;        // (n_sel) plastic entry of each synapse of the set
    const int32_t* pre_k;      // (n_sel) its presynaptic trace index
    const int32_t* post_x;     // (n_sel) its column of x
    const float* trace;        // (B, n_tr)
    const float* x;            // (B, n_x)
    const float* coef;         // (B)
    const int32_t* fly_ptr;    // (n_flies + 1) slots of each fly: fly_slots[fly_ptr[f] .. fly_ptr[f+1])
    const int32_t* fly_slots;
    const float* sign;         // (n_pl)
    const float* wmax;         // (n_pl)
    float* pw;                 // (B, n_pl)
};

__device__ __forceinline__ void delta_clip(const DeltaArgs& a, int32_t b, int32_t j, float d, float sg, float mx)
{
    float* w = a.pw + (int64_t)b * a.n_pl + j;
    const float v = __fmul_rn(sg, __fadd_rn(*w, d));
    *w = __fmul_rn(sg, fminf(fmaxf(v, 0.0f), mx));
}

// One thread per synapse of the set and DELTA_FLIES flies (blockIdx.y: which). Consecutive threads take
// consecutive synapses: `sel` ascends, so a warp's weights are one run of pw and its traces a handful
// of values (a presynaptic neuron's synapses are neighbours). With the flies fastest instead, each
// weight was a sector of its own (64 slots, 793 k synapses: 406 us against 206). Staging the slots'
// tables, or the rows of x, in shared memory to load more at once measured slower (269, 304 us).
constexpr int DELTA_FLIES = 8;
__global__ void __launch_bounds__(256) k_delta_apply(const DeltaArgs a)
{
    const int32_t s = (int32_t)(blockIdx.x * blockDim.x + threadIdx.x);
    if (s >= a.n_sel) return;
    const int32_t j = a.sel[s], pk = a.pre_k[s], px = a.post_x[s];
    for (int32_t f0 = blockIdx.y * DELTA_FLIES; f0 < a.n_flies; f0 += gridDim.y * DELTA_FLIES)
        for (int32_t f = f0; f < min(a.n_flies, f0 + DELTA_FLIES); f++) {
            const int32_t q0 = a.fly_ptr[f], q1 = a.fly_ptr[f + 1];
            float d = 0.0f;
            for (int32_t q = q0; q < q1; q++) {
                const int32_t b = a.fly_slots[q];
                const float c = a.coef[b];
                if (c != 0.0f)
                    d = __fadd_rn(d, __fmul_rn(__fmul_rn(c, a.trace[(int64_t)b * a.n_tr + pk]), a.x[(int64_t)b * a.n_x + px]));
            }
            if (d == 0.0f) continue;
            const float sg = a.sign[j], mx = a.wmax[j];
            for (int32_t q = q0; q < q1; q++) delta_clip(a, a.fly_slots[q], j, d, sg, mx);
        }
}

__global__ void __launch_bounds__(256) k_backprop(int32_t B, int32_t n_sel, const int32_t* sel, const int32_t* pre_l,
                                                  const int32_t* post_x, const float* x, int32_t n_x, const float* pw,
                                                  int64_t n_pl, float w_syn, float* delta, int32_t n_delta)
{
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n_sel) return;
    const int32_t j = sel[s], to = pre_l[s], from = post_x[s];
    for (int32_t b = blockIdx.y; b < B; b += gridDim.y) {
        const float v = __fmul_rn(__fdiv_rn(pw[(int64_t)b * n_pl + j], w_syn), x[(int64_t)b * n_x + from]);
        atomicAdd(delta + (int64_t)b * n_delta + to, v);
    }
}

}  // namespace fb
