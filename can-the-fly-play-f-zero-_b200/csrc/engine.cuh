// Device-resident layout of one engine (a connectome shared by B instances) and the
// step engine's kernels. Layout in HBM:
//
//   connectome  rowptr[n+1] i64 (rows padded to 8 entries), col[nnz_pad] i32,
//               cnt[nnz_pad] i16 (INT32 mode) or wfx[nnz_pad] i64 (Q32.32 mode)
//   plastic     pl_rowptr[n+1] i64 (by presynaptic neuron), pl_pidx[n_pl] i32 (compact target),
//               pl_q0[n_pl] i64, ppost_of[n] i32 (compact target index or -1), pw[B][n_pl] f32.
//               Plastic entries keep their connectome weight in the fixed CSR; an instance's
//               weight pw enters as the Q32.32 delta q32(pw) - q32(w0), pushed at spike time.
//   state       v[B][n], g[B][n] (f32 or f64), ref[B][n] i8
//   inputs      ext_idx[n] i32, p_ext[B][n_ext] f32, bias_ext[B][n_ext] f32
//   delay line  acc[S][B][n_pad] (i16, i32 or i64): synaptic input of the next S ticks (slot = tick mod
//               S, S = 2 x the persistent engine's epoch, at least 2; 2 in the step engine's own array where
//               the persistent engine's is 16 bits wide), rows padded to 16 entries so that every row
//               starts on a 16-byte boundary at any accumulator width;
//               items[R][n_groups][cap_c] int2: spike work lists of the last R = n_delay + 1 steps, one per
//               instance group (a list is overwritten after its arrivals were pushed);
//               item_count[R_pl][n_groups], R_pl = n_delay + K (K: the persistent engine's epoch, 1
//               without it): a count is zeroed K steps before its list is filled again;
//               pring[R_pl][B][n_ppost] i64: plastic input (a slot is cleared by its reader at least
//               one epoch before anyone pushes into it again);
//               with pull propagation also masks[R][n][ceil(B/64)] u64: which instances each
//               neuron spiked in, and the connectome by postsynaptic neuron (colptr, cpre, ccnt/cwfx)
//
// The delay line is "deferred push": the fixed-weight rows of the spikes of step s are scattered
// into acc only shortly before they arrive (the step engine at step s + n_delay - 1, the
// persistent engine one epoch ahead), so only S accumulator slots (instead of n_delay) are live.
// Fixed weights never change during a run and integer addition is order-free, so this equals the
// reference's push-at-spike-time ring (brain.py:54-56) exactly.
// Plastic weights may change between runs, so their rows are pushed at spike time.
#pragma once
#include "chain.cuh"
#include "common.cuh"

namespace fb {

struct DevNet {
    int64_t n, n_pad;
    int32_t B, n_delay, R, n_ref;
    int32_t R_pl;              // slots of the plastic input and of the list lengths: n_delay + the persistent engine's epoch
    const int64_t* rowptr;
    const int32_t* col;
    const int16_t* cnt;
    const int64_t* wfx;
    int64_t n_pl;
    int32_t n_ppost;
    const int64_t* pl_rowptr;
    const int32_t* pl_pidx;
    const int64_t* pl_q0;      // q32 of each plastic entry's connectome weight
    const int32_t* ppost_of;
    const int64_t* colptr;     // pull propagation: the connectome by postsynaptic neuron (or nullptr)
    const int32_t* cpre;
    const int16_t* ccnt;
    const int64_t* cwfx;
    Lif<float> L32;
    Lif<double> L64;
};

struct DevState {
    void* v;
    void* g;
    int8_t* ref;
    const float* pw;
    const int32_t* ext_idx;
    int32_t n_ext;
    const float* p_ext;
    const float* bias_ext;
    void* acc;                 // [n_slots][B][n_pad]
    int32_t n_slots;
    int64_t* pring;
    int2* items;               // [R][n_groups][cap_c]
    int32_t* item_count;       // [R_pl][n_groups]
    int64_t cap_c;             // items per (step, group) list
    int32_t group;             // instances per group (group of instance b = b / group)
    int32_t n_groups;
    const int64_t* reset_tick;
    const int64_t* stop_tick;
    unsigned long long* masks; // pull propagation: [R][n][mask_words] spiking instances per neuron (or nullptr)
    int32_t mask_words;        // ceil(B / 64)
    int32_t* err;              // [0] overflow, [1] barrier timeout step (host-mapped)
    uint32_t seed;
};

struct StepArgs {
    int64_t t;                 // tick of this step
    uint32_t step_no;          // Poisson hash counter
    int32_t s;                 // index of this step within the run
    const uint32_t* kicks;     // raster of this run or nullptr
    int32_t words;             // raster words per instance-step
    int32_t* counts;           // (B, n) this run's counts
    int32_t* step_counts;      // (steps, B) or nullptr
    uint64_t* step_digest;     // (steps, B) or nullptr
};

__device__ __forceinline__ int64_t pos_mod(int64_t a, int64_t m) { int64_t r = a % m; return r < 0 ? r + m : r; }

__device__ __forceinline__ bool bits_differ(float a, float b) { return __float_as_uint(a) != __float_as_uint(b); }
__device__ __forceinline__ bool bits_differ(double a, double b)
{
    return __double_as_longlong(a) != __double_as_longlong(b);
}

// accumulator slot of tick t
template <typename AccT> __device__ __forceinline__ AccT* acc_slot(const DevNet& N, const DevState& S, int64_t t)
{
    return reinterpret_cast<AccT*>(S.acc) + pos_mod(t, S.n_slots) * (int64_t)N.B * N.n_pad;
}

template <typename Real> __device__ __forceinline__ const Lif<Real>& lif_of(const DevNet& N);
template <> __device__ __forceinline__ const Lif<float>& lif_of<float>(const DevNet& N) { return N.L32; }
template <> __device__ __forceinline__ const Lif<double>& lif_of<double>(const DevNet& N) { return N.L64; }

// the work list of step t and group q, and its length
__device__ __forceinline__ int2* list_of(const DevNet& N, const DevState& S, int64_t t, int32_t q)
{
    return S.items + (pos_mod(t, N.R) * S.n_groups + q) * S.cap_c;
}
__device__ __forceinline__ int32_t* count_of(const DevNet& N, const DevState& S, int64_t t, int32_t q)
{
    return S.item_count + pos_mod(t, N.R_pl) * S.n_groups + q;
}

// Fire-and-forget reductions into global memory (no value comes back; the address is converted to
// the global window explicitly, so the hardware never falls back to a returning generic atomic).
// No "memory" clobber: the reduced words are never read in the phase that reduces into them, and
// leaving the clobber out lets the compiler issue the next edges' loads before these reductions.
__device__ __forceinline__ void red_add(int32_t* p, int32_t x)
{
    asm volatile("red.relaxed.gpu.global.add.s32 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "r"(x));
}
__device__ __forceinline__ void red_add(int64_t* p, int64_t x)
{
    asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "l"(x));
}

// A work item: up to CHUNK consecutive entries of a spiking row, {first entry in the padded CSR,
// (instance << CHUNK_BITS) | number of entries}.
__device__ __forceinline__ int2 make_item(const DevNet& N, int32_t i, int32_t b, int c)
{
    const int64_t r0 = N.rowptr[i], r1 = N.rowptr[i + 1];
    const int64_t k0 = r0 + (int64_t)c * CHUNK;
    return make_int2((int32_t)k0, (b << CHUNK_BITS) | (int32_t)min((int64_t)CHUNK, r1 - k0));
}

// Append `nch` work items (this lane's spike: chunks 0..nch-1 of row i of instance b) to the list of
// the lane's group; one atomic per warp and list (the ballot/shuffle compaction). The step engine's blocks hold
// one instance, so one list; written without the search for others its step was slower (100 steps of 16 x 16,384 in
// FP64: 756 us and 729).
__device__ __forceinline__ void warp_append(const DevNet& N, const DevState& S, int64_t t, int nch, int32_t i,
                                            int32_t b)
{
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    unsigned todo = __ballot_sync(FULL, nch > 0);
    if (!todo) return;
    const int32_t key = nch > 0 ? b / S.group : -1;
    while (todo) {
        const int leader = __ffs(todo) - 1;
        const int32_t kk = __shfl_sync(FULL, key, leader);
        const bool mine = nch > 0 && key == kk;
        int incl = mine ? nch : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += y;
        }
        const int total = __shfl_sync(FULL, incl, 31);
        int base = 0;
        if (lane == 31) base = atomicAdd(count_of(N, S, t, kk), total);
        base = __shfl_sync(FULL, base, 31);
        if (mine) {
            int2* list = list_of(N, S, t, kk);
            const int64_t start = (int64_t)base + incl - nch;
            for (int ch = 0; ch < nch; ch++) {
                const int64_t p = start + ch;
                if (p < S.cap_c) list[p] = make_item(N, i, b, ch);
                else atomicExch(S.err, 1);
            }
        }
        todo &= ~__ballot_sync(FULL, mine);
    }
}

// Plastic row of a spiking neuron, pushed at spike time into the ring slot it arrives from.
__device__ __forceinline__ void push_plastic_row(const DevNet& N, const DevState& S, int64_t t, int32_t b, int32_t i)
{
    const int64_t p0 = N.pl_rowptr[i], p1 = N.pl_rowptr[i + 1];
    if (p0 == p1) return;
    unsigned long long* dst = reinterpret_cast<unsigned long long*>(
        S.pring + (pos_mod(t + N.n_delay, N.R_pl) * N.B + b) * (int64_t)N.n_ppost);
    const float* w = S.pw + (int64_t)b * N.n_pl;
    for (int64_t k = p0; k < p1; k++) {
        const int64_t d = to_q32(w[k]) - N.pl_q0[k];
        if (d != 0) red_add(reinterpret_cast<int64_t*>(dst) + N.pl_pidx[k], d);
    }
}

// The same for networks whose plastic rows are long (several plastic synapses per presynaptic
// neuron): four entries at a time, their loads in flight together, then their reductions (a
// reduction between two loads keeps the second from being issued early). Same sums.
__device__ __forceinline__ void push_plastic_row_batched(const DevNet& N, const DevState& S, int64_t t, int32_t b,
                                                         int32_t i)
{
    const int64_t p0 = N.pl_rowptr[i], p1 = N.pl_rowptr[i + 1];
    if (p0 == p1) return;
    int64_t* dst = S.pring + (pos_mod(t + N.n_delay, N.R_pl) * N.B + b) * (int64_t)N.n_ppost;
    const float* w = S.pw + (int64_t)b * N.n_pl;
    for (int64_t k0 = p0; k0 < p1; k0 += 4) {
        float wv[4];
        int64_t q0[4];
        int32_t pi[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int64_t k = min(k0 + u, p1 - 1);
            wv[u] = w[k];
            q0[u] = N.pl_q0[k];
            pi[u] = N.pl_pidx[k];
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int64_t d = to_q32(wv[u]) - q0[u];
            if (k0 + u < p1 && d != 0) red_add(dst + pi[u], d);
        }
    }
}

// Arriving plastic input of (b, i) at tick t, read and cleared (L2 only: other SMs wrote it).
template <typename Real>
__device__ __forceinline__ Real take_plastic(const DevNet& N, const DevState& S, int64_t t, int32_t b, int32_t i)
{
    const int32_t pp = N.ppost_of[i];
    int64_t* q = S.pring + (pos_mod(t, N.R_pl) * N.B + b) * (int64_t)N.n_ppost + pp;
    const int64_t px = __ldcg(reinterpret_cast<const long long*>(q));
    if (px != 0) *q = 0;
    return from_q32<Real>(px);
}

// Poisson kick of ext slot j of instance b at run step s (raster) or hash draw.
template <bool RASTER>
__device__ __forceinline__ bool kick_of(const DevState& S, const uint32_t* kicks, int32_t words, int32_t B, int32_t s,
                                        int32_t b, int32_t j, uint32_t tid, uint32_t step_no)
{
    if (RASTER) {
        const uint32_t w = kicks[((int64_t)s * B + b) * words + (j >> 5)];
        return (w >> (j & 31)) & 1u;
    }
    const float p = S.p_ext[(int64_t)b * S.n_ext + j];
    return p > 0.0f && hash_kick(tid, step_no, S.seed, (uint32_t)b, p);
}

// Step engine, one part: the pairs (b, i) of a warp advance one step; spikes become work items.
template <typename Real, typename AccT, bool RASTER, bool PLASTIC, bool RECORD>
__device__ __forceinline__ void update_pair(const DevNet& N, const DevState& S, const StepArgs& A, int32_t b, int64_t i64)
{
    const int64_t n = N.n, t = A.t;
    const Lif<Real>& L = lif_of<Real>(N);
    const int32_t i = (int32_t)i64;
    int nch = 0;
    if (i64 < n && t < S.stop_tick[b]) {
        const int64_t pair = (int64_t)b * n + i;
        AccT* ap = acc_slot<AccT>(N, S, t) + (int64_t)b * N.n_pad + i;
        Real* pv = reinterpret_cast<Real*>(S.v) + pair;
        Real* pg = reinterpret_cast<Real*>(S.g) + pair;
        const AccT x = *ap;                              // (independent loads: in flight together)
        Real v = *pv, g = *pg;
        const int r0 = S.ref[pair];
        const int32_t j = S.ext_idx[i];
        const bool target = PLASTIC && N.ppost_of[i] >= 0;
        if (x != 0) *ap = 0;
        Real buf = acc_to_real<Real>(x, L.w_syn);
        if (target) buf = add_rn(buf, take_plastic<Real>(N, S, t, b, i));
        const Real v0 = v, g0 = g;
        int r = r0;
        float bias = 0.0f;
        bool kicked = false;
        if (j >= 0) {
            bias = S.bias_ext[(int64_t)b * S.n_ext + j];
            kicked = kick_of<RASTER>(S, A.kicks, A.words, N.B, A.s, b, j, (uint32_t)pair, A.step_no);
        }
        // the engine always fuses the two multiply-adds, as the shipped reference kernel does
        const bool spk = lif_step<Real>(v, g, r, buf, j >= 0, bias, kicked, L, N.n_ref, true);
        if (bits_differ(g, g0)) *pg = g;
        if (bits_differ(v, v0)) *pv = v;
        if (r != r0) S.ref[pair] = (int8_t)r;
        if (spk) {
            A.counts[pair] += 1;
            if (S.masks) atomicOr(S.masks + (pos_mod(t, N.R) * n + i) * S.mask_words + (b >> 6), 1ull << (b & 63));
            const int64_t len = N.rowptr[i + 1] - N.rowptr[i];
            nch = (int)((len + CHUNK - 1) / CHUNK);
            if (PLASTIC) push_plastic_row(N, S, t, b, i);
            if (RECORD) {
                if (A.step_counts) atomicAdd(A.step_counts + (int64_t)A.s * N.B + b, 1);
                if (A.step_digest)
                    atomicAdd(reinterpret_cast<unsigned long long*>(A.step_digest + (int64_t)A.s * N.B + b),
                              (unsigned long long)spike_tag((uint64_t)i));
            }
        }
    }
    warp_append(N, S, t, nch, i, b);
}

// 8 consecutive CSR entries of one lane: weights (one or four 16-byte loads) and columns (two).
template <typename AccT> struct Edges8;
template <> struct Edges8<int32_t> {
    int32_t w[8];
    int32_t c[8];
    __device__ __forceinline__ void load(const DevNet& N, int64_t k)
    {
        const int4 cw = __ldg(reinterpret_cast<const int4*>(N.cnt + k));
        const int4 c0 = __ldg(reinterpret_cast<const int4*>(N.col + k));
        const int4 c1 = __ldg(reinterpret_cast<const int4*>(N.col + k + 4));
        const uint32_t u[4] = {(uint32_t)cw.x, (uint32_t)cw.y, (uint32_t)cw.z, (uint32_t)cw.w};
#pragma unroll
        for (int q = 0; q < 4; q++) {
            w[2 * q] = (int32_t)(int16_t)(u[q] & 0xffffu);
            w[2 * q + 1] = (int32_t)(int16_t)(u[q] >> 16);
        }
        c[0] = c0.x; c[1] = c0.y; c[2] = c0.z; c[3] = c0.w;
        c[4] = c1.x; c[5] = c1.y; c[6] = c1.z; c[7] = c1.w;
    }
};
template <> struct Edges8<int64_t> {
    int64_t w[8];
    int32_t c[8];
    __device__ __forceinline__ void load(const DevNet& N, int64_t k)
    {
        const longlong2* p = reinterpret_cast<const longlong2*>(N.wfx + k);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const longlong2 x = __ldg(p + q);
            w[2 * q] = x.x;
            w[2 * q + 1] = x.y;
        }
        const int4 c0 = __ldg(reinterpret_cast<const int4*>(N.col + k));
        const int4 c1 = __ldg(reinterpret_cast<const int4*>(N.col + k + 4));
        c[0] = c0.x; c[1] = c0.y; c[2] = c0.z; c[3] = c0.w;
        c[4] = c1.x; c[5] = c1.y; c[6] = c1.z; c[7] = c1.w;
    }
};

// Scatter one work item (<= CHUNK entries of a spiking row) with LANES lanes, 8 entries a lane.
template <typename AccT, int LANES>
__device__ __forceinline__ void push_item(const DevNet& N, AccT* acc_b, int64_t k0, int32_t len, int lane)
{
    const int64_t k1 = k0 + len;
#pragma unroll 2
    for (int64_t k = k0 + (int64_t)lane * 8; k < k1; k += LANES * 8) {
        Edges8<AccT> e;
        e.load(N, k);
#pragma unroll
        for (int q = 0; q < 8; q++)
            if (e.w[q] != 0) red_add(acc_b + e.c[q], e.w[q]);
    }
}

// Items of the list of step t and group q: its count, clamped to the capacity (L2: other SMs appended to it)
__device__ __forceinline__ int32_t list_length(const DevNet& N, const DevState& S, int64_t t, int32_t q)
{
    return (int32_t)min((int64_t)max(__ldcg(count_of(N, S, t, q)), 0), S.cap_c);
}

// Scatter the items [g0, g1) of the list of spike step s = t+1-n_delay and group q into acc_next; lane
// group `lg` of `n_lg` (LANES lanes each, lane `lane` within it) takes items g0+lg, g0+lg+n_lg, ...
// Items of instance b are skipped unless reset_tick[b] <= s and t+1 < stop_tick[b].
template <typename AccT, int LANES>
__device__ __forceinline__ void push_range(const DevNet& N, const DevState& S, int64_t t, int32_t q, AccT* acc_next,
                                           int64_t g0, int64_t g1, int64_t lg, int64_t n_lg, int lane)
{
    const int64_t s = t + 1 - N.n_delay;
    const int2* list = list_of(N, S, s, q);
    for (int64_t g = g0 + lg; g < g1; g += n_lg) {
        const int2 item = __ldcg(list + g);
        const int32_t b = item.y >> CHUNK_BITS;
        if (s < S.reset_tick[b] || t + 1 >= S.stop_tick[b]) continue;
        push_item<AccT, LANES>(N, acc_next + (int64_t)b * N.n_pad, (int64_t)(uint32_t)item.x,
                               item.y & ((1 << CHUNK_BITS) - 1), lane);
    }
}

// The spike-mask slot that step t+1 records into starts empty (it last held step t-n_delay, whose
// propagation ran at step t-1).
__device__ __forceinline__ void clear_mask_slot(const DevNet& N, const DevState& S, int64_t t, int blk, int n_blk)
{
    if (!S.masks) return;
    const int64_t words = N.n * S.mask_words;
    unsigned long long* m = S.masks + pos_mod(t + 1, N.R) * words;
    for (int64_t k = (int64_t)blk * blockDim.x + threadIdx.x; k < words; k += (int64_t)n_blk * blockDim.x) m[k] = 0ull;
}

// Step engine, the other part, block `blk` of `n_blk`: the spikes of step t+1-n_delay (they arrive at
// step t+1) are scattered into the accumulator that step t+1 reads; each block takes a contiguous
// share of every list.
template <typename AccT>
__device__ __forceinline__ void push_lists(const DevNet& N, const DevState& S, int64_t t, int lanes, int blk, int n_blk)
{
    AccT* acc = acc_slot<AccT>(N, S, t + 1);
    __shared__ int32_t s_total;
    for (int32_t q = 0; q < S.n_groups; q++) {
        if (threadIdx.x == 0) s_total = list_length(N, S, t + 1 - N.n_delay, q);     // (one load per block: they all hit one address)
        __syncthreads();
        const int64_t total = s_total;
        const int64_t g0 = total * blk / n_blk, g1 = total * (blk + 1) / n_blk;
        const int64_t lg = threadIdx.x / lanes, n_lg = blockDim.x / lanes;
        const int lane = threadIdx.x % lanes;
        if (lanes == 8) push_range<AccT, 8>(N, S, t, q, acc, g0, g1, lg, n_lg, lane);
        else if (lanes == 16) push_range<AccT, 16>(N, S, t, q, acc, g0, g1, lg, n_lg, lane);
        else push_range<AccT, 32>(N, S, t, q, acc, g0, g1, lg, n_lg, lane);
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------------------------
// Step engine: one launch per step. The first n_push blocks scatter the spikes that arrive at t+1, the
// others advance every (instance, neuron) through step t, `per` blocks an instance and `tiles` pairs a thread. The two touch
// different accumulator slots (t+1 and t) and, with n_delay >= 2, different lists: the pushed one
// (step t+1-n_delay) was filled by an earlier launch, the one that starts empty here held step t-n_delay,
// pushed by the launch before. With n_delay = 1 the pushed spikes are this step's own, so the host
// launches the two parts one after the other (n_push = 0, then pushing blocks alone).
// `do_push` 0: the arrivals of t+1 were pushed ahead already (by the persistent engine); only the mask
// slot is cleared.
// Small networks are bound by a launch's chain of dependent loads (list length, item, edges;
// accumulator, state, kick): 16 x 16,384 FP64 took 14.6 us a step as two ordinary launches and takes 7.0,
// 4 x 1,000 11.7 and 4.0. Large ones are bound by the state's traffic in L2: 16 x 138,639 FP64 30.7 as two
// launches and 22.8, 64 x 138,639 FP32 123 and 94 (one launch, but a tile a block: 28.5 and 127).
// ---------------------------------------------------------------------------------------------
struct StepGrid {
    int32_t n_push, per;       // pushing blocks; updating blocks per instance
    int32_t tiles;             // 256 neurons each of an updating block
    int32_t do_push, lanes;
};

template <typename Real, typename AccT, bool RASTER, bool PLASTIC, bool RECORD>
__global__ void __launch_bounds__(256) k_step(const __grid_constant__ DevNet N, const __grid_constant__ DevState S,
                                              const __grid_constant__ StepArgs A, const StepGrid G)
{
    pdl_chain();
    if ((int)blockIdx.x < G.n_push) {
        clear_mask_slot(N, S, A.t, (int)blockIdx.x, G.n_push);
        if (G.do_push && A.t + 1 - N.n_delay >= 0) push_lists<AccT>(N, S, A.t, G.lanes, (int)blockIdx.x, G.n_push);
        return;
    }
    const uint32_t u = blockIdx.x - (uint32_t)G.n_push;
    const int32_t b = (int32_t)(u / (uint32_t)G.per);
    if (u == 0)                // the lists consumed by the push at t-1 start empty again
        for (int32_t k = threadIdx.x; k < S.n_groups; k += blockDim.x) *count_of(N, S, A.t - N.n_delay, k) = 0;
    const int64_t i0 = (int64_t)(u % (uint32_t)G.per) * G.tiles * 256 + threadIdx.x;
#pragma unroll 1
    for (int k = 0; k < G.tiles; k++) update_pair<Real, AccT, RASTER, PLASTIC, RECORD>(N, S, A, b, i0 + k * 256);
}

// ---------------------------------------------------------------------------------------------
// Pull propagation (step engine, in place of the pushing blocks): every postsynaptic neuron j gathers its
// incoming entries whose presynaptic neuron spiked at step s = t+1-n_delay, for the instances of
// one 64-bit mask word per thread. The sums are exact integers, so push and pull give identical
// accumulators; pull reads the whole connectome once per step for all instances, push only the
// rows of the spikes (it pays off only when a large share of neurons fires every step).
// ---------------------------------------------------------------------------------------------
template <typename AccT> __device__ __forceinline__ AccT pull_weight(const DevNet& N, int64_t e);
template <> __device__ __forceinline__ int32_t pull_weight<int32_t>(const DevNet& N, int64_t e) { return N.ccnt[e]; }
template <> __device__ __forceinline__ int64_t pull_weight<int64_t>(const DevNet& N, int64_t e) { return N.cwfx[e]; }

template <typename AccT>
__global__ void __launch_bounds__(256) k_pull(const DevNet N, const DevState S, int64_t t)
{
    clear_mask_slot(N, S, t, (int)blockIdx.x, (int)gridDim.x);
    const int64_t s = t + 1 - N.n_delay;
    if (s < 0) return;
    AccT* acc = acc_slot<AccT>(N, S, t + 1);
    const int W = S.mask_words;
    const unsigned long long* M = S.masks + pos_mod(s, N.R) * N.n * W;
    const int64_t total = N.n * W;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < total; p += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = p / W;
        const int w = (int)(p - j * W);
        const int64_t e1 = N.colptr[j + 1];
        for (int64_t e = N.colptr[j]; e < e1; e++) {
            unsigned long long m = __ldg(M + (int64_t)N.cpre[e] * W + w);
            if (!m) continue;
            const AccT c = pull_weight<AccT>(N, e);
            while (m) {
                const int32_t b = w * 64 + __ffsll((long long)m) - 1;
                m &= m - 1;
                if (s < S.reset_tick[b] || t + 1 >= S.stop_tick[b]) continue;
                acc[(int64_t)b * N.n_pad + j] += c;     // (b, j) belongs to this thread alone
            }
        }
    }
}

}  // namespace fb
