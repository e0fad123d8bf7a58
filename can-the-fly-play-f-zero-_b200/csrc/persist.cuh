// Persistent engine: one cooperative launch runs all steps of a run for one group of instances.
//
// Instances are independent, so B is split into groups small enough that a group's neuron state
// (v, g f32 + refractory/flag byte = 9 B per instance-neuron) fits in the shared memory of the whole
// GPU (148 x ~227 KB). Each CTA owns a contiguous slice of the group's (instance, neuron) pairs and
// keeps their state in shared memory for the whole run.
//
// Epochs: the spikes of a step arrive n_delay steps later, so with 2K <= n_delay everything that
// arrives during an epoch of K steps (at most MAX_EPOCH) is known one epoch ahead, and with 3K <=
// n_delay there is an epoch to spare for listing. In epoch e, which covers the ticks [T, T + K), the
// warps of a CTA
//   advance   every pair through all K steps at once: its K accumulator values are read from L2
//             (and cleared), its state is loaded and stored once, and no barrier separates the
//             steps. The pairs are taken in tiles of 128 from a shared counter;
//   list      (LIST_WARPS) the spikes of epoch e - 1: counts, plastic rows, and the work items of
//             the group's list of each step. With 3K > n_delay the whole CTA lists the epoch's own
//             spikes after the advance instead: no list is late, and the epoch is 2-3 us longer;
//   push      (PUSH_WARPS, or BUSY_PUSH_WARPS) the work items that arrive in [T + K, T + 2K), into the other K of the 2K
//             accumulator slots (slot = tick mod 2K). The items were listed in epoch e - 1 at the
//             latest: T + 2K - 1 - n_delay < T - K (< T where epochs list their own spikes).
// The listing and pushing warps take tiles too when they are done. One grid barrier ends an epoch;
// between arriving at it and waiting for it a CTA draws the next epoch's Poisson kicks.
//
// What bounds an epoch (16 instances of 138,639 neurons, K = 6: 27 us or 4.5 us per step, against 8.4 in the
// step-by-step kernel before): the advance reads 27 MB of accumulators from L2 and the pushes reduce 1.4 M
// entries into them, each about half of the 22 us they take together; the barrier takes 3-4 us.
// Advancing an epoch at a time takes the state's shared-memory traffic (22 B per pair and step) and
// three CTA-level barriers out of every step. 512 threads: with 128 registers each nothing of the
// advance is spilled; at 1,024 threads its spills, behind the queued reductions, made an epoch of 4
// steps 34 us instead of 22, and a routine called from the advance that needs more than half of the
// registers does the same (advance_pairs with two quads per lane group: 40 us per 6 steps).
//
// Every wait is bounded: after ~4 s a CTA raises the timeout flag and every CTA returns (the others
// read the flag in the grid barrier).
#pragma once
#include "engine.cuh"

namespace fb {

constexpr int PT = 512;                 // threads per CTA (128 registers each: nothing of the advance is spilled)
constexpr int TILE = 128;               // pairs a warp advances at a time: a quad of consecutive pairs per lane
constexpr int EV_BUF = 192;             // quads a warp keeps for the pair-by-pair advance
constexpr int SPK_BUF = 1024;           // spikes of one CTA and epoch buffered for the listing warps
constexpr int IN_BUF = 2048;            // input pairs of one CTA with their kick thresholds in shared memory, at least
constexpr long long BARRIER_TIMEOUT_CYCLES = 8000000000LL;   // ~4 s at 1.9 GHz
constexpr int MAX_EPOCH = 6;            // steps per epoch at most
constexpr int K_BITS = 18;              // bits of a local pair index (per < 2^18)

constexpr int PUSH_WARPS = 5;                              // warps that scatter arriving items ...
constexpr int LIST_WARPS = 2;                              // ... and that list the previous epoch's spikes
constexpr int BUSY_PUSH_WARPS = 7;                         // scattering warps in an epoch that follows one with ...
constexpr int BUSY_ENTRIES = 12000;                        // ... more arriving entries than this per step for its CTA
constexpr int PUSH_LANES = 16;                             // lanes that scatter an item
constexpr int LIST_THREADS = 32 * LIST_WARPS;

struct PersistPlan {
    int32_t group = 0;        // instances per launch (0: engine unavailable)
    int32_t n_groups = 1;
    int32_t ctas = 0;
    int64_t per = 0;          // pairs per CTA (multiple of 16)
    int32_t inputs = IN_BUF;  // input pairs of a CTA held in shared memory
    size_t smem = 0;
    size_t smem_max = 0;      // ... that a block can have
    int32_t launches_per_run = 0;
};

struct PersistArgs {
    int64_t t0;
    uint32_t step0;
    int32_t steps;
    const uint32_t* kicks;
    int32_t words;
    int32_t* counts;
    int32_t* step_counts;
    uint64_t* step_digest;
    unsigned int* bar;        // zeroed before the launch
    int32_t* abort_flag;      // zeroed before the launch
    const int2* ext_tab;      // per CTA: input pairs {k | instance << 18, ext slot}
    const int32_t* ext_off;   // (ctas + 1) offsets into ext_tab
    long long* trace;         // nullptr, or (steps, ctas, TRACE_SLOTS) clock64 stamps of each step's phases
    int64_t pushed_until;     // the arrivals of every tick < pushed_until are in the accumulators
    int32_t epoch;            // K: steps between grid barriers (at most n_slots / 2, 2K <= n_delay or K = 1)
    int32_t list_late;        // an epoch's spikes are listed in the next one (3K <= n_delay), else at its own end
    long long barrier_cycles; // the grid barrier's wait budget (SM clock cycles) before it times out
};

// Phase stamps (per step and CTA; SM clock cycles, compare within a CTA), in step order. An epoch's
// steps run together, so its span is divided evenly between them: 0 and 4 a step's share begins (its
// kicks were drawn before the epoch), 1 and 2 likewise, 3 it ends; 8 the listing of the previous
// epoch done. Per epoch, at its first step: 7 push warps start, 10 push warps done; at its last
// step: 5 grid-barrier arrival, 9 the next epoch's kicks drawn, 6 grid-barrier exit.
constexpr int TRACE_SLOTS = 11;

__device__ __forceinline__ unsigned int ld_acquire_u32(const unsigned int* p)
{
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// one pair's accumulator: its value, and the word that holds it cleared
__device__ __forceinline__ int32_t* word_of(int16_t* p) { return reinterpret_cast<int32_t*>((uintptr_t)p & ~(uintptr_t)3); }
__device__ __forceinline__ int32_t ld_acc(int32_t* p) { return __ldcg(p); }
__device__ __forceinline__ int64_t ld_acc(int64_t* p) { return __ldcg(reinterpret_cast<const long long*>(p)); }
__device__ __forceinline__ int32_t ld_acc(int16_t* p)
{
    const int32_t w = __ldcg(word_of(p)), lo = (int32_t)(int16_t)w;
    return ((uintptr_t)p & 2) ? (w - lo) >> 16 : lo;
}
template <typename T> __device__ __forceinline__ void clear_acc(T* p) { *p = 0; }
__device__ __forceinline__ void clear_acc(int16_t* p) { *word_of(p) = 0; }
// the reduction of one entry into its target's accumulator
__device__ __forceinline__ void red_acc(int32_t* p, int32_t w) { red_add(p, w); }
__device__ __forceinline__ void red_acc(int64_t* p, int64_t w) { red_add(p, w); }
__device__ __forceinline__ void red_acc(int16_t* p, int32_t w)
{
    red_add(word_of(p), (int32_t)((uint32_t)w << (8 * ((uint32_t)(uintptr_t)p & 2u))));
}
// what a connectome entry adds, and what a pair's accumulator holds
template <typename AccT> struct SumOf { using T = AccT; };
template <> struct SumOf<int16_t> { using T = int32_t; };
__device__ __forceinline__ int ld_volatile_i32(const int32_t* p) { return *reinterpret_cast<const volatile int32_t*>(p); }

__device__ __forceinline__ long long* trace_at(const PersistArgs& A, int32_t s, int slot)
{
    return A.trace + ((int64_t)s * gridDim.x + blockIdx.x) * TRACE_SLOTS + slot;
}
__device__ __forceinline__ void stamp(const PersistArgs& A, int32_t s, int slot)
{
    if (A.trace) *trace_at(A, s, slot) = clock64();
}

// The grid barrier in two halves, for one thread per CTA with a CTA barrier before the arrival and
// after the wait. The wait is bounded and returns true if the run must stop (timeout here or
// elsewhere).
__device__ __forceinline__ void grid_arrive(const PersistArgs& A)
{
    __threadfence();
    atomicAdd(A.bar, 1u);
}
__device__ __forceinline__ bool grid_wait(const PersistArgs& A, unsigned int target, long long t0, int32_t* err, int tag)
{
    bool stop = false;
    while (ld_acquire_u32(A.bar) < target) {
        if (ld_volatile_i32(A.abort_flag)) { stop = true; break; }
        if (clock64() - t0 > A.barrier_cycles) {
            stop = true;
            atomicExch(A.abort_flag, 1);
            atomicCAS(err + 1, 0, tag);
            break;
        }
    }
    __threadfence();
    return stop;
}

// Shared-memory layout of one CTA (bytes), for `per` pairs.
struct PersistSmem {
    int32_t v, g, ref, kick, special, events, inputs, spk, hash, ticks, misc, total;
    int32_t n_inputs;
    PersistSmem() = default;
    explicit PersistSmem(int32_t per, int32_t n_in = IN_BUF) : n_inputs(n_in)
    {
        const int32_t per4 = (per + 3) / 4;  // quads
        v = 0;
        g = v + per * 4;
        kick = g + per * 4;                  // two words per quad (epoch parity): bit 4 s + j = kick of pair j at step s
        inputs = kick + 2 * per4 * 4;        // n_inputs inputs {local pair | instance << 18, threshold}
        inputs = (inputs + 15) / 16 * 16;
        spk = inputs + 8 * n_inputs;         // two buffers (epoch parity) of SPK_BUF spikes {local pair | step << 18}
        hash = spk + 2 * 4 * SPK_BUF;        // kick hash seeds of (step, instance); per instance the pair-number offset
        ticks = hash + 4 * (MAX_EPOCH + 1) * 64; // reset and stop ticks of up to 64 instances; active steps (epoch parity)
        misc = ticks + 2 * 64 * 8 + 2 * 64 * 4;  // counters
        events = misc + 512;                 // per warp: quad indices (16-bit: per < 2^18) for the pair-by-pair advance
        special = events + PT / 32 * EV_BUF * 2; // quad indices with a plastic target or a bias
        ref = special + per4 * 2;
        ref = (ref + 15) / 16 * 16;          // bits 0-5 refractory, 6 plastic target, 7 nonzero bias
        total = ref + (per + 15) / 16 * 16;
    }
};

// The counters of PersistSmem::misc
struct PersistCnt {
    int32_t n_special;
    int32_t stops[2];                        // an instance stops in (or before) the epoch (epoch parity)
    int32_t tile[2];                         // next tile (epoch parity)
    int32_t n_spk[2];                        // spikes buffered (epoch parity)
    int32_t entries[2];                      // entries scattered in the last epoch (epoch parity)
    int32_t stop;
    int32_t list_at, count_at;               // where the epoch's first step lies in the rings of lists and of their lengths
    int32_t cursor[MAX_EPOCH], base[MAX_EPOCH];  // a listing batch's items per step, and where they start in the lists
};
static_assert(sizeof(PersistCnt) <= 512, "counters fit their block");

// Everything a launch's kernel is given, as one parameter block: the routines of an epoch that stay out
// of line (so that the advance keeps its registers) read it through a reference
struct PersistParams {
    DevNet N;
    DevState S;
    PersistArgs A;
    PersistSmem lay;
    int32_t b0, G, q;         // first instance, instances, index of the group
    int32_t per;              // pairs per CTA
};
__device__ __forceinline__ int64_t first_pair(const PersistParams& P) { return (int64_t)blockIdx.x * P.per; }
// the block's dynamic shared memory (named here, not passed, so that every routine addresses it as such)
extern __shared__ __align__(128) uint8_t persist_smem[];
template <typename T> __device__ __forceinline__ T* smem_at(int32_t offset)
{
    return reinterpret_cast<T*>(persist_smem + offset);
}

__device__ __forceinline__ void list_sync() { asm volatile("bar.sync 3, %0;" ::"n"(LIST_THREADS) : "memory"); }

__device__ __forceinline__ float max3(float a, float b, float c)
{
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// four consecutive accumulators: loaded from L2 (other SMs reduce into them), tested, cleared
struct Acc4i {
    int4 a;
    __device__ __forceinline__ void load(const int32_t* p) { a = __ldcg(reinterpret_cast<const int4*>(p)); }
    __device__ __forceinline__ void zero() { a = make_int4(0, 0, 0, 0); }
    __device__ __forceinline__ bool any() const { return (a.x | a.y | a.z | a.w) != 0; }
    __device__ __forceinline__ static void clear(int32_t* p) { *reinterpret_cast<int4*>(p) = make_int4(0, 0, 0, 0); }
    __device__ __forceinline__ int32_t at(int j) const { return j == 0 ? a.x : j == 1 ? a.y : j == 2 ? a.z : a.w; }
};
struct Acc4l {
    longlong2 a, b;
    __device__ __forceinline__ void load(const int64_t* p)
    {
        a = __ldcg(reinterpret_cast<const longlong2*>(p));
        b = __ldcg(reinterpret_cast<const longlong2*>(p) + 1);
    }
    __device__ __forceinline__ void zero() { a = b = make_longlong2(0, 0); }
    __device__ __forceinline__ bool any() const { return (a.x | a.y | b.x | b.y) != 0; }
    __device__ __forceinline__ static void clear(int64_t* p)
    {
        reinterpret_cast<longlong2*>(p)[0] = make_longlong2(0, 0);
        reinterpret_cast<longlong2*>(p)[1] = make_longlong2(0, 0);
    }
    __device__ __forceinline__ int64_t at(int j) const { return j == 0 ? a.x : j == 1 ? a.y : j == 2 ? b.x : b.y; }
};
// 16-bit accumulators, two pairs to a 32-bit word: a pair's count is added at its half of the word
// (w << 16 for the odd pair), so the word is S_hi * 2^16 + S_lo mod 2^32, which determines both sums as
// long as each fits in 16 signed bits (fb_create checks the connectome's largest input sum).
__device__ __forceinline__ int32_t lo16(int32_t w) { return (int32_t)(int16_t)w; }
__device__ __forceinline__ int32_t hi16(int32_t w) { return (w - lo16(w)) >> 16; }
struct Acc4s {
    int2 a;
    __device__ __forceinline__ void load(const int16_t* p) { a = __ldcg(reinterpret_cast<const int2*>(p)); }
    __device__ __forceinline__ void zero() { a = make_int2(0, 0); }
    __device__ __forceinline__ bool any() const { return (a.x | a.y) != 0; }
    __device__ __forceinline__ static void clear(int16_t* p) { *reinterpret_cast<int2*>(p) = make_int2(0, 0); }
    __device__ __forceinline__ int32_t at(int j) const { return j == 0 ? lo16(a.x) : j == 1 ? hi16(a.x) : j == 2 ? lo16(a.y) : hi16(a.y); }
};
template <typename AccT> struct Acc4Of;
template <> struct Acc4Of<int16_t> { using T = Acc4s; };
template <> struct Acc4Of<int32_t> { using T = Acc4i; };
template <> struct Acc4Of<int64_t> { using T = Acc4l; };

// Kick threshold of an input of probability p: with u = h >> 8 < 2^24 the draw u * 2^-24 < p of
// hash_kick holds exactly when u < ceil(p * 2^24) (the product is exact in float); 0 for p <= 0.
__device__ __forceinline__ int32_t kick_threshold(float p)
{
    return p > 0.0f ? (int32_t)fminf(ceilf(__fmul_rn(p, 16777216.0f)), 16777217.0f) : 0;
}

// One spike of the listing: pair k of this CTA fired at run step s. Counts it, pushes its plastic row and
// records it; its row is [r0, r1) of the padded CSR and its instance b.
template <bool PLASTIC, bool RECORD>
__device__ __forceinline__ void list_one(const PersistParams& P, int32_t k, int32_t s, int64_t& r0, int64_t& r1, int32_t& b)
{
    const DevNet& N = P.N;
    const uint32_t np = (uint32_t)N.n_pad, lp = (uint32_t)(first_pair(P) + k);
    const int32_t bl = (int32_t)(lp / np), i = (int32_t)(lp - (uint32_t)bl * np);
    b = P.b0 + bl;
    r0 = __ldg(N.rowptr + i);
    r1 = __ldg(N.rowptr + i + 1);
    red_add(P.A.counts + (int64_t)b * N.n + i, 1);
    if (PLASTIC) push_plastic_row_batched(N, P.S, P.A.t0 + s, b, i);
    if (RECORD) {
        if (P.A.step_counts) atomicAdd(P.A.step_counts + (int64_t)s * N.B + b, 1);
        if (P.A.step_digest)
            atomicAdd(reinterpret_cast<unsigned long long*>(P.A.step_digest + (int64_t)s * N.B + b),
                      (unsigned long long)spike_tag((uint64_t)i));
    }
}

// A place in a ring of m at most m - 1 before or behind it
__device__ __forceinline__ int32_t wrap(int32_t at, int32_t m) { return at < 0 ? at + m : at >= m ? at - m : at; }
// The list of the step `ds` steps after (before: < 0) the epoch's first and its length. By the tick, list_of and count_of
// take a 64-bit remainder each, and an epoch's chain of listing, pushing and advancing had six of them
__device__ __forceinline__ int2* list_from(const PersistParams& P, int32_t ds)
{
    return P.S.items + ((int64_t)wrap(smem_at<PersistCnt>(P.lay.misc)->list_at + ds, P.N.R) * P.S.n_groups + P.q) * P.S.cap_c;
}
__device__ __forceinline__ int32_t* count_from(const PersistParams& P, int32_t ds)
{
    return P.S.item_count + wrap(smem_at<PersistCnt>(P.lay.misc)->count_at + ds, P.N.R_pl) * P.S.n_groups + P.q;
}

// Its work items at `base`, .. of its step's list
__device__ __forceinline__ void write_items(const PersistParams& P, int2* list, int32_t base, int64_t r0, int64_t r1, int32_t b)
{
    for (int64_t r = r0; r < r1; r += CHUNK, base++) {
        if (base < P.S.cap_c) list[base] = make_int2((int32_t)r, (b << CHUNK_BITS) | (int32_t)min((int64_t)CHUNK, r1 - r));
        else atomicExch(P.S.err, 1);
    }
}
__device__ __forceinline__ int row_items(int64_t r0, int64_t r1) { return (int)((r1 - r0 + CHUNK - 1) / CHUNK); }

// A spike that finds its epoch's buffer full, listed where it is found
template <bool PLASTIC, bool RECORD>
__device__ __noinline__ void list_overflow(const PersistParams& P, int32_t k, int32_t s)
{
    int64_t r0, r1;
    int32_t b;
    list_one<PLASTIC, RECORD>(P, k, s, r0, r1, b);
    const int64_t t = P.A.t0 + s;
    const int nch = row_items(r0, r1);
    if (nch) write_items(P, list_of(P.N, P.S, t, P.q), atomicAdd(count_of(P.N, P.S, t, P.q), nch), r0, r1, b);
}

// The spikes of local pair k (bit 4 s: at step s of the epoch whose first step is s0) into the buffer of
// the epoch's parity; the spikes that find it full are listed at once
template <bool PLASTIC, bool RECORD>
__device__ __forceinline__ void record_spikes(const PersistParams& P, int par, int32_t k, int32_t s0, uint32_t hits)
{
    PersistCnt* C = smem_at<PersistCnt>(P.lay.misc);
    uint32_t* spk = smem_at<uint32_t>(P.lay.spk) + par * SPK_BUF;
    int32_t at = atomicAdd(&C->n_spk[par], __popc(hits));
    for (; hits; hits &= hits - 1, at++) {
        const int ds = (__ffs(hits) - 1) >> 2;
        if (at < SPK_BUF) spk[at] = (uint32_t)k | ((uint32_t)ds << K_BITS);
        else list_overflow<PLASTIC, RECORD>(P, k, s0 + ds);
    }
}

// The buffered spikes (parity par) of the epoch whose first step is s0 (kc steps): counts, plastic rows,
// records, work items. A batch of `stride` spikes (one per thread) reserves its items with one atomic
// per step. Threads tid0 = 0..stride-1: the listing warps, or (`all`) the whole block; the counters of
// the parity are zero again afterwards. `back`: steps from that epoch to the present one.
template <bool PLASTIC, bool RECORD>
__device__ __noinline__ void list_epoch(const PersistParams& P, int par, int32_t s0, int32_t kc, int32_t back, bool all)
{
    PersistCnt* C = smem_at<PersistCnt>(P.lay.misc);
    const uint32_t* spk = smem_at<uint32_t>(P.lay.spk) + par * SPK_BUF;
    const int tid0 = threadIdx.x, stride = all ? PT : LIST_THREADS;
    const int32_t m = min(C->n_spk[par], SPK_BUF);
    auto sync = [&]() {
        if (all) __syncthreads();
        else list_sync();
    };
    for (int32_t j0 = 0; j0 < m; j0 += stride) {
        const int32_t j = j0 + tid0;
        int64_t r0 = 0, r1 = 0;
        int32_t b = 0, at = 0, ds = 0;
        if (j < m) {
            const uint32_t e = spk[j];
            ds = (int32_t)(e >> K_BITS);
            list_one<PLASTIC, RECORD>(P, (int32_t)(e & ((1u << K_BITS) - 1)), s0 + ds, r0, r1, b);
            at = atomicAdd(&C->cursor[ds], row_items(r0, r1));
        }
        sync();
        if (tid0 < kc) {
            const int32_t n = C->cursor[tid0];
            C->cursor[tid0] = 0;
            C->base[tid0] = n ? atomicAdd(count_from(P, tid0 - back), n) : 0;
        }
        sync();
        if (r1 > r0) write_items(P, list_from(P, ds - back), C->base[ds] + at, r0, r1, b);
    }
    sync();
    if (tid0 == 0) C->n_spk[par] = 0;
}

// Kick hash seeds and active steps (parity par) of the epoch of kc steps whose first is s0
template <bool RASTER>
__device__ __forceinline__ void prepare_epoch(const PersistParams& P, int32_t s0, int32_t kc, int par,
                                              int tid0, int stride)
{
    const int64_t* s_stop = smem_at<int64_t>(P.lay.ticks) + 64;
    int32_t* act = reinterpret_cast<int32_t*>(const_cast<int64_t*>(s_stop) + 64) + par * 64;
    uint32_t* s_hash = smem_at<uint32_t>(P.lay.hash);
    if (!RASTER)
        for (int w = tid0; w < kc * 64; w += stride)
            s_hash[w] = mix32((P.A.step0 + (uint32_t)(s0 + (w >> 6))) * 0x9e3779b9u ^ mix32(P.S.seed + (uint32_t)(P.b0 + (w & 63))));
    if (tid0 < 32) {                                            // (whole warps call: the first one)
        bool some = false;
        for (int w = tid0; w < 64; w += 32) {
            act[w] = (int32_t)max((int64_t)0, min((int64_t)kc, s_stop[w] - (P.A.t0 + s0)));
            some = some || (w < P.G && act[w] < kc);
        }
        some = __any_sync(0xffffffffu, some);
        if (tid0 == 0) smem_at<PersistCnt>(P.lay.misc)->stops[par] = some;
    }
}

// The Poisson kicks of that epoch into its bitmap (all threads): bit 4 s + j of quad word k / 4. The
// hash seed depends on (step, instance) only, so a draw is one mix32 of the pair number
template <bool RASTER, int KB>
__device__ __noinline__ void draw_kicks(const PersistParams& P, int32_t s0, int par)
{
    const int tid = threadIdx.x;
    uint32_t* map = smem_at<uint32_t>(P.lay.kick) + par * ((P.per + 3) / 4);
    const int32_t* act = reinterpret_cast<const int32_t*>(smem_at<int64_t>(P.lay.ticks) + 128) + par * 64;
    const uint32_t* s_hash = smem_at<uint32_t>(P.lay.hash);
    const uint32_t* s_off = s_hash + MAX_EPOCH * 64;
    const int2* s_in = smem_at<int2>(P.lay.inputs);
    const int32_t e0 = P.A.ext_off[blockIdx.x], e1 = P.A.ext_off[blockIdx.x + 1];
    const int32_t n_in = RASTER ? 0 : min(e1 - e0, P.lay.n_inputs);
    for (int32_t e = tid; e < n_in; e += PT) {
        const int2 en = s_in[e];
        const int32_t k = en.x & 0x3ffff, bl = en.x >> 18, na = act[bl];
        const uint32_t id = (uint32_t)k + s_off[bl];
        uint32_t bits = 0;
#pragma unroll
        for (int s = 0; s < KB; s++)
            if (s < na && (int32_t)(mix32(id ^ s_hash[s * 64 + bl]) >> 8) < en.y) bits |= 1u << (4 * s);
        if (bits) atomicOr(map + (k >> 2), bits << (k & 3));
    }
    for (int32_t e = e0 + n_in + tid; e < e1; e += PT) {
        const int2 en = __ldg(P.A.ext_tab + e);
        const int32_t k = en.x & 0x3ffff, bl = en.x >> 18;
        if (bl >= P.G) continue;
        const int32_t na = act[bl];
        uint32_t bits = 0;
        for (int s = 0; s < na; s++)
            if (kick_of<RASTER>(P.S, P.A.kicks, P.A.words, P.N.B, s0 + s, P.b0 + bl, en.y, (uint32_t)k + s_off[bl],
                                P.A.step0 + (uint32_t)(s0 + s)))
                bits |= 1u << (4 * s);
        if (bits) atomicOr(map + (k >> 2), bits << (k & 3));
    }
}

// Push warps: this CTA's shares of the lists arriving at ticks [a0, a1) (at most MAX_EPOCH lists, the
// spikes of n_delay ticks before) scattered into their accumulator slots. Warp w of n_w takes a
// contiguous run of the CTA's items: 32 items are loaded at once (one per lane; those of instances that
// were reset or have stopped are dropped), then two at a time are scattered, each by half of the warp, 8
// entries per lane: a row of 60 entries leaves 24 lanes of a warp idle, and a chain of loads and
// reductions a row is what a warp waits for. ms per 166 steps of 16 x 50,000 neurons with 60 entries, all
// driven at 100 Hz, by lanes an item and pushing warps: 32 lanes 1.58 (5 warps), 1.33 (7), 1.37 (9);
// 16 lanes 1.14, 1.20, 1.41; 8 lanes 1.16, 1.27, 1.47. Rows of 110 entries do not mind (64 whole
// brains 1.82 with 32 and 16 lanes, 1.85 with 8). More warps than 5 slow the advance by as much as they
// gain, for their loads and its loads queue up behind the reductions (~0.7 per SM clock), until
// pushing is by far the longest part. So two more warps push after an epoch with more than BUSY_ENTRIES a
// step and CTA. ms with 5 and 7 warps, by entries: 35 thousand (16 whole brains, 30 % driven at 100 Hz) 9.9 and
// 7.8; 15 thousand (16 x 20,000, 300 entries a row, all at 60 Hz) 2.35 and 2.18; 10 thousand (16 x 50,000, all
// at 400 Hz) 2.29 and 2.29; 5 thousand (half of them) 1.38 and 1.60. Sums are whole numbers: who pushes
// an item does not matter. `ahead`: steps from the present epoch's first tick to a0; `slot0`: the accumulator slot of
// that tick; `next`: the coming epoch's parity.
template <typename AccT>
__device__ __noinline__ void push_epoch(const PersistParams& P, int64_t a0, int64_t a1, int ahead, int slot0, int w, int n_w, int next)
{
    constexpr unsigned FULL = 0xffffffffu;
    const DevNet& N = P.N;
    const DevState& S = P.S;
    const int lane = threadIdx.x & 31, nl = (int)(a1 - a0);
    const int64_t* s_reset = smem_at<int64_t>(P.lay.ticks);
    const int64_t* s_stop = s_reset + 64;
    // this CTA's share of each list, flattened
    int32_t from = 0, len_k = 0;
    if (lane < nl && a0 + lane >= N.n_delay) {
        // total * block / blocks in 32 bits: by its quotient and remainder
        const uint32_t total = (uint32_t)min((int64_t)max(__ldcg(count_from(P, ahead + lane - N.n_delay)), 0), S.cap_c);
        const uint32_t n_c = gridDim.x, c = blockIdx.x, each = total / n_c, rest = total - each * n_c;
        from = (int32_t)(each * c + rest * c / n_c);
        len_k = (int32_t)(each * (c + 1) + rest * (c + 1) / n_c) - from;
    }
    int32_t first[MAX_EPOCH], off[MAX_EPOCH + 1];
    off[0] = 0;
#pragma unroll
    for (int k = 0; k < MAX_EPOCH; k++) {
        first[k] = __shfl_sync(FULL, from, k);
        off[k + 1] = off[k] + __shfl_sync(FULL, len_k, k);
    }
    const uint32_t M = (uint32_t)off[MAX_EPOCH];                // (at most six lists of 2^31 by 148: 16 M fits)
    const int64_t np = N.n_pad, slot_stride = (int64_t)N.B * np;
    AccT* acc0 = reinterpret_cast<AccT*>(S.acc) + (int64_t)P.b0 * np;
    const int32_t list0 = wrap(smem_at<PersistCnt>(P.lay.misc)->list_at + ahead - N.n_delay, N.R);
    slot0 = wrap(slot0 + ahead, S.n_slots);
    const int32_t j1 = (int32_t)(M * (uint32_t)(w + 1) / (uint32_t)n_w);
    int32_t mine = 0;
    for (int32_t j0 = (int32_t)(M * (uint32_t)w / (uint32_t)n_w); j0 < j1; j0 += 32) {
        int32_t start = 0, len = 0;
        int64_t to = 0;                                         // offset of the item's row of accumulators
        if (j0 + lane < j1) {
            const int32_t j = j0 + lane;
            int k = 0;
            int32_t g = first[0] + j;
#pragma unroll
            for (int u = 1; u < MAX_EPOCH; u++)
                if (off[u] <= j) { k = u; g = first[u] + (j - off[u]); }
            const int32_t ls = list0 + k < N.R ? list0 + k : list0 + k - N.R;
            const int2 item = __ldcg(S.items + ((int64_t)ls * S.n_groups + P.q) * S.cap_c + g);
            const int32_t bl = (item.y >> CHUNK_BITS) - P.b0;
            start = item.x;
            if (a0 + k - N.n_delay >= s_reset[bl] && a0 + k < s_stop[bl]) len = item.y & ((1 << CHUNK_BITS) - 1);
            const int32_t sl = slot0 + k < S.n_slots ? slot0 + k : slot0 + k - S.n_slots;
            to = sl * slot_stride + (int64_t)bl * np;
            mine += len;
        }
        const int n = min(32, j1 - j0);
        for (int u0 = 0; u0 < n; u0 += 32 / PUSH_LANES) {
            const int u = u0 + lane / PUSH_LANES;               // (u = n <= 31 where n is odd: an item of length 0)
            const int32_t r = __shfl_sync(FULL, start, u), l = __shfl_sync(FULL, len, u);
            AccT* acc = acc0 + __shfl_sync(FULL, to, u);
            for (int32_t q = 8 * (lane % PUSH_LANES); q < l; q += 8 * PUSH_LANES) {
                Edges8<typename SumOf<AccT>::T> e;
                e.load(N, (int64_t)(uint32_t)r + q);
#pragma unroll
                for (int c = 0; c < 8; c++)
                    if (e.w[c] != 0) red_acc(acc + e.c[c], e.w[c]);
            }
        }
    }
    if (M > BUSY_ENTRIES / CHUNK) {                             // (fewer items cannot hold that many entries)
        mine = __reduce_add_sync(FULL, mine);
        if (lane == 0 && mine) atomicAdd(&smem_at<PersistCnt>(P.lay.misc)->entries[next], mine);
    }
}

// The pair-by-pair advance of up to 8 quads through the kc steps of the epoch whose first is s0, four
// lanes per quad (`quad`: this lane's, or -1): the quads that the tiles' advance passes over because
// they have a plastic target or a bias, or a kick or a spike in this epoch. Every load of the epoch is
// issued before the first step; what was read is cleared.
template <typename AccT, bool PLASTIC, bool RECORD, int KB>
__device__ __noinline__ void advance_pairs(const PersistParams& P, int32_t quad, int32_t s0, int32_t kc, int par, int slot0,
                                           int ring0)
{
    const DevNet& N = P.N;
    const DevState& S = P.S;
    const int j = threadIdx.x & 3;
    const int32_t k = 4 * quad + j;
    const uint32_t np = (uint32_t)N.n_pad, lp = (uint32_t)(first_pair(P) + (quad < 0 ? 0 : k));
    const int32_t bl = (int32_t)(lp / np), i = (int32_t)(lp - (uint32_t)bl * np);
    const bool on = quad >= 0 && i < N.n;
    AccT* const acc = reinterpret_cast<AccT*>(S.acc) + (int64_t)P.b0 * np + lp;
    const int64_t slot_stride = (int64_t)N.B * np;
    typename SumOf<AccT>::T x[KB];
#pragma unroll
    for (int s = 0; s < KB; s++) {
        const int sl = slot0 + s < S.n_slots ? slot0 + s : slot0 + s - S.n_slots;
        x[s] = on && s < kc ? ld_acc(acc + sl * slot_stride) : 0;
    }
    uint32_t* kw = smem_at<uint32_t>(P.lay.kick) + par * ((P.per + 3) / 4) + (quad < 0 ? 0 : quad);
    const uint32_t kick = on ? *kw >> j : 0u;
    __syncwarp();                                               // (a quad's words are read before they are cleared)
    if (on && j == 0 && *kw != 0u) *kw = 0u;
    if (!on) return;
    float* sv = smem_at<float>(P.lay.v) + k;
    float* sg = smem_at<float>(P.lay.g) + k;
    uint8_t* sr = smem_at<uint8_t>(P.lay.ref) + k;
    const int32_t b = P.b0 + bl;
    const int na = smem_at<int32_t>(P.lay.ticks + 1024)[par * 64 + bl];
    const uint32_t f = *sr;
    const Lif<float> L = N.L32;
    int64_t px[KB];
    int64_t* ring = nullptr;
    if (PLASTIC) {
        if (f & 0x40) ring = S.pring + (int64_t)b * N.n_ppost + __ldg(N.ppost_of + i);
#pragma unroll
        for (int s = 0; s < KB; s++) {
            const int at = ring0 + s < N.R_pl ? ring0 + s : ring0 + s - N.R_pl;
            px[s] = ring && s < na ? (int64_t)__ldcg(reinterpret_cast<const long long*>(ring + (int64_t)at * N.B * N.n_ppost)) : 0;
        }
    }
    const float bias = (f & 0x80) ? S.bias_ext[(int64_t)b * S.n_ext + __ldg(S.ext_idx + i)] : 0.0f;
    float v = *sv, g = *sg;
    int r = (int)(f & 0x3fu);
    uint32_t hits = 0;
#pragma unroll
    for (int s = 0; s < KB; s++) {
        const int sl = slot0 + s < S.n_slots ? slot0 + s : slot0 + s - S.n_slots;
        if (x[s] != 0) clear_acc(acc + sl * slot_stride);
        if (s < na) {
            float buf = acc_to_real<float>(x[s], L.w_syn);
            if (PLASTIC && ring) {
                const int at = ring0 + s < N.R_pl ? ring0 + s : ring0 + s - N.R_pl;
                buf = add_rn(buf, from_q32<float>(px[s]));
                if (px[s] != 0) ring[(int64_t)at * N.B * N.n_ppost] = 0;
            }
            // the engine always fuses the two multiply-adds, as the shipped reference does
            if (lif_step<float>(v, g, r, buf, (f & 0x80u) != 0, bias, (kick >> (4 * s)) & 1u, L, N.n_ref, true))
                hits |= 1u << (4 * s);
        }
    }
    *sv = v;
    *sg = g;
    *sr = (uint8_t)((f & 0xc0u) | (uint32_t)r);
    if (hits) record_spikes<PLASTIC, RECORD>(P, par, k, s0, hits);
}

// The advance of this CTA's tiles through the kc steps of the epoch whose first is s0 (FULL: kc = KB, and no
// instance stops in it or has stopped), a quad of consecutive pairs per lane. Quads of an instance that
// stops take their own number of steps here: handed to advance_pairs, they made every epoch after
// the stop slow (a frame of 16 whole brains in which one run ends: 2.0 ms against 0.8). The arithmetic is lif_step's without kicks, plastic input,
// biases and spikes, in straight-line code: the refractory counters of the whole epoch are known at
// its start, and a quad that takes a kick or reaches the threshold (one in thirty) is left as it was
// and handed to advance_pairs, together with those that do not qualify from the start. Testing for
// kicks and spikes at every step took 27 of 110 instructions per quad and step; two quads per lane, and
// two-float arithmetic (fma.rn.f32x2), whose register pairs cost more moves than they saved, were
// slower. `turn`: this warp's next turn of the CTA's counter (`first_turn`: tile 0).
template <typename AccT, bool PLASTIC, bool RECORD, int KB, bool FULL>
__device__ __forceinline__ void advance_tiles(const PersistParams& P, int32_t turn, int32_t first_turn, uint16_t* ev,
                                              int32_t cnt, int32_t kc, int32_t s0, int par, int slot0, int ring0)
{
    using Acc4 = typename Acc4Of<AccT>::T;
    PersistCnt* C = smem_at<PersistCnt>(P.lay.misc);
    const int lane = threadIdx.x & 31;
    const int32_t np = (int32_t)P.N.n_pad, end = first_turn + (cnt + TILE - 1) / TILE;
    AccT* slot[KB];                                             // this CTA's accumulators at each step
#pragma unroll
    for (int s = 0; s < KB; s++) {
        const int sl = slot0 + s < P.S.n_slots ? slot0 + s : slot0 + s - P.S.n_slots;
        slot[s] = reinterpret_cast<AccT*>(P.S.acc) + ((int64_t)P.b0 * np + first_pair(P)) + (int64_t)sl * P.N.B * np;
    }
    const Lif<float> L = P.N.L32;
    // what decides about a lane's quad and its accumulators, loaded one tile ahead (an L2 round trip is as
    // long as the arithmetic of a tile)
    struct Ahead {
        Acc4 x[KB];
        uint32_t rb;                                            // the four refractory counters
        int32_t on;                                             // steps of the epoch that its instance advances (!FULL)
        bool ok;                                                // advanced here
    };
    auto fetch = [&](Ahead& a, int32_t k) {
        a.rb = k < cnt ? *smem_at<uint32_t>(P.lay.ref + k) : 0xc0u;
        a.ok = !(a.rb & 0xc0c0c0c0u);                           // neither a special quad nor padding
        a.on = kc;
        if (!FULL && a.ok)
            a.on = smem_at<int32_t>(P.lay.ticks + 1024)[par * 64 + (int32_t)((uint32_t)(first_pair(P) + k) / (uint32_t)np)];
#pragma unroll
        for (int s = 0; s < KB; s++) {
            a.x[s].zero();
            if (a.ok && (FULL || s < kc)) a.x[s].load(slot[s] + k);
        }
    };
    auto take_turn = [&]() {
        if (lane == 0) turn = atomicAdd(&C->tile[par], 1);
        turn = __shfl_sync(0xffffffffu, turn, 0);
    };
    while (turn < end) {
        // tiles while the quads they set aside surely fit this warp's buffer; no call inside, so that what
        // is loaded ahead stays in registers
        int pending = 0;
        Ahead next;
        int32_t k_next = (turn - first_turn) * TILE + 4 * lane;
        fetch(next, k_next);
        for (bool go = true; go;) {
            const int32_t k = k_next;
            const Ahead a = next;
            take_turn();
            go = turn < end && pending + 2 * 32 <= EV_BUF;
            if (go) {
                k_next = (turn - first_turn) * TILE + 4 * lane;
                fetch(next, k_next);
            }
            bool aside = false;                                 // for advance_pairs
            if (a.ok) {
                const float4 v4 = *smem_at<float4>(P.lay.v + 4 * k), g4 = *smem_at<float4>(P.lay.g + 4 * k);
                const uint32_t kick = *smem_at<uint32_t>(P.lay.kick + par * ((P.per + 3) / 4) * 4 + k);
                float g[4] = {g4.x, g4.y, g4.z, g4.w}, v[4] = {v4.x, v4.y, v4.z, v4.w};
                int r[4];
#pragma unroll
                for (int j = 0; j < 4; j++) r[j] = (int)((a.rb >> (8 * j)) & 0xffu);
                float top = L.v_rest;
#pragma unroll
                for (int s = 0; s < KB; s++) {
                    if (!FULL && s >= a.on) break;
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        g[j] = fma_rn(g[j], L.ds, acc_to_real<float>(a.x[s].at(j), L.w_syn));
                        const float e = sub_rn(g[j], sub_rn(v[j], L.v_rest));
                        if (r[j] <= s) v[j] = fma_rn(e, L.dm, v[j]);
                    }
                    top = s == 0 ? max3(v[0], v[1], max3(v[2], v[3], v[3])) : max3(max3(top, v[0], v[1]), v[2], v[3]);
                }
                aside = kick != 0u || top >= L.v_th;
                if (!aside) {
                    *smem_at<float4>(P.lay.v + 4 * k) = make_float4(v[0], v[1], v[2], v[3]);
                    *smem_at<float4>(P.lay.g + 4 * k) = make_float4(g[0], g[1], g[2], g[3]);
                    if (a.rb) *smem_at<uint32_t>(P.lay.ref + k) = __vsubus4(a.rb, 0x01010101u * (uint32_t)(FULL ? kc : a.on));
#pragma unroll
                    for (int s = 0; s < KB; s++)
                        if ((FULL || s < kc) && a.x[s].any()) Acc4::clear(slot[s] + k);
                }
            }
            const uint32_t m = __ballot_sync(0xffffffffu, aside);
            if (aside) ev[pending + __popc(m & ((1u << lane) - 1u))] = (uint16_t)(k >> 2);
            pending += __popc(m);
        }
        __syncwarp();
        for (; pending > 0; pending -= 8) {
            const int e = pending - 8 + (lane >> 2);
            advance_pairs<AccT, PLASTIC, RECORD, KB>(P, e >= 0 ? (int32_t)ev[e] : -1, s0, kc, par, slot0, ring0);
        }
    }
}

// This CTA's state into shared memory, its tables and counters, and the first epoch's kicks
template <bool RASTER, bool PLASTIC, int KB>
__device__ __noinline__ void load_state(const PersistParams& P, int32_t cnt)
{
    const DevNet& N = P.N;
    const DevState& S = P.S;
    const int tid = threadIdx.x;
    const int32_t n = (int32_t)N.n, np = (int32_t)N.n_pad, b0 = P.b0, G = P.G;
    const int64_t lo = first_pair(P);
    float* sv = smem_at<float>(P.lay.v);
    float* sg = smem_at<float>(P.lay.g);
    uint8_t* sr = smem_at<uint8_t>(P.lay.ref);
    PersistCnt* C = smem_at<PersistCnt>(P.lay.misc);
    const uint32_t lp0 = (uint32_t)lo + (uint32_t)tid;
    int32_t bl = (int32_t)(lp0 / (uint32_t)np), i = (int32_t)(lp0 - (uint32_t)bl * (uint32_t)np);
    for (int32_t k = tid; k < cnt; k += PT) {
        uint8_t f = (i & ~3) < n ? 0 : 0xc0;                     // a quad of padding is passed over like a special one
        float v = N.L32.v_rest, g = 0.0f;
        if (i < n) {
            const int64_t gp = (int64_t)(b0 + bl) * n + i;
            v = reinterpret_cast<const float*>(S.v)[gp];
            g = reinterpret_cast<const float*>(S.g)[gp];
            f = (uint8_t)S.ref[gp];
            if (PLASTIC && N.ppost_of[i] >= 0) f |= 0x40;
        }
        sv[k] = v;
        sg[k] = g;
        sr[k] = f;
        for (i += PT; i >= np; i -= np) bl++;
    }
    uint32_t* s_kick = smem_at<uint32_t>(P.lay.kick);
    for (int32_t w = tid; w < 2 * ((P.per + 3) / 4); w += PT) s_kick[w] = 0u;
    for (int w = tid; w < (int)(sizeof(PersistCnt) / 4); w += PT) reinterpret_cast<int32_t*>(C)[w] = 0;
    if (tid < 64) {                                              // the ticks stay constant during a launch
        int64_t* s_reset = smem_at<int64_t>(P.lay.ticks);
        s_reset[tid] = tid < G ? S.reset_tick[b0 + tid] : 0;
        s_reset[64 + tid] = tid < G ? S.stop_tick[b0 + tid] : 0;
        // the pair number (instance * n + neuron) of local pair k of instance tid is k + this
        smem_at<uint32_t>(P.lay.hash)[MAX_EPOCH * 64 + tid] = (uint32_t)((int64_t)(b0 + tid) * n + lo - (int64_t)tid * np);
    }
    __syncthreads();
    if (tid == 0) {
        C->list_at = (int32_t)pos_mod(P.A.t0, N.R);
        C->count_at = (int32_t)pos_mod(P.A.t0, N.R_pl);
    }
    prepare_epoch<RASTER>(P, 0, min(P.A.epoch, P.A.steps), 0, tid, PT);
    const int32_t e0 = P.A.ext_off[blockIdx.x], e1 = P.A.ext_off[blockIdx.x + 1];
    int2* s_in = smem_at<int2>(P.lay.inputs);
    for (int32_t e = e0 + tid; e < e1; e += PT) {               // biases and probabilities are constant during a launch
        const int2 en = __ldg(P.A.ext_tab + e);
        const int32_t k = en.x & 0x3ffff, bi = en.x >> 18;
        const int64_t at = (int64_t)(b0 + bi) * S.n_ext + en.y;
        if (bi < G && S.bias_ext[at] != 0.0f) sr[k] |= 0x80;
        if (!RASTER && e - e0 < P.lay.n_inputs) s_in[e - e0] = make_int2(en.x, bi < G ? kick_threshold(S.p_ext[at]) : 0);
    }
    __syncthreads();
    for (int32_t k = 4 * tid; k < cnt; k += 4 * PT)
        if ((*reinterpret_cast<const uint32_t*>(sr + k) & 0xc0c0c0c0u) && (int32_t)((uint32_t)(lo + k) % (uint32_t)np) < n)
            smem_at<uint16_t>(P.lay.special)[atomicAdd(&C->n_special, 1)] = (uint16_t)(k >> 2);
    draw_kicks<RASTER, KB>(P, 0, 0);
    __syncthreads();
}

__device__ __noinline__ void store_state(const PersistParams& P, int32_t cnt)
{
    const int32_t n = (int32_t)P.N.n, np = (int32_t)P.N.n_pad;
    const float* sv = smem_at<float>(P.lay.v);
    const float* sg = smem_at<float>(P.lay.g);
    const uint8_t* sr = smem_at<uint8_t>(P.lay.ref);
    const uint32_t lp0 = (uint32_t)first_pair(P) + threadIdx.x;
    int32_t bl = (int32_t)(lp0 / (uint32_t)np), i = (int32_t)(lp0 - (uint32_t)bl * (uint32_t)np);
    for (int32_t k = threadIdx.x; k < cnt; k += PT) {
        if (i < n) {
            const int64_t gp = (int64_t)(P.b0 + bl) * n + i;
            reinterpret_cast<float*>(P.S.v)[gp] = sv[k];
            reinterpret_cast<float*>(P.S.g)[gp] = sg[k];
            P.S.ref[gp] = (int8_t)(sr[k] & 0x3f);
        }
        for (i += PT; i >= np; i -= np) bl++;
    }
}

// One launch runs `A.steps` steps of the instances [b0, b0 + G) (group q) in epochs of A.epoch <= KB
// steps; the warp roles are described at the top of this file.
template <typename AccT, bool RASTER, bool PLASTIC, bool RECORD, int KB>
__global__ void __launch_bounds__(PT, 1) k_persist(const __grid_constant__ PersistParams P)
{
    const PersistArgs& A = P.A;
    PersistCnt* C = smem_at<PersistCnt>(P.lay.misc);
    const int tid = threadIdx.x, lane = tid & 31;
    const int32_t np = (int32_t)P.N.n_pad;
    const int32_t cnt = (int32_t)max((int64_t)0, min((int64_t)P.per, (int64_t)P.G * np - first_pair(P)));
    load_state<RASTER, PLASTIC, KB>(P, cnt);

    // An epoch is known by its first step: what else a warp needs between the routines is derived again
    // from the parameters, so that few registers stay live across the advance
    const int K = A.epoch;
    const bool is_l = tid < LIST_THREADS;
    const int n_slots = P.S.n_slots;
    int slot0 = (int)pos_mod(A.t0, n_slots);                    // accumulator slot of the epoch's first tick
    int ring0 = PLASTIC ? (int)pos_mod(A.t0, P.N.R_pl) : 0;     // ... and its slot of the plastic ring
    unsigned int bar_target = 0;
    int par = 0;
    bool stop = false;

    // ---- prologue: the arrivals of the first epoch not in the accumulators yet -----------------
    {
        const int64_t a1 = min(A.t0 + K, A.t0 + A.steps + 1);
        if (A.pushed_until < a1) {
            push_epoch<AccT>(P, A.pushed_until, a1, (int)(A.pushed_until - A.t0), slot0, tid >> 5, PT / 32, 0);
            __syncthreads();
            bar_target += gridDim.x;
            if (tid == 0) {
                const long long c0 = clock64();
                grid_arrive(A);
                C->stop = grid_wait(A, bar_target, c0, P.S.err, 1);
            }
            __syncthreads();
            stop = C->stop != 0;
        }
    }
    // ---- epochs of K steps, one grid barrier each ---------------------------------------------
    int32_t ep0 = 0;
    for (; ep0 < A.steps && !stop; ep0 += K, par ^= 1) {
        long long c_begin = 0;
        if (tid == PT - 1 && A.trace) c_begin = clock64();
        if (is_l) {
            const int32_t kc = min(K, A.steps - ep0);
            if (A.list_late && ep0 > 0) list_epoch<PLASTIC, RECORD>(P, par ^ 1, ep0 - K, K, K, false);
            // the lists whose items arrive in this epoch were pushed before it: their lengths are zero when the
            // slots serve again, K steps after the ticks of this epoch
            if (blockIdx.x == 0 && tid < kc) *count_from(P, tid - P.N.n_delay) = 0;
            if (ep0 + kc < A.steps) prepare_epoch<RASTER>(P, ep0 + kc, min(K, A.steps - ep0 - kc), par ^ 1, tid, LIST_THREADS);
            if (tid == 0) {
                C->tile[par ^ 1] = 0;
                if (A.trace)
                    for (int32_t s = 0; s < kc; s++) stamp(A, ep0 + s, 8);
            }
        } else if (const int n_w = C->entries[par] > BUSY_ENTRIES * K ? BUSY_PUSH_WARPS : PUSH_WARPS; tid < LIST_THREADS + 32 * n_w) {
            // the arrivals of the next epoch (and of the tick after the run) not pushed yet
            const int64_t end = A.t0 + A.steps + 1, T = A.t0 + ep0;
            const int64_t pa0 = max(A.pushed_until, min(T + K, end)), pa1 = min(T + 2 * K, end);
            if (tid == LIST_THREADS) stamp(A, ep0, 7);
            if (pa0 < pa1) push_epoch<AccT>(P, pa0, pa1, (int)(pa0 - T), slot0, (tid - LIST_THREADS) >> 5, n_w, par ^ 1);
            if (tid == LIST_THREADS) stamp(A, ep0, 10);
        }
        // ---- advance: the special quads first (8 of them per turn), then the tiles ---------------------
        const int32_t kc = min(K, A.steps - ep0);
        const int32_t n_sp = C->n_special, sp_turns = (n_sp + 7) / 8;
        int32_t turn = 0;
        for (;;) {
            if (lane == 0) turn = atomicAdd(&C->tile[par], 1);
            turn = __shfl_sync(0xffffffffu, turn, 0);
            if (turn >= sp_turns) break;
            const int32_t e = turn * 8 + (lane >> 2);
            advance_pairs<AccT, PLASTIC, RECORD, KB>(P, e < n_sp ? (int32_t)smem_at<uint16_t>(P.lay.special)[e] : -1, ep0, kc, par,
                                                     slot0, ring0);
        }
        uint16_t* ev = smem_at<uint16_t>(P.lay.events) + (tid >> 5) * EV_BUF;   // this warp's quads for advance_pairs
        if (kc == KB && !C->stops[par]) advance_tiles<AccT, PLASTIC, RECORD, KB, true>(P, turn, sp_turns, ev, cnt, kc, ep0, par, slot0, ring0);
        else advance_tiles<AccT, PLASTIC, RECORD, KB, false>(P, turn, sp_turns, ev, cnt, kc, ep0, par, slot0, ring0);
        if (tid == PT - 1 && A.trace) {                         // the epoch's span, divided between its steps
            const long long d = max((clock64() - c_begin) / kc, 2LL);
            for (int32_t s = 0; s < kc; s++) {
                const long long c0 = c_begin + s * d;
                *trace_at(A, ep0 + s, 0) = *trace_at(A, ep0 + s, 4) = c0;
                *trace_at(A, ep0 + s, 1) = *trace_at(A, ep0 + s, 2) = c0;
                *trace_at(A, ep0 + s, 3) = c0 + d - 1;
            }
        }
        slot0 += kc;
        if (slot0 >= n_slots) slot0 -= n_slots;
        ring0 += kc;
        if (ring0 >= P.N.R_pl) ring0 -= P.N.R_pl;
        if (!A.list_late) {
            __syncthreads();                                    // every spike of the epoch is buffered
            list_epoch<PLASTIC, RECORD>(P, par, ep0, kc, 0, true);
        }
        if (ep0 + K < A.steps) {                                // another epoch follows
            __syncthreads();                                    // this epoch's work of the CTA is done
            long long c0 = 0;
            if (tid == 0) {
                c0 = clock64();
                grid_arrive(A);
                stamp(A, ep0 + K - 1, 5);
                C->entries[par] = 0;                            // (the coming epoch adds to it)
                C->list_at = wrap(C->list_at + K, P.N.R);
                C->count_at = wrap(C->count_at + K, P.N.R_pl);
            }
            draw_kicks<RASTER, KB>(P, ep0 + K, par ^ 1);
            bar_target += gridDim.x;
            if (tid == 0) {
                stamp(A, ep0 + K - 1, 9);
                C->stop = grid_wait(A, bar_target, c0, P.S.err, ep0 + K + 1);
                stamp(A, ep0 + K - 1, 6);
            }
            __syncthreads();
            stop = C->stop != 0;
        }
    }
    // the last epoch's spikes are listed before the launch ends (the next launch scatters them)
    __syncthreads();
    if (!stop && A.list_late) list_epoch<PLASTIC, RECORD>(P, par ^ 1, ep0 - K, A.steps - (ep0 - K), 0, true);
    store_state(P, cnt);
}

// Largest group whose state fits in shared memory of `ctas` CTAs; 0 if not even one instance does.
inline PersistPlan plan_persistent(int64_t n, int64_t n_pad, int32_t B, bool f64, int n_ref, int n_delay,
                                   int sm_count, int device)
{
    PersistPlan P{};
    if (f64 || n_ref > 63 || n_delay < 3) return P;
    int smem_optin = 0;
    cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    if (smem_optin <= 0) smem_optin = 232448;
    int64_t per_max = 0;
    for (int64_t lo = 16, hi = (int64_t)1 << K_BITS; lo <= hi;) {  // largest `per` whose layout fits
        const int64_t mid = (lo + hi) / 2 / 16 * 16;
        if (mid < 16) break;
        if (PersistSmem((int32_t)mid).total <= smem_optin) { per_max = mid; lo = mid + 16; }
        else hi = mid - 16;
    }
    if (per_max <= 0) return P;
    const int ctas = sm_count;
    int64_t gmax = std::min<int64_t>((int64_t)ctas * per_max / n_pad, 63);
    if (gmax < 1) return P;
    const int32_t n_groups = (int32_t)((B + gmax - 1) / gmax);
    const int32_t G = (B + n_groups - 1) / n_groups;
    int64_t per = ((int64_t)G * n_pad + ctas - 1) / ctas;
    per = (per + 15) / 16 * 16;
    if (per > per_max || per >= ((int64_t)1 << K_BITS)) return P;
    P.group = G;
    P.n_groups = n_groups;
    P.ctas = ctas;
    P.per = per;
    P.smem = (size_t)PersistSmem((int32_t)per).total;
    P.smem_max = (size_t)smem_optin;
    P.launches_per_run = n_groups;
    (void)n;
    return P;
}

// Room for the `most` input pairs that a CTA has, as far as shared memory goes (an even number: what follows is
// aligned to 16 bytes). Beyond it a kick draws its threshold from two dependent global loads: an epoch's kicks of
// 5,400 inputs per CTA took 5.0 us with 2,048 of them in shared memory and 2.8 with all (16 x 50,000, all
// driven at 100 Hz: 2.41 ms per 166 steps and 1.83 with K = 1, 1.16 and 0.99 with K = 6).
inline void plan_inputs(PersistPlan& P, int32_t most)
{
    const int32_t spare = (int32_t)(P.smem_max - (size_t)PersistSmem((int32_t)P.per).total) / 8;
    P.inputs = std::min((std::max(most, IN_BUF) + 1) & ~1, (IN_BUF + spare) & ~1);
    P.smem = (size_t)PersistSmem((int32_t)P.per, P.inputs).total;
}

// Steps per epoch. Longer epochs mean fewer barriers, but the 2K accumulator slots of the group are to stay
// in L2: in 16 bits K = 6 takes 53 MB for 16 whole brains (4.53 us per step, 4.80 with K = 4; 18 brains
// 2.95 and 3.46); in 32 bits it takes 106 MB and was slower (7.9 us per step, 5.5 with K = 4).
// Listing an epoch's spikes in the next one takes 3K <= n_delay, at its own end 2K <= n_delay and 2-3 us.
// The longer epoch is worth it from a third more steps on: ms per 166 steps of 64 whole brains with
// K = 1 late / 2 own 5.71 / 3.93, 2 / 3 3.39 / 2.98, 3 / 4 2.55 / 2.47, 4 / 6 2.16 / 2.05, but 5 / 6 1.98 / 2.05.
struct EpochPlan {
    int32_t late = 1;         // the longest that can be listed late
    int32_t steps = 1;        // K of a run
};
inline EpochPlan plan_epochs(int n_delay, int acc_bytes)
{
    const int most = acc_bytes == 2 ? MAX_EPOCH : 4, own = std::min(most, n_delay / 2);
    EpochPlan E;
    E.late = std::max(1, std::min(most, n_delay / 3));
    E.steps = 3 * own >= 4 * E.late ? own : E.late;
    return E;
}

template <typename AccT, bool RASTER, bool PLASTIC, bool RECORD, int KB>
cudaError_t launch_persist_one(const PersistPlan& P, const DevNet& N, const DevState& S, const PersistArgs& A,
                               cudaStream_t st)
{
    auto kern = k_persist<AccT, RASTER, PLASTIC, RECORD, KB>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)P.smem_max);
    if (e != cudaSuccess) return e;
    for (int32_t q = 0; q < P.n_groups; q++) {
        const int32_t b0 = q * P.group;
        const int32_t G = std::min<int32_t>(P.group, N.B - b0);
        e = cudaMemsetAsync(A.bar, 0, sizeof(unsigned int), st);
        if (e != cudaSuccess) return e;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(P.ctas);
        cfg.blockDim = dim3(PT);
        cfg.dynamicSmemBytes = P.smem;
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, kern, PersistParams{N, S, A, PersistSmem((int32_t)P.per, P.inputs), b0, G, q, (int32_t)P.per});
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

template <typename AccT, int KB>
cudaError_t launch_persist_acc(const PersistPlan& P, const DevNet& N, const DevState& S, const PersistArgs& A,
                               bool plastic, bool raster, bool record, cudaStream_t st)
{
#define LP_(R_, P_, C_) return launch_persist_one<AccT, R_, P_, C_, KB>(P, N, S, A, st)
    if (raster) {
        if (plastic) { if (record) LP_(true, true, true); LP_(true, true, false); }
        if (record) LP_(true, false, true);
        LP_(true, false, false);
    }
    if (plastic) {
        if (record) LP_(false, true, true);
        LP_(false, true, false);
    }
    if (record) LP_(false, false, true);
    LP_(false, false, false);
#undef LP_
}

inline cudaError_t launch_persistent(const PersistPlan& P, const DevNet& N, const DevState& S, const PersistArgs& A,
                                     int acc_bytes, bool plastic, bool raster, bool record, cudaStream_t st)
{
    // KB = K: an advance with room for more steps than an epoch has takes the form for instances that stop, and
    // reads and tests slots it does not use (64 whole brains, 166 steps at K = 2: 4.06 ms with KB = 4, 3.33 with 2)
#define LK_(T_, K_) case K_: return launch_persist_acc<T_, K_>(P, N, S, A, plastic, raster, record, st)
    if (acc_bytes == 8) switch (A.epoch) { LK_(int64_t, 1); LK_(int64_t, 2); LK_(int64_t, 3); LK_(int64_t, 4); }
    if (acc_bytes == 4) switch (A.epoch) { LK_(int32_t, 1); LK_(int32_t, 2); LK_(int32_t, 3); LK_(int32_t, 4); }
    if (acc_bytes == 2) switch (A.epoch) { LK_(int16_t, 1); LK_(int16_t, 2); LK_(int16_t, 3); LK_(int16_t, 4); LK_(int16_t, 5); LK_(int16_t, 6); }
#undef LK_
    return cudaErrorInvalidValue;
}

}  // namespace fb
