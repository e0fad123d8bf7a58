// Motion-vision front end on the device (flyzero/vision.py:142-191, MotionEye.see) for every
// instance at once, writing the eye neurons' Poisson probabilities straight into p_ext: the
// frames are already on the device, so no rates cross the bus and no host loop runs per frame.
//
// The default is two launches: k_eye_grid (a thread per instance and grid cell: luminance, high-pass,
// delay arms, colours) and k_eye_neurons (several blocks per instance, its grids in shared memory); small eyes
// take k_eye_neurons alone, one block per instance, which forms the grids itself. Grids too large for
// shared memory take four grid-wide kernels, which state the steps one by one:
//   k_eye_cells    one thread per (instance, grid cell):
//                  lum = mean over the cell x cell block of mean(R, G, B) / 255 (vision.py:136-140),
//                  each block row summed with NumPy's pairwise rule, the row sums added in order;
//                  blue / green grids the same way from one channel (chromatic channels);
//                  high-pass lp += a_hp (lum - lp), hp = lum - lp, sig_on = max(hp, 0),
//                  sig_off = max(-hp, 0). An instance whose restart flag is set starts from this
//                  frame: lp = lum, delay arms 0 (vision.py:145-147).
//   k_eye_integral one block per instance: the integral image of the zero-padded lum grid,
//                  cumsum down the columns then along the rows (vision.py:170), float32.
//   k_eye_rates    one thread per (instance, eye neuron): its channel at its grid cell,
//                  motion = the Hassenstein-Reichardt correlator delayed(A) B - A delayed(B) of its
//                  polarity, B the cell `shift` to the right / below, rectified for its screen
//                  direction (vision.py:151-162); columnar channels as vision.py:164-186 (the
//                  sustained contrast in float64, as NumPy promotes it); 0 above y_min;
//                  p_ext[b][slot] = f32(max_rate * clip(gain * rate, 0, 1)) * p_scale. A neuron
//                  whose cell, channel or slot is out of range is skipped.
//   k_eye_delay    one thread per (instance, polarity, cell): d += a_d (sig - d); clears the
//                  instance's restart flag.
// One rounding per operation in the order NumPy evaluates it, no contraction.
#pragma once
#include "chain.cuh"
#include "common.cuh"

namespace fb {

enum EyeChannel : uint8_t {
    EYE_ON_RIGHT = 0, EYE_ON_LEFT, EYE_ON_DOWN, EYE_ON_UP,
    EYE_OFF_RIGHT, EYE_OFF_LEFT, EYE_OFF_DOWN, EYE_OFF_UP,
    EYE_ON_TRANSIENT, EYE_OFF_TRANSIENT, EYE_ON_SUSTAINED, EYE_OFF_SUSTAINED, EYE_BLUE, EYE_GREEN,
    EYE_CHANNELS
};

struct EyeArgs {
    int32_t B, H, W, cell, gh, gw, shift, surround, chromatic;
    float a_hp, a_d, gain_f, max_rate, p_scale, transient_f, chromatic_f;
    double gain, sustained;
    const uint8_t* frames;      // (B, H, W, 3)
    const uint8_t* flip;        // (B) mirror the frame left-right, or nullptr
    uint8_t* restart;           // (B) start the filters from this frame; cleared when it is done
    float* lum;                 // (B, gh, gw)
    float* lp;                  // (B, gh, gw)
    float* sig;                 // (B, 2, gh, gw)  ON, OFF
    float* dly;                 // (B, 2, gh, gw)
    float* col;                 // (B, 2, gh, gw)  blue, green
    float* ii;                  // (B, gh + 1, gw + 1)
    int32_t n_cells;
    const int32_t* gx;          // (n_cells) grid column
    const int32_t* gy;          // (n_cells) grid row
    const uint8_t* chan;        // (n_cells) EyeChannel
    const uint8_t* visible;     // (n_cells) 0 above y_min
    const int32_t* slot;        // (n_cells) ext slot
    float* p_ext;               // (B, n_ext)
    int32_t n_ext;
    float* rates;               // (B, n_cells) rates in Hz, or nullptr
};

// NumPy's pairwise float32 sum of n values with the given stride (sequential below 8, eight
// accumulators up to 128 values, then the tail).
template <typename F>
__device__ __forceinline__ float np_row_sum(int32_t n, F at)
{
    if (n < 8) {
        float r = 0.0f;
        for (int32_t i = 0; i < n; i++) r = __fadd_rn(r, at(i));
        return r;
    }
    float a[8];
#pragma unroll
    for (int32_t j = 0; j < 8; j++) a[j] = at(j);
    int32_t i = 8;
    for (; i < n - n % 8; i += 8)
#pragma unroll
        for (int32_t j = 0; j < 8; j++) a[j] = __fadd_rn(a[j], at(i + j));
    float r = __fadd_rn(__fadd_rn(__fadd_rn(a[0], a[1]), __fadd_rn(a[2], a[3])),
                        __fadd_rn(__fadd_rn(a[4], a[5]), __fadd_rn(a[6], a[7])));
    for (; i < n; i++) r = __fadd_rn(r, at(i));
    return r;
}

__global__ void k_eye_cells(const EyeArgs a)
{
    const int64_t cells = (int64_t)a.gh * a.gw;
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= (int64_t)a.B * cells) return;
    const int32_t b = (int32_t)(p / cells);
    const int64_t q = p - (int64_t)b * cells;
    const int32_t y = (int32_t)(q / a.gw), x = (int32_t)(q - (int64_t)y * a.gw);
    const bool fl = a.flip && a.flip[b];
    const uint8_t* fr = a.frames + (int64_t)b * a.H * a.W * 3;
    auto px = [&](int32_t yy, int32_t xx) {
        const int32_t c = x * a.cell + xx;
        return fr + ((int64_t)(y * a.cell + yy) * a.W + (fl ? a.W - 1 - c : c)) * 3;
    };
    float s = 0.0f, sb = 0.0f, sg = 0.0f;
    for (int32_t yy = 0; yy < a.cell; yy++) {
        s = __fadd_rn(s, np_row_sum(a.cell, [&](int32_t xx) {
                          const uint8_t* v = px(yy, xx);
                          const float m = __fdiv_rn(__fadd_rn(__fadd_rn((float)v[0], (float)v[1]), (float)v[2]), 3.0f);
                          return __fdiv_rn(m, 255.0f);
                      }));
        if (a.chromatic) {
            sb = __fadd_rn(sb, np_row_sum(a.cell, [&](int32_t xx) { return __fdiv_rn((float)px(yy, xx)[2], 255.0f); }));
            sg = __fadd_rn(sg, np_row_sum(a.cell, [&](int32_t xx) { return __fdiv_rn((float)px(yy, xx)[1], 255.0f); }));
        }
    }
    const float area = (float)(a.cell * a.cell);
    const float lum = __fdiv_rn(s, area);
    a.lum[p] = lum;
    if (a.chromatic) {
        a.col[((int64_t)b * 2 + 0) * cells + q] = __fdiv_rn(sb, area);
        a.col[((int64_t)b * 2 + 1) * cells + q] = __fdiv_rn(sg, area);
    }
    float lp = a.lp[p];
    if (a.restart[b]) {
        lp = lum;
        a.dly[((int64_t)b * 2 + 0) * cells + q] = 0.0f;
        a.dly[((int64_t)b * 2 + 1) * cells + q] = 0.0f;
    }
    lp = __fadd_rn(lp, __fmul_rn(a.a_hp, __fsub_rn(lum, lp)));
    a.lp[p] = lp;
    const float hp = __fsub_rn(lum, lp);
    a.sig[((int64_t)b * 2 + 0) * cells + q] = fmaxf(hp, 0.0f);
    a.sig[((int64_t)b * 2 + 1) * cells + q] = fmaxf(-hp, 0.0f);
}

// blockDim.x >= max(gw, gh) + 1
__global__ void k_eye_integral(const EyeArgs a)
{
    const int32_t b = blockIdx.x, W1 = a.gw + 1;
    const float* lum = a.lum + (int64_t)b * a.gh * a.gw;
    float* ii = a.ii + (int64_t)b * (a.gh + 1) * W1;
    const int32_t t = threadIdx.x;
    if (t <= a.gw) {                       // column t of the padded grid, down the rows
        float c = 0.0f;
        ii[t] = 0.0f;
        for (int32_t i = 1; i <= a.gh; i++) {
            c = __fadd_rn(c, t == 0 ? 0.0f : lum[(int64_t)(i - 1) * a.gw + t - 1]);
            ii[(int64_t)i * W1 + t] = c;
        }
    }
    __syncthreads();
    if (t <= a.gh) {                       // row t, along the columns
        float* r = ii + (int64_t)t * W1;
        float c = r[0];
        for (int32_t j = 1; j <= a.gw; j++) {
            c = __fadd_rn(c, r[j]);
            r[j] = c;
        }
    }
}

__device__ __forceinline__ float eye_motion(const EyeArgs& a, int32_t b, int32_t pol, int32_t dir, int32_t y, int32_t x)
{
    const int64_t cells = (int64_t)a.gh * a.gw;
    const float* sg = a.sig + ((int64_t)b * 2 + pol) * cells;
    const float* dl = a.dly + ((int64_t)b * 2 + pol) * cells;
    const int32_t s = a.shift;
    float corr = 0.0f;
    const int64_t i0 = (int64_t)y * a.gw + x;
    if (dir < 2) {
        if (x < a.gw - s) corr = __fsub_rn(__fmul_rn(dl[i0], sg[i0 + s]), __fmul_rn(sg[i0], dl[i0 + s]));
    } else if (y < a.gh - s) {
        const int64_t i1 = i0 + (int64_t)s * a.gw;
        corr = __fsub_rn(__fmul_rn(dl[i0], sg[i1]), __fmul_rn(sg[i0], dl[i1]));
    }
    return (dir & 1) ? fmaxf(-corr, 0.0f) : fmaxf(corr, 0.0f);
}

// the centre-minus-surround contrast, float64 after the float32 box sum (vision.py:167-174)
__device__ __forceinline__ double eye_contrast(const EyeArgs& a, int32_t b, int32_t y, int32_t x)
{
    const int32_t W1 = a.gw + 1, r = a.surround;
    const float* ii = a.ii + (int64_t)b * (a.gh + 1) * W1;
    const int32_t y0 = min(max(y - r, 0), a.gh), y1 = min(max(y + r + 1, 0), a.gh);
    const int32_t x0 = min(max(x - r, 0), a.gw), x1 = min(max(x + r + 1, 0), a.gw);
    const float num = __fadd_rn(__fsub_rn(__fsub_rn(ii[(int64_t)y1 * W1 + x1], ii[(int64_t)y0 * W1 + x1]),
                                          ii[(int64_t)y1 * W1 + x0]), ii[(int64_t)y0 * W1 + x0]);
    const double sur = __ddiv_rn((double)num, (double)((int64_t)(y1 - y0) * (x1 - x0)));
    return __dsub_rn((double)a.lum[((int64_t)b * a.gh + y) * a.gw + x], sur);
}

__global__ void k_eye_rates(const EyeArgs a)
{
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= (int64_t)a.B * a.n_cells) return;
    const int32_t b = (int32_t)(p / a.n_cells), k = (int32_t)(p - (int64_t)b * a.n_cells);
    const int32_t c = a.chan[k], x = a.gx[k], y = a.gy[k], s = a.slot[k];
    if (x < 0 || x >= a.gw || y < 0 || y >= a.gh || c >= EYE_CHANNELS || s < 0 || s >= a.n_ext) return;
    const int64_t cell = ((int64_t)b * a.gh + y) * a.gw + x, cells = (int64_t)a.gh * a.gw;
    float r = 0.0f;
    if (c < EYE_ON_TRANSIENT) {
        r = eye_motion(a, b, c >> 2, c & 3, y, x);
    } else if (c <= EYE_OFF_TRANSIENT) {
        const float hp = a.sig[((int64_t)b * 2 + (c - EYE_ON_TRANSIENT)) * cells + (cell - (int64_t)b * cells)];
        r = __fdiv_rn(__fmul_rn(a.transient_f, hp), a.gain_f);
    } else if (c <= EYE_OFF_SUSTAINED) {
        if (a.sustained != 0.0) {
            const double con = eye_contrast(a, b, y, x);
            const double m = c == EYE_ON_SUSTAINED ? fmax(con, 0.0) : fmax(-con, 0.0);
            r = __double2float_rn(__ddiv_rn(__dmul_rn(a.sustained, m), a.gain));
        }
    } else if (a.chromatic) {
        const float v = a.col[((int64_t)b * 2 + (c - EYE_BLUE)) * cells + (cell - (int64_t)b * cells)];
        r = __fdiv_rn(__fmul_rn(a.chromatic_f, v), a.gain_f);
    }
    if (!a.visible[k]) r = 0.0f;
    const float rate = __fmul_rn(a.max_rate, fminf(fmaxf(__fmul_rn(a.gain_f, r), 0.0f), 1.0f));
    if (a.rates) a.rates[p] = rate;
    a.p_ext[(int64_t)b * a.n_ext + s] = __fmul_rn(rate, a.p_scale);
}

__global__ void k_eye_delay(const EyeArgs a)
{
    const int64_t cells = (int64_t)a.gh * a.gw;
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= (int64_t)a.B * 2 * cells) return;
    a.dly[p] = __fadd_rn(a.dly[p], __fmul_rn(a.a_d, __fsub_rn(a.sig[p], a.dly[p])));
    if (p % (2 * cells) == 0) a.restart[p / (2 * cells)] = 0;
}

// ---- the same eye in two launches or one (the default) ---------------------------------------------------
// The grid of every instance by one thread per cell, then the neurons of an instance by several blocks.
// One block per instance for all of it (its grid in shared memory) kept 64 instances on 64 of the 148 SMs and
// waited through its phases one after the other: 38.5 us for 64 frames of 224 x 256; these two take 7.4 and 16,
// 20.8 together as a dependent chain whose second kernel reads its tables beside the first. The neuron kernel lets
// the next call's grid kernel go when its blocks are done: let go at once, all the grid's blocks settled on the few SMs
// that its own blocks had left free (62 eyes of 19 x 19 cells of 8 x 8 pixels: 19.4 us a call, now 10.5). Small
// eyes, and as many as there are SMs, lose more by the second launch than they gain: they take one
// block per instance again (fb_motion_eye says where the line lies).

// x / 3 and x / 255 rounded to nearest for the values a pixel can take (R + G + B and its third, a byte): one
// Newton correction of the quotient by its exact remainder (Markstein 1990). Checked against the
// division for all 766 sums and 256 bytes. Tables of the quotients in shared memory cost 3.5 bank cycles a
// lookup: 9.1 us per 64 frames of 224 x 256 against 7.4.
__device__ __forceinline__ float eye_quotient(float x, float d, float r)
{
    const float q = __fmul_rn(x, r);
    return __fmaf_rn(__fmaf_rn(-q, d, x), r, q);
}
__device__ __forceinline__ float eye_lum(float sum) { return eye_quotient(eye_quotient(sum, 3.0f, 1.0f / 3.0f), 255.0f, 1.0f / 255.0f); }
__device__ __forceinline__ float eye_channel(float byte) { return eye_quotient(byte, 255.0f, 1.0f / 255.0f); }

// The sums of one cell: luminance, blue, green (the colours when `chrom`).
// VEC4: cell 4 and W a multiple of 4, so a cell row is three aligned 32-bit words.
template <bool VEC4>
__device__ __forceinline__ void cell_sums(const EyeArgs& a, const uint8_t* fr, bool fl, int32_t y, int32_t x, bool chrom,
                                          float& s, float& sb, float& sg)
{
    s = sb = sg = 0.0f;
    if constexpr (VEC4) {
        const int32_t c0 = fl ? a.W - 4 - 4 * x : 4 * x;
        uint32_t w[4][3];
#pragma unroll
        for (int32_t yy = 0; yy < 4; yy++) {
            const uint32_t* p = reinterpret_cast<const uint32_t*>(fr + ((int64_t)(4 * y + yy) * a.W + c0) * 3);
#pragma unroll
            for (int j = 0; j < 3; j++) w[yy][j] = p[j];
        }
#pragma unroll
        for (int32_t yy = 0; yy < 4; yy++) {
            float lum[4], blue[4], green[4];
#pragma unroll
            for (int p = 0; p < 4; p++) {
                float ch[3];
#pragma unroll
                for (int c = 0; c < 3; c++) ch[c] = (float)((w[yy][(3 * p + c) >> 2] >> (8 * ((3 * p + c) & 3))) & 255u);
                lum[p] = eye_lum(__fadd_rn(__fadd_rn(ch[0], ch[1]), ch[2]));
                blue[p] = chrom ? eye_channel(ch[2]) : 0.0f;
                green[p] = chrom ? eye_channel(ch[1]) : 0.0f;
            }
            // a row of fewer than eight values is summed in order; the mirrored frame's pixel xx is this
            // segment's 3 - xx
            auto row = [&](const float (&v)[4]) {
                const float r0 = fl ? v[3] : v[0], r1 = fl ? v[2] : v[1], r2 = fl ? v[1] : v[2], r3 = fl ? v[0] : v[3];
                return __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(0.0f, r0), r1), r2), r3);
            };
            s = __fadd_rn(s, row(lum));
            if (chrom) {
                sb = __fadd_rn(sb, row(blue));
                sg = __fadd_rn(sg, row(green));
            }
        }
    } else {
        auto px = [&](int32_t yy, int32_t xx) {
            const int32_t c = x * a.cell + xx;
            return fr + ((int64_t)(y * a.cell + yy) * a.W + (fl ? a.W - 1 - c : c)) * 3;
        };
        for (int32_t yy = 0; yy < a.cell; yy++) {
            s = __fadd_rn(s, np_row_sum(a.cell, [&](int32_t xx) {
                              const uint8_t* v = px(yy, xx);
                              return eye_lum((float)(v[0] + v[1] + v[2]));
                          }));
            if (chrom) {
                sb = __fadd_rn(sb, np_row_sum(a.cell, [&](int32_t xx) { return eye_channel((float)px(yy, xx)[2]); }));
                sg = __fadd_rn(sg, np_row_sum(a.cell, [&](int32_t xx) { return eye_channel((float)px(yy, xx)[1]); }));
            }
        }
    }
}

// One grid cell q of instance b (p = b * cells + q): luminance, colours (when chromatic), high-pass signal (hp itself; ON is
// max(hp, 0), OFF max(-hp, 0)) and this frame's delay arms; the filters go on to the next frame's.
struct EyeCell {
    float lum, blue, green, hp, on, off;
};
template <bool VEC4>
__device__ __forceinline__ EyeCell eye_cell(const EyeArgs& a, int32_t b, int32_t q, int64_t p, bool restart, bool fl)
{
    const int32_t y = q / a.gw, x = q - y * a.gw;
    const int64_t cells = (int64_t)a.gh * a.gw;
    float* dly = a.dly + (int64_t)b * 2 * cells + q;
    EyeCell c;
    float lp, s, sb, sg;
    auto filters = [&]() {
        lp = a.lp[p];
        c.on = dly[0];
        c.off = dly[cells];
    };
    if (VEC4) filters();                                           // (in flight beside the pixels)
    cell_sums<VEC4>(a, a.frames + (int64_t)b * a.H * a.W * 3, fl, y, x, a.chromatic != 0, s, sb, sg);
    if (!VEC4) filters();                                          // (beside cells of any size they were spilled)
    const float area = (float)(a.cell * a.cell);
    c.lum = __fdiv_rn(s, area);
    if (a.chromatic) {
        c.blue = __fdiv_rn(sb, area);
        c.green = __fdiv_rn(sg, area);
    }
    if (restart) {
        lp = c.lum;
        c.on = c.off = 0.0f;
    }
    lp = __fadd_rn(lp, __fmul_rn(a.a_hp, __fsub_rn(c.lum, lp)));
    a.lp[p] = lp;
    c.hp = __fsub_rn(c.lum, lp);
    dly[0] = __fadd_rn(c.on, __fmul_rn(a.a_d, __fsub_rn(fmaxf(c.hp, 0.0f), c.on)));
    dly[cells] = __fadd_rn(c.off, __fmul_rn(a.a_d, __fsub_rn(fmaxf(-c.hp, 0.0f), c.off)));
    return c;
}

// One thread per (instance, grid cell), the results for k_eye_neurons in the scratch arrays (hp: the ON half of
// `sig`; the delay arms: its OFF half and the integral image's place).
// Bound by instruction issue: twenty instructions a pixel.
template <bool VEC4>
__global__ void __launch_bounds__(256) k_eye_grid(const EyeArgs a)
{
    pdl_chain_behind();
    const int64_t cells = (int64_t)a.gh * a.gw;
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= (int64_t)a.B * cells) return;
    const int32_t b = (int32_t)(p / cells), q = (int32_t)(p - (int64_t)b * cells);
    const EyeCell c = eye_cell<VEC4>(a, b, q, p, a.restart[b] != 0, a.flip && a.flip[b]);
    a.lum[p] = c.lum;
    if (a.chromatic) {
        a.col[(int64_t)b * 2 * cells + q] = c.blue;
        a.col[((int64_t)b * 2 + 1) * cells + q] = c.green;
    }
    a.sig[(int64_t)b * 2 * cells + q] = c.hp;
    a.sig[((int64_t)b * 2 + 1) * cells + q] = c.on;
    a.ii[(int64_t)b * (a.gh + 1) * (a.gw + 1) + q] = c.off;
}

// The neurons [blockIdx.x * run, ...) of instance blockIdx.y. The block keeps the instance's grids in shared
// memory (a neuron gathers up to four cells of them), forms the integral image there (every block of an
// instance for itself: sharing it would cost a launch), and takes the neurons in chunks. SORT: a chunk's are
// sorted by the kind of their channel, so that a warp works on one kind, and their rates go out in neuron
// order through shared memory; without it a thread takes its own. Gathered from L1 and unsorted, 64 x
// 12,246 neurons took 25.7 us, now 16.5; what bounds it is instruction issue (~200 a neuron, 60 of them
// the sort, which pays where the contrast's FP64 is long: fb_motion_eye). 64 registers, so one block of
// 1,024 threads an SM, or two of 512.
constexpr int EYE_THREADS = 1024, EYE_UNROLL = 4;              // (a chunk's entries are numbered in 12 bits)

constexpr int EYE_SMEM_MAX = 227 * 1024;                          // of a block, all of it dynamic: the kernel has no static arrays
struct EyeSmem {                                                   // offsets in floats (a grid has at most 1023 x 1023 cells)
    int32_t hp, on, off, lum, ii, col, rate, order, kind, total;
    EyeSmem() = default;
    EyeSmem(int32_t threads, int32_t cells, int32_t ii_cells, bool sust, bool chrom)
    {
        hp = 0;
        on = hp + cells;
        off = on + cells;
        lum = off + cells;
        ii = lum + (sust ? cells : 0);
        col = ii + (sust ? ii_cells : 0);
        rate = col + (chrom ? 2 * cells : 0);
        order = rate + EYE_UNROLL * threads;
        kind = order + EYE_UNROLL * threads;
        total = kind + 4;
    }
};

// running sums of n values `stride` apart, eight loaded at a time
__device__ __forceinline__ void running_sum(float* v, int32_t n, int32_t stride)
{
    float c = 0.0f;
    int32_t i = 0;
    for (; i + 8 <= n; i += 8) {
        float x[8];
#pragma unroll
        for (int u = 0; u < 8; u++) x[u] = v[(i + u) * stride];
#pragma unroll
        for (int u = 0; u < 8; u++) v[(i + u) * stride] = c = __fadd_rn(c, x[u]);
    }
    for (; i < n; i++) v[i * stride] = c = __fadd_rn(c, v[i * stride]);
}

// where a block's grids come from: k_eye_grid's results, or its own pixels (one block per instance then)
enum { EYE_GRID_READ = 0, EYE_GRID_OWN = 1, EYE_GRID_OWN4 = 2 };
template <int GRID, bool SORT, int T>                             // T threads; as a variable it cost 5 %
__global__ void __launch_bounds__(T, EYE_THREADS / T) k_eye_neurons(const EyeArgs a, const EyeSmem S, int32_t run)
{
    constexpr int32_t chunk = EYE_UNROLL * T;
    extern __shared__ float sm[];
    const int32_t b = blockIdx.y, W1 = a.gw + 1, tid = threadIdx.x, lane = tid & 31;
    const int32_t cells = a.gh * a.gw;
    float *s_hp = sm + S.hp, *s_on = sm + S.on, *s_off = sm + S.off, *s_lum = sm + S.lum, *s_ii = sm + S.ii;
    float *s_col = sm + S.col, *s_rate = sm + S.rate;
    uint32_t* s_order = reinterpret_cast<uint32_t*>(sm + S.order); // per sorted place: entry | channel << 12 | visible << 16 | y << 17
    int32_t* s_kind = reinterpret_cast<int32_t*>(sm + S.kind);     // neurons of each kind in the chunk
    const bool sust = a.sustained != 0.0;
    const int32_t k1 = min(a.n_cells, (int32_t)(blockIdx.x + 1) * run);
    // a chunk's neurons, loaded ahead (the first one's beside the grids): cell (-1: out of range, or no neuron),
    // channel, visibility and row (no division by gw later: 5 % of the instructions), ext slot
    int32_t cell[EYE_UNROLL], chan[EYE_UNROLL], slot[EYE_UNROLL];
    auto fetch = [&](int32_t first) {
#pragma unroll
        for (int u = 0; u < EYE_UNROLL; u++) {
            const int32_t k = first + tid + u * T;
            cell[u] = -1;
            chan[u] = slot[u] = 0;
            if (k >= k1) continue;
            const int32_t x = __ldg(a.gx + k), y = __ldg(a.gy + k), c = __ldg(a.chan + k);
            const int32_t seen = __ldg(a.visible + k) != 0;
            slot[u] = __ldg(a.slot + k);
            const bool in = x >= 0 && x < a.gw && y >= 0 && y < a.gh && c < EYE_CHANNELS && slot[u] >= 0 && slot[u] < a.n_ext;
            if (in) cell[u] = y * a.gw + x;
            chan[u] = (c & 15) | (seen << 4) | ((y & 1023) << 5);
        }
    };
    if (GRID != EYE_GRID_READ) pdl_chain();
    fetch(blockIdx.x * run);                                       // (EYE_GRID_READ: the caller's tables are older than k_eye_grid)
    if (GRID == EYE_GRID_READ) pdl_wait();
    {
        const bool restart = GRID != EYE_GRID_READ && a.restart[b] != 0, fl = GRID != EYE_GRID_READ && a.flip && a.flip[b];
        const float* hp = a.sig + (int64_t)b * 2 * cells;
        const float* off = a.ii + (int64_t)b * (a.gh + 1) * W1;
        const float* lum = a.lum + (int64_t)b * cells;
        const float* col = a.col + (int64_t)b * 2 * cells;
        for (int32_t q = tid; q < cells; q += T) {
            if constexpr (GRID == EYE_GRID_READ) {
                s_hp[q] = hp[q];
                s_on[q] = hp[cells + q];
                s_off[q] = off[q];
                if (sust) {
                    const float l = lum[q];
                    const int32_t y = q / a.gw, x = q - y * a.gw;
                    s_lum[q] = l;
                    s_ii[(y + 1) * W1 + x + 1] = l;
                }
                if (a.chromatic) {
                    s_col[q] = col[q];
                    s_col[cells + q] = col[cells + q];
                }
            } else {
                const EyeCell c = eye_cell<GRID == EYE_GRID_OWN4>(a, b, q, (int64_t)b * cells + q, restart, fl);
                s_hp[q] = c.hp;
                s_on[q] = c.on;
                s_off[q] = c.off;
                if (sust) {
                    const int32_t y = q / a.gw, x = q - y * a.gw;
                    s_lum[q] = c.lum;
                    s_ii[(y + 1) * W1 + x + 1] = c.lum;
                }
                if (a.chromatic) {
                    s_col[q] = c.blue;
                    s_col[cells + q] = c.green;
                }
            }
        }
        if (sust) {                                                // a border of zeros
            for (int32_t t = tid; t <= a.gw; t += T) s_ii[t] = 0.0f;
            for (int32_t t = tid; t <= a.gh; t += T) s_ii[t * W1] = 0.0f;
            __syncthreads();
            for (int32_t t = tid; t <= a.gw; t += T) running_sum(s_ii + t, a.gh + 1, W1);      // down the rows,
            __syncthreads();
            for (int32_t t = tid; t <= a.gh; t += T) running_sum(s_ii + t * W1, W1, 1);        // then along them
        }
    }
    if (!SORT) __syncthreads();                                    // the grids are in place
    for (int32_t first = blockIdx.x * run; first < k1; first += chunk) {
        int32_t count = min(chunk, k1 - first), kind[EYE_UNROLL];
        if (SORT) {
            if (tid < 4) s_kind[tid] = 0;
            __syncthreads();                                           // (the grids are in place, the last chunk is out)
            // the neurons' places, sorted by kind: ballots count a warp's, one atomic per kind and warp reserves theirs
            int32_t at[EYE_UNROLL], mine = 0;
#pragma unroll
            for (int u = 0; u < EYE_UNROLL; u++) {
                const int32_t c = chan[u] & 15;
                kind[u] = cell[u] < 0 ? -1 : c < EYE_ON_TRANSIENT ? 0 : c <= EYE_OFF_TRANSIENT ? 1 : c <= EYE_OFF_SUSTAINED ? 2 : 3;
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                int32_t n = 0;
#pragma unroll
                for (int u = 0; u < EYE_UNROLL; u++) {
                    const uint32_t m = __ballot_sync(0xffffffffu, kind[u] == i);
                    if (kind[u] == i) at[u] = n + __popc(m & ((1u << lane) - 1u));
                    n += __popc(m);
                }
                if (lane == i) mine = n;
            }
            int32_t base = 0;
            if (lane < 4 && mine) base = atomicAdd(&s_kind[lane], mine);
#pragma unroll
            for (int u = 0; u < EYE_UNROLL; u++) {
                const int32_t from = __shfl_sync(0xffffffffu, base, kind[u] & 3);
                if (kind[u] >= 0) at[u] += from;
            }
            __syncthreads();
            int32_t before[4];
            count = 0;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                before[i] = count;
                count += s_kind[i];
            }
#pragma unroll
            for (int u = 0; u < EYE_UNROLL; u++)
                if (kind[u] >= 0) {
                    const int32_t e = tid + u * T;
                    const int32_t bf = kind[u] == 0 ? before[0] : kind[u] == 1 ? before[1] : kind[u] == 2 ? before[2] : before[3];
                    s_order[bf + at[u]] = (uint32_t)e | ((uint32_t)chan[u] << 12);
                    s_rate[e] = __int_as_float(cell[u]);               // its cell, until its rate takes the place
                }
            __syncthreads();
        } else {
#pragma unroll
            for (int u = 0; u < EYE_UNROLL; u++) {                 // (a thread's own entries, in neuron order)
                const int32_t e = tid + u * T;
                s_order[e] = (uint32_t)e | ((uint32_t)chan[u] << 12);
                s_rate[e] = __int_as_float(cell[u]);
                kind[u] = cell[u];
            }
        }
        // (in turn, so that the code of one neuron is not unrolled four times)
#pragma unroll 1
        for (int32_t at_e = tid; at_e < count; at_e += T) {
            const uint32_t o = s_order[at_e];
            const int32_t e = (int32_t)(o & 4095u), c = (int32_t)((o >> 12) & 15u), q = __float_as_int(s_rate[e]);
            if (!SORT && q < 0) continue;
            const int32_t y = (int32_t)(o >> 17), x = q - y * a.gw;
            float r = 0.0f;
            if (c < EYE_ON_TRANSIENT) {
                const int32_t dir = c & 3, sh = a.shift;
                const float sgn = (c >> 2) ? -1.0f : 1.0f;         // (a sign change is exact)
                const float* dl = (c >> 2) ? s_off : s_on;
                float corr = 0.0f;
                if (dir < 2 ? x < a.gw - sh : y < a.gh - sh) {
                    const int32_t q1 = dir < 2 ? q + sh : q + sh * a.gw;
                    const float s0 = fmaxf(sgn * s_hp[q], 0.0f), s1 = fmaxf(sgn * s_hp[q1], 0.0f);
                    corr = __fsub_rn(__fmul_rn(dl[q], s1), __fmul_rn(s0, dl[q1]));
                }
                r = (dir & 1) ? fmaxf(-corr, 0.0f) : fmaxf(corr, 0.0f);
            } else if (c <= EYE_OFF_TRANSIENT) {
                const float h = s_hp[q];
                r = __fdiv_rn(__fmul_rn(a.transient_f, fmaxf(c == EYE_ON_TRANSIENT ? h : -h, 0.0f)), a.gain_f);
            } else if (c <= EYE_OFF_SUSTAINED) {
                if (sust) {
                    const int32_t rr = a.surround;
                    const int32_t y0 = min(max(y - rr, 0), a.gh), y1 = min(max(y + rr + 1, 0), a.gh);
                    const int32_t x0 = min(max(x - rr, 0), a.gw), x1 = min(max(x + rr + 1, 0), a.gw);
                    const float num = __fadd_rn(__fsub_rn(__fsub_rn(s_ii[y1 * W1 + x1], s_ii[y0 * W1 + x1]), s_ii[y1 * W1 + x0]),
                                                s_ii[y0 * W1 + x0]);
                    const double sur = __ddiv_rn((double)num, (double)((int64_t)(y1 - y0) * (x1 - x0)));
                    const double con = __dsub_rn((double)s_lum[q], sur);
                    const double m = c == EYE_ON_SUSTAINED ? fmax(con, 0.0) : fmax(-con, 0.0);
                    r = __double2float_rn(__ddiv_rn(__dmul_rn(a.sustained, m), a.gain));
                }
            } else if (a.chromatic) {
                r = __fdiv_rn(__fmul_rn(a.chromatic_f, s_col[(c - EYE_BLUE) * cells + q]), a.gain_f);
            }
            if (!((o >> 16) & 1u)) r = 0.0f;
            s_rate[e] = __fmul_rn(a.max_rate, fminf(fmaxf(__fmul_rn(a.gain_f, r), 0.0f), 1.0f));
        }
        if (SORT) __syncthreads();
#pragma unroll
        for (int u = 0; u < EYE_UNROLL; u++) {
            if (kind[u] < 0) continue;
            const int32_t e = tid + u * T;
            const float rate = s_rate[e];
            if (a.rates) a.rates[(int64_t)b * a.n_cells + first + e] = rate;
            a.p_ext[(int64_t)b * a.n_ext + slot[u]] = __fmul_rn(rate, a.p_scale);
        }
        if (first + chunk < k1) fetch(first + chunk);
    }
    if (GRID == EYE_GRID_READ) pdl_launch();
    if (blockIdx.x == 0 && tid == 0) a.restart[b] = 0;
}

}  // namespace fb
