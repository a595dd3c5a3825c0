// xcorr_kernel.cuh -- the fused correlation + peak kernel (FP32 SIMT path).
//
// One launch replaces, for a section of windows, the reference's
//   organize_data_fft2d_multi(_deformed)  X/xcorr2d_multi_grid.cu:497, 654
//   cufftExecC2C FORWARD x2               :1334-1341, 1649-1656
//   multiply_conjugate                    :519
//   cufftExecC2C INVERSE                  :1347, 1662
//   complex2amp_xcorr2d                   :536
//   fftshift2d_xcorr2d_row/col            :547, 566
//   find_local_max_2d                     :585
//   reduce_max_index_general/final x4     :32, 103
//   replace_local_max_2d                  :298
//   peak_subpixel_4peak_2d                :309
//   kernel_remove_nan                     :457
// The correlation planes never leave shared memory.
//
// Per CTA: a batch of B windows (B even).  Every transform is one thread's, on packed FP32
// pairs (fft_reg.cuh); shared memory is laid out so that each phase's pairs come in with one
// 16-byte load per two elements (Plane below).  Data flow:
//   P1  the windows' pixel rows are staged in shared memory by cp.async (Raw below); row task
//       (window, row): read both frames' rows, pack z = f1 + i*f2, row FFT in registers, store.
//   P2  column task: column FFT in registers -> Z = FFT2(f1) + i*FFT2(f2).
//   P3  column task (window pair, column): the cross spectrum conj(F1)*F2 follows
//       from Z(k) and Z(-k) as  C = Im(Z(k)Z(-k))/2 + i(|Z(-k)|^2 - |Z(k)|^2)/4;
//       it is Hermitian, so two windows share one inverse transform:
//       W = 4 (C_a + i*C_b), inverse column FFT in registers.
//   P4  row task (pair, row): inverse row FFT -> Re = 4 corr_a, Im = 4 corr_b;
//       |.|/(4N) written as fftshifted FP32 planes.
//   P5  warp per window (two warps for windows taller than 32 rows when the CTA has
//       them): 4-neighbour local maxima inside the search region,
//       count, register top-K (value desc, then lower index), 3-point Gaussian fit
//       with an accurate log-ratio denominator, predictor, limits, NaN/Inf removal.
#pragma once
#include <cfloat>
#include <climits>

#include "fft_reg.cuh"
#include "piv_common.cuh"

namespace piv {

// Bytes b and b + 1 of w as floats: each byte is placed into the low mantissa bits of 2^23
// (0x4B0000bb), then 2^23 is subtracted from both -- exact for 0..255.
template <int b>
__device__ __forceinline__ float2 bytes_to_floats(uint32_t w)
{
    return __fadd2_rn(make_float2(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u | b)),
                                  __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u | (b + 1)))),
                      make_float2(-8388608.0f, -8388608.0f));
}

// ------------------------------------------------------------------------------
// Staging of the windows' pixels.  A row task reads one row, so its loads straight from global
// memory touch 32 different lines per instruction: 394 of the kernel's 997 L1 wavefronts per
// 32x32 window, with L1 at 77 % the bound.  Instead a warp copies a window's rows into shared
// memory (cp.async, neighbouring lanes on neighbouring addresses: about 70 wavefronts), in the
// place where the window's spectrum goes later, and the row tasks read them there.
//   float rows lie an odd number of 16-byte chunks apart, byte rows an odd number of 8-byte
//   chunks, so that 32 consecutive rows are read without bank conflicts.
// Rows start at any pixel: 16-byte copies of float rows need a spacing of 4 (f16), 8-byte copies
// of byte rows an 8-aligned start for every window (b8); the other forms copy 4 bytes at a time,
// byte rows from the word that holds the first pixel.
// ------------------------------------------------------------------------------
template <int N>
__device__ __forceinline__ void copy_async(uint32_t dst, const void *src)
{
    if constexpr (N == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(N) : "memory");
}

constexpr int twice_odd(int n)
{
    while (n % 4 != 2) ++n;
    return n;
}
template <int WSX, int WSY, bool DEF>
struct Raw {
    static constexpr int F = (WSX / 4) | 1;               // float rows: 16-byte chunks apart
    static constexpr int U = twice_odd(WSX / 4 + 1);      // byte rows: words apart
    static constexpr int F_WORDS = DEF ? WSY * F * 4 : WSY * U;
    static constexpr int CELLS = (F_WORDS + WSY * U + 3) / 4;

    // Rows [r0, WSY) of a frame, by the lanes of one warp: a lane keeps its chunk column and
    // steps down the rows that the warp covers at a time.
    template <int BYTES, int C, int PITCH, class T>
    static __device__ __forceinline__ void rows(uint32_t dst, const T *src, int pitch, int r0, int lane)
    {
        constexpr int RPI = 32 / C < WSY ? 32 / C : WSY;  // rows per step
        const int r = lane / C, c = lane - r * C;
        const T *p = src + (ptrdiff_t)(r * pitch + c * (BYTES / (int)sizeof(T)));
        const ptrdiff_t step = (ptrdiff_t)RPI * pitch;
        dst += r * PITCH + c * BYTES;
#pragma unroll
        for (int k = 0; k < (WSY + RPI - 1) / RPI; ++k) {
            const int row = k * RPI + r;
            if ((32 == C * RPI || r < RPI) && (WSY % RPI == 0 || row < WSY) && (r0 == 0 || row >= r0))
                copy_async<BYTES>(dst + k * RPI * PITCH, p);
            p += step;
        }
    }
    static __device__ __forceinline__ void bytes(uint32_t dst, const uint8_t *src, int pitch, int r0, int lane, bool b8)
    {
        if (WSX % 8 == 0 && b8) {
            rows<8, WSX / 8 ? WSX / 8 : 1, U * 4>(dst, src, pitch, r0, lane);
        } else {
            constexpr int C = WSX / 4 + 1;
            src = reinterpret_cast<const uint8_t *>(reinterpret_cast<uintptr_t>(src) & ~(uintptr_t)3);
#pragma unroll 1
            for (int e = r0 * C + lane; e < WSY * C; e += 32) {
                const int r = e / C, c = e - r * C;
                copy_async<4>(dst + (r * U + c) * 4, src + (size_t)r * pitch + 4 * c);
            }
        }
    }
    static __device__ __forceinline__ void floats(uint32_t dst, const float *src, int pitch, int r0, int lane, bool f16)
    {
        if (f16) {
            rows<16, WSX / 4, F * 16>(dst, src, pitch, r0, lane);
        } else {
#pragma unroll 1
            for (int e = r0 * WSX + lane; e < WSY * WSX; e += 32) {
                const int r = e / WSX, c = e - r * WSX;
                copy_async<4>(dst + (r * F * 4 + c) * 4, src + (size_t)r * pitch + c);
            }
        }
    }
    // a staged row as neighbouring pairs v[j] = (row[2j], row[2j + 1]); shift: the byte of the
    // first word that holds pixel 0 (the same for all rows of a window)
    static __device__ __forceinline__ void read_bytes(const uint32_t *row, int shift, bool b8, float2 (&v)[WSX / 2])
    {
        uint32_t w[WSX / 4];
        if (WSX % 8 == 0 && b8) {
#pragma unroll
            for (int q = 0; q < WSX / 8; ++q) {
                const uint2 u = reinterpret_cast<const uint2 *>(row)[q];
                w[2 * q] = u.x;
                w[2 * q + 1] = u.y;
            }
        } else {
            uint32_t lo = row[0];
#pragma unroll
            for (int q = 0; q < WSX / 4; ++q) {
                const uint32_t hi = row[q + 1];
                w[q] = __funnelshift_r(lo, hi, 8 * shift);
                lo = hi;
            }
        }
#pragma unroll
        for (int q = 0; q < WSX / 4; ++q) {
            v[2 * q] = bytes_to_floats<0>(w[q]);
            v[2 * q + 1] = bytes_to_floats<2>(w[q]);
        }
    }
    static __device__ __forceinline__ void read_floats(const float4 *row, float2 (&v)[WSX / 2])
    {
#pragma unroll
        for (int q = 0; q < WSX / 4; ++q) {
            const float4 u = row[q];
            v[2 * q] = make_float2(u.x, u.y);
            v[2 * q + 1] = make_float2(u.z, u.w);
        }
    }
};

// ------------------------------------------------------------------------------
// Shared-memory layout of the spectra.  Unit: a 16-byte cell (re0, re1, im0, im1) of two
// neighbouring elements of a line, so that one load gives both packed pairs of an element
// pair.  A line of N elements has N/2 cells, which are written element by element by threads
// that each hold one position of many lines:
//   window (P1..P3)  cell (j, c) = rows 2j, 2j + 1 of column c, at j * ZS + c; written by row
//                    threads (P1), read and rewritten by column threads (P2, P3);
//   pair (P3, P4)    cell (r, j) = columns 2j, 2j + 1 of row r, at r * DS + j; written by
//                    column threads (P3), read by row threads (P4).
// Bank conflicts: the 4-byte stores of 32 consecutive rows (columns) go to 16 cells, whose
// 4-bank groups repeat after 8; the upper cells of each 16 (8 for lines of 16, 4 for lines
// of 8) therefore hold (im0, im1, re0, re1), and windows (pairs) are padded apart by the
// line's length in banks.  Odd ZS and DS keep the 16-byte accesses conflict-free.
// ------------------------------------------------------------------------------
constexpr int cells_apart(int cells, int len)
{
    while ((4 * cells) % 32 != len % 32) ++cells;
    return cells;
}
// cell j of a line of N: true where the imaginary parts come first
template <int N>
__host__ __device__ constexpr bool im_first(int j) { return (j & (N >= 24 ? 8 : N >= 12 ? 4 : 2)) != 0; }

// async copies of this thread: all but the newest PENDING groups have landed
template <int PENDING>
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory"); }
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

template <int WSX, int WSY>
struct Plane {
    static constexpr int ZS = WSX + 1, DS = WSX / 2 + 1;
    static constexpr int ZW = cells_apart((WSY / 2) * ZS, WSY);  // cells of a window
    // float stride of the correlation planes' rows: 16-byte rows, an odd number of cells
    static constexpr int LDF = (WSX / 4) % 2 ? WSX : WSX + 4;
    static constexpr int PLANES = 2 * WSY * LDF / 4;  // cells of a pair's two planes
    static constexpr int D = WSY * DS;                // cells of a pair's spectrum
    static constexpr int SCRATCH = 17;                // cells of a pair's peak scratch (PeakPart[2][2])
    // cells of a pair: two windows, then the pair's spectrum, then its planes and peak scratch
    static constexpr int PW = cells_apart(
        2 * ZW > D ? (2 * ZW > PLANES + SCRATCH ? 2 * ZW : PLANES + SCRATCH) : (D > PLANES + SCRATCH ? D : PLANES + SCRATCH),
        WSX);
};

// cell j of a line of N as the packed pair it holds, and back
template <int N, int j>
__device__ __forceinline__ cplx<float2> from_cell(float4 v)
{
    if constexpr (im_first<N>(j)) return {make_float2(v.z, v.w), make_float2(v.x, v.y)};
    else return {make_float2(v.x, v.y), make_float2(v.z, v.w)};
}
template <int N, int j>
__device__ __forceinline__ float4 to_cell(cplx<float> a, cplx<float> b)
{
    if constexpr (im_first<N>(j)) return make_float4(a.im, b.im, a.re, b.re);
    else return make_float4(a.re, b.re, a.im, b.im);
}

// Inserts a candidate into a lane's descending list (value desc, then lower index).  A lane
// meets its candidates in ascending index order, so an equal value never goes above a listed
// one and the values alone decide.
template <int K>
__device__ __forceinline__ void topk_insert(float (&tv)[K], int (&ti)[K], float v, int i)
{
    if (!(v > tv[K - 1])) return;
#pragma unroll
    for (int s = K - 1; s >= 1; --s) {
        const bool up = v > tv[s - 1], here = v > tv[s];  // v goes above slot s - 1, above slot s
        tv[s] = up ? tv[s - 1] : (here ? v : tv[s]);
        ti[s] = up ? ti[s - 1] : (here ? i : ti[s]);
    }
    if (v > tv[0]) {
        tv[0] = v;
        ti[0] = i;
    }
}

// ------------------------------------------------------------------------------
// Peak stage of one window: 4-neighbour local maxima inside the search region, count,
// top-Npeak_save, 3-point Gaussian fit, predictor, limits, NaN/Inf removal
// (find_local_max_2d, reduce_max_index_*, replace_local_max_2d, peak_subpixel_4peak_2d,
// kernel_remove_nan).  P: the window's fftshifted plane in shared memory with row
// stride LDF floats.  One warp per window (peak_window), or, for windows of more than 32
// rows, two warps that each scan half of the rows and merge their top-N through shared
// memory (peak_window_part, then peak_window_merge after a barrier).
// ------------------------------------------------------------------------------

// Region rows first, first + step, ... scanned by this lane into its sorted top-K
// (value desc, index asc); returns the lane's count of maxima.
template <int WSX, int WSY, int K, int LDF>
__device__ __forceinline__ int peak_scan(const GridGeom &g, const float *P, int first, int step, float (&tv)[K],
                                         int (&ti)[K])
{
    const int rows = WSY - 2 * g.by;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        tv[k] = -1.f;
        ti[k] = INT_MAX;
    }
    // columns allowed by the border (and by the 4-neighbour stencil) as a bitmask
    constexpr int NWRD = (WSX + 31) / 32;
    const int lo = g.bx > 1 ? g.bx : 1, hi = (WSX - 1 - g.bx) < (WSX - 2) ? (WSX - 1 - g.bx) : (WSX - 2);
    uint32_t allow[NWRD];
#pragma unroll
    for (int q = 0; q < NWRD; ++q) {
        // bits [lo, hi] of word q
        const int l = lo - 32 * q, h = hi - 32 * q;
        const uint32_t upto = h >= 31 ? 0xffffffffu : (h < 0 ? 0u : ((2u << h) - 1u));
        const uint32_t from = l <= 0 ? 0xffffffffu : (l > 31 ? 0u : ~((1u << l) - 1u));
        allow[q] = upto & from;
    }
    // v > 0 and v >= all four neighbours  <=>  v >= max(neighbours, smallest subnormal)
    const float tiny = __int_as_float(1);
    int cnt = 0;
    for (int jj = first; jj < rows; jj += step) {
        const int j = g.by + jj;
        const float *pm = P + j * LDF;
        float mid[WSX];
        // local-maximum test of every column without branches, as a bitmask
        uint32_t mk[NWRD];
#pragma unroll
        for (int q = 0; q < NWRD; ++q) mk[q] = 0;
        auto test = [&](int i, const float (&row)[WSX], float up, float down) {
            const float m = fmaxf(fmaxf(row[i - 1], row[i + 1]), fmaxf(fmaxf(up, down), tiny));
            if (row[i] >= m) mk[i >> 5] |= 1u << (i & 31);
        };
        if constexpr (LDF % 4 == 0) {
            // 16-byte rows: four columns a load
#pragma unroll
            for (int q = 0; q < WSX / 4; ++q) {
                const float4 v = reinterpret_cast<const float4 *>(pm)[q];
                mid[4 * q] = v.x;
                mid[4 * q + 1] = v.y;
                mid[4 * q + 2] = v.z;
                mid[4 * q + 3] = v.w;
            }
#pragma unroll
            for (int q = 0; q < WSX / 4; ++q) {
                const float4 u = reinterpret_cast<const float4 *>(pm - LDF)[q];
                const float4 d = reinterpret_cast<const float4 *>(pm + LDF)[q];
                if (q > 0) test(4 * q, mid, u.x, d.x);
                test(4 * q + 1, mid, u.y, d.y);
                test(4 * q + 2, mid, u.z, d.z);
                if (q < WSX / 4 - 1) test(4 * q + 3, mid, u.w, d.w);
            }
        } else {
#pragma unroll
            for (int i = 0; i < WSX; ++i) mid[i] = pm[i];
#pragma unroll
            for (int i = 1; i < WSX - 1; ++i) test(i, mid, pm[i - LDF], pm[i + LDF]);
        }
        // the row's maxima in column order into the lane's top-K
#pragma unroll
        for (int q = 0; q < NWRD; ++q) {
            uint32_t m = mk[q] & allow[q];
            cnt += __popc(m);
            while (m) {
                const int i = 32 * q + __ffs(m) - 1;
                m &= m - 1;
                topk_insert<K>(tv, ti, pm[i], j * WSX + i);
            }
        }
    }
    return cnt;
}

// Nps rounds of a warp arg-max over the lanes' list heads; lane k < Nps receives the
// k-th best (value, index), -1 / INT_MAX when there are fewer candidates.  Candidates
// are positive, so their bit patterns order as unsigned integers: the largest value
// is one warp max-reduction, the lowest index holding it one min-reduction (value
// desc, then lower index).  Indices are unique, so exactly one lane owns each winner and pops it.
template <int K>
__device__ __forceinline__ void peak_pop(float (&tv)[K], int (&ti)[K])
{
#pragma unroll
    for (int s = 0; s < K - 1; ++s) {
        tv[s] = tv[s + 1];
        ti[s] = ti[s + 1];
    }
    tv[K - 1] = -1.f;
    ti[K - 1] = INT_MAX;
}
template <int K>
__device__ __forceinline__ void peak_select(int Nps, int lane, float (&tv)[K], int (&ti)[K], float &v, int &idx)
{
    v = -1.f;
    idx = INT_MAX;
    for (int k = 0; k < Nps; ++k) {
        const uint32_t key = tv[0] > 0.f ? __float_as_uint(tv[0]) : 0u;
        const uint32_t kmax = __reduce_max_sync(0xffffffffu, key);
        const uint32_t imin = __reduce_min_sync(0xffffffffu, key == kmax ? (uint32_t)ti[0] : 0xffffffffu);
        const float bv = kmax ? __uint_as_float(kmax) : -1.f;
        const int bi = kmax ? (int)imin : INT_MAX;
        if (lane == k) {
            v = bv;
            idx = bi;
        }
        if (bi == ti[0] && bv > 0.f) peak_pop(tv, ti);
    }
}
// The same for two windows at once, one per half-warp (windows of at most 16 rows, which would
// leave half of a warp idle): lane k < Nps of each half receives its window's k-th.  A 16x16
// launch at 2048x1536, 50 % overlap: 66 -> 61 us, 8x8: 125 -> 109, 32x16: 54 -> 49.
template <int K>
__device__ __forceinline__ void peak_select_half(int Nps, int lane, float (&tv)[K], int (&ti)[K], float &v, int &idx)
{
    v = -1.f;
    idx = INT_MAX;
    for (int k = 0; k < Nps; ++k) {
        float bv = tv[0];
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) bv = fmaxf(bv, __shfl_xor_sync(0xffffffffu, bv, o));
        int bi = tv[0] == bv ? ti[0] : INT_MAX;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) bi = min(bi, __shfl_xor_sync(0xffffffffu, bi, o));
        if ((lane & 15) == k) {
            v = bv;
            idx = bi;
        }
        if (bi == ti[0] && bv > 0.f) peak_pop(tv, ti);
    }
}

// ln(fm fp / c^2), the Gaussian fit's denominator, which cancels near flat peaks (the
// reference's ln fm + ln fp - 2 ln c in FP32 loses most of its bits there).  fm fp - c^2 is
// formed exactly, up to one rounding, from the two products and their FMA residuals, divided
// by c^2 and passed to log1pf: about 2 ulp of the true value, as FP64 would give after the
// final rounding to FP32, without FP64 arithmetic.  Products below 2^-100, where they would
// lose bits to underflow, take the FP64 form.
__device__ __forceinline__ float fit_denominator(float fm, float fp, float c)
{
    const float p = fm * fp, q = c * c;
    if (!(p >= 7.8886091e-31f && q >= 7.8886091e-31f))  // 2^-100; also zeros and NaN
        return (float)log(((double)fm * (double)fp) / ((double)c * (double)c));
    const float ep = fmaf(fm, fp, -p), eq = fmaf(c, c, -q);
    return log1pf(((p - q) + (ep - eq)) / q);
}

// One direction (step 1: x, LDF: y) of the sub-pixel fit of the candidate at idx with value c
// on plane P: half of the numerator ln f- - ln f+ (FP32 as the reference) over the cancelling
// denominator ln(f- f+ / c^2) (fit_denominator).  false on the plane's edge.
template <int WSX, int WSY, int LDF>
__device__ __forceinline__ bool peak_shift(const float *P, int idx, float c, int step, float &sh)
{
    const int j = idx / WSX, i = idx - j * WSX;
    if (i == 0 || i == WSX - 1 || j == 0 || j == WSY - 1) return false;
    const float *pc = P + j * LDF + i;
    const float f0 = pc[-step], f2 = pc[step];
    const float nn = logf(f0) - logf(f2);
    sh = nn / fit_denominator(f0, f2, c) * 0.5f;
    return true;
}

// limits and NaN/Inf removal of a fitted displacement
__device__ __forceinline__ bool peak_limits(const GridGeom &g, float &ox, float &oy)
{
    if (ox < g.lx1 || ox > g.lx2 || oy < g.ly1 || oy > g.ly2 || isnan(ox) || isnan(oy) || isinf(ox) || isinf(oy)) {
        ox = 0.f;
        oy = 0.f;
        return false;
    }
    return true;
}

// Sub-pixel fit of the candidates held by lanes < Nps, limits, NaN/Inf removal and the
// stores of the window's outputs; cnt is the window's count of maxima.  Called by whole
// warps (the fits' x and y halves run on separate lanes and meet by shuffle).
template <int WSX, int WSY, int LDF>
__device__ __forceinline__ void peak_fit_store(const XcorrArgs &a, const float *P, int w, int lane, float v, int idx,
                                               int cnt, float pred_x, float pred_y)
{
    const GridGeom &g = a.g;
    const int Nps = g.Nps;
    // lanes [0, Nps) fit x and lanes [Nps, 2 Nps) fit y of the same candidates
    const int comp = lane < Nps ? 0 : (lane < 2 * Nps ? 1 : 2);
    const int k = comp == 1 ? lane - Nps : lane;
    const float cv = __shfl_sync(0xffffffffu, v, k & 31);
    const int cidx = __shfl_sync(0xffffffffu, idx, k & 31);
    float sh = 0.f;
    const bool inner = comp < 2 && cv > 0.f && peak_shift<WSX, WSY, LDF>(P, cidx, cv, comp ? LDF : 1, sh);
    const float sy = __shfl_sync(0xffffffffu, sh, (lane + Nps) & 31);
    if (lane < Nps) {
        float ox = 0.f, oy = 0.f;
        bool ok = false;
        if (inner) {
            const int j = idx / WSX, i = idx - j * WSX;
            ox = (float)i + sh - (float)WSX / 2 + pred_x;
            oy = (float)j + sy - (float)WSY / 2 + pred_y;
            ok = peak_limits(g, ox, oy);
        }
        const size_t o = (size_t)w * Nps + lane;
        a.cdx[o] = ox;
        a.cdy[o] = oy;
        a.cvalid[o] = ok ? 1 : 0;
        a.pidx[o] = (v > 0.f) ? idx : -1;
        a.pval[o] = (v > 0.f) ? v : 0.f;
    }
    if (lane == 0) a.count[w] = cnt;
}

// The picks of the CTA's windows (value, index; value <= 0: none), fitted together: a window's
// fit takes 2 Nps lanes, so one warp fits several windows at once instead of each warp running
// the whole fit for 8 of its lanes.
template <int B, int K>
struct PeakPicks {
    float v[B][K];
    int idx[B][K];
};

// Fits and stores picks t = (window b, k, direction), called by NT threads (whole warps).
template <int WSX, int WSY, int LDF, int B, int K, int NT, class PlaneOf, class Win>
__device__ __forceinline__ void peak_fit_all(const XcorrArgs &a, const PeakPicks<B, K> &picks, PlaneOf plane_of,
                                             Win win, int tid)
{
    const GridGeom &g = a.g;
    const int Nps = g.Nps, n = 2 * Nps * B;
    for (int t0 = tid & ~31; t0 < n; t0 += NT) {
        const int t = t0 + (tid & 31), comp = t & 1;
        const int b = (t >> 1) / Nps, k = (t >> 1) - b * Nps;
        const int w = t < n ? win(b) : -1;
        const bool live = w >= a.w_first && w < a.w_end;
        float v = -1.f, o = 0.f;
        int idx = 0;
        bool ok = false;
        if (live) {
            v = picks.v[b][k];
            idx = picks.idx[b][k];
            float sh;
            if (v > 0.f && peak_shift<WSX, WSY, LDF>(plane_of(b), idx, v, comp ? LDF : 1, sh)) {
                const int j = idx / WSX, i = idx - j * WSX;
                const float pred = comp ? a.pred_y[w] : a.pred_x[w];
                o = comp ? (float)j + sh - (float)WSY / 2 + pred : (float)i + sh - (float)WSX / 2 + pred;
                ok = true;
            }
        }
        float other = __shfl_xor_sync(0xffffffffu, o, 1);
        if (ok) ok = comp ? peak_limits(g, other, o) : peak_limits(g, o, other);
        if (live) {
            const size_t q = (size_t)w * Nps + k;
            if (comp == 0) {
                a.cdx[q] = o;
                a.cvalid[q] = ok ? 1 : 0;
                a.pidx[q] = (v > 0.f) ? idx : -1;
            } else {
                a.cdy[q] = o;
                a.pval[q] = (v > 0.f) ? v : 0.f;
            }
        }
    }
}

// diagnostic mode: the plane only, the pass outputs stay untouched
template <int WSX, int WSY, int LDF>
__device__ __forceinline__ void peak_dump(const XcorrArgs &a, const float *P, int w, int lane)
{
    float *dst = a.cc_dump + (size_t)(w - a.w_first) * (WSX * WSY);
    for (int t = lane; t < WSX * WSY; t += 32) {
        const int j = t / WSX, i = t - j * WSX;
        dst[t] = P[j * LDF + i];
    }
}

__device__ __forceinline__ int warp_sum(int x)
{
    return __reduce_add_sync(0xffffffffu, x);
}

// One warp per window: its count of maxima and its picks (lane k < Nps: the k-th).
template <int WSX, int WSY, int K, int LDF>
__device__ __forceinline__ int peak_pick(const GridGeom &g, const float *P, int lane, float &v, int &idx)
{
    float tv[K];
    int ti[K];
    const int cnt = warp_sum(peak_scan<WSX, WSY, K, LDF>(g, P, lane, 32, tv, ti));
    peak_select<K>(g.Nps, lane, tv, ti, v, idx);
    return cnt;
}

// Two windows of at most 16 rows, one per half-warp (P: the half's window).
template <int WSX, int WSY, int K, int LDF>
__device__ __forceinline__ int peak_pick_half(const GridGeom &g, const float *P, int lane, float &v, int &idx)
{
    float tv[K];
    int ti[K];
    int cnt = peak_scan<WSX, WSY, K, LDF>(g, P, lane & 15, 16, tv, ti);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    peak_select_half<K>(g.Nps, lane, tv, ti, v, idx);
    return cnt;
}

// One warp per window.
template <int WSX, int WSY, int K, int LDF = WSX + 1>
__device__ __forceinline__ void peak_window(const XcorrArgs &a, const float *P, int w, int lane)
{
    if (a.cc_dump) {
        peak_dump<WSX, WSY, LDF>(a, P, w, lane);
        return;
    }
    // the predictor of the window, fetched early (used by the Nps fitting lanes)
    float pred_x = 0.f, pred_y = 0.f;
    if (lane < a.g.Nps) {
        pred_x = a.pred_x[w];
        pred_y = a.pred_y[w];
    }
    float v;
    int idx;
    const int cnt = peak_pick<WSX, WSY, K, LDF>(a.g, P, lane, v, idx);
    peak_fit_store<WSX, WSY, LDF>(a, P, w, lane, v, idx, cnt, pred_x, pred_y);
}

// Two warps per window: one warp's half of the rows and its top-Nps.
struct PeakPart {
    float v[8];
    int idx[8];
    int cnt;
};

template <int WSX, int WSY, int K, int LDF = WSX + 1>
__device__ __forceinline__ void peak_window_part(const XcorrArgs &a, const float *P, int part, int lane,
                                                 PeakPart &out)
{
    if (a.cc_dump) return;
    float tv[K];
    int ti[K];
    const int cnt = warp_sum(peak_scan<WSX, WSY, K, LDF>(a.g, P, 32 * part + lane, 64, tv, ti));
    float v;
    int idx;
    peak_select<K>(a.g.Nps, lane, tv, ti, v, idx);
    if (lane < a.g.Nps) {
        out.v[lane] = v;
        out.idx[lane] = idx;
    }
    if (lane == 0) out.cnt = cnt;
}

// After a barrier, one warp merges the two halves' top-Nps (one entry per lane).
__device__ __forceinline__ int peak_merge(int Nps, int lane, const PeakPart (&parts)[2], float &v, int &idx)
{
    float tv[1] = {-1.f};
    int ti[1] = {INT_MAX};
    if (lane < 2 * Nps) {
        const PeakPart &pp = parts[lane >= Nps];
        const int k = lane >= Nps ? lane - Nps : lane;
        tv[0] = pp.v[k];
        ti[0] = pp.idx[k];
    }
    peak_select<1>(Nps, lane, tv, ti, v, idx);
    return parts[0].cnt + parts[1].cnt;
}

// ... and fits them.
template <int WSX, int WSY, int LDF = WSX + 1>
__device__ __forceinline__ void peak_window_merge(const XcorrArgs &a, const float *P, int w, int lane,
                                                  const PeakPart (&parts)[2])
{
    if (a.cc_dump) {
        peak_dump<WSX, WSY, LDF>(a, P, w, lane);
        return;
    }
    float pred_x = 0.f, pred_y = 0.f;
    if (lane < a.g.Nps) {
        pred_x = a.pred_x[w];
        pred_y = a.pred_y[w];
    }
    float v;
    int idx;
    const int cnt = peak_merge(a.g.Nps, lane, parts, v, idx);
    peak_fit_store<WSX, WSY, LDF>(a, P, w, lane, v, idx, cnt, pred_x, pred_y);
}

// Residency asked of the register allocation (the second __launch_bounds__ argument), where
// the compiler's own choice leaves the SM's shared memory unused: 64x64 with 2 windows per CTA
// of 128 threads (68 KB: 3 CTAs at 168 registers, 0.551 ms a grid-1 launch at 6600x4400; unbounded
// 217 registers and 2 CTAs, 0.685), 32x64 with 4 windows per 128 threads or 2 per 64 (12 warps at
// 168 registers; a launch at 4096x2160 and spacing 8x16 668 and 692 us, unbounded at 213 registers
// 726 and 712, 1024x768 and spacing 16x32 19.3 and 20.8 us against 24.1 and 23.7), 32x32 with 4 windows per CTA of 128
// threads (5 CTAs at 96 registers).
template <int WSX, int WSY, int B, int NT>
constexpr int xcorr_min_ctas()
{
    if (WSX == 32 && WSY == 32 && B == 4 && NT == 128) return 5;
    if (WSX == 64 && WSY == 64 && B == 2 && NT == 128) return 3;
    if (WSX == 32 && WSY == 64 && B == 4 && NT == 128) return 3;
    if (WSX == 32 && WSY == 64 && B == 2 && NT == 64) return 6;
    return 1;
}

template <int WSX, int WSY, int B, int NT, int K, bool DEF>
__global__ void __launch_bounds__(NT, (xcorr_min_ctas<WSX, WSY, B, NT>())) xcorr_peak_kernel(const XcorrArgs a)
{
    chain_start();
    constexpr int VB = 1;
    const unsigned blk = blockIdx.x;
#include "xcorr_body.inc"
}

// 2x2-block form: a CTA takes two horizontally adjacent window pairs in two consecutive window
// rows, whose overlapping pixel rows are gathered and row-transformed once (at 50 % overlap 3/4
// of the row transforms of the row-major form).  Same arithmetic per window, so the same bits.
template <int WSX, int WSY, int NT, int K, bool DEF>
__global__ void __launch_bounds__(NT, (xcorr_min_ctas<WSX, WSY, 4, NT>())) xcorr_block_kernel(const XcorrArgs a)
{
    chain_start();
    constexpr int B = 4, VB = 2;
    const unsigned blk = blockIdx.x;
#include "xcorr_body.inc"
}

// the pair of a batch that owns item `it`
__device__ __forceinline__ int batch_pair(const XcorrBatch &b, int it)
{
    int lo = 0, hi = b.n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (b.first[mid] <= it) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Warp form for 32x32 windows: every warp takes one window pair through all phases on its own,
// without a CTA barrier and with all of its lanes busy in each (32 rows, 32 columns).  Z never
// goes back to shared memory: lane c keeps column c in registers and takes the partner column
// -c from lane -c by shuffle.  Window a's cross spectrum waits for window b's half in registers,
// half in shared memory, which lets 16 warps share an SM (12.6 KB of shared memory and 128
// registers a thread each; the CTA form's 16.9 KB a pair allow 12).  113,300 windows of the
// 6600x4400 grid 2 take 0.344 ms; the best CTA form (8 windows, 128 threads) 0.407 ms, and
// 0.464 ms before packed transforms and staged loads.  What bounds it: issue slots (2,310 warp
// instructions per window, 59 % of the slots used), then latency: 14 of 16 possible warps active.
template <int K>
struct PairShared {
    using L = Plane<32, 32>;
    static constexpr int PARK = 8 * 32;  // parked half of window a's cross spectrum
    static constexpr int PICKS = (int)((sizeof(PeakPicks<2, K>) + 15) / 16);
    static constexpr int CELLS = L::ZW + PARK > L::PLANES + PICKS ? L::ZW + PARK : L::PLANES + PICKS;
    static_assert(L::D <= CELLS, "the pair's spectrum fits");
};
template <int NW, int K, bool DEF>
__global__ void __launch_bounds__(32 * NW, 16 / NW) xcorr_pair_kernel(const XcorrArgs a)
{
    chain_start();
    const unsigned blk = blockIdx.x;
#include "xcorr_pair_body.inc"
}
template <int NW, int K, bool DEF>
__global__ void __launch_bounds__(32 * NW, 16 / NW) xcorr_pair_batch_kernel(const __grid_constant__ XcorrBatch b)
{
    chain_start();
    const int lo = batch_pair(b, blockIdx.x);
    const XcorrArgs &a = b.pairs[lo];
    const unsigned blk = blockIdx.x - b.first[lo];
#include "xcorr_pair_body.inc"
}

// Batch form: the CTA-sized window batches ("items") of many pairs with the same window
// shape in one launch, one CTA per item.  Pair i owns items [first[i], first[i+1]); a
// CTA finds its pair by bisection and reads the pair's arguments from the parameter
// (constant bank; read from global memory instead, the kernel ran 2.8 % slower).
// (A persistent grid whose CTAs loop over items was measured against this: the loop made
// the compiler hold loop-invariant state through every phase, 62 -> 106 registers at
// 16x16 and 152 -> 216 at 64x64, and lose occupancy; the hardware scheduler balances
// one-item CTAs as well.)
template <int WSX, int WSY, int B, int NT, int K, bool DEF>
__global__ void __launch_bounds__(NT, (xcorr_min_ctas<WSX, WSY, B, NT>())) xcorr_batch_kernel(const __grid_constant__ XcorrBatch b)
{
    chain_start();
    const int lo = batch_pair(b, blockIdx.x);
    const XcorrArgs &a = b.pairs[lo];
    const unsigned blk = blockIdx.x - b.first[lo];
    constexpr int VB = 1;
#include "xcorr_body.inc"
}

// ------------------------------------------------------------------------------
// Launch of one instantiated shape, K saved peaks at most (explicitly instantiated in
// xcorr_shape_*.cu).
// ------------------------------------------------------------------------------
template <int WSX, int WSY, int B, int NT, int K>
cudaError_t launch_shape(const XcorrArgs &a, bool deformed, cudaStream_t s)
{
    if (a.w_end <= a.w_first) return cudaSuccess;
    const int n = a.w_end - (a.w_first & ~1);  // CTAs start at an even window (pairing)
    const size_t smem = (size_t)(B / 2) * Plane<WSX, WSY>::PW * sizeof(float4);
    dim3 grid((n + B - 1) / B);
    cudaError_t e = cudaSuccess;
    auto go = [&](auto kern) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return;
        kern<<<grid, NT, smem, s>>>(a);
        e = cudaGetLastError();
    };
    if (deformed) go(xcorr_peak_kernel<WSX, WSY, B, NT, K, true>);
    else go(xcorr_peak_kernel<WSX, WSY, B, NT, K, false>);
    return e;
}

// Launch of the 2x2-block form (four windows per CTA): the blocks of the launch's window rows
// (rounded out to whole block rows; windows outside [w_first, w_end) are computed, not
// written).  An odd row of windows has no whole pairs of columns: the row-major form then.
template <int WSX, int WSY, int NT, int K>
cudaError_t launch_shape_block(const XcorrArgs &a, bool deformed, cudaStream_t s)
{
    if (a.w_end <= a.w_first) return cudaSuccess;
    const int nx = a.g.Nx_vec;
    if (nx % 2) return launch_shape<WSX, WSY, 4, NT, K>(a, deformed, s);
    const int by0 = (a.w_first / nx) >> 1, by1 = ((a.w_end - 1) / nx) >> 1;
    const size_t smem = (size_t)2 * Plane<WSX, WSY>::PW * sizeof(float4);
    dim3 grid((unsigned)((nx >> 1) * (by1 - by0 + 1)));
    cudaError_t e = cudaSuccess;
    auto go = [&](auto kern) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return;
        kern<<<grid, NT, smem, s>>>(a);
        e = cudaGetLastError();
    };
    if (deformed) go(xcorr_block_kernel<WSX, WSY, NT, K, true>);
    else go(xcorr_block_kernel<WSX, WSY, NT, K, false>);
    return e;
}

// Launch of a batch: items = sum over pairs of ceil(windows / B), first[] their prefix
// sums; one CTA per item.
template <int WSX, int WSY, int B, int NT, int K>
cudaError_t launch_shape_batch(const XcorrBatch &b, bool deformed, cudaStream_t s)
{
    if (b.items <= 0) return cudaSuccess;
    const size_t smem = (size_t)(B / 2) * Plane<WSX, WSY>::PW * sizeof(float4);
    cudaError_t e = cudaSuccess;
    auto go = [&](auto kern) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return;
        kern<<<b.items, NT, smem, s>>>(b);
        e = cudaGetLastError();
    };
    if (deformed) go(xcorr_batch_kernel<WSX, WSY, B, NT, K, true>);
    else go(xcorr_batch_kernel<WSX, WSY, B, NT, K, false>);
    return e;
}

// Launches of the warp form (two windows per warp, NW warps per CTA).
template <int NW, int K>
cudaError_t launch_pair(const XcorrArgs &a, bool deformed, cudaStream_t s)
{
    if (a.w_end <= a.w_first) return cudaSuccess;
    const int pairs = (a.w_end - (a.w_first & ~1) + 1) / 2;  // warps start at an even window
    cudaError_t e = cudaSuccess;
    auto go = [&](auto kern, int cells) {
        const size_t smem = (size_t)NW * cells * sizeof(float4);
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return;
        kern<<<(pairs + NW - 1) / NW, 32 * NW, smem, s>>>(a);
        e = cudaGetLastError();
    };
    if (deformed) go(xcorr_pair_kernel<NW, K, true>, PairShared<K>::CELLS);
    else go(xcorr_pair_kernel<NW, K, false>, PairShared<K>::CELLS);
    return e;
}

template <int NW, int K>
cudaError_t launch_pair_batch(const XcorrBatch &b, bool deformed, cudaStream_t s)
{
    if (b.items <= 0) return cudaSuccess;
    cudaError_t e = cudaSuccess;
    auto go = [&](auto kern, int cells) {
        const size_t smem = (size_t)NW * cells * sizeof(float4);
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return;
        kern<<<b.items, 32 * NW, smem, s>>>(b);
        e = cudaGetLastError();
    };
    if (deformed) go(xcorr_pair_batch_kernel<NW, K, true>, PairShared<K>::CELLS);
    else go(xcorr_pair_batch_kernel<NW, K, false>, PairShared<K>::CELLS);
    return e;
}

// A shape's kernels are compiled in parts (PIV_K 4 or 8 saved peaks, PIV_BATCH 0 or 1), because the
// driver loads a whole module with the first of its kernels and a program rarely needs two parts.
// The first use in a process of 64x64 took 25.5 ms in one module, 9.5 in parts; 32x32 15.5 -> 7.1,
// 48x48 18.4 -> 7.2.
#ifdef PIV_K
#if PIV_BATCH
#define PIV_SHAPE(WX, WY, B, NT)
#define PIV_SHAPE_BATCH(WX, WY, B, NT) \
    template cudaError_t launch_shape_batch<WX, WY, B, NT, PIV_K>(const XcorrBatch &, bool, cudaStream_t);
#else
#define PIV_SHAPE(WX, WY, B, NT) \
    template cudaError_t launch_shape<WX, WY, B, NT, PIV_K>(const XcorrArgs &, bool, cudaStream_t);
#define PIV_SHAPE_BATCH(WX, WY, B, NT)
#endif
#endif

}  // namespace piv
