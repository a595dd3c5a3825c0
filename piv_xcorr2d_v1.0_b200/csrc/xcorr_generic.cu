// xcorr_generic.cu -- the correlation + peak kernel for every window shape the reference
// accepts (ws_x, ws_y multiples of 4 from 4 to 1024, X/xcorr2d_multi_grid.cu:896-920) and
// any Npeak_save, where the fused register-FFT kernels (xcorr_kernel.cuh, 8..64 px, top-8)
// have no instance.  It replaces the same reference steps as those kernels:
//   organize_data_fft2d_multi(_deformed)  X/xcorr2d_multi_grid.cu:497, 654
//   cufftExecC2C FORWARD x2 / INVERSE     :1334-1347, 1649-1662
//   multiply_conjugate, complex2amp       :519, 536
//   fftshift2d_xcorr2d_row/col            :547, 566
//   find_local_max_2d                     :585
//   reduce_max_index_*, replace_local_max :32, 103, 298 (Npeak_save rounds)
//   peak_subpixel_4peak_2d, remove_nan    :309, 457
//
// One CTA per window, persistent over the launch's windows.  The window's complex plane
// lives in shared memory when it fits (up to 20,480 points, e.g. 128x128 or 160x128), else
// in the CTA's slab of an engine-owned global workspace.
//   load     z = f1 + i*f2 written at the digit-reversed position of the forward
//            transform (mixed radix 4, 2, 3, 5, 7 and any other prime, outermost first);
//   forward  in-place decimation-in-time stages along x, then along y (natural output);
//   spectrum C(k) = conj(F1)F2 from Z(k), Z(-k) as in the fused kernels, C(-k) = conj C(k);
//   inverse  in-place decimation-in-frequency stages (natural input, digit-reversed output,
//            the same permutation), then |.|/N in place;
//   peaks    the fftshifted plane is read through index maps: 4-neighbour local maxima
//            inside the search region, their count, one scan with a top-list per thread (up to
//            8 saved peaks) or Npeak_save rounds of a block arg-max (more), value desc, then
//            lower index; the 3-point Gaussian fit with the FP64 log-ratio denominator,
//            predictor, limits, NaN/Inf removal.
// What bounds it: shared-memory passes and their index arithmetic.  All index maps are tables
// or multiply-high divisions by per-stage constants, and the peaks are found in one scan: a runtime
// division or remainder per point and stage and a scan per saved peak took 0.946 ms for the 7,676
// 40x40 windows and 0.892 ms for the 1,333 96x96 windows of a 2048x1536 frame at 50 % overlap,
// now 0.394 and 0.293 ms.
// Twiddles are exp(-2 pi i t/N) tables computed per CTA in FP64 and rounded once to FP32.
#include <cfloat>
#include <climits>

#include "piv_common.cuh"
#include "xcorr_kernel.cuh"

namespace piv {

// Radices of the two dimensions (outermost first) and where the plane lives; the constants of
// the index divisions (div_by): mx[s], my[s] by M of stage s (the product of the radices after
// it), px[s], py[s] by the butterflies per line N / radix, dx by ws_x.
struct GenericPlan {
    int nfx, nfy;
    int fx[12], fy[12];
    uint32_t mx[12], my[12], px[12], py[12], dx;
    int in_smem;  // 1: the plane in shared memory, 0: in the CTA's workspace slab
    int rows;     // rows that a warp covers in one step
    int any;      // a radix above 7 (prime up to 251): the local-array stage
};

namespace {

constexpr int kGenThreads = kGenericThreads;
constexpr int kGenWarps = kGenThreads / 32;

// n / d by a multiply-high with ceil(2^32 / d) (0 for d = 1): exact while n * d < 2^32, and the
// kernel's n stay below 2^20 points with d up to 1024.
__device__ __forceinline__ int div_by(int n, uint32_t magic) { return magic ? (int)__umulhi((uint32_t)n, magic) : n; }

// a * w
__device__ __forceinline__ float2 gmul(float2 a, float2 w)
{
    return make_float2(__fmaf_rn(a.x, w.x, -__fmul_rn(a.y, w.y)), __fmaf_rn(a.y, w.x, __fmul_rn(a.x, w.y)));
}

// W_N^t (forward) or its conjugate (inverse) from the forward table
template <bool INV>
__device__ __forceinline__ float2 gtw(const float2 *W, int t)
{
    const float2 w = W[t];
    return INV ? make_float2(w.x, -w.y) : w;
}

// R-point DFT of x in place: y[k] = sum_q x[q] W_R^(q k), W_R^e = W_N^(e N/R)
template <int R, bool INV>
__device__ __forceinline__ void gdft(float2 (&x)[R], const float2 *W, int N)
{
    if constexpr (R == 2) {
        const float2 a = x[0], b = x[1];
        x[0] = make_float2(a.x + b.x, a.y + b.y);
        x[1] = make_float2(a.x - b.x, a.y - b.y);
    } else if constexpr (R == 4) {
        const float2 a = x[0], b = x[1], c = x[2], d = x[3];
        const float2 t0 = make_float2(a.x + c.x, a.y + c.y), t1 = make_float2(a.x - c.x, a.y - c.y);
        const float2 t2 = make_float2(b.x + d.x, b.y + d.y), u = make_float2(b.x - d.x, b.y - d.y);
        // (b - d) times -i (forward) or +i (inverse)
        const float2 t3 = INV ? make_float2(-u.y, u.x) : make_float2(u.y, -u.x);
        x[0] = make_float2(t0.x + t2.x, t0.y + t2.y);
        x[1] = make_float2(t1.x + t3.x, t1.y + t3.y);
        x[2] = make_float2(t0.x - t2.x, t0.y - t2.y);
        x[3] = make_float2(t1.x - t3.x, t1.y - t3.y);
    } else {
        const int st = N / R;
        float2 w[R], y[R];
#pragma unroll
        for (int q = 1; q < R; ++q) w[q] = gtw<INV>(W, q * st);
#pragma unroll
        for (int k = 0; k < R; ++k) {
            float2 acc = x[0];
#pragma unroll
            for (int q = 1; q < R; ++q) {
                const float2 p = (q * k) % R ? gmul(x[q], w[(q * k) % R]) : x[q];
                acc.x = __fadd_rn(acc.x, p.x);
                acc.y = __fadd_rn(acc.y, p.y);
            }
            y[k] = acc;
        }
#pragma unroll
        for (int k = 0; k < R; ++k) x[k] = y[k];
    }
}

// Where a stage works: one dimension of the plane, for all lines.  Elements of a line are
// estride apart, lines lstride apart.
struct GLines {
    int N, estride, lines, lstride;
    uint32_t by_lines;  // div_by constant of `lines` (used when lines are the fast index)
    const float2 *W;
};

// One stage along one dimension.  DIT (forward): blocks of L points combine R sub-transforms of
// M = L/R points: inputs at q*M + k1 are twiddled by W_L^(q k1) and transformed, outputs to
// k1 + M*k2.  DIF (inverse): inputs at m + M*q are transformed and the outputs twiddled by
// W_L^(m k2), to m + M*k2.  LINE_FAST: consecutive threads take consecutive lines (columns:
// contiguous addresses) rather than consecutive points.  by_m, by_pl: div_by constants of M and
// of the butterflies per line.
template <int R, bool INV, bool LINE_FAST>
__device__ __forceinline__ void gstage(float2 *buf, const GLines &d, int L, uint32_t by_m, uint32_t by_pl)
{
    const int M = L / R, tws = d.N / L, per_line = d.N / R, total = d.lines * per_line, step = M * d.estride;
    for (int b = threadIdx.x; b < total; b += kGenThreads) {
        int line, t;
        if constexpr (LINE_FAST) {
            t = div_by(b, d.by_lines);
            line = b - t * d.lines;
        } else {
            line = div_by(b, by_pl);
            t = b - line * per_line;
        }
        const int blk = div_by(t, by_m), k1 = t - blk * M;
        float2 *base = buf + line * d.lstride + (blk * L + k1) * d.estride;
        float2 x[R];
#pragma unroll
        for (int q = 0; q < R; ++q) x[q] = base[q * step];
        const float2 *w = d.W + k1 * tws;  // q k1 tws < N
        if constexpr (!INV) {
            if (M > 1) {
#pragma unroll
                for (int q = 1; q < R; ++q) x[q] = gmul(x[q], gtw<false>(w, (q - 1) * k1 * tws));
            }
            gdft<R, false>(x, d.W, d.N);
        } else {
            gdft<R, true>(x, d.W, d.N);
            if (M > 1) {
#pragma unroll
                for (int q = 1; q < R; ++q) x[q] = gmul(x[q], gtw<true>(w, (q - 1) * k1 * tws));
            }
        }
#pragma unroll
        for (int q = 0; q < R; ++q) base[q * step] = x[q];
    }
}

// A stage of a prime radix above 7 (up to 251): the R-point DFT runs from a local array.
template <bool INV, bool LINE_FAST>
__device__ __noinline__ void gstage_any(float2 *buf, int R, const GLines d, int L, uint32_t by_m, uint32_t by_pl)
{
    const int M = L / R, tws = d.N / L, per_line = d.N / R, total = d.lines * per_line, st = d.N / R;
    float2 x[256];
    for (int b = threadIdx.x; b < total; b += kGenThreads) {
        int line, t;
        if constexpr (LINE_FAST) {
            t = div_by(b, d.by_lines);
            line = b - t * d.lines;
        } else {
            line = div_by(b, by_pl);
            t = b - line * per_line;
        }
        const int blk = div_by(t, by_m), k1 = t - blk * M, step = M * d.estride;
        float2 *base = buf + line * d.lstride + (blk * L + k1) * d.estride;
        for (int q = 0; q < R; ++q) {
            x[q] = base[q * step];
            if (!INV && q > 0) x[q] = gmul(x[q], gtw<false>(d.W, q * k1 * tws));
        }
        for (int k = 0; k < R; ++k) {
            float2 acc = x[0];
            int e = 0;  // (q k) mod R
            for (int q = 1; q < R; ++q) {
                e += k;
                if (e >= R) e -= R;
                const float2 p = gmul(x[q], gtw<INV>(d.W, e * st));
                acc.x = __fadd_rn(acc.x, p.x);
                acc.y = __fadd_rn(acc.y, p.y);
            }
            if (INV && k > 0) acc = gmul(acc, gtw<true>(d.W, k * k1 * tws));
            base[k * step] = acc;  // inputs are all in x already
        }
    }
}

// ANY: the instance that also carries the local-array stage for primes above 7 (its
// 2 KB per-thread stack is reserved only when such a window shape is launched)
template <bool ANY, bool INV, bool LF>
__device__ __forceinline__ void gstage_r(float2 *buf, int R, const GLines &d, int L, uint32_t by_m, uint32_t by_pl)
{
    switch (R) {
    case 2: gstage<2, INV, LF>(buf, d, L, by_m, by_pl); break;
    case 3: gstage<3, INV, LF>(buf, d, L, by_m, by_pl); break;
    case 4: gstage<4, INV, LF>(buf, d, L, by_m, by_pl); break;
    case 5: gstage<5, INV, LF>(buf, d, L, by_m, by_pl); break;
    case 7: gstage<7, INV, LF>(buf, d, L, by_m, by_pl); break;
    default:
        if constexpr (ANY) {
            if (R == 11) gstage<11, INV, LF>(buf, d, L, by_m, by_pl);
            else if (R == 13) gstage<13, INV, LF>(buf, d, L, by_m, by_pl);
            else gstage_any<INV, LF>(buf, R, d, L, by_m, by_pl);
        }
        break;
    }
}

// Forward (DIT, innermost radix first) or inverse (DIF, outermost first) transform of
// every line of one dimension.  f: radices, outermost first.
template <bool ANY, bool INV, bool LF>
__device__ void gfft_dim(float2 *buf, const int *f, int nf, const uint32_t *by_m, const uint32_t *by_pl,
                         const GLines &d)
{
    if constexpr (!INV) {
        int L = 1;
        for (int s = nf - 1; s >= 0; --s) {
            L *= f[s];
            gstage_r<ANY, false, LF>(buf, f[s], d, L, by_m[s], by_pl[s]);
            __syncthreads();
        }
    } else {
        int L = d.N;
        for (int s = 0; s < nf; ++s) {
            gstage_r<ANY, true, LF>(buf, f[s], d, L, by_m[s], by_pl[s]);
            __syncthreads();
            L /= f[s];
        }
    }
}

// position of natural index n in the digit-reversed order of radices f (outermost first)
__device__ __forceinline__ int gperm(int n, const int *f, int nf, int N)
{
    int pos = 0, size = N;
    for (int s = 0; s < nf; ++s) {
        const int M = size / f[s];
        pos += (n % f[s]) * M;
        n /= f[s];
        size = M;
    }
    return pos;
}

__device__ __forceinline__ bool gbetter(float v1, int i1, float v2, int i2)
{
    return v1 > v2 || (v1 == v2 && i1 < i2);
}

// block-wide best (value desc, index asc) and, optionally, sum; every thread gets them
__device__ __forceinline__ void gblock_best(float &v, int &i, int &cnt, float *rv, int *ri, int *rc)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_down_sync(0xffffffffu, v, o);
        const int oi = __shfl_down_sync(0xffffffffu, i, o);
        cnt += __shfl_down_sync(0xffffffffu, cnt, o);
        if (gbetter(ov, oi, v, i)) {
            v = ov;
            i = oi;
        }
    }
    __syncthreads();  // the previous round's readers are done with rv/ri/rc
    if (lane == 0) {
        rv[warp] = v;
        ri[warp] = i;
        rc[warp] = cnt;
    }
    __syncthreads();
    v = rv[0];
    i = ri[0];
    cnt = rc[0];
    for (int q = 1; q < nw; ++q) {
        if (gbetter(rv[q], ri[q], v, i)) {
            v = rv[q];
            i = ri[q];
        }
        cnt += rc[q];
    }
}

// How a warp covers rows of nx points: one row at a time, or 32 / nx rows where they are narrower
// than the warp (one row at a time left 28 of 32 lanes idle at 4 x 1024: a launch at 2048x1536 503
// us, 212 this way).  A lane's row of those and its first column are a table in shared memory, 2
// bytes each: kept in registers over the windows they spilled others, and 12 bytes each cost some
// windows a resident CTA.
__device__ __forceinline__ uint16_t row_lane(int nx, int rows, int lane)
{
    const int row = rows > 1 ? lane / nx : 0, col = lane - row * nx;
    return (uint16_t)(row < rows ? row << 10 | col : 1023);  // past every column: an idle lane
}

// The search region's local maxima, top-K list per thread (rows by warp, columns by lane, so a
// thread meets them in ascending index order), then per warp, then over the warps: pv, pi get
// the Nps best.  Returns the count (thread 0).
template <int K, class Plane>
__device__ __forceinline__ int gpeaks(const Plane &P, int rows, const uint16_t *lanes, int Nps, int nx, int ilo, int ihi, int jlo,
                                      int jhi, float *pv, int *pi, PeakPart *parts)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float tiny = __int_as_float(1);  // v >= max(neighbours, tiny)  <=>  v > 0 and a local maximum
    float tv[K];
    int ti[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        tv[k] = -1.f;
        ti[k] = INT_MAX;
    }
    int cnt = 0;
    const int at = lanes[lane];
    for (int j = jlo + warp * rows + (at >> 10); j <= jhi; j += kGenWarps * rows)
        for (int i = ilo + (at & 1023); i <= ihi; i += 32) {
            const float v = P(i, j);
            const float m = fmaxf(fmaxf(P(i - 1, j), P(i + 1, j)), fmaxf(fmaxf(P(i, j - 1), P(i, j + 1)), tiny));
            if (v >= m) {
                ++cnt;
                topk_insert<K>(tv, ti, v, j * nx + i);
            }
        }
    cnt = warp_sum(cnt);
    float v;
    int idx;
    peak_select<K>(Nps, lane, tv, ti, v, idx);
    if (lane < Nps) {
        parts[warp].v[lane] = v;
        parts[warp].idx[lane] = idx;
    }
    if (lane == 0) parts[warp].cnt = cnt;
    __syncthreads();
    cnt = 0;
    if (warp == 0) {
        // two list entries per lane hold the warps' up to 8 x 8 picks, best first
        static_assert(kGenWarps * 8 <= 64, "two entries per lane");
        float mv[2] = {-1.f, -1.f};
        int mi[2] = {INT_MAX, INT_MAX};
        for (int e = lane; e < kGenWarps * Nps; e += 32) {
            const int q = e / Nps, k = e - q * Nps;
            const float ev = parts[q].v[k];
            const int ei = parts[q].idx[k];
            if (gbetter(ev, ei, mv[0], mi[0])) {
                mv[1] = mv[0];
                mi[1] = mi[0];
                mv[0] = ev;
                mi[0] = ei;
            } else {
                mv[1] = ev;
                mi[1] = ei;
            }
        }
        peak_select<2>(Nps, lane, mv, mi, v, idx);
        if (lane < Nps) {
            pv[lane] = v;
            pi[lane] = idx;
        }
        cnt = warp_sum(lane < kGenWarps ? parts[lane].cnt : 0);
    }
    return cnt;
}

}  // namespace

// SMEM: the plane in shared memory (known at compile time, so that its accesses are 32-bit
// shared-memory instructions rather than generic ones).
template <bool DEF, bool ANY, bool SMEM>
__global__ void __launch_bounds__(kGenThreads, ANY ? 2 : 3) xcorr_generic_kernel(const XcorrArgs a,
                                                                                 const GenericPlan pl, float2 *gplane)
{
    chain_start();
    const GridGeom &g = a.g;
    const int nx = g.ws_x, ny = g.ws_y, N = nx * ny, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    extern __shared__ __align__(16) unsigned char gsm[];
    __shared__ PeakPart parts[kGenWarps];
    __shared__ uint16_t s_lanes[32];
    float2 *Wx = reinterpret_cast<float2 *>(gsm);
    float2 *Wy = Wx + nx;
    int *Sx = reinterpret_cast<int *>(Wy + ny);  // shifted column -> storage column
    int *Sy = Sx + nx;                            // shifted row -> storage row offset
    int *Px = Sy + ny;                            // column -> digit-reversed column
    int *Py = Px + nx;                            // row -> digit-reversed row offset
    float *rv = reinterpret_cast<float *>(Py + ny);
    int *ri = reinterpret_cast<int *>(rv + 32);
    int *rc = ri + 32;
    float *pv = reinterpret_cast<float *>(rc + 32);  // the window's picks
    int *pi = reinterpret_cast<int *>(pv + g.Nps);
    float2 *plane;
    if constexpr (SMEM)
        plane = reinterpret_cast<float2 *>(gsm + (((size_t)(nx + ny) * 16 + 96 * 4 + (size_t)g.Nps * 8 + 15) & ~(size_t)15));
    else
        plane = gplane + (size_t)blockIdx.x * N;

    if (tid < 32) s_lanes[tid] = row_lane(nx, pl.rows, tid);
    // tables: forward twiddles (FP64, rounded once) and the index maps
    for (int t = tid; t < nx; t += kGenThreads) {
        double s, c;
        sincospi(2.0 * (double)t / (double)nx, &s, &c);
        Wx[t] = make_float2((float)c, (float)(-s));
        Sx[t] = gperm((t + nx / 2) % nx, pl.fx, pl.nfx, nx);
        Px[t] = gperm(t, pl.fx, pl.nfx, nx);
    }
    for (int t = tid; t < ny; t += kGenThreads) {
        double s, c;
        sincospi(2.0 * (double)t / (double)ny, &s, &c);
        Wy[t] = make_float2((float)c, (float)(-s));
        Sy[t] = gperm((t + ny / 2) % ny, pl.fy, pl.nfy, ny) * nx;
        Py[t] = gperm(t, pl.fy, pl.nfy, ny) * nx;
    }
    __syncthreads();

    const float tiny = __int_as_float(1);
    const int ilo = g.bx > 1 ? g.bx : 1, ihi = min(nx - 1 - g.bx, nx - 2);
    const int jlo = g.by > 1 ? g.by : 1, jhi = min(ny - 1 - g.by, ny - 2);
    const int rw = ihi - ilo + 1, rh = jhi - jlo + 1, region = (rw > 0 && rh > 0) ? rw * rh : 0;
    const GLines rows = {nx, 1, ny, nx, 0u, Wx}, cols = {ny, nx, nx, 1, pl.dx, Wy};

    for (int w = a.w_first + blockIdx.x; w < a.w_end; w += gridDim.x) {
        const int iy = w / g.Nx_vec, ix = w - iy * g.Nx_vec;
        // ---- load at the digit-reversed positions of the forward transform: rows by warp ----
        {
            const size_t px = (size_t)(iy * g.sp_y - g.Ny_left + a.f1.my) * a.f1.pitch + ix * g.sp_x - g.Nx_left + a.f1.mx;
            const uint8_t *p1 = a.f1.base + px, *p2 = a.f2.base + px;
            const float *pd = DEF ? a.def + (size_t)(iy * g.sp_y) * a.def_pitch + ix * g.sp_x : nullptr;
            const int at = s_lanes[lane];
            for (int r = warp * pl.rows + (at >> 10); r < ny; r += kGenWarps * pl.rows) {
                float2 *row = plane + Py[r];
#pragma unroll 4
                for (int i = at & 1023; i < nx; i += 32) {
                    const float v1 = (float)p1[(size_t)r * a.f1.pitch + i];
                    float v2;
                    if constexpr (DEF) v2 = pd[(size_t)r * a.def_pitch + i];
                    else v2 = (float)p2[(size_t)r * a.f2.pitch + i];
                    row[Px[i]] = make_float2(v1, v2);
                }
            }
        }
        __syncthreads();
        // ---- forward 2D transform: rows (x), then columns (y) ----
        gfft_dim<ANY, false, false>(plane, pl.fx, pl.nfx, pl.mx, pl.px, rows);
        gfft_dim<ANY, false, true>(plane, pl.fy, pl.nfy, pl.my, pl.py, cols);
        // ---- cross spectrum, in place over (k, -k) pairs.  Z(0,0) = (sum f1, sum f2) is
        //      exactly zero iff a frame's window is all zero; the reference's correlation is
        //      then exactly 0 (no candidate), so the spectrum is set to 0 ----
        const float2 dc = plane[0];
        const bool dead = dc.x == 0.f || dc.y == 0.f;
        __syncthreads();  // every thread has read the DC term before it is overwritten
        const int at = s_lanes[lane];
        for (int ky = warp * pl.rows + (at >> 10); ky <= ny / 2; ky += kGenWarps * pl.rows) {
            const int my = ky ? ny - ky : 0;
            for (int kx = at & 1023; kx < nx; kx += 32) {
                const int mx = kx ? nx - kx : 0, t = ky * nx + kx, tm = my * nx + mx;
                if (tm < t) continue;
                const float2 A = plane[t], M = plane[tm];
                const float im2 = __fmaf_rn(A.y, M.x, __fmul_rn(A.x, M.y));
                const float pw = __fsub_rn(__fmaf_rn(M.y, M.y, __fmul_rn(M.x, M.x)), __fmaf_rn(A.y, A.y, __fmul_rn(A.x, A.x)));
                const float2 C = dead ? make_float2(0.f, 0.f) : make_float2(0.5f * im2, 0.25f * pw);
                plane[t] = C;
                if (tm != t) plane[tm] = make_float2(C.x, -C.y);
            }
        }
        __syncthreads();
        // ---- inverse 2D transform (natural in, digit-reversed out), then |.|/N ----
        gfft_dim<ANY, true, true>(plane, pl.fy, pl.nfy, pl.my, pl.py, cols);
        gfft_dim<ANY, true, false>(plane, pl.fx, pl.nfx, pl.mx, pl.px, rows);
        for (int t = tid; t < N; t += kGenThreads) {
            const float2 z = plane[t];
            plane[t].x = __fdiv_rn(sqrtf(__fmaf_rn(z.x, z.x, __fmul_rn(z.y, z.y))), (float)N);
        }
        __syncthreads();
        auto P = [&](int i, int j) -> float { return plane[Sy[j] + Sx[i]].x; };
        if (a.cc_dump) {
            float *dst = a.cc_dump + (size_t)(w - a.w_first) * N;
            for (int j = warp; j < ny; j += kGenWarps)
                for (int i = lane; i < nx; i += 32) dst[j * nx + i] = P(i, j);
            __syncthreads();
            continue;
        }
        int cnt = 0;
        if (g.Nps <= 4) {
            cnt = gpeaks<4>(P, pl.rows, s_lanes, g.Nps, nx, ilo, ihi, jlo, jhi, pv, pi, parts);
        } else if (g.Nps <= 8) {
            cnt = gpeaks<8>(P, pl.rows, s_lanes, g.Nps, nx, ilo, ihi, jlo, jhi, pv, pi, parts);
        } else {
            // Npeak_save rounds of a block arg-max over the local maxima
            float prev_v = FLT_MAX;
            int prev_i = -1;
            for (int k = 0; k < g.Nps; ++k) {
                float bv = -1.f;
                int bi = INT_MAX, c = 0;
                if (prev_v > 0.f) {
                    for (int t = tid; t < region; t += kGenThreads) {
                        const int jj = t / rw, j = jlo + jj, i = ilo + (t - jj * rw);
                        const float v = P(i, j);
                        const float m = fmaxf(fmaxf(P(i - 1, j), P(i + 1, j)), fmaxf(fmaxf(P(i, j - 1), P(i, j + 1)), tiny));
                        if (!(v >= m)) continue;
                        if (k == 0) ++c;
                        const int idx = j * nx + i;
                        if (gbetter(prev_v, prev_i, v, idx) && gbetter(v, idx, bv, bi)) {
                            bv = v;
                            bi = idx;
                        }
                    }
                }
                gblock_best(bv, bi, c, rv, ri, rc);
                if (k == 0) cnt = c;
                if (tid == 0) {
                    pv[k] = bv;
                    pi[k] = bi;
                }
                prev_v = bv;
                prev_i = bi;
            }
        }
        __syncthreads();
        // ---- fit and store; the x and y halves of a pick on neighbouring lanes ----
        for (int e0 = tid & ~31; e0 < 2 * g.Nps; e0 += kGenThreads) {
            const int e = e0 + lane, k = e >> 1, comp = e & 1;
            const bool live = k < g.Nps;
            const float v = live ? pv[k] : -1.f;
            const int idx = live ? pi[k] : 0;
            float o = 0.f;
            bool ok = false;
            if (v > 0.f) {
                const int j = idx / nx, i = idx - j * nx;
                if (i != 0 && i != nx - 1 && j != 0 && j != ny - 1) {
                    const float f0 = comp ? P(i, j - 1) : P(i - 1, j);
                    const float f2 = comp ? P(i, j + 1) : P(i + 1, j);
                    const double dv = (double)v * (double)v;
                    const float nn = logf(f0) - logf(f2);
                    const double den = log(((double)f0 * (double)f2) / dv);
                    const float sh = (float)((double)nn / den / 2.0);
                    o = comp ? (float)j + sh - (float)ny / 2 + a.pred_y[w] : (float)i + sh - (float)nx / 2 + a.pred_x[w];
                    ok = true;
                }
            }
            float other = __shfl_xor_sync(0xffffffffu, o, 1);
            if (ok) ok = comp ? peak_limits(g, other, o) : peak_limits(g, o, other);
            if (live) {
                const size_t q = (size_t)w * g.Nps + k;
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
        if (tid == 0) a.count[w] = cnt;
        __syncthreads();
    }
}

// The launch of one instance.  ANY and SMEM have a module each (PIV_PART 2 * ANY + !SMEM), as the
// driver loads a whole module with the first of its kernels: the first 40x40 pair of a process
// waited 4.5 ms for one module of all, 1.6 for its own.
template <bool ANY, bool SMEM>
cudaError_t launch_generic(const XcorrArgs &a, const GenericPlan &pl, bool deformed, float2 *workspace, int ctas,
                           size_t smem, cudaStream_t s)
{
    cudaError_t e = cudaSuccess;
    auto go = [&](auto kern) {
        // the largest any launch asks for: a captured launch of another grid's (larger) windows
        // keeps running under the attribute set last
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 224 * 1024);
        if (e != cudaSuccess) return;
        kern<<<ctas, kGenThreads, smem, s>>>(a, pl, workspace);
        e = cudaGetLastError();
    };
    if (deformed) go(xcorr_generic_kernel<true, ANY, SMEM>);
    else go(xcorr_generic_kernel<false, ANY, SMEM>);
    return e;
}
#define PIV_GENERIC(ANY, SMEM) \
    template cudaError_t launch_generic<ANY, SMEM>(const XcorrArgs &, const GenericPlan &, bool, float2 *, int, size_t, \
                                                   cudaStream_t);

#if PIV_PART
PIV_GENERIC((PIV_PART >> 1) != 0, (PIV_PART & 1) == 0)
#else
extern PIV_GENERIC(false, false)
extern PIV_GENERIC(true, true)
extern PIV_GENERIC(true, false)

// ---------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------

namespace {
constexpr int kGenSmemPlane = 20480;  // complex points of a plane kept in shared memory

// the constant of div_by
uint32_t div_magic32(int d) { return d > 1 ? (uint32_t)((0x100000000ull + (uint64_t)d - 1) / (uint64_t)d) : 0u; }

int radices(int n, int *f)
{
    int nf = 0;
    while (n % 4 == 0 && n > 4) {
        f[nf++] = 4;
        n /= 4;
    }
    for (int p = 2; n > 1; ++p)
        while (n % p == 0) {
            f[nf++] = p;
            n /= p;
        }
    return nf;
}

size_t table_bytes(int nx, int ny, int nps)
{
    return (((size_t)(nx + ny) * 16 + 96 * 4 + (size_t)nps * 8 + 15) & ~(size_t)15);
}
}  // namespace

GenericPlan generic_plan(int wsx, int wsy)
{
    GenericPlan pl{};
    pl.nfx = radices(wsx, pl.fx);
    pl.nfy = radices(wsy, pl.fy);
    pl.in_smem = wsx * wsy <= kGenSmemPlane ? 1 : 0;
    pl.any = 0;
    auto constants = [&](int n, const int *f, int nf, uint32_t *by_m, uint32_t *by_pl) {
        int M = n;
        for (int s = 0; s < nf; ++s) {
            pl.any |= f[s] > 7;
            M /= f[s];
            by_m[s] = div_magic32(M);
            by_pl[s] = div_magic32(n / f[s]);
        }
    };
    constants(wsx, pl.fx, pl.nfx, pl.mx, pl.px);
    constants(wsy, pl.fy, pl.nfy, pl.my, pl.py);
    pl.dx = div_magic32(wsx);
    pl.rows = wsx < 32 ? 32 / wsx : 1;
    return pl;
}

bool xcorr_generic_needs_workspace(int wsx, int wsy) { return wsx * wsy > kGenSmemPlane; }

int xcorr_generic_ctas(int wsx, int wsy, int nps)
{
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 148;
    }
    if (xcorr_generic_needs_workspace(wsx, wsy)) return 2 * sms;
    // 228 KB an SM; a CTA also holds the kernel's own arrays and 1 KB of the system's
    const size_t smem = table_bytes(wsx, wsy, nps) + (size_t)wsx * wsy * sizeof(float2) +
                        kGenWarps * sizeof(PeakPart) + 32 * sizeof(uint16_t);
    const int by_smem = (int)((228 * 1024) / (smem + 1024));
    const int per_sm = by_smem < 1 ? 1 : (by_smem > 8 ? 8 : by_smem);
    return per_sm * sms;
}

cudaError_t launch_xcorr_generic(const XcorrArgs &a, bool deformed, float2 *workspace, int workspace_ctas,
                                 cudaStream_t s)
{
    const int n = a.w_end - a.w_first;
    if (n <= 0) return cudaSuccess;
    const GenericPlan pl = generic_plan(a.g.ws_x, a.g.ws_y);
    if (!pl.in_smem && (!workspace || workspace_ctas < 1)) return cudaErrorInvalidValue;
    const size_t smem = table_bytes(a.g.ws_x, a.g.ws_y, a.g.Nps) +
                        (pl.in_smem ? (size_t)a.g.ws_x * a.g.ws_y * sizeof(float2) : 0);
    int ctas = pl.in_smem ? xcorr_generic_ctas(a.g.ws_x, a.g.ws_y, a.g.Nps) : workspace_ctas;
    if (ctas > n) ctas = n;
    const auto launch = pl.any ? (pl.in_smem ? launch_generic<true, true> : launch_generic<true, false>)
                               : (pl.in_smem ? launch_generic<false, true> : launch_generic<false, false>);
    return launch(a, pl, deformed, workspace, ctas, smem, s);
}
#endif

}  // namespace piv
