// field_kernels.cu -- window deformation, grid upsampling and vector validation.
//
// The vector-field "extension" of the reference (extend_filtered_vecfield_p1/p2,
// X/xcorr2d_multi_grid.cu:1547-1618: thousands of 1-float device copies that pad the
// field with a 3-cell edge-replicated border) is not materialised: every read of the
// extended field at (m, n) reads the field at (clamp(m-3), clamp(n-3)), which is the
// same value.
#include "fft_reg.cuh"
#include "piv_common.cuh"

namespace piv {

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// Extended-field value at ext index (m, n) of a field with Nx x Ny vectors.
__device__ __forceinline__ float ext_field(const float *f, int Nx, int Ny, int m, int n)
{
    return *(f + clampi(n - 3, 0, Ny - 1) * Nx + clampi(m - 3, 0, Nx - 1));
}

// ------------------------------------------------------------------------------
// Kernel_Window_Deformation_2d (X/xcorr2d_multi_grid.cu:608-652, launched at :1300
// and :1624): bilinear displacement of every pixel of the [Ny_aug][Nx_aug] extent, then
// bilinear interpolation of frame 2 there.  Every product and sum is rounded as the
// reference's, written out because neighbouring pixels share packed FP32 instructions.
// Frame-2 taps outside the padded frame read 0 (the reference reads its zero padding there,
// or out of bounds).
//
// What bounds it: instructions, the conversion pipe and the latency of the byte gathers.  Against
// one scalar pixel after another (83 instructions and 7 conversions a pixel, every tap's bounds
// checked):
//   - floor(x) in integer and float form comes from one addition: x + 1.5 * 2^23 rounded down
//     holds it in its low bits (|x| < 2^22), so only the bytes go through the conversion pipe;
//   - a cell's displacements lie between its corners', so one test of the corners clears a whole
//     run of pixels; runs near the frame's border, and displacements that are no small numbers,
//     take deform_any.
// Two mappings, 6600x4400 at spacing 16: 82 us before, 70 by deform_cell8_kernel, 82 by
// deform_kernel; 4096x2160 at 12: 47 -> 28 us by deform_kernel; 2048x1536 at 4 (20): 21.5 -> 13
// (22.5 -> 12).
// ------------------------------------------------------------------------------
constexpr int kDeformRows = 32, kDeformThreads = 128, kDeformMinCtas = 600;
constexpr int kDeformFar = 1 << 21;  // positions that the addition of 1.5 * 2^23 splits, with room to spare

// One pixel at (px, py): taps may lie outside the frame, and the position may be any number or none.
// Without the first line a predictor with NaN in 1 % of its vectors took 28.6 us at 2048x1536 and
// spacing 16 (15.0 with it, 14.7 without NaN): eight such calls in a row for a run of pixels.
__device__ __noinline__ float deform_any(const Frame8 &f, float px, float py, int col_off, int row_off)
{
    const float inf = __int_as_float(0x7f800000);
    // no number: an infinite position's taps lie outside, and its weights times their zeros are NaN
    if (!(fabsf(px) < inf && fabsf(py) < inf)) return __int_as_float(0x7fffffff);
    const int i_x = (int)floorf(px), i_y = (int)floorf(py);
    const float a_x = __fsub_rn(px, (float)i_x), a_y = __fsub_rn(py, (float)i_y);
    float p[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        const int c = i_x + col_off + (t & 1), r = i_y + row_off + (t >> 1);
        p[t] = (c >= 0 && c < f.cols && r >= 0 && r < f.rows) ? (float)*(f.base + (size_t)r * f.pitch + c) : 0.f;
    }
    const float b_x = __fsub_rn(1.f, a_x), b_y = __fsub_rn(1.f, a_y);
    const float s = __fmaf_rn(__fmul_rn(b_x, b_y), p[0], __fmul_rn(__fmul_rn(a_x, b_y), p[1]));
    return __fmaf_rn(__fmul_rn(a_x, a_y), p[3], __fmaf_rn(__fmul_rn(b_x, a_y), p[2], s));
}

// Any spacing: a thread makes two neighbouring columns and walks down `rows` rows.  What depends on
// the column alone (the cell's column, the weights, the divisions by the spacing) is done once, the
// rows' weights come from a table, and the field is read where the rows enter the next cell.
template <class Off>
__global__ void __launch_bounds__(kDeformThreads) deform_kernel(const __grid_constant__ DeformArgs a, const int rows)
{
    __shared__ float4 s_row[kDeformRows];  // (a_y, a_y, 1 - a_y, 1 - a_y)
    const int X0 = (blockIdx.x * kDeformThreads + threadIdx.x) * 2;
    const int Y0 = blockIdx.y * rows, Y1 = min(Y0 + rows, a.Ny_aug);
    const int st_x = a.hfws_x - a.sp_x * 3, st_y = a.hfws_y - a.sp_y * 3;  // origin of the extended field
    auto cell = [](int v, int st, int sp) { return ((float)v - (float)st) / (float)sp; };
    if (threadIdx.x < rows) {
        const float y = cell(Y0 + threadIdx.x, st_y, a.sp_y), a_y = y - floorf(y);
        s_row[threadIdx.x] = make_float4(a_y, a_y, 1.f - a_y, 1.f - a_y);
    }
    __syncthreads();
    if (X0 >= a.Nx_aug) return;
    const int col_off = a.f2.mx - a.Nx_left, row_off = a.f2.my - a.Ny_left;
    const float xa = cell(X0, st_x, a.sp_x), xb = cell(X0 + 1, st_x, a.sp_x);
    const float fa = floorf(xa), fb = floorf(xb);
    const float2 one = make_float2(1.f, 1.f), minus = make_float2(-1.f, -1.f);
    const float2 a_x = make_float2(xa - fa, xb - fb), b_x = __fadd2_rn(one, make_float2(-a_x.x, -a_x.y));
    // the clamped field columns of both pixels' cells
    const int ca = clampi((int)fa - 3, 0, a.Nx_vec - 1), ca1 = clampi((int)fa - 2, 0, a.Nx_vec - 1);
    const int cb = clampi((int)fb - 3, 0, a.Nx_vec - 1), cb1 = clampi((int)fb - 2, 0, a.Nx_vec - 1);
    chain_start();
    float2 u1, u2, u3, u4, v1, v2, v3, v4;
    auto field_row = [&](int n, float2 &ul, float2 &ur, float2 &vl, float2 &vr) {
        const size_t o = (size_t)clampi(n - 3, 0, a.Ny_vec - 1) * a.Nx_vec;
        const float *u = a.fx + o, *v = a.fy + o;
        ul = make_float2(*(u + ca), *(u + cb));
        ur = make_float2(*(u + ca1), *(u + cb1));
        vl = make_float2(*(v + ca), *(v + cb));
        vr = make_float2(*(v + ca1), *(v + cb1));
    };
    const float2 X = make_float2((float)X0, (float)(X0 + 1));
    const float kMagic = 12582912.f;  // 1.5 * 2^23
    const float2 magic = make_float2(kMagic, kMagic), unmagic = make_float2(-kMagic, -kMagic);
    const int pitch = a.f2.pitch;
    const uint8_t *base = a.f2.base, *base1 = base + pitch;
    const Off k0 = (Off)(row_off - 0x4B400000) * (Off)pitch + (Off)(col_off - 0x4B400000);
    const bool both = X0 + 1 < a.Nx_aug;
    float *dst = a.out + (size_t)Y0 * a.out_pitch + X0;

    auto position = [&](int Y, float2 fy, float2 &px, float2 &py) {
        const float4 w = s_row[Y - Y0];
        const float2 a_y = make_float2(w.x, w.y), b_y = make_float2(w.z, w.w);
        const float2 c1 = __fmul2_rn(b_x, b_y), c2 = __fmul2_rn(a_x, b_y);
        const float2 c3 = __fmul2_rn(b_x, a_y), c4 = __fmul2_rn(a_x, a_y);
        px = __ffma2_rn(c4, u4, __ffma2_rn(c3, u3, __ffma2_rn(c2, u2, __ffma2_rn(c1, u1, X))));
        py = __ffma2_rn(c4, v4, __ffma2_rn(c3, v3, __ffma2_rn(c2, v2, __ffma2_rn(c1, v1, fy))));
    };
    auto store = [&](float2 res) {
        if (both) *reinterpret_cast<float2 *>(dst) = res;
        else *dst = res.x;
        dst += a.out_pitch;
    };
    // N rows whose taps all lie in the frame: all loads before their use
    auto run = [&](auto nc, int Y, float2 fy) {
        constexpr int N = decltype(nc)::value;
        float2 px[N], py[N], tx[N], ty[N];
        unsigned char p[N][8];
#pragma unroll
        for (int i = 0; i < N; ++i) {
            position(Y + i, fy, px[i], py[i]);
            fy = __fadd2_rn(fy, one);
            tx[i] = __fadd2_rd(px[i], magic);
            ty[i] = __fadd2_rd(py[i], magic);
            const Off oa = (Off)__float_as_int(ty[i].x) * (Off)pitch + ((Off)__float_as_int(tx[i].x) + k0);
            const Off ob = (Off)__float_as_int(ty[i].y) * (Off)pitch + ((Off)__float_as_int(tx[i].y) + k0);
            const uint8_t *pa = base + oa, *pb = base + ob, *pa1 = base1 + oa, *pb1 = base1 + ob;
            p[i][0] = *(pa);
            p[i][1] = *(pb);
            p[i][2] = *(pa + 1);
            p[i][3] = *(pb + 1);
            p[i][4] = *(pa1);
            p[i][5] = *(pb1);
            p[i][6] = *(pa1 + 1);
            p[i][7] = *(pb1 + 1);
        }
#pragma unroll
        for (int i = 0; i < N; ++i) {
            auto tap = [&](int t) { return make_float2((float)p[i][2 * t], (float)p[i][2 * t + 1]); };
            const float2 ax = __ffma2_rn(__fadd2_rn(tx[i], unmagic), minus, px[i]);
            const float2 ay = __ffma2_rn(__fadd2_rn(ty[i], unmagic), minus, py[i]);
            const float2 bx = __ffma2_rn(ax, minus, one), by = __ffma2_rn(ay, minus, one);
            const float2 s = __ffma2_rn(__fmul2_rn(bx, by), tap(0), __fmul2_rn(__fmul2_rn(ax, by), tap(1)));
            store(__ffma2_rn(__fmul2_rn(ax, ay), tap(3), __ffma2_rn(__fmul2_rn(bx, ay), tap(2), s)));
        }
    };

    int Y = Y0, i_y = (int)floorf(cell(Y0, st_y, a.sp_y));
    float2 fy = make_float2((float)Y0, (float)Y0);
    field_row(i_y, u3, u4, v3, v4);
    while (true) {
        u1 = u3;
        u2 = u4;
        v1 = v3;
        v2 = v4;
        field_row(i_y + 1, u3, u4, v3, v4);
        // the rows of this cell; their displacements lie between the corners'
        const int end = min(Y1, st_y + (i_y + 1) * a.sp_y);
        auto lowest = [](float2 p, float2 q, float2 r, float2 s) {
            return fminf(fminf(fminf(p.x, p.y), fminf(q.x, q.y)), fminf(fminf(r.x, r.y), fminf(s.x, s.y)));
        };
        auto highest = [](float2 p, float2 q, float2 r, float2 s) {
            return fmaxf(fmaxf(fmaxf(p.x, p.y), fmaxf(q.x, q.y)), fmaxf(fmaxf(r.x, r.y), fmaxf(s.x, s.y)));
        };
        // a NaN corner makes sum NaN
        const float2 uv = __fadd2_rn(__fadd2_rn(__fadd2_rn(u1, u2), __fadd2_rn(u3, u4)),
                                     __fadd2_rn(__fadd2_rn(v1, v2), __fadd2_rn(v3, v4)));
        const float sum = uv.x + uv.y;
        const bool inside = X.x + lowest(u1, u2, u3, u4) >= (float)(1 - col_off) &&
                            X.y + highest(u1, u2, u3, u4) < (float)(min(a.f2.cols, kDeformFar) - 3 - col_off) &&
                            fy.x + lowest(v1, v2, v3, v4) >= (float)(1 - row_off) &&
                            (float)end + highest(v1, v2, v3, v4) < (float)(min(a.f2.rows, kDeformFar) - 3 - row_off) &&
                            sum == sum;
        if (inside) {
            for (; Y + 2 <= end; Y += 2) {
                run(std::integral_constant<int, 2>{}, Y, fy);
                fy = __fadd2_rn(fy, make_float2((float)(2), (float)(2)));
            }
            for (; Y < end; ++Y) {
                run(std::integral_constant<int, 1>{}, Y, fy);
                fy = __fadd2_rn(fy, one);
            }
        } else {
#pragma unroll 1
            for (; Y < end; ++Y) {
                float2 px, py;
                position(Y, fy, px, py);
                const float left = deform_any(a.f2, px.x, py.x, col_off, row_off);
                store(make_float2(left, deform_any(a.f2, px.y, py.y, col_off, row_off)));
                fy = __fadd2_rn(fy, one);
            }
        }
        if (Y >= Y1) break;
        ++i_y;
    }
}

// Spacings and origins that are multiples of 8: runs of 8 pixels of a row share a cell, whose 8
// values are loaded once for a thread's one run.  Bounded to 40 registers (6 CTAs per SM): the
// gathers' latency wants the warps (4 CTAs 76 us, 6 CTAs 70, unbounded 93 at 6600x4400).
template <class Off, bool POW2>
__global__ void __launch_bounds__(256, 6) deform_cell8_kernel(const __grid_constant__ DeformArgs a)
{
    chain_start();
    const int X0 = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
    const int Y = blockIdx.y;
    if (X0 >= a.Nx_aug) return;
    const float x_st = (float)(a.hfws_x - a.sp_x * 3), y_st = (float)(a.hfws_y - a.sp_y * 3);
    const int col_off = a.f2.mx - a.Nx_left, row_off = a.f2.my - a.Ny_left;
    // a power of two's reciprocal is exact, and so is the quotient by it
    const float ix = 1.f / (float)a.sp_x, iy = 1.f / (float)a.sp_y;
    auto cell = [](float v, float st, float sp, float inv) { return POW2 ? (v - st) * inv : (v - st) / sp; };
    const float y = cell((float)Y, y_st, (float)a.sp_y, iy), fy = floorf(y), a_y = y - fy, b_y = 1.f - a_y;
    const float fx = floorf(cell((float)X0, x_st, (float)a.sp_x, ix));
    const int i_x = (int)fx, i_y = (int)fy;
    auto field = [&](const float *f, int m, int n) { return ext_field(f, a.Nx_vec, a.Ny_vec, i_x + m, i_y + n); };
    const float u1 = field(a.fx, 0, 0), u2 = field(a.fx, 1, 0), u3 = field(a.fx, 0, 1), u4 = field(a.fx, 1, 1);
    const float v1 = field(a.fy, 0, 0), v2 = field(a.fy, 1, 0), v3 = field(a.fy, 0, 1), v4 = field(a.fy, 1, 1);
    const float2 one = make_float2(1.f, 1.f), minus = make_float2(-1.f, -1.f);
    const float kMagic = 12582912.f;  // 1.5 * 2^23
    const float2 magic = make_float2(kMagic, kMagic), unmagic = make_float2(-kMagic, -kMagic);
    float2 px[4], py[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float2 X = make_float2((float)(X0 + 2 * q), (float)(X0 + 2 * q + 1));
        const float xa = cell(X.x, x_st, (float)a.sp_x, ix), xb = cell(X.y, x_st, (float)a.sp_x, ix);
        const float2 a_x = make_float2(xa - fx, xb - fx);
        const float2 b_x = __ffma2_rn(a_x, minus, one);
        const float2 c1 = vmul(b_x, b_y), c2 = vmul(a_x, b_y), c3 = vmul(b_x, a_y), c4 = vmul(a_x, a_y);
        px[q] = vfma(c4, u4, vfma(c3, u3, vfma(c2, u2, vfma(c1, u1, X))));
        py[q] = vfma(c4, v4, vfma(c3, v3, vfma(c2, v2, vfma(c1, v1, make_float2((float)Y, (float)Y)))));
    }
    // the displacements lie between the corners' (a NaN corner makes the sum NaN)
    const float sum = ((u1 + u2) + (u3 + u4)) + ((v1 + v2) + (v3 + v4));
    const bool inside = (float)X0 + fminf(fminf(u1, u2), fminf(u3, u4)) >= (float)(1 - col_off) &&
                        (float)X0 + fmaxf(fmaxf(u1, u2), fmaxf(u3, u4)) <
                            (float)(min(a.f2.cols, kDeformFar) - 10 - col_off) &&
                        (float)Y + fminf(fminf(v1, v2), fminf(v3, v4)) >= (float)(1 - row_off) &&
                        (float)Y + fmaxf(fmaxf(v1, v2), fmaxf(v3, v4)) <
                            (float)(min(a.f2.rows, kDeformFar) - 3 - row_off) &&
                        sum == sum;
    float2 res[4];
    if (inside) {
        const int pitch = a.f2.pitch;
        const uint8_t *base = a.f2.base, *base1 = base + pitch;
        const Off k0 = (Off)(row_off - 0x4B400000) * (Off)pitch + (Off)(col_off - 0x4B400000);
        unsigned char p[4][8];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float2 tx = __fadd2_rd(px[q], magic), ty = __fadd2_rd(py[q], magic);
            const Off oa = (Off)__float_as_int(ty.x) * (Off)pitch + ((Off)__float_as_int(tx.x) + k0);
            const Off ob = (Off)__float_as_int(ty.y) * (Off)pitch + ((Off)__float_as_int(tx.y) + k0);
            const uint8_t *pa = base + oa, *pb = base + ob, *pa1 = base1 + oa, *pb1 = base1 + ob;
            p[q][0] = *(pa);
            p[q][1] = *(pb);
            p[q][2] = *(pa + 1);
            p[q][3] = *(pb + 1);
            p[q][4] = *(pa1);
            p[q][5] = *(pb1);
            p[q][6] = *(pa1 + 1);
            p[q][7] = *(pb1 + 1);
            // the fractions
            px[q] = __ffma2_rn(__fadd2_rn(tx, unmagic), minus, px[q]);
            py[q] = __ffma2_rn(__fadd2_rn(ty, unmagic), minus, py[q]);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            auto tap = [&](int t) { return make_float2((float)p[q][2 * t], (float)p[q][2 * t + 1]); };
            const float2 ax = px[q], ay = py[q], bx = __ffma2_rn(ax, minus, one), by = __ffma2_rn(ay, minus, one);
            const float2 s = __ffma2_rn(__fmul2_rn(bx, by), tap(0), __fmul2_rn(__fmul2_rn(ax, by), tap(1)));
            res[q] = __ffma2_rn(__fmul2_rn(ax, ay), tap(3), __ffma2_rn(__fmul2_rn(bx, ay), tap(2), s));
        }
    } else {
#pragma unroll
        for (int q = 0; q < 4; ++q)
            res[q] = make_float2(deform_any(a.f2, px[q].x, py[q].x, col_off, row_off),
                                 deform_any(a.f2, px[q].y, py[q].y, col_off, row_off));
    }
    float *dst = a.out + (size_t)Y * a.out_pitch + X0;
    if (X0 + 7 < a.Nx_aug) {
        reinterpret_cast<float4 *>(dst)[0] = make_float4(res[0].x, res[0].y, res[1].x, res[1].y);
        reinterpret_cast<float4 *>(dst)[1] = make_float4(res[2].x, res[2].y, res[3].x, res[3].y);
    } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (X0 + 2 * q < a.Nx_aug) dst[2 * q] = res[q].x;
            if (X0 + 2 * q + 1 < a.Nx_aug) dst[2 * q + 1] = res[q].y;
        }
    }
}

template <class Off>
void launch_deform_as(const DeformArgs &a, cudaStream_t s)
{
    // the cell edges x_st + m * sp are multiples of 8; the cell index is then exact for every pixel
    // of a run (its float quotient is exact for these small integers)
    const int x_st = a.hfws_x - a.sp_x * 3;
    if (a.sp_x % 8 == 0 && x_st % 8 == 0) {
        const dim3 grid(((a.Nx_aug + 7) / 8 + 255) / 256, a.Ny_aug);
        const bool pow2 = (a.sp_x & (a.sp_x - 1)) == 0 && (a.sp_y & (a.sp_y - 1)) == 0;
        if (pow2) launch_chained(deform_cell8_kernel<Off, true>, grid, dim3(256), 0, s, a);
        else launch_chained(deform_cell8_kernel<Off, false>, grid, dim3(256), 0, s, a);
        return;
    }
    // rows per thread: as many as leave four CTAs per SM (a CTA's start is 2 to 3 us of latency)
    const int gx = (a.Nx_aug + 2 * kDeformThreads - 1) / (2 * kDeformThreads);
    int rows = kDeformRows;
    while (rows > 2 && gx * ((a.Ny_aug + rows - 1) / rows) < kDeformMinCtas) rows /= 2;
    launch_chained(deform_kernel<Off>, dim3(gx, (a.Ny_aug + rows - 1) / rows), dim3(kDeformThreads), 0, s, a, rows);
}

cudaError_t launch_deform(const DeformArgs &a, cudaStream_t s)
{
    if ((uint64_t)a.f2.pitch * a.f2.rows <= UINT32_MAX) launch_deform_as<uint32_t>(a, s);
    else launch_deform_as<uint64_t>(a, s);
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------
// Autotuning input: a particle-like pattern (sparse bright pixels on a dark
// background) so that the timed correlation does its full candidate work.
// ------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t hash2(uint32_t x, uint32_t y)
{
    uint32_t h = x * 0x9E3779B1u ^ (y + 0x7F4A7C15u) * 0x85EBCA77u;
    h ^= h >> 15;
    h *= 0x2C1B3C6Du;
    h ^= h >> 12;
    return h;
}

__global__ void pattern_kernel(uint8_t *u8, float *f32, int pitch, int cols, int rows, uint32_t seed)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x >= cols || y >= rows) return;
    const uint32_t h = hash2((uint32_t)x + seed, (uint32_t)y);
    const float v = (h % 23u == 0u) ? (float)(120u + (h >> 24) % 136u) : (float)(8u + (h >> 28));
    if (u8) u8[(size_t)y * pitch + x] = (uint8_t)v;
    if (f32) f32[(size_t)y * pitch + x] = v;
}

cudaError_t launch_pattern(uint8_t *u8, float *f32, int pitch, int cols, int rows, uint32_t seed, cudaStream_t s)
{
    dim3 grid((cols + 255) / 256, rows);
    pattern_kernel<<<grid, 256, 0, s>>>(u8, f32, pitch, cols, rows, seed);
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------
// Upsampling_vecfield_kernel_2d (X/xcorr2d_multi_grid.cu:675-704) with the launch
// arguments of Upsampling_vector_field (:1580-1581).
// ------------------------------------------------------------------------------
__global__ void upsample_kernel(const UpsampleArgs a)
{
    chain_start();
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    if (tid >= a.Nx2 * a.Ny2) return;
    const float x_st_vec1 = (float)(a.sp_x1 / 2 - 3 * a.sp_x1), y_st_vec1 = (float)(a.sp_y1 / 2 - 3 * a.sp_y1);
    const float vs1x = (float)a.sp_x1, vs1y = (float)a.sp_y1;
    int idy = tid / a.Nx2;
    int idx = tid - idy * a.Nx2;
    idx = idx * a.sp_x2 + a.sp_x2 / 2;
    idy = idy * a.sp_y2 + a.sp_y2 / 2;
    float a_x = (float)(idx - x_st_vec1) / vs1x;
    float a_y = (float)(idy - y_st_vec1) / vs1y;
    const int i_x = (int)floorf(a_x);
    const int i_y = (int)floorf(a_y);
    a_x = a_x - (float)i_x;
    a_y = a_y - (float)i_y;
    const float ce1 = (1 - a_x) * (1 - a_y);
    const float ce2 = a_x * (1 - a_y);
    const float ce3 = (1 - a_x) * a_y;
    const float ce4 = a_x * a_y;
    a.fx2[tid] = ce1 * ext_field(a.fx1, a.Nx1, a.Ny1, i_x, i_y) + ce2 * ext_field(a.fx1, a.Nx1, a.Ny1, i_x + 1, i_y) +
                 ce3 * ext_field(a.fx1, a.Nx1, a.Ny1, i_x, i_y + 1) +
                 ce4 * ext_field(a.fx1, a.Nx1, a.Ny1, i_x + 1, i_y + 1);
    a.fy2[tid] = ce1 * ext_field(a.fy1, a.Nx1, a.Ny1, i_x, i_y) + ce2 * ext_field(a.fy1, a.Nx1, a.Ny1, i_x + 1, i_y) +
                 ce3 * ext_field(a.fy1, a.Nx1, a.Ny1, i_x, i_y + 1) +
                 ce4 * ext_field(a.fy1, a.Nx1, a.Ny1, i_x + 1, i_y + 1);
}

cudaError_t launch_upsample(const UpsampleArgs &a, cudaStream_t s)
{
    const int n = a.Nx2 * a.Ny2;
    launch_chained(upsample_kernel, dim3((n + 255) / 256), dim3(256), 0, s, a);
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------
// Validation.
// ------------------------------------------------------------------------------

// Calc_median (X/xcorr2d_multi_grid.cu:174-207) on a thread-private slice: (N+2)/2
// bubble passes move the largest values to the end, leaving the middle in place.
__device__ float median_bubble(float *d, int n, int stride)
{
    int cnt = n;
    for (int i = 0; i < (n + 2) / 2; i++) {
        cnt -= 1;
        float t1 = d[0];
        for (int j = 0; j < cnt; j++) {
            const float t2 = d[(1 + j) * stride];
            if (t1 > t2) {
                d[(1 + j) * stride] = t1;
                d[j * stride] = t2;
            } else {
                t1 = t2;
            }
        }
    }
    if (n % 2 == 0) return (d[(n / 2) * stride] + d[(n / 2 - 1) * stride]) / 2;
    return d[((n - 1) / 2) * stride];
}

// Ascending bitonic sort of a register array (N a power of two, all indices compile-time).
template <int N, int K, int J>
__device__ __forceinline__ void bitonic_step(float (&a)[N])
{
    static_for<0, N>([&](auto ic) {
        constexpr int i = decltype(ic)::value, l = i ^ J;
        if constexpr (l > i) {
            const float x = a[i], y = a[l];
            if constexpr ((i & K) == 0) {
                a[i] = fminf(x, y);
                a[l] = fmaxf(x, y);
            } else {
                a[i] = fmaxf(x, y);
                a[l] = fminf(x, y);
            }
        }
    });
    if constexpr (J > 1) bitonic_step<N, K, J / 2>(a);
}

template <int N, int K = 2>
__device__ __forceinline__ void bitonic_sort(float (&a)[N])
{
    bitonic_step<N, K, K / 2>(a);
    if constexpr (K < N) bitonic_sort<N, K * 2>(a);
}

// Median of the first n (<= N) entries of a sorted array, as Calc_median defines it
// (mean of the two middle values for even n, FP32).
// a[idx] for a runtime idx by a binary select tree over compile-time indices (keeps the
// array in registers; a compare-and-select loop is turned back into a local-memory load).
template <int N>
__device__ __forceinline__ float select_dyn(const float (&a)[N], int idx)
{
    if constexpr (N == 1) {
        return a[0];
    } else {
        float t[N / 2];
        const bool up = (idx & (N / 2)) != 0;
#pragma unroll
        for (int i = 0; i < N / 2; ++i) t[i] = up ? a[i + N / 2] : a[i];
        return select_dyn<N / 2>(t, idx);
    }
}

template <int N>
__device__ __forceinline__ float median_sorted(const float (&a)[N], int n)
{
    const float hi = select_dyn<N>(a, n / 2);  // n odd: (n-1)/2 == n/2
    if (n % 2 != 0) return hi;
    const float lo = select_dyn<N>(a, n / 2 - 1);
    return (hi + lo) / 2;
}

struct MedianPass {
    const float *cdx, *cdy;
    const uint8_t *cvalid;
    int Nps;
    const float *ix, *iy;  // input field; NULL -> candidate 0 (median_filter_data_prep)
    const uint8_t *iv;
    float *ox, *oy;
    uint8_t *ov;
    int Nx, Ny, wx, wy, minN;
    float thr;
    int median;        // 0: only copy candidate 0 (Npass_median == 0)
    int *list, *list_n;  // append invalid outputs here when non-NULL (fill work list)
    int *zero_n;         // set to 0 by a pass before the one that appends
};

// Neighbours are gathered in raster stencil order with the centre slot (wx*wy-1)/2 skipped.
__device__ __forceinline__ void median_neighbour(const MedianPass &a, int id, bool &ok, float &fxv, float &fyv)
{
    if (a.ix) {
        ok = a.iv[id] != 0;
        fxv = a.ix[id];
        fyv = a.iy[id];
    } else {
        ok = a.cvalid[(size_t)id * a.Nps] != 0;
        fxv = a.cdx[(size_t)id * a.Nps];
        fyv = a.cdy[(size_t)id * a.Nps];
    }
}

// median_filtering's decision: the first valid candidate whose normalised residuals are
// both below the insert threshold replaces the vector, else (0, 0, invalid).
__device__ __forceinline__ void median_decide(const MedianPass &a, int v, float mx, float my, float dmx, float dmy,
                                              float &rx, float &ry, uint8_t &rv)
{
    const float epsilon = 0.1f;  // X/xcorr2d_multi_grid.cuh:192
    for (int i = 0; i < a.Nps; ++i) {
        const size_t c = (size_t)v * a.Nps + i;
        if (!a.cvalid[c]) continue;
        const float cx = a.cdx[c], cy = a.cdy[c];
        const float devix = __fdiv_rn(fabsf(cx - mx), dmx + epsilon);
        const float deviy = __fdiv_rn(fabsf(cy - my), dmy + epsilon);
        if (devix < a.thr && deviy < a.thr) {
            rv = 1;
            rx = cx;
            ry = cy;
            return;
        }
    }
}

// The register form of one vector (stencils of at most 32 cells).
__device__ __forceinline__ void median_vector32(const MedianPass &a, int v, float &rx, float &ry, uint8_t &rv)
{
    const int Ntm = a.wx * a.wy, centre = (Ntm - 1) / 2;
    const int vy = v / a.Nx, vx = v - vy * a.Nx;
    const int hfwx = (a.wx - 1) / 2, hfwy = (a.wy - 1) / 2;
    const float inf = __int_as_float(0x7f800000);
    float xs[32], ys[32];
    int n = 0;
    int tx = 0, ty = 0;  // stencil column and row of slot t (no division per slot)
#pragma unroll
    for (int t = 0; t < 32; ++t) {
        const int x = vx - hfwx + tx, y = vy - hfwy + ty;
        const bool inb = (t < Ntm) & (t != centre) & (x >= 0) & (x <= a.Nx - 1) & (y >= 0) & (y <= a.Ny - 1);
        bool ok;
        float px, py;
        median_neighbour(a, inb ? y * a.Nx + x : v, ok, px, py);  // always a valid address
        ok = ok & inb;
        xs[t] = ok ? px : inf;
        ys[t] = ok ? py : inf;
        n += ok;
        const bool wrap = ++tx == a.wx;
        tx = wrap ? 0 : tx;
        ty += wrap;
    }
    if (n >= a.minN && n >= 1) {
        bitonic_sort<32>(xs);
        bitonic_sort<32>(ys);
        const float mx = median_sorted<32>(xs, n), my = median_sorted<32>(ys, n);
        // |x - median| over a sorted x falls, then rises (then +inf): a bitonic
        // sequence, which the final merge stage of the network sorts on its own
#pragma unroll
        for (int q = 0; q < 32; ++q) {
            xs[q] = (q < n) ? fabsf(xs[q] - mx) : inf;
            ys[q] = (q < n) ? fabsf(ys[q] - my) : inf;
        }
        bitonic_step<32, 32, 16>(xs);
        bitonic_step<32, 32, 16>(ys);
        const float dmx = median_sorted<32>(xs, n), dmy = median_sorted<32>(ys, n);
        median_decide(a, v, mx, my, dmx, dmy, rx, ry, rv);
    }
}

// One pass of organize_median_filter_data + median_validity + Calc_median x4 +
// Calc_devi x2 + median_filtering (X/xcorr2d_multi_grid.cu:209-296, 1464-1513), one
// thread per vector.  The medians are order statistics, so how they are found does not
// change them: REG (stencils of at most 32 cells) keeps one register slot per stencil
// cell (+inf when the neighbour is absent) and sorts with a bitonic network; larger
// stencils use the reference's partial bubble sort on a thread-private shared slice.
template <bool REG>
__global__ void __launch_bounds__(128) median_pass_kernel(const MedianPass a)
{
    chain_start();
    extern __shared__ float sl[];
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    const int Nt = a.Nx * a.Ny;
    if (a.zero_n && v == 0) *a.zero_n = 0;
    if (v >= Nt) return;
    const int Ntm = a.wx * a.wy;
    float rx = 0.f, ry = 0.f;
    uint8_t rv = 0;
    if (!a.median) {
        rx = a.cdx[(size_t)v * a.Nps];
        ry = a.cdy[(size_t)v * a.Nps];
        rv = a.cvalid[(size_t)v * a.Nps];
    } else {
        if constexpr (REG) {
            median_vector32(a, v, rx, ry, rv);
        } else {
            const int vy = v / a.Nx, vx = v - vy * a.Nx;
            const int hfwx = (a.wx - 1) / 2, hfwy = (a.wy - 1) / 2;
            const int centre = (Ntm - 1) / 2;
            // thread-private slices interleaved across threads: element k of thread t at k*blockDim + t
            const int stride = blockDim.x;
            float *xs = sl + threadIdx.x, *ys = sl + (size_t)Ntm * blockDim.x + threadIdx.x;
            int n = 0;
            for (int t = 0; t < Ntm; ++t) {
                if (t == centre) continue;
                const int ty = t / a.wx, tx = t - ty * a.wx;
                const int x = vx - hfwx + tx, y = vy - hfwy + ty;
                if (x >= 0 && x <= a.Nx - 1 && y >= 0 && y <= a.Ny - 1) {
                    bool ok;
                    float fxv, fyv;
                    median_neighbour(a, y * a.Nx + x, ok, fxv, fyv);
                    if (ok) {
                        xs[n * stride] = fxv;
                        ys[n * stride] = fyv;
                        n++;
                    }
                }
            }
            if (n >= a.minN && n >= 1) {
                const float mx = median_bubble(xs, n, stride), my = median_bubble(ys, n, stride);
                for (int q = 0; q < n; ++q) {
                    xs[q * stride] = fabsf(xs[q * stride] - mx);
                    ys[q * stride] = fabsf(ys[q * stride] - my);
                }
                const float dmx = median_bubble(xs, n, stride), dmy = median_bubble(ys, n, stride);
                median_decide(a, v, mx, my, dmx, dmy, rx, ry, rv);
            }
        }
    }
    a.ox[v] = rx;
    a.oy[v] = ry;
    a.ov[v] = rv;
    if (a.list && !rv) a.list[atomicAdd(a.list_n, 1)] = v;
}

// Batcher's merge exchange (Knuth, The Art of Computer Programming 3, algorithm 5.2.2 M):
// ascending sort of N registers, all indices compile-time.
template <int N, int P, int Q, int R, int D>
__device__ __forceinline__ void merge_exchange(float (&a)[N])
{
    static_for<0, N - D>([&](auto ic) {
        constexpr int i = decltype(ic)::value;
        if constexpr ((i & P) == R) {
            const float x = a[i], y = a[i + D];
            a[i] = fminf(x, y);
            a[i + D] = fmaxf(x, y);
        }
    });
    if constexpr (Q != P) merge_exchange<N, P, Q / 2, P, Q - P>(a);
}
template <int N, int P>
__device__ __forceinline__ void merge_exchange_sort(float (&a)[N])
{
    constexpr int T = N <= 32 ? 16 : 0;  // 2^(t - 1), t = ceil(log2 N)
    static_assert(N > 16 && N <= 32, "one network size class");
    merge_exchange<N, P, T, 0, P>(a);
    if constexpr (P > 1) merge_exchange_sort<N, P / 2>(a);
}

// Median and MAD of one component of the 5x5 neighbourhood of (vx, vy) by a whole warp, slot q of
// median_pass_kernel's network in lane q.  For NaN (candidates set by the caller) and medians that
// are no number: what fminf and fmaxf make of those depends on the exchanges, so these are the
// network's own.  About 100 instructions a neighbourhood; every lane gets the result.
__device__ __forceinline__ float2 median5_warp(const float *src, const uint8_t *flag, int step, int Nx, int Ny, int vx,
                                               int vy, int lane)
{
    const unsigned all = 0xffffffffu;
    const float inf = __int_as_float(0x7f800000);
    const int x = vx + lane % 5 - 2, y = vy + lane / 5 - 2;
    bool ok = lane < 25 && lane != 12 && x >= 0 && x < Nx && y >= 0 && y < Ny;
    const size_t id = (size_t)(ok ? y * Nx + x : 0) * step;
    ok = ok && flag[id];
    float w = ok ? src[id] : inf;
    const int n = __popc(__ballot_sync(all, ok));
    auto merge = [&](int k) {  // the exchanges of size k
#pragma unroll
        for (int j = k / 2; j > 0; j /= 2) {
            const float o = __shfl_xor_sync(all, w, j);
            w = ((lane & k) != 0) != ((lane & j) != 0) ? fmaxf(w, o) : fminf(w, o);
        }
    };
    auto median = [&]() {
        const float hi = __shfl_sync(all, w, n / 2), lo = __shfl_sync(all, w, (n / 2 - 1) & 31);
        return n % 2 ? hi : (hi + lo) / 2;
    };
#pragma unroll
    for (int k = 2; k <= 32; k *= 2) merge(k);
    const float med = median();
    w = lane < n ? fabsf(w - med) : inf;
    merge(32);
    return make_float2(med, median());
}

// The components of a warp's neighbourhoods that need median5_warp, one after another: those with a
// NaN, and those whose median is no number.  odd: this lane's neighbourhood holds an infinity or NaN.
__device__ __noinline__ float2 median5_special(const float *px, const float *py, const uint8_t *flag, int step, int Nx,
                                               int Ny, int v, bool odd, float med, float mad)
{
    const int lane = threadIdx.x & 31, vy = v / Nx, vx = v - vy * Nx;
    bool special = odd && !(fabsf(med) < __int_as_float(0x7f800000));
    if (odd && !special) {
        const float *src = lane & 1 ? py : px;
        for (int q = 0; q < 25 && !special; ++q) {
            const int x = vx + q % 5 - 2, y = vy + q / 5 - 2;
            if (q == 12 || x < 0 || x >= Nx || y < 0 || y >= Ny) continue;
            const size_t id = (size_t)(y * Nx + x) * step;
            special = flag[id] && src[id] != src[id];
        }
    }
    for (unsigned todo = __ballot_sync(0xffffffffu, special); todo; todo &= todo - 1) {
        const int q = __ffs(todo) - 1;  // component q & 1, as this lane's by its own parity
        const int qx = __shfl_sync(0xffffffffu, vx, q), qy = __shfl_sync(0xffffffffu, vy, q);
        const float2 m = median5_warp(q & 1 ? py : px, flag, step, Nx, Ny, qx, qy, lane);
        if (lane == q) {
            med = m.x;
            mad = m.y;
        }
    }
    return make_float2(med, mad);
}

// The 5x5 stencil (the usual one): two threads per vector, one for each component, which meet by
// shuffle for the decision.  A component's 24 neighbours are sorted by merge exchange (123
// exchanges; the 32-slot bitonic network of median_pass_kernel has 240).  With all 24 present,
// which all but the border vectors have, the median and the MAD need no further sort: the
// deviations of the lower and the upper half are two sorted lists, whose 12 smallest are
// min(lower[i], upper[11 - i]).  What bounds it: the latency of the straight-line code on small
// grids, issue slots on large ones.  Validation of a grid (two median passes, fill, smoothing), one
// thread per vector with the general network -> this: 21 x 16 vectors 34 -> 23 us, 411 x 274
// 64 -> 43 us, 384 x 509 98 -> 63 us.  Neighbourhoods with infinities or
// NaN go through median5_special, out of line so that the others pay one vote for it: 511 x 269
// vectors take 51 us without any, 67 to 86 with 1 to 20 % infinities, 87 and 113 with 1 and 5 % NaN
// (one thread per vector and the general network 84 to 104; a thread's own loops over local memory
// 166 to 212).  Other stencils keep median_pass_kernel: the exchanges and the two halves of the MAD
// are laid out for exactly 24 neighbours.
__global__ void __launch_bounds__(128) median5_pass_kernel(const MedianPass a)
{
    chain_start();
    const int t = blockIdx.x * 128 + threadIdx.x, comp = t & 1, Nt = a.Nx * a.Ny;
    const bool live = (t >> 1) < Nt;
    const int v = live ? t >> 1 : Nt - 1;
    if (a.zero_n && t == 0) *a.zero_n = 0;
    const int vy = v / a.Nx, vx = v - vy * a.Nx;
    const float *src = a.ix ? (comp ? a.iy : a.ix) : (comp ? a.cdy : a.cdx);
    const uint8_t *flag = a.ix ? a.iv : a.cvalid;
    const int step = a.ix ? 1 : a.Nps;
    const float inf = __int_as_float(0x7f800000);
    float s[24];
    int n = 0;
    bool odd = false;  // an infinity or a NaN
#pragma unroll
    for (int q = 0; q < 25; ++q) {
        if (q == 12) continue;  // the centre
        const int x = vx + q % 5 - 2, y = vy + q / 5 - 2;
        const bool inb = (unsigned)x < (unsigned)a.Nx && (unsigned)y < (unsigned)a.Ny;
        const size_t id = (size_t)(inb ? y * a.Nx + x : v) * step;
        const bool ok = inb && flag[id] != 0;
        const float f = src[id];
        s[q < 12 ? q : q - 1] = ok ? f : inf;
        n += ok;
        odd |= ok && !(fabsf(f) < inf);
    }
    merge_exchange_sort<24, 16>(s);
    float med, mad;
    if (n == 24) {
        med = (s[12] + s[11]) / 2;
        float lo = 0.f, hi = inf;
#pragma unroll
        for (int i = 0; i < 12; ++i) {
            const float l = fabsf(s[11 - i] - med), u = fabsf(s[23 - i] - med);  // lower[i], upper[11 - i]
            lo = fmaxf(lo, fminf(l, u));
            hi = fminf(hi, fmaxf(l, u));
        }
        mad = (hi + lo) / 2;
    } else {
        float w[32];
#pragma unroll
        for (int q = 0; q < 32; ++q) w[q] = q < 24 ? s[q < 24 ? q : 0] : inf;
        med = median_sorted<32>(w, n);
        // |x - median| over a sorted x falls, then rises (then +inf): the network's final merge
        // stage sorts it
#pragma unroll
        for (int q = 0; q < 32; ++q) w[q] = q < n ? fabsf(w[q] - med) : inf;
        bitonic_step<32, 32, 16>(w);
        mad = median_sorted<32>(w, n);
    }
    if (__any_sync(0xffffffffu, odd)) {
        const float2 m = median5_special(a.ix ? a.ix : a.cdx, a.ix ? a.iy : a.cdy, flag, step, a.Nx, a.Ny, v, odd, med, mad);
        med = m.x;
        mad = m.y;
    }
    // median_filtering's decision (median_decide): the first valid candidate with both residuals
    // below the threshold
    const float epsilon = 0.1f;
    bool found = !(n >= a.minN && n >= 1), ok = false;
    float r = 0.f;
    for (int i = 0; i < a.Nps; ++i) {
        const size_t c = (size_t)v * a.Nps + i;
        float cand = 0.f;
        bool pass = false;
        if (!found && a.cvalid[c]) {
            cand = comp ? a.cdy[c] : a.cdx[c];
            pass = __fdiv_rn(fabsf(cand - med), mad + epsilon) < a.thr;
        }
        const bool both = __shfl_xor_sync(0xffffffffu, (int)pass, 1) && pass;
        if (both) {
            r = cand;
            ok = found = true;
        }
        if (__all_sync(0xffffffffu, found)) break;
    }
    if (!live) return;
    (comp ? a.oy : a.ox)[v] = r;
    if (comp == 0) {
        a.ov[v] = ok;
        if (a.list && !ok) a.list[atomicAdd(a.list_n, 1)] = v;
    }
}

// fill_blank_vecfield + fill_blank_vecfield_update repeated until nothing changes
// (X/xcorr2d_multi_grid.cu:352-397, host loop :1514-1528), on the device without host
// polling: one CTA iterates over the list of invalid vectors.  valid codes: 0
// invalid, 1 valid, 2 filled in this iteration (not yet a source, as in the
// reference's two-kernel update).  The iteration count is capped at Nx+Ny+2 (the
// fill front advances at least one cell per iteration while anything changes); the
// cap sets a status bit instead of spinning.  cap_override > 0 lowers the cap (fault
// injection: a wide hole then hits it).
__global__ void __launch_bounds__(1024) fill_kernel(float *fx, float *fy, uint8_t *fv, int Nx, int Ny,
                                                    const int *list, const int *list_n, int *status,
                                                    int cap_override)
{
    chain_start();
    __shared__ int s_cnt[2];
    const int n = *list_n;
    const int cap = cap_override > 0 ? cap_override : Nx + Ny + 2;
    if (threadIdx.x < 2) s_cnt[threadIdx.x] = 0;
    __syncthreads();
    for (int it = 0; it < cap; ++it) {
        int local = 0;
        for (int q = threadIdx.x; q < n; q += blockDim.x) {
            const int v = list[q];
            if (fv[v] != 0) continue;
            const int vy = v / Nx, vx = v - vy * Nx;
            int cnt = 0;
            float sumx = 0.f, sumy = 0.f;
            for (int j = max(0, vy - 1); j <= min(Ny - 1, vy + 1); j++)
                for (int k = max(0, vx - 1); k <= min(Nx - 1, vx + 1); k++) {
                    const int id = j * Nx + k;
                    if (fv[id] == 1) {
                        cnt += 1;
                        sumx += fx[id];
                        sumy += fy[id];
                    }
                }
            if (cnt > 0) {
                local++;
                fx[v] = __fdiv_rn(sumx, (float)cnt);
                fy[v] = __fdiv_rn(sumy, (float)cnt);
                fv[v] = 2;
            }
        }
        if (local) atomicAdd(&s_cnt[it & 1], local);
        __syncthreads();
        for (int q = threadIdx.x; q < n; q += blockDim.x) {
            const int v = list[q];
            if (fv[v] == 2) fv[v] = 1;
        }
        const int total = s_cnt[it & 1];
        if (threadIdx.x == 0) s_cnt[(it + 1) & 1] = 0;
        __syncthreads();
        if (total == 0) return;
    }
    if (threadIdx.x == 0) atomicOr(status, kStatusFillCap);
}

// organize_smooth_filter_data + smoothing_tophat (X/xcorr2d_multi_grid.cu:399-443):
// mean over the in-bounds wx x wy stencil, centre included, summed in raster order
// (the reference sums in atomic-arrival order).  The validity is carried along unchanged.
__global__ void smooth_kernel(const float *ix, const float *iy, const uint8_t *iv, float *ox, float *oy, uint8_t *ov,
                              int Nx, int Ny, int wx, int wy)
{
    chain_start();
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= Nx * Ny) return;
    const int vy = v / Nx, vx = v - vy * Nx;
    const int hfwx = (wx - 1) / 2, hfwy = (wy - 1) / 2;
    float sx = 0.f, sy = 0.f;
    int n = 0;
    for (int ty = 0; ty < wy; ++ty)
        for (int tx = 0; tx < wx; ++tx) {
            const int x = vx - hfwx + tx, y = vy - hfwy + ty;
            if (x >= 0 && x <= Nx - 1 && y >= 0 && y <= Ny - 1) {
                sx += ix[y * Nx + x];
                sy += iy[y * Nx + x];
                n++;
            }
        }
    ox[v] = __fdiv_rn(sx, (float)n);
    oy[v] = __fdiv_rn(sy, (float)n);
    if (ov != iv) ov[v] = iv[v];
}

// MedianFilter_Smoothing_p1/p2: median passes (ping-pong), fill in place, smoothing
// passes (ping-pong); the buffer order is chosen so the result lands in (fx, fy, fv).
cudaError_t launch_validate(const ValidateArgs &a, cudaStream_t s)
{
    const int Nt = a.Nx_vec * a.Ny_vec;
    const int steps_med = a.Npass_median > 0 ? a.Npass_median : 1;
    const int n_steps = steps_med + a.Npass_smooth;
    auto dst_is_canon = [&](int step) { return ((n_steps - step) % 2) == 0; };  // step is 1-based
    const float *cx = nullptr, *cy = nullptr;
    const uint8_t *cv = nullptr;
    cudaError_t e = cudaSuccess;
    int *list = a.iffill ? a.list : nullptr;
    // the work list's length starts at 0: an earlier median pass clears it, or a memset
    if (list && steps_med == 1) {
        e = cudaMemsetAsync(a.list_n, 0, sizeof(int), s);
        if (e != cudaSuccess) return e;
    }
    const int tb = 128;
    for (int st = 1; st <= steps_med; ++st) {
        MedianPass m;
        m.cdx = a.cdx;
        m.cdy = a.cdy;
        m.cvalid = a.cvalid;
        m.Nps = a.Nps;
        m.ix = cx;
        m.iy = cy;
        m.iv = cv;
        const bool canon = dst_is_canon(st);
        m.ox = canon ? a.fx : a.tx;
        m.oy = canon ? a.fy : a.ty;
        m.ov = canon ? a.fv : a.tv;
        m.Nx = a.Nx_vec;
        m.Ny = a.Ny_vec;
        m.wx = a.wx_med;
        m.wy = a.wy_med;
        m.minN = a.minNneigh;
        m.thr = a.insert_threshold;
        m.median = a.Npass_median > 0;
        m.list = (st == steps_med) ? list : nullptr;
        m.list_n = a.list_n;
        m.zero_n = (list && st == 1 && steps_med > 1) ? a.list_n : nullptr;
        if (m.median && a.wx_med == 5 && a.wy_med == 5) {
            launch_chained(median5_pass_kernel, dim3((2 * Nt + 127) / 128), dim3(128), 0, s, m);
        } else if (a.wx_med * a.wy_med <= 32) {
            launch_chained(median_pass_kernel<true>, dim3((Nt + tb - 1) / tb), dim3(tb), 0, s, m);
        } else {
            const size_t smem = m.median ? (size_t)2 * a.wx_med * a.wy_med * tb * sizeof(float) : 0;
            if (smem > 48 * 1024) {
                e = cudaFuncSetAttribute(median_pass_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
                if (e != cudaSuccess) return e;
            }
            launch_chained(median_pass_kernel<false>, dim3((Nt + tb - 1) / tb), dim3(tb), smem, s, m);
        }
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        cx = m.ox;
        cy = m.oy;
        cv = m.ov;
    }
    if (a.iffill) {
        launch_chained(fill_kernel, dim3(1), dim3(1024), 0, s, const_cast<float *>(cx), const_cast<float *>(cy),
                       const_cast<uint8_t *>(cv),
                       a.Nx_vec, a.Ny_vec, a.list, a.list_n, a.status, a.fill_cap);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    for (int k = 0; k < a.Npass_smooth; ++k) {
        const int st = steps_med + 1 + k;
        const bool canon = dst_is_canon(st);
        float *ox = canon ? a.fx : a.tx, *oy = canon ? a.fy : a.ty;
        uint8_t *ov = canon ? a.fv : a.tv;
        launch_chained(smooth_kernel, dim3((Nt + 255) / 256), dim3(256), 0, s, cx, cy, cv, ox, oy, ov, a.Nx_vec,
                       a.Ny_vec, a.wx_sm, a.wy_sm);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        cx = ox;
        cy = oy;
        cv = ov;
    }
    return cudaSuccess;
}

}  // namespace piv
