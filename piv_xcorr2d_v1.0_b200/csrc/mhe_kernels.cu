// mhe_kernels.cu -- MHE contrast enhancement (X/MHE7_4_gpu.cu), integer and
// bit-exact with the reference.  Two kernels, one warp per ws x ws tile:
//   mhe_hist_kernel   MakeHist_kernel (:66) with per-warp shared-memory histograms
//                     instead of global atomics; written into a zero-ringed tile grid.
//   mhe_apply_kernel  CreateTransfer_kernel (:85) + prescan_kernel (:5) +
//                     Calc_Enhanced_value_kernel (:103) + Enhanced_kernel (:121):
//                     9-tile transfer histogram, inclusive prefix sum, threshold
//                     stretch to a 256-entry LUT, LUT applied to the tile's pixels.
// The neighbour count of Calc_cnt_neigh_kernel (:45) is computed inline.
#include <cmath>

#include "piv_common.cuh"

namespace piv {

bool mhe_geometry(int Nx, int Ny, int ws, float thresh, MheGeom &m)
{
    if (Nx < 1 || Ny < 1 || ws < 1) return false;
    m.Nx = Nx;
    m.Ny = Ny;
    m.ws = ws;
    // mhe_gpu::init (X/MHE7_4_gpu.cu:157-178)
    if (Nx % ws == 0 && Ny % ws == 0) {
        m.height = Ny;
        m.width = Nx;
        m.xs = 0;
        m.ys = 0;
    } else {
        m.width = ws * (Nx / ws);
        m.xs = (Nx - m.width) / 2;
        m.height = ws * (Ny / ws);
        m.ys = (Ny - m.height) / 2;
    }
    m.maxI = m.height / ws;
    m.maxJ = m.width / ws;
    m.Ntrash = (int)roundf((float)(ws * ws) * thresh);
    m.Nnontrash = ws * ws - m.Ntrash;
    return m.maxI >= 1 && m.maxJ >= 1 && m.Nnontrash > 0;
}

// One warp per ws x ws tile, 8 tiles per CTA, and no CTA-wide barrier: a tile's work is
// short, so a CTA per tile spent most of its life in launch and barrier latency.
// A tile's pixels are read as 4-byte words when the tile start, the width and the pitch
// allow it (the usual case), else byte by byte; each lane fetches a batch of kBatch
// elements before using any of them, so the loads overlap (16 instead of 8: more registers, no faster).
constexpr int kTilesPerCta = 8;
constexpr int kBatch = 8;

__device__ __forceinline__ bool mhe_words(const uint8_t *p, int pitch, int ws)
{
    return ((reinterpret_cast<uintptr_t>(p) & 3) == 0) && (pitch % 4 == 0) && (ws % 4 == 0);
}

// One frame, or both of a pair in one launch (blockIdx.y): on small frames, where a launch is a
// few CTAs, the second frame then costs nothing (enhancement of a pair by two such launches
// instead of four: 333x251 40 -> 19 us, 1024x1024 21 -> 15).
struct MheFrames {
    const uint8_t *in[2];
    uint8_t *out[2];
    int *levels[2];
    // the word form's mapping: a step of the warp covers row_step rows of wpr words (one row, or a
    // part of one, when a row has 32 words or more); lane / wpr = (lane * lane_magic) >> 16
    int wpr, row_step, lane_magic;
    uint32_t lut_magic[3];  // ceil(2^32 / divisor) of the LUT for 4, 6 and 9 tiles, 0: divide
};

// The rows of a tile in words, as one lane visits them: column c0 (then every 32nd), rows r0,
// r0 + row_step, ...; n of them (0: an idle lane).  The kernels are bound by instructions (817 and
// 1340 per 40x40 tile with a division per word and per LUT entry), so a lane only steps down its
// column, bytes become shared-memory addresses by one or two logic instructions, and the LUT
// multiplies.  Bounded to 64 registers: 4 CTAs per SM (5 and 6 spill; unbounded 43 -> 49 us).  One
// frame of 4096x2160: 27.6 -> 21.4 us, of 6600x4400: 52.5 -> 43.  Tiles whose rows are not
// 4-byte aligned (the odd widths) go byte by byte (ByteLane).
struct WordLane {
    int c0, r0, n;
    __device__ WordLane(const MheFrames &f, int ws, int lane)
    {
        r0 = (lane * f.lane_magic) >> 16;
        c0 = lane - r0 * f.wpr;
        n = r0 < f.row_step && c0 < f.wpr ? (ws - r0 + f.row_step - 1) / f.row_step : 0;
    }
};

// The pixels of a tile one byte at a time, as one lane visits them: every 32nd in row order.  A step
// is some whole rows and a part of one, which passes the row's end at most once, so nothing is
// divided after the first pixel.  A warp has one tile, so the latency of its chain of batches is
// what bounds tiles of 32 px and more, and a division per pixel (two in the second kernel) was twice
// as long a chain.  One frame of 4095x2159: 25 px tiles 44.3 -> 34.0 us, 40 px 40.2 -> 27.9, 128 px
// 113.3 -> 60.2, 300 px 592 -> 301.
template <class T>
struct ByteLane {
    T *p;
    int c, ws, rest;
    ptrdiff_t step_bytes, wrap;
    __device__ ByteLane(T *tile, int pitch, int w, int lane) : ws(w)
    {
        const int r = lane / w, rows = 32 / w;
        c = lane - r * w;
        p = tile + (ptrdiff_t)r * pitch + c;
        rest = 32 - rows * w;
        step_bytes = (ptrdiff_t)rows * pitch + rest;
        wrap = pitch - w;
    }
    __device__ void step()
    {
        p += step_bytes;
        c += rest;
        if (c >= ws) {
            c -= ws;
            p += wrap;
        }
    }
};

template <bool PAIR>
__global__ void __launch_bounds__(256, 4) mhe_hist_kernel(const MheGeom m, const MheFrames f, int in_pitch)
{
    chain_start();
    const uint8_t *in = PAIR && blockIdx.y ? f.in[1] : f.in[0];
    int *levels = PAIR && blockIdx.y ? f.levels[1] : f.levels[0];
    __shared__ __align__(1024) int h[kTilesPerCta + 1][256];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.x * kTilesPerCta + warp;
    int *hw = h[warp];
    reinterpret_cast<int4 *>(hw)[lane] = reinterpret_cast<int4 *>(hw)[lane + 32] = make_int4(0, 0, 0, 0);
    __syncwarp();
    if (tile >= m.maxI * m.maxJ) return;  // warp-uniform
    const int ty = tile / m.maxJ, tx = tile - ty * m.maxJ;
    const uint8_t *src = in + (size_t)(m.ys + ty * m.ws) * in_pitch + m.xs + tx * m.ws;
    if (mhe_words(src, in_pitch, m.ws)) {
        const uint32_t base = (uint32_t)__cvta_generic_to_shared(hw);  // 1024-byte aligned
        // Bin 4 * byte, or-ed into the histogram's base.  No branches: a word past the lane's last
        // counts the bytes (lane, lane, lane, lane) in a histogram that nobody reads.
        const uint32_t none = (uint32_t)__cvta_generic_to_shared(h[kTilesPerCta]);
        auto count = [&](uint32_t shifted, uint32_t to) {
            asm volatile("red.shared.add.u32 [%0], 1;" ::"r"((shifted & 0x3fcu) | to) : "memory");
        };
        const WordLane l(f, m.ws, lane);
        const size_t step = (size_t)f.row_step * in_pitch;
        for (int c = l.c0; c < f.wpr; c += 32) {
            const uint8_t *p = src + (size_t)l.r0 * in_pitch + 4 * c;
            for (int k0 = 0; k0 < l.n; k0 += kBatch) {
                uint32_t v[kBatch];
#pragma unroll
                for (int k = 0; k < kBatch; ++k) {
                    v[k] = 0x01010101u * lane;
                    if (k0 + k < l.n) v[k] = *reinterpret_cast<const uint32_t *>(p);
                    p += step;
                }
#pragma unroll
                for (int k = 0; k < kBatch; ++k) {
                    const uint32_t to = k0 + k < l.n ? base : none;
                    count(v[k] << 2, to);
                    count(v[k] >> 6, to);
                    count(v[k] >> 14, to);
                    count(v[k] >> 22, to);
                }
            }
        }
    } else {
        const int npx = m.ws * m.ws;
        ByteLane<const uint8_t> l(src, in_pitch, m.ws, lane);
        for (int base = lane; base < npx; base += 32 * kBatch) {
            int v[kBatch];
#pragma unroll
            for (int k = 0; k < kBatch; ++k) {
                v[k] = -1;
                if (base + 32 * k < npx) v[k] = *l.p;
                l.step();
            }
#pragma unroll
            for (int k = 0; k < kBatch; ++k)
                if (v[k] >= 0) atomicAdd(&hw[v[k]], 1);
        }
    }
    __syncwarp();
    int4 *dst = reinterpret_cast<int4 *>(levels + ((size_t)(ty + 1) * (m.maxJ + 2) + 1 + tx) * 256);
    dst[lane] = reinterpret_cast<int4 *>(hw)[lane];
    dst[lane + 32] = reinterpret_cast<int4 *>(hw)[lane + 32];
}

__device__ __forceinline__ void mhe_apply(const MheGeom &m, const MheFrames &f, const uint8_t *in, int in_pitch,
                                          const int *levels, uint8_t *out, int out_pitch, int ox, int oy)
{
    __shared__ __align__(256) uint8_t lut_all[kTilesPerCta][256];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.x * kTilesPerCta + warp;
    if (tile >= m.maxI * m.maxJ) return;  // warp-uniform; nothing below syncs the CTA
    uint8_t *lut = lut_all[warp];
    const int ty = tile / m.maxJ, tx = tile - ty * m.maxJ;
    const int W = m.maxJ + 2;
    const int c = (ty + 1) * W + 1 + tx;
    const uint8_t *src = in + (size_t)(m.ys + ty * m.ws) * in_pitch + m.xs + tx * m.ws;
    uint8_t *dst = out + (size_t)(oy + m.ys + ty * m.ws) * out_pitch + ox + m.xs + tx * m.ws;
    const bool words = mhe_words(src, in_pitch, m.ws) && mhe_words(dst, out_pitch, m.ws);
    const WordLane l(f, m.ws, lane);
    const size_t step = (size_t)f.row_step * in_pitch;
    const uint8_t *p = src + (size_t)l.r0 * in_pitch + 4 * l.c0;
    chain_start();
    // the first batch of the tile's pixels is fetched before the LUT is built (before the wait as well it
    // gained 0.2 of 17 us, but read pixels that only the kernel before had waited for)
    uint32_t v[kBatch];
    if (words) {
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            v[k] = 0;
            if (k < l.n) v[k] = *reinterpret_cast<const uint32_t *>(p);
            p += step;
        }
    }
    // CreateTransfer_kernel: 3x3 tile neighbourhood of the zero-ringed grid; this lane
    // owns bins [8 lane, 8 lane + 8)
    int tr[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
        for (int dx = -1; dx <= 1; ++dx) {
            const int4 *h = reinterpret_cast<const int4 *>(levels + (size_t)(c + dy * W + dx) * 256 + 8 * lane);
            const int4 u = *(h), w = *(h + 1);
            tr[0] += u.x;
            tr[1] += u.y;
            tr[2] += u.z;
            tr[3] += u.w;
            tr[4] += w.x;
            tr[5] += w.y;
            tr[6] += w.z;
            tr[7] += w.w;
        }
    // inclusive prefix sum over the 256 bins (prescan_kernel + its one-element shift):
    // within the lane, then an exclusive warp scan of the lane totals
#pragma unroll
    for (int i = 1; i < 8; ++i) tr[i] += tr[i - 1];
    int incl = tr[7];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int n = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += n;
    }
    const int excl = incl - tr[7];
    // Calc_cnt_neigh_kernel with (Nx, Ny) = (maxJ, maxI)
    int cnt;
    if (tx >= 1 && tx <= m.maxJ - 2 && ty >= 1 && ty <= m.maxI - 2)
        cnt = 9;
    else if ((tx == 0 && ty == 0) || (tx == 0 && ty == m.maxI - 1) || (tx == m.maxJ - 1 && ty == 0) ||
             (tx == m.maxJ - 1 && ty == m.maxI - 1))
        cnt = 4;
    else
        cnt = 6;
    // Calc_Enhanced_value_kernel.  cum <= cnt * Nnontrash = d, so n = 255 cum <= 255 d and the
    // product with ceil(2^32 / d) gives the exact quotient while 255 d^2 < 2^32
    const uint32_t magic = cnt == 9 ? f.lut_magic[2] : (cnt == 6 ? f.lut_magic[1] : f.lut_magic[0]);
    const int d = cnt * m.Nnontrash, trash = cnt * m.Ntrash;
    uint32_t lv[2] = {0u, 0u};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int b = 8 * lane + i;
        int cum = max(tr[i] + excl - trash, 0);
        cum = min(255, magic ? (int)__umulhi((uint32_t)(cum * 255), magic) : cum * 255 / d);
        if (b == 0) cum = 0;
        if (b == 255) cum = 255;
        lv[i >> 2] |= (uint32_t)cum << (8 * (i & 3));
    }
    reinterpret_cast<uint2 *>(lut)[lane] = make_uint2(lv[0], lv[1]);
    __syncwarp();
    // Enhanced_kernel on this tile
    if (words) {
        const uint32_t base = (uint32_t)__cvta_generic_to_shared(lut);  // 256-byte aligned
        // the LUT's entry of byte B of w: the byte takes the place of the base's lowest
        auto entry = [&](uint32_t w, auto bc) {
            uint32_t e;
            asm volatile("ld.shared.u8 %0, [%1];"
                         : "=r"(e)
                         : "r"(__byte_perm(w, base, 0x7650u | decltype(bc)::value))
                         : "memory");
            return e;
        };
        using std::integral_constant;
        const size_t out_step = (size_t)f.row_step * out_pitch;
        for (int c = l.c0; c < f.wpr; c += 32) {
            uint8_t *o = dst + (size_t)l.r0 * out_pitch + 4 * c;
            if (c != l.c0) p = src + (size_t)l.r0 * in_pitch + 4 * c;
            for (int k0 = 0; k0 < l.n; k0 += kBatch) {
                if (k0 > 0 || c != l.c0) {
#pragma unroll
                    for (int k = 0; k < kBatch; ++k) {
                        v[k] = 0;
                        if (k0 + k < l.n) v[k] = *reinterpret_cast<const uint32_t *>(p);
                        p += step;
                    }
                }
#pragma unroll
                for (int k = 0; k < kBatch; ++k) {
                    const uint32_t lo = __byte_perm(entry(v[k], integral_constant<int, 0>{}),
                                                    entry(v[k], integral_constant<int, 1>{}), 0x0040);
                    const uint32_t hi = __byte_perm(entry(v[k], integral_constant<int, 2>{}),
                                                    entry(v[k], integral_constant<int, 3>{}), 0x0040);
                    if (k0 + k < l.n) *reinterpret_cast<uint32_t *>(o) = __byte_perm(lo, hi, 0x5410);
                    o += out_step;
                }
            }
        }
    } else {
        const int npx = m.ws * m.ws;
        ByteLane<const uint8_t> from(src, in_pitch, m.ws, lane);
        ByteLane<uint8_t> to(dst, out_pitch, m.ws, lane);
        for (int base = lane; base < npx; base += 32 * kBatch) {
            int px[kBatch];
#pragma unroll
            for (int k = 0; k < kBatch; ++k) {
                px[k] = 0;
                if (base + 32 * k < npx) px[k] = *from.p;
                from.step();
            }
#pragma unroll
            for (int k = 0; k < kBatch; ++k) {
                if (base + 32 * k < npx) *to.p = lut[px[k]];
                to.step();
            }
        }
    }
}

__global__ void __launch_bounds__(256, 4) mhe_apply_kernel(const MheGeom m, const MheFrames f, int in_pitch,
                                                           int out_pitch, int ox, int oy)
{
    mhe_apply(m, f, f.in[0], in_pitch, f.levels[0], f.out[0], out_pitch, ox, oy);
}
__global__ void __launch_bounds__(256, 4) mhe_apply_pair_kernel(const MheGeom m, const MheFrames f, int in_pitch,
                                                                int out_pitch, int ox, int oy)
{
    const bool q = blockIdx.y != 0;
    mhe_apply(m, f, q ? f.in[1] : f.in[0], in_pitch, q ? f.levels[1] : f.levels[0], q ? f.out[1] : f.out[0], out_pitch,
              ox, oy);
}

template <bool PAIR>
static cudaError_t launch_frames(const MheGeom &m, MheFrames f, int in_pitch, int out_pitch, int ox, int oy,
                                 cudaStream_t s)
{
    f.wpr = m.ws / 4;
    f.row_step = f.wpr >= 1 && f.wpr <= 32 ? 32 / f.wpr : 1;
    f.lane_magic = f.wpr >= 1 && f.wpr <= 32 ? (65536 + f.wpr - 1) / f.wpr : 0;
    for (int q = 0; q < 3; ++q) {
        const uint64_t d = (uint64_t)(q == 2 ? 9 : 4 + 2 * q) * m.Nnontrash;
        f.lut_magic[q] = d > 1 && 255 * d * d < (1ull << 32) ? (uint32_t)(((1ull << 32) + d - 1) / d) : 0;
    }
    const dim3 ctas((m.maxI * m.maxJ + kTilesPerCta - 1) / kTilesPerCta, PAIR ? 2 : 1);
    launch_chained(mhe_hist_kernel<PAIR>, ctas, dim3(32 * kTilesPerCta), 0, s, m, f, in_pitch);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const auto apply = PAIR ? mhe_apply_pair_kernel : mhe_apply_kernel;
    launch_chained(apply, ctas, dim3(32 * kTilesPerCta), 0, s, m, f, in_pitch, out_pitch, ox, oy);
    return cudaGetLastError();
}

cudaError_t launch_mhe(const MheGeom &m, const uint8_t *in, int in_pitch, int *levels, uint8_t *out, int out_pitch,
                       int ox, int oy, cudaStream_t s)
{
    const MheFrames f{{in, in}, {out, out}, {levels, levels}, 0, 0, 0, {0, 0, 0}};
    return launch_frames<false>(m, f, in_pitch, out_pitch, ox, oy, s);
}

cudaError_t launch_mhe_pair(const MheGeom &m, const uint8_t *in1, const uint8_t *in2, int in_pitch, int *levels,
                            uint8_t *out1, uint8_t *out2, int out_pitch, int ox, int oy, cudaStream_t s)
{
    int *second = levels + (size_t)(m.maxI + 2) * (m.maxJ + 2) * 256;
    const MheFrames f{{in1, in2}, {out1, out2}, {levels, second}, 0, 0, 0, {0, 0, 0}};
    return launch_frames<true>(m, f, in_pitch, out_pitch, ox, oy, s);
}

}  // namespace piv
