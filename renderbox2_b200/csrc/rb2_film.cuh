// Film reconstruction on the device: every output pixel gathers the samples
// of its neighbourhood in a fixed order (rows, columns, then samples), so the
// image does not depend on scheduling.  The weights follow the reference's
// splat (renderers/samplerrenderer.cu:103-168): a sample with raster position
// s contributes to pixel x when ceil(s - 0.5 - width) <= x <= floor(s - 0.5 +
// width), with weight table[min(floor(|x - (s - 0.5)| / width * 16), 15)].
// Arithmetic is IEEE single precision with no contraction (the oracle's
// rb2o_film restates it operation by operation).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "rb2_shading.cuh"

namespace rb2dev {

struct FilmArgs {
    float gx[16], gy[16];       // the 16 x 16 table is gy[iy] * gx[ix], rounded once
    float xw, yw, inv_xw, inv_yw;
    int rx, ry;                 // neighbourhood half-size in pixels
    uint32_t width, height;
};

// A pixel's sums (rgb and weight), out of the kernel: accum == nullptr: write
// max(0, sum(wL) / sum(w)) to rgb; otherwise add the sums to accum.
__device__ __forceinline__ void film_store(uint32_t pix, float ax, float ay, float az, float aw, float4* accum,
                                           float* rgb)
{
    if (accum) {
        const float4 a = accum[pix];
        accum[pix] = make_float4(__fadd_rn(a.x, ax), __fadd_rn(a.y, ay), __fadd_rn(a.z, az), __fadd_rn(a.w, aw));
    } else {
        const float inv = aw != 0.0f ? __fdiv_rn(1.0f, aw) : 0.0f;
        rgb[3 * (size_t)pix + 0] = fmaxf(0.0f, __fmul_rn(ax, inv));
        rgb[3 * (size_t)pix + 1] = fmaxf(0.0f, __fmul_rn(ay, inv));
        rgb[3 * (size_t)pix + 2] = fmaxf(0.0f, __fmul_rn(az, inv));
    }
}

// One thread per output pixel, any filter width and sample count: the path of
// films that k_film_strip does not take (film_gather in rb2_film.cu).
// Samples are sample-major (sample j of pixel p at j * npix + p).
//
// Bound: the loads of the candidates' positions (L1 and L2).  As many blocks as
// the film has pixels for, so that the hardware evens out the last wave: 40
// registers leave 6 blocks per SM, and a grid of 8 per SM ran a second,
// third-full wave (1280 x 720 x 16, Gaussian of half-width 16: 43.8 -> 29.8 ms;
// of 8: 11.9 -> 8.2 ms).  The pixel loop takes one step; as a plain test of the
// index the kernel is 10 % slower (the compiler then pipelines the samples'
// loads less), a bound of 32 registers (8 blocks per SM) 20 %.
static __global__ void __launch_bounds__(256, 1)
    k_film_gather(const __grid_constant__ FilmArgs f, const float2* xy, const float4* L, uint32_t per_pixel,
                  float4* accum, float* rgb)
{
    __shared__ float tab[256];
    tab[threadIdx.x] = __fmul_rn(f.gx[threadIdx.x & 15], f.gy[threadIdx.x >> 4]);
    __syncthreads();
    const uint32_t W = f.width, H = f.height, npix = W * H;
    for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < npix; p += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t pix = (uint32_t)p;
        const int x = (int)(pix % W), y = (int)(pix / W);
        const float xf = (float)x, yf = (float)y;
        float ax = 0.0f, ay = 0.0f, az = 0.0f, aw = 0.0f;
        const int qy0 = max(0, y - f.ry), qy1 = min((int)H - 1, y + f.ry);
        const int qx0 = max(0, x - f.rx), qx1 = min((int)W - 1, x + f.rx);
        for (int qy = qy0; qy <= qy1; qy++) {
            for (int qx = qx0; qx <= qx1; qx++) {
                const uint32_t q = (uint32_t)qy * W + (uint32_t)qx;
                for (uint32_t j = 0; j < per_pixel; j++) {
                    const float2 s = xy[(size_t)j * npix + q];
                    const float dx = __fsub_rn(s.x, 0.5f), dy = __fsub_rn(s.y, 0.5f);
                    if (x < (int)ceilf(__fsub_rn(dx, f.xw)) || x > (int)floorf(__fadd_rn(dx, f.xw)) ||
                        y < (int)ceilf(__fsub_rn(dy, f.yw)) || y > (int)floorf(__fadd_rn(dy, f.yw)))
                        continue;
                    const float fx = fabsf(__fmul_rn(__fmul_rn(__fsub_rn(xf, dx), f.inv_xw), 16.0f));
                    const float fy = fabsf(__fmul_rn(__fmul_rn(__fsub_rn(yf, dy), f.inv_yw), 16.0f));
                    const int ix = min((int)floorf(fx), 15), iy = min((int)floorf(fy), 15);
                    const float w = tab[iy * 16 + ix];
                    const float4 l = L[(size_t)j * npix + q];
                    ax = __fadd_rn(ax, __fmul_rn(w, l.x));
                    ay = __fadd_rn(ay, __fmul_rn(w, l.y));
                    az = __fadd_rn(az, __fmul_rn(w, l.z));
                    aw = __fadd_rn(aw, w);
                }
            }
        }
        film_store(pix, ax, ay, az, aw, accum, rgb);
    }
}

// Two IEEE additions in one instruction.  (The products stay scalar: a paired
// mul.rn.f32x2 before a paired add was contracted to one rounding.)
__device__ __forceinline__ float2 add2(float2 a, float2 b)
{
    unsigned long long x = *reinterpret_cast<unsigned long long*>(&a), y = *reinterpret_cast<unsigned long long*>(&b);
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(x) : "l"(y));
    return *reinterpret_cast<float2*>(&x);
}
// Table index of a distance in [0, 16) table cells (or beyond: 15): floor by
// adding 2^23 toward minus infinity, so no conversion instruction.
__device__ __forceinline__ int film_cell(float d)
{
    return __float_as_int(__fadd_rd(fminf(fabsf(d), 15.0f), 8388608.0f)) & 15;
}

constexpr uint32_t kFilmStripCols = 32;  // output columns of a k_film_strip block (one warp)

// Shared bytes of a k_film_strip block.
__host__ __device__ constexpr size_t film_strip_smem(int rx, int ry, uint32_t per_pixel)
{
    return (size_t)(kFilmStripCols + 2 * rx) * per_pixel * (16 + 4 * (2 * ry + 1));
}

// One warp per strip of 32 columns x `rows` output rows.  It walks down the
// source rows; each row's samples (32 + 2 rx pixels) go to shared memory once,
// with the sample's weight for each of the 2 RY + 1 output rows it can reach
// (NaN: outside the window), and each lane then adds the 2 rx + 1 columns
// around its own to 2 RY + 1 output rows held in registers (a ring; the row
// that has seen its last source row leaves it).  Each output pixel still adds
// its samples by rows, then columns, then samples, with the operations of
// k_film_gather, so the sums are bit-identical to it.
//
// Bound: instruction issue at the 9 to 10 warps per SM that the staged rows
// leave room for (36 bytes per sample; 5-bit table cells instead of weights
// doubled the warps but lengthened the inner loop, 619 against 449 us).  One
// thread per pixel over all 49 candidate pixels loaded and tested each sample
// 49 times, with two float-to-int conversions each (XU pipe at 60 %).  Here a
// sample is read 5 times, its row weights are found once per strip, and
// candidates that only rounding could reach are left out.  Gaussian of
// half-width 2, 1280 x 720 x 16 samples: 1221 -> 449 us (365 MB of samples and
// image: 813 GB/s); box of 0.5: 392 -> 208 us; 120 x 90 x 4: 49 -> 33 us.
template <int RY>
__global__ void __launch_bounds__(kFilmStripCols)
    k_film_strip(const __grid_constant__ FilmArgs f, const float2* xy, const float4* L, uint32_t per_pixel,
                 uint32_t rows, float4* accum, float* rgb)
{
    constexpr int R = 2 * RY + 1;
    const float kOutside = __int_as_float(0x7fffffff);  // NaN: outside the window (weights are finite)
    extern __shared__ float4 s_film[];
    __shared__ float s_gx[16], s_gy[16];
    const int lane = (int)threadIdx.x, W = (int)f.width, H = (int)f.height;
    const uint32_t npix = f.width * f.height;
    const int ncols = (int)kFilmStripCols + 2 * f.rx, n = ncols * (int)per_pixel;
    float4* s_l = s_film;                                    // rgb, x position less 0.5
    float* s_w = reinterpret_cast<float*>(s_film + n);       // R weights per sample, [k][sample]
    if (lane < 16) {
        s_gx[lane] = f.gx[lane];
        s_gy[lane] = f.gy[lane];
    }
    const int x0 = (int)(blockIdx.x * kFilmStripCols), x = x0 + lane;
    const int y0 = (int)(blockIdx.y * rows), y1 = min(H, y0 + (int)rows);
    const float xf = (float)x;
    float2 rg[R], bw[R];
#pragma unroll
    for (int k = 0; k < R; k++) rg[k] = bw[k] = make_float2(0.0f, 0.0f);
    __syncwarp();

    // Source row i (qy = y0 - RY + i) reaches output rows y0 + i - 2 RY .. y0 + i;
    // output row y0 + o is ring entry o mod R.
    for (int i0 = 0; y0 - RY + i0 < y1 + RY; i0 += R) {
#pragma unroll
        for (int ph = 0; ph < R; ph++) {
            const int i = i0 + ph, qy = y0 - RY + i;
            if (qy >= 0 && qy < min(H, y1 + RY)) {
                __syncwarp();
                // Loads in groups, so that a group's latency is paid once.
                constexpr int G = 6;
                int col = lane, j = 0;
                while (col >= ncols) { col -= ncols; j++; }
                for (int k0 = lane; k0 < n; k0 += G * (int)kFilmStripCols) {
                    float4 l[G];
                    float2 p[G];
#pragma unroll
                    for (int g = 0; g < G; g++) {
                        const int qx = x0 - f.rx + col;
                        l[g] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        p[g] = make_float2(0.0f, 0.0f);
                        if (k0 + g * (int)kFilmStripCols < n && qx >= 0 && qx < W) {
                            const size_t at = (size_t)j * npix + (size_t)qy * W + qx;
                            l[g] = __ldg(L + at);
                            p[g] = __ldg(xy + at);
                        }
                        col += (int)kFilmStripCols;
                        while (col >= ncols) { col -= ncols; j++; }
                    }
#pragma unroll
                    for (int g = 0; g < G; g++) {
                        const int k = k0 + g * (int)kFilmStripCols;
                        if (k < n) {
                            s_l[k] = make_float4(l[g].x, l[g].y, l[g].z, __fsub_rn(p[g].x, 0.5f));
                            const float dy = __fsub_rn(p[g].y, 0.5f);
                            const float lo = __fsub_rn(dy, f.yw), hi = __fadd_rn(dy, f.yw);
#pragma unroll
                            for (int r = 0; r < R; r++) {
                                const float yf = (float)(qy - RY + r);
                                const float w =
                                    s_gy[film_cell(__fmul_rn(__fmul_rn(__fsub_rn(yf, dy), f.inv_yw), 16.0f))];
                                s_w[r * n + k] = yf >= lo && yf <= hi ? w : kOutside;
                            }
                        }
                    }
                }
                __syncwarp();
                for (int c = 0; c <= 2 * f.rx; c++) {
                    const int qx = x - f.rx + c;
                    if (qx < 0 || qx >= W) continue;
#pragma unroll 2
                    for (int k = lane + c; k < n; k += ncols) {
                        const float4 l = s_l[k];
                        const bool in = xf >= __fsub_rn(l.w, f.xw) && xf <= __fadd_rn(l.w, f.xw);
                        const float gx = s_gx[film_cell(__fmul_rn(__fmul_rn(__fsub_rn(xf, l.w), f.inv_xw), 16.0f))];
                        const float wx = in ? gx : kOutside;
#pragma unroll
                        for (int r = 0; r < R; r++) {
                            const int a = (ph + r + 1) % R;
                            const float w = __fmul_rn(wx, s_w[r * n + k]);
                            if (w == w) {
                                rg[a] = add2(rg[a], make_float2(__fmul_rn(w, l.x), __fmul_rn(w, l.y)));
                                bw[a] = add2(bw[a], make_float2(__fmul_rn(w, l.z), w));
                            }
                        }
                    }
                }
            }
            const int y = y0 + i - 2 * RY;  // complete
            const int a = (ph + 1) % R;
            if (y >= y0 && y < y1 && x < W)
                film_store((uint32_t)y * (uint32_t)W + (uint32_t)x, rg[a].x, rg[a].y, bw[a].x, bw[a].y, accum, rgb);
            rg[a] = bw[a] = make_float2(0.0f, 0.0f);
        }
    }
}

// Final image of an accumulated film.
static __global__ void k_film_resolve(const float4* accum, uint32_t npix, float* rgb)
{
    for (uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x; pix < npix; pix += gridDim.x * blockDim.x) {
        const float4 a = accum[pix];
        const float inv = a.w != 0.0f ? __fdiv_rn(1.0f, a.w) : 0.0f;
        rgb[3 * (size_t)pix + 0] = fmaxf(0.0f, __fmul_rn(a.x, inv));
        rgb[3 * (size_t)pix + 1] = fmaxf(0.0f, __fmul_rn(a.y, inv));
        rgb[3 * (size_t)pix + 2] = fmaxf(0.0f, __fmul_rn(a.z, inv));
    }
}

}  // namespace rb2dev
