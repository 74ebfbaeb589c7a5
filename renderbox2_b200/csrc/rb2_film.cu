// Film: filtered, deterministic image reconstruction (rb2_film_develop, the
// integrators' filtered accumulation) and the PFM image writer.
#include "rb2.h"
#include "rb2_devmem.h"
#include "rb2_film.cuh"
#include "rb2_internal.h"
#include "rb2_render.h"
#include "rb2_render_internal.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>

namespace rb2dev {

// The integrators' default (RB2_FILTER_NONE): mean of the pixel's own samples.
__global__ void k_film_mean(const float4* L, uint32_t npix, uint32_t spp, float* rgb)
{
    const float inv = 1.0f / (float)spp;
    for (uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x; pix < npix; pix += gridDim.x * blockDim.x) {
        float ax = 0.0f, ay = 0.0f, az = 0.0f;
        for (uint32_t j = 0; j < spp; j++) {
            const float4 l = L[(size_t)j * npix + pix];
            ax = __fadd_rn(ax, l.x);
            ay = __fadd_rn(ay, l.y);
            az = __fadd_rn(az, l.z);
        }
        rgb[3 * (size_t)pix + 0] = __fmul_rn(ax, inv);
        rgb[3 * (size_t)pix + 1] = __fmul_rn(ay, inv);
        rgb[3 * (size_t)pix + 2] = __fmul_rn(az, inv);
    }
}

}  // namespace rb2dev

using namespace rb2;

namespace {

int cuda_fail(cudaError_t e, const char* what) { return fail(rb2::cuda_status(e), std::string(what) + ": " + cudaGetErrorString(e)); }

}  // namespace

namespace rb2 {

int film_args(const rb2_filter& f, uint32_t width, uint32_t height, rb2dev::FilmArgs& out)
{
    int rc = filter_axes(f, out.gx, out.gy);
    if (rc) return rc;
    out.xw = f.xwidth;
    out.yw = f.ywidth;
    out.inv_xw = 1.0f / f.xwidth;
    out.inv_yw = 1.0f / f.ywidth;
    // A sample of pixel q lies within 0.5 + width of q's centre row/column,
    // plus what rounding of s - 0.5 -/+ width adds at the image's far end
    // (a few units in the last place of the largest coordinate).
    const float slack = ((float)std::max(width, height) + std::max(f.xwidth, f.ywidth)) * 0x1p-21f;
    out.rx = (int)std::floor(f.xwidth + 0.5f + slack);
    out.ry = (int)std::floor(f.ywidth + 0.5f + slack);
    out.width = width;
    out.height = height;
    return RB2_OK;
}

namespace {

// Largest staged row of k_film_strip: one block per SM.
constexpr size_t kStripMaxSmem = 226 * 1024;

template <int RY>
cudaError_t launch_strip(const rb2dev::FilmArgs& fa, const float2* xy, const float4* L, uint32_t per_pixel, int sms,
                         float4* accum, float* rgb, cudaStream_t s)
{
    const size_t smem = rb2dev::film_strip_smem(fa.rx, fa.ry, per_pixel);
    cudaError_t e;
    // The limit belongs to the kernel on this device, not to this launch: always
    // the same value, since another thread may be between its own two calls.
    if (smem > 40 * 1024 && (e = cudaFuncSetAttribute(rb2dev::k_film_strip<RY>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                      (int)kStripMaxSmem)) != cudaSuccess)
        return e;
    int per_sm = 0;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, rb2dev::k_film_strip<RY>, rb2dev::kFilmStripCols,
                                                           smem)) != cudaSuccess)
        return e;
    // Rows per strip: a strip of n rows reads n + 2 RY.  As many as leave a warp
    // for every resident slot, and at least 2 RY where the film has 8 warps per
    // SM of them; smaller films are bound by the longest warp and take shorter
    // strips (half-width 3, 64 x 64 x 4: 88 us with strips of 6 rows, 53 us with
    // 1; 640 x 360 x 4: 96 us with 6, 113 us with 2).
    const uint32_t gx = (fa.width + rb2dev::kFilmStripCols - 1) / rb2dev::kFilmStripCols;
    const uint64_t lines = (uint64_t)fa.height * gx, slots = (uint64_t)sms * (uint64_t)std::max(1, per_sm);
    const uint64_t least = std::min<uint64_t>(2 * RY, (lines + 8 * sms - 1) / (8 * sms));
    const uint32_t rows = (uint32_t)std::min<uint64_t>(64, std::max<uint64_t>(least, (lines + slots - 1) / slots));
    const dim3 grid(gx, (fa.height + rows - 1) / rows);
    rb2dev::k_film_strip<RY><<<grid, rb2dev::kFilmStripCols, smem, s>>>(fa, xy, L, per_pixel, rows, accum, rgb);
    return cudaGetLastError();
}

// Whether k_film_strip takes a film.  It holds 2 ry + 1 rows of sums in
// registers and a source row's samples in shared memory, so half-heights must
// reach 1 to 3 pixels and a row must fit.  Its row and column numbers are exact
// as floats below 2^22, and its grid has at most 65,535 strips in y.
//
// Of those films it takes the ones it develops faster.  It finds a sample's
// weights once where k_film_gather finds them for each of the (2 rx + 1) x
// (2 ry + 1) candidates, but it adds to 2 ry + 1 rows per column whatever the
// window covers of them, runs one warp per staged row, and pays a row's latency
// per sample row.  So (microseconds, gather : strip, half-widths x/y, width x
// height x samples):
//   one sample: wide windows on large films only (2/2 320x180 18 : 23, 1280x720
//     82 : 67; 3/3 640x360 43 : 52);
//   films whose strips run in few waves: several samples (64x64: 0.5/0.5 x 2
//     12 : 12, x 16 42 : 27; 0.5/3 320x180 x 2 22 : 35), or a wide window;
//   larger films: by the window's share of the rows, and the more the fewer
//     warps fit (0.5/0.5, share 0.33: 1280x720 x 16 190 : 215; 0.6/0.6, 0.48:
//     336 : 217; 2/2, 3.2: 1280x720 x 64, 2 warps 8.99 : 5.87 ms; 640x360 x 128,
//     1 warp 4.2 : 4.9 ms; 16/2, 25.6: 1280x720 x 64, 1 warp 59 : 39 ms).
// Over 1218 films (20 windows, 64x64 to 1920x1080, 1 to 128 samples) the choice
// costs 1.6 % against the better of the two.
bool strip_wins(const rb2dev::FilmArgs& fa, uint32_t per_pixel, int sms)
{
    const size_t smem = rb2dev::film_strip_smem(fa.rx, fa.ry, per_pixel);
    if (fa.ry < 1 || fa.ry > 3 || fa.width > (1u << 22) || fa.height > (1u << 16) || smem > kStripMaxSmem) return false;
    const uint64_t npix = (uint64_t)fa.width * fa.height, taps = (uint64_t)(2 * fa.rx + 1) * (2 * fa.ry + 1);
    const float window = 4.0f * fa.xw * fa.yw, share = window / (float)(2 * fa.ry + 1);
    if (per_pixel == 1) return window >= 16.0f && npix * taps >= 20000000;
    const uint64_t lines = (uint64_t)fa.height * ((fa.width + rb2dev::kFilmStripCols - 1) / rb2dev::kFilmStripCols);
    const uint64_t warps = std::min<uint64_t>(32, 227 * 1024 / (smem + 1024));  // per SM
    if (lines <= 6 * sms * warps) return per_pixel >= 3 || share >= 2.0f;
    return share >= (warps >= 3 ? 0.45f : warps == 2 ? 0.7f : 3.3f);
}

}  // namespace

int film_gather(const rb2dev::FilmArgs& fa, const float2* xy, const float4* L, uint32_t per_pixel, int sms,
                float4* accum, float* rgb, cudaStream_t s)
{
    cudaError_t e;
    const bool strip = strip_wins(fa, per_pixel, sms);
    if (strip && fa.ry == 1) e = launch_strip<1>(fa, xy, L, per_pixel, sms, accum, rgb, s);
    else if (strip && fa.ry == 2) e = launch_strip<2>(fa, xy, L, per_pixel, sms, accum, rgb, s);
    else if (strip) e = launch_strip<3>(fa, xy, L, per_pixel, sms, accum, rgb, s);
    else {
        const uint64_t npix = (uint64_t)fa.width * fa.height;
        rb2dev::k_film_gather<<<(unsigned)((npix + 255) / 256), 256, 0, s>>>(fa, xy, L, per_pixel, accum, rgb);
        e = cudaGetLastError();
    }
    return e == cudaSuccess ? RB2_OK : cuda_fail(e, "film gather");
}

}  // namespace rb2

extern "C" {

int rb2_film_develop(const rb2_filter* f, uint32_t width, uint32_t height, uint32_t spp, const float* d_xy,
                     const float* d_L, float* d_rgb, void* stream)
{
    int rc = validate_filter(f);
    if (rc) return rc;
    const uint64_t npix = (uint64_t)width * height;
    if (npix == 0 || spp == 0) return RB2_OK;
    if (npix * spp > 0xFFFFFFFFull) return fail(RB2_EINVAL, "width x height x spp must be < 2^32");
    if (!d_L || !d_rgb || (f->kind != RB2_FILTER_NONE && !d_xy)) return fail(RB2_EINVAL, "null buffer");
    if (((uintptr_t)d_L & 15u) || ((uintptr_t)d_xy & 7u)) return fail(RB2_EINVAL, "L must be 16-byte and xy 8-byte aligned");
    const cudaStream_t s = (cudaStream_t)stream;
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (f->kind == RB2_FILTER_NONE) {
        const unsigned g = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((npix + 255) / 256, (uint64_t)sms * 8));
        rb2dev::k_film_mean<<<g, 256, 0, s>>>(reinterpret_cast<const float4*>(d_L), (uint32_t)npix, spp, d_rgb);
        const cudaError_t e = cudaGetLastError();
        return e == cudaSuccess ? RB2_OK : cuda_fail(e, "film launch");
    }
    rb2dev::FilmArgs fa{};
    if ((rc = film_args(*f, width, height, fa))) return rc;
    return film_gather(fa, reinterpret_cast<const float2*>(d_xy), reinterpret_cast<const float4*>(d_L), spp, sms,
                       nullptr, d_rgb, s);
}

int rb2_integrator_set_filter(rb2_integrator* it, const rb2_filter* f)
{
    if (!it) return fail(RB2_EINVAL, "null integrator");
    if (!f) {
        it->filter = rb2_filter{RB2_FILTER_NONE, 0.5f, 0.5f, 0.0f};
        return RB2_OK;
    }
    const int rc = validate_filter(f);
    if (rc) return rc;
    it->filter = *f;
    return RB2_OK;
}

int rb2_image_write_pfm(const char* path, const float* h_rgb, uint32_t width, uint32_t height)
{
    if (!path || (!h_rgb && width && height)) return fail(RB2_EINVAL, "null argument");
    FILE* fp = std::fopen(path, "wb");
    if (!fp) return fail(RB2_EIO, std::string("cannot open ") + path);
    // PFM: "PF", dimensions, negative scale = little-endian, rows bottom to top.
    const int ok_header = std::fprintf(fp, "PF\n%u %u\n-1.0\n", width, height) > 0;
    bool ok = ok_header;
    for (uint32_t row = 0; ok && row < height; row++) {
        const float* src = h_rgb + 3 * (size_t)(height - 1 - row) * width;
        ok = std::fwrite(src, sizeof(float), 3 * (size_t)width, fp) == 3 * (size_t)width;
    }
    ok = (std::fclose(fp) == 0) && ok;
    return ok ? RB2_OK : fail(RB2_EIO, std::string("write failed: ") + path);
}

}  // extern "C"
