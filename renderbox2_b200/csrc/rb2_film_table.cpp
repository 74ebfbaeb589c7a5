// Filter table of the film (core/film.cpp:36-60 with core/filter.h:46-132),
// computed on the host in IEEE single precision without contraction.  The
// table is indexed [y][x] with fx taken from x (the reference took it from y,
// core/film.cpp:56, so its table did not vary along x).
#include "rb2_internal.h"
#include "rb2_render.h"

#include <cmath>

namespace {

// The two factors of the filter at offset (x, y).
void eval_axes(const rb2_filter& f, float x, float y, float& gx, float& gy)
{
    switch (f.kind) {
    case RB2_FILTER_TRIANGLE:
        gx = std::fmax(0.0f, f.xwidth - std::fabs(x));
        gy = std::fmax(0.0f, f.ywidth - std::fabs(y));
        return;
    case RB2_FILTER_GAUSSIAN:
        gx = std::fmax(0.0f, std::exp(-f.alpha * x * x) - std::exp(-f.alpha * f.xwidth * f.xwidth));
        gy = std::fmax(0.0f, std::exp(-f.alpha * y * y) - std::exp(-f.alpha * f.ywidth * f.ywidth));
        return;
    default:
        gx = gy = 1.0f;  // box (and "none", unused)
    }
}

}  // namespace

namespace rb2 {

int validate_filter(const rb2_filter* f)
{
    if (!f) return fail(RB2_EINVAL, "null filter");
    if (f->kind > RB2_FILTER_GAUSSIAN) return fail(RB2_EINVAL, "unknown filter kind");
    if (f->kind == RB2_FILTER_NONE) return RB2_OK;
    if (!(f->xwidth > 0.0f && f->xwidth <= 16.0f && f->ywidth > 0.0f && f->ywidth <= 16.0f))
        return fail(RB2_EINVAL, "filter half-widths must be in (0, 16]");
    if (f->kind == RB2_FILTER_GAUSSIAN && !(f->alpha > 0.0f && std::isfinite(f->alpha)))
        return fail(RB2_EINVAL, "Gaussian alpha must be positive");
    return RB2_OK;
}

// The 16 factors per axis: table entry [y][x] is gx[x] * gy[y].
int filter_axes(const rb2_filter& f, float gx[16], float gy[16])
{
    const int rc = validate_filter(&f);
    if (rc) return rc;
    for (int i = 0; i < 16; ++i)
        eval_axes(f, ((float)i + 0.5f) * f.xwidth / 16.0f, ((float)i + 0.5f) * f.ywidth / 16.0f, gx[i], gy[i]);
    return RB2_OK;
}

}  // namespace rb2

extern "C" int rb2_filter_table(const rb2_filter* f, float* table256)
{
    if (!table256) return rb2::fail(RB2_EINVAL, "null table");
    if (const int rc = rb2::validate_filter(f)) return rc;
    float gx[16], gy[16];
    if (const int rc = rb2::filter_axes(*f, gx, gy)) return rc;
    for (int y = 0; y < 16; ++y)
        for (int x = 0; x < 16; ++x) table256[y * 16 + x] = gx[x] * gy[y];
    return RB2_OK;
}
