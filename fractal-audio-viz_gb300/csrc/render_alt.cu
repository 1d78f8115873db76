// Plain form for julia / burning-ship / tricorn: FP64-mantissa perturbation
// with the formula-aware real 2x2 linear BLA, one thread per pixel.
//
// Restates render_alternate_reference_impl and alternate_delta_step
// (renderer.cpp:11933-12448): the image series for Julia, the signed escape
// margin built on the MPFR margin of each reference step, block acceptance
// only when the endpoint stays inside (else an exact replay), the Burning
// Ship axis-crossing step in FloatExp components, the exact scaled formula
// step once the reference orbit ends, and the Jacobian carried for the
// analytic-DE plane.  Compiled with --fmad=false like the Mandelbrot plain
// form, so results match the reference release build bit for bit.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "device.h"

namespace fgb {
namespace {

using namespace fx;

constexpr int kAltPastTurns = 16;  // formula steps per turn past the orbit's end
constexpr double kTwoPi = 6.283185307179586476925286766559005768;
constexpr double kLogTwo = 0.693147180559945309417232121458176568;

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ double pixel_offset(int index, int dimension, int mode) {
    const double origin = mode == 1 ? static_cast<double>(dimension / 2) : static_cast<double>(dimension - 1) / 2.0;
    return static_cast<double>(index) - origin;
}

__device__ __forceinline__ float nan_f() { return __int_as_float(0x7fc00000); }

__device__ __forceinline__ Sc ld_sc(const Sc* s) { return sc_make(__ldg(&s->re), __ldg(&s->im), __ldg(&s->e)); }
__device__ __forceinline__ Fe ld_fe(const Fe* f) { return fe_make(__ldg(&f->m), __ldg(&f->e)); }

__device__ float smooth_escape(int iteration, const Nrm& norm, double bias) {
    if (is_zero(norm.m)) return static_cast<float>(static_cast<double>(iteration) - bias);
    const double log_mag = 0.5 * (log(norm.m) + static_cast<double>(norm.e) * kLogTwo);
    if (!(log_mag > 0.0) || !is_finite(log_mag)) return static_cast<float>(static_cast<double>(iteration) - bias);
    return static_cast<float>((static_cast<double>(iteration) - log(log_mag) / kLogTwo) - bias);
}

// Real Jacobian [xa xb; ya yb] of the pixel map (renderer.cpp:7912-8073).
struct Jac {
    Fe xa, xb, ya, yb;
};

__device__ Jac jac_identity() { return Jac{fe_from(1.0, 0), fe_zero(), fe_zero(), fe_from(1.0, 0)}; }

__device__ Jac jac_holomorphic(const Sc& d) {
    const Fe re = fe_from(d.re, d.e);
    const Fe im = fe_from(d.im, d.e);
    return Jac{re, fe_neg(im), im, re};
}

__device__ __forceinline__ bool negative(const Fe& a) { return hi_of(a.m) < 0 && !is_zero(a.m); }

__device__ Jac jac_step(int formula, const Sc& total, const Jac& p, bool parameter_plane) {
    const Fe re = fe_from(total.re, total.e);
    const Fe im = fe_from(total.im, total.e);
    Fe m00, m01, m10, m11;
    if (formula == kFormulaTricorn) {
        m00 = fe_twice(re, false);
        m01 = fe_twice(im, true);
        m10 = m01;
        m11 = fe_twice(re, true);
    } else if (formula == kFormulaBurningShip) {
        const Fe ar = fe_abs(re), ai = fe_abs(im);
        const bool rneg = negative(re), ineg = negative(im);
        m00 = fe_twice(ar, rneg);
        m01 = fe_twice(ai, !ineg);
        m10 = fe_twice(ai, rneg);
        m11 = fe_twice(ar, ineg);
    } else {
        m00 = fe_twice(re, false);
        m01 = fe_twice(im, true);
        m10 = fe_twice(im, false);
        m11 = m00;
    }
    const Fe one = parameter_plane ? fe_from(1.0, 0) : fe_zero();
    return Jac{fe_add(fe_add(fe_mul(m00, p.xa), fe_mul(m01, p.ya)), one),
               fe_add(fe_add(fe_mul(m00, p.xb), fe_mul(m01, p.yb)), fe_zero()),
               fe_add(fe_add(fe_mul(m10, p.xa), fe_mul(m11, p.ya)), fe_zero()),
               fe_add(fe_add(fe_mul(m10, p.xb), fe_mul(m11, p.yb)), one)};
}

__device__ __noinline__ Jac jac_bla(const AltStep* s, const Jac j, bool parameter_plane) {
    const Jac p{fe_from(j.xa.m, j.xa.e), fe_from(j.xb.m, j.xb.e), fe_from(j.ya.m, j.ya.e), fe_from(j.yb.m, j.yb.e)};
    Fe c[8];
    for (int k = 0; k < 8; ++k) c[k] = ld_fe(&s->c[k]);
    return Jac{fe_add(fe_add(fe_mul(c[0], p.xa), fe_mul(c[1], p.ya)), parameter_plane ? c[4] : fe_zero()),
               fe_add(fe_add(fe_mul(c[0], p.xb), fe_mul(c[1], p.yb)), parameter_plane ? c[5] : fe_zero()),
               fe_add(fe_add(fe_mul(c[2], p.xa), fe_mul(c[3], p.ya)), parameter_plane ? c[6] : fe_zero()),
               fe_add(fe_add(fe_mul(c[2], p.xb), fe_mul(c[3], p.yb)), parameter_plane ? c[7] : fe_zero())};
}

// render_plane_de_matrix (renderer.cpp:7936-7990).
__device__ bool de_matrix(const Sc& total, const Jac& j, const Fe& spacing, double& ox, double& oy) {
    const double mag = hypot(total.re, total.im);
    if (!(mag > 0.0) || !is_finite(mag)) return false;
    const double lm = log(mag) + static_cast<double>(total.e) * kLogTwo;
    if (!(lm > 0.0) || !is_finite(lm)) return false;
    const double ur = total.re / mag, ui = total.im / mag;
    const Fe sxa = fe_mul(j.xa, spacing), sxb = fe_mul(j.xb, spacing);
    const Fe sya = fe_mul(j.ya, spacing), syb = fe_mul(j.yb, spacing);
    const Fe dr = fe_add(fe_mul(sxa, ur), fe_mul(sya, ui));
    const Fe di = fe_add(fe_mul(sxb, ur), fe_mul(syb, ui));
    const Fe d2 = fe_add(fe_sqr(dr), fe_sqr(di));
    if (fe_is_zero(d2) || !fe_finite(d2)) return false;
    const Fe num = fe_from(mag * lm, total.e);
    const Fe rr = fe_div(fe_mul(num, dr), d2);
    const Fe ri = fe_div(fe_neg(fe_mul(num, di)), d2);
    ox = scale2(rr.m, rr.e);
    oy = scale2(ri.m, ri.e);
    return is_finite(ox) && is_finite(oy);
}

struct Planes {
    std::int64_t* iter;
    double *phase, *dex, *dey, *t1, *t2;
    __device__ void clear(long long i, int max_iter) const {
        iter[i] = max_iter;
        phase[i] = dex[i] = dey[i] = t1[i] = t2[i] = 0.0;
    }
    __device__ void escape(long long i, int raw, const Sc& total, const Nrm& test2, const Jac& j,
                           const Fe& spacing) const {
        iter[i] = raw;
        const double re = sc_re_d(total), im = sc_im_d(total);
        double ph = 0.0;
        if (is_finite(re) && is_finite(im)) {
            ph = atan2(im, re) / kTwoPi;
            ph -= floor(ph);
            if (!is_finite(ph)) ph = 0.0;
        }
        phase[i] = ph;
        double ox = 0.0, oy = 0.0;
        if (de_matrix(total, j, spacing, ox, oy)) {
            dex[i] = ox;
            dey[i] = oy;
        } else {
            dex[i] = 0.0;
            dey[i] = 0.0;
        }
        t1[i] = nrm_to_d(sc_norm2(total));
        t2[i] = nrm_to_d(test2);
    }
};

// Signed escape margin from the MPFR margin of step i (renderer.cpp:8427-8443).
__device__ __noinline__ Fe alt_margin(const AltParams& p, int i, Sc d) {
    sc_normalize(d);
    const OrbitRec* r = p.orbit + i;
    const Fe m0 = ld_fe(&r->margin);
    const Fe zr = fe_make(__ldg(&r->parts.re.m), __ldg(&r->parts.re.e));
    const Fe zi = fe_make(__ldg(&r->parts.im.m), __ldg(&r->parts.im.e));
    const Fe cross = fe_twice(fe_add(fe_mul(zr, fe_from(d.re, d.e)), fe_mul(zi, fe_from(d.im, d.e))), false);
    const Nrm dn = sc_norm2(d);
    return fe_add(fe_add(m0, cross), fe_make(dn.m, dn.e));
}

// Whether the pixel Z_i + d lies inside the escape radius by so much that
// the signed margin above cannot come out positive, decided in FP32.  With
// |d|^2 < 16 R^2 (so |Z| <= 5 R for an accepted total) the estimate of
// |Z + d|^2 is off by less than 4e-6 R^2 (operands truncated to 2^-23) and
// the FP64 margin by less than 1e-13 R^2, both far below the 2^-14 R^2 kept
// free; a NaN or an overflow fails.  The margin, the norm and the total cost
// 11 FP64 instructions (880 cycles of a sub-partition) and only the sign
// matters until the pixel escapes.
__device__ __forceinline__ bool alt_inside(const AltParams& p, int i, const Sc& d) {
    const float2 z = __ldg(reinterpret_cast<const float2*>(&p.orbit[i].zf_re));
    const int e = imax(imin(d.e, 64), -4096);
    const float dx = float_of(d.re, e), dy = float_of(d.im, e);
    const float tx = z.x + dx, ty = z.y + dy;
    const float r2 = p.escape_mode == 1 ? 1.0e8f : 4.0f;
    return tx * tx + ty * ty < r2 * (1.0f - 0x1p-14f) && dx * dx + dy * dy < r2 * 16.0f;
}

// Whether adding d to r changes which side of zero it is on (zero counts
// with the positive side), as the sign of the rounded sum has it: the sum of
// two finite values is negative exactly when the larger magnitude is.
__device__ __forceinline__ bool crosses_zero(const Fe& r, const Fe& d) {
    if (is_zero(d.m)) return false;
    const bool rn = hi_of(r.m) < 0 && !is_zero(r.m), dn = hi_of(d.m) < 0;
    if (is_zero(r.m)) return dn;
    if (rn == dn) return false;
    const int larger = d.e != r.e ? (d.e > r.e ? 1 : -1) : order_of(fabs_(d.m), fabs_(r.m));
    return rn ? larger >= 0 : larger > 0;
}

// alternate_delta_step (renderer.cpp:11933-12034).
// The general form, on normalised values; out of line, since few steps
// need it.
template <int Formula>
__device__ __noinline__ Sc alt_step(const AltParams& p, int i, Sc d, Sc pd) {
    sc_normalize(d);
    sc_normalize(pd);
    const Sc z = ld_sc(&p.orbit[i].z);
    if constexpr (Formula == kFormulaTricorn) {
        const Sc zc = sc_conj(z), dcj = sc_conj(d);
        return sc_add(sc_twice(sc_mul(zc, dcj)), sc_add(sc_sqr(dcj), pd));
    }
    if constexpr (Formula == kFormulaBurningShip) {
        const Fe rr = fe_from(z.re, z.e), ri = fe_from(z.im, z.e);
        const Fe dr = fe_from(d.re, d.e), di = fe_from(d.im, d.e);
        const Fe ar = fe_abs(rr), ai = fe_abs(ri);
        if (crosses_zero(rr, dr) || crosses_zero(ri, di)) {
            const Fe tr = fe_add(rr, dr), ti = fe_add(ri, di);
            const Fe atr = fe_abs(tr), ati = fe_abs(ti);
            const Sc zn = ld_sc(&p.orbit[i + 1].z);
            const Fe por = fe_sub(fe_from(p.parameter.re, p.parameter.e), fe_from(zn.re, zn.e));
            const Fe poi = fe_sub(fe_from(p.parameter.im, p.parameter.e), fe_from(zn.im, zn.e));
            const Fe nr = fe_add(fe_sub(fe_sqr(atr), fe_sqr(ati)), fe_add(por, fe_from(pd.re, pd.e)));
            const Fe ni = fe_add(fe_twice(fe_mul(atr, ati), false), fe_add(poi, fe_from(pd.im, pd.e)));
            return sc_from_fe(nr, ni);
        }
        const bool rneg = negative(rr), ineg = negative(ri);
        const Fe lr = fe_sub(fe_twice(fe_mul(ar, dr), rneg), fe_twice(fe_mul(ai, di), ineg));
        const Fe li = fe_add(fe_twice(fe_mul(ar, di), ineg), fe_twice(fe_mul(ai, dr), rneg));
        const Fe sr = fe_sub(fe_sqr(dr), fe_sqr(di));
        const Fe si = fe_twice(fe_mul(dr, di), rneg != ineg);
        return sc_from_fe(fe_add(fe_add(lr, sr), fe_from(pd.re, pd.e)), fe_add(fe_add(li, si), fe_from(pd.im, pd.e)));
    }
    return sc_add(sc_twice(sc_mul(z, d)), sc_add(sc_sqr(d), pd));
}

// scaled_formula_step (renderer.cpp:11917-11931).
template <int Formula>
__device__ __noinline__ Sc formula_step(Sc v, Sc c) {
    sc_normalize(v);
    sc_normalize(c);
    if constexpr (Formula == kFormulaBurningShip) {
        return sc_add(sc_sqr(sc_make(fabs_(v.re), fabs_(v.im), v.e)), c);
    }
    return sc_add(sc_sqr(Formula == kFormulaTricorn ? sc_conj(v) : v), c);
}

// The Jacobian after a general step, its entries on one shared exponent
// again where they allow it (raw_double.h).
__device__ Jac jac_pack(const Jac& j) {
    int e = INT_MIN;
    if (!is_zero(j.xa.m)) e = imax(e, j.xa.e);
    if (!is_zero(j.xb.m)) e = imax(e, j.xb.e);
    if (!is_zero(j.ya.m)) e = imax(e, j.ya.e);
    if (!is_zero(j.yb.m)) e = imax(e, j.yb.e);
    auto fits = [&](const Fe& v) {
        return is_zero(v.m) || (bexp(v.m) == 1022 && static_cast<unsigned>(e) - static_cast<unsigned>(v.e) <= 380u);
    };
    if (e == INT_MIN || !fits(j.xa) || !fits(j.xb) || !fits(j.ya) || !fits(j.yb)) return j;
    auto shared = [&](const Fe& v) { return fe_make(is_zero(v.m) ? v.m : add_exp(v.m, v.e - e), e); };
    return Jac{shared(j.xa), shared(j.xb), shared(j.ya), shared(j.yb)};
}

__device__ Jac jac_normal(const Jac& j) {
    return Jac{fe_from(j.xa.m, j.xa.e), fe_from(j.xb.m, j.xb.e), fe_from(j.ya.m, j.ya.e), fe_from(j.yb.m, j.yb.e)};
}

__device__ __noinline__ Jac jac_step_general(int formula, Sc total, const Jac j, bool parameter_plane) {
    sc_normalize(total);
    return jac_pack(jac_step(formula, total, jac_normal(j), parameter_plane));
}

__device__ __forceinline__ bool jac_part(double v) {
    return static_cast<unsigned>(bexp(v) - kRawLow) <= kJacSpan || is_zero(v);
}

// jac_step on the values themselves: total raw (a part may have cancelled to
// zero), entries on one exponent k.  The parameter plane's +1 is 2^-k in the
// entries' unit; below 2^-600 of it, it cannot move a sum that is above
// 2^-463.  Returns false, with nothing changed, where the ranges do not fit.
template <int Formula>
__device__ __forceinline__ bool jac_step_raw(const Sc& total, Jac& j) {
    constexpr bool parameter_plane = Formula != kFormulaJulia;
    const int k = j.xa.e;
    const bool fits = k == j.xb.e && k == j.ya.e && k == j.yb.e && k >= -400 && jac_part(j.xa.m) && jac_part(j.xb.m)
        && jac_part(j.ya.m) && jac_part(j.yb.m);
    if (!fits) return false;
    const double tr = is_zero(total.re) ? total.re : add_exp(total.re, 1);
    const double ti = is_zero(total.im) ? total.im : add_exp(total.im, 1);
    // Rows of M (jac_step): real part 2 (tr, -ti); imaginary part 2 (ti, tr)
    // with each formula's signs.
    bool s0 = false, s1 = false;  // signs of (ti, tr) in the second row
    if constexpr (Formula == kFormulaTricorn) {
        s0 = s1 = true;
    } else if constexpr (Formula == kFormulaBurningShip) {
        const bool rn = hi_of(tr) < 0 && !is_zero(tr), in = hi_of(ti) < 0 && !is_zero(ti);
        s0 = s1 = rn != in;
    }
    const double m00 = tr, m01 = neg_(ti), m10 = flip(ti, s0), m11 = flip(tr, s1);
    double xa = m00 * j.xa.m + m01 * j.ya.m, xb = m00 * j.xb.m + m01 * j.yb.m;
    double ya = m10 * j.xa.m + m11 * j.ya.m, yb = m10 * j.xb.m + m11 * j.yb.m;
    if constexpr (parameter_plane) {
        if (k <= 600) {
            const double one = from_hilo((1023 - k) << 20, 0);
            xa = xa + one;
            yb = yb + one;
        } else if (bexp(xa) < 560 || bexp(yb) < 560) {
            return false;
        }
    }
    const int top = imax(imax(bexp(xa), bexp(xb)), imax(bexp(ya), bexp(yb)));
    int shift = 0;
    if (top > 1023 + 300) {
        const auto low = [](double v) { return is_zero(v) ? 2046 : bexp(v); };
        const int least = imin(imin(low(xa), low(xb)), imin(low(ya), low(yb)));
        if (least - 300 >= kRawLow) shift = 300;
    }
    const auto entry = [&](double v) { return fe_make(is_zero(v) ? v : add_exp(v, -shift), k + shift); };
    j = Jac{entry(xa), entry(xb), entry(ya), entry(yb)};
    return true;
}

template <int Formula>
__device__ __forceinline__ void jac_advance(const Sc& total, bool raw, Jac& j) {
    if (raw && jac_step_raw<Formula>(total, j)) return;
    j = jac_step_general(Formula, total, j, Formula != kFormulaJulia);
}

// alt_step on raw values.  For the burning ship, away from a fold (no part of
// Z + d on the other side of zero from Z's) the signs of |Z| cancel to one
// sign on the imaginary part: 7 products and 7 sums, as for the others.
template <int Formula>
__device__ __forceinline__ Sc alt_step_raw(double zr, double zi, const Sc& d, const Sc& pd) {
    const double z2r = add_exp(zr, 1), z2i = add_exp(zi, 1);
    const double lr = z2r * d.re - z2i * d.im;
    const double li = z2r * d.im + z2i * d.re;
    const double sr = d.re * d.re - d.im * d.im;
    const double si = add_exp(d.re * d.im, 1);
    if constexpr (Formula == kFormulaBurningShip) {
        const bool s = (hi_of(zr) ^ hi_of(zi)) < 0;
        return sc_make((lr + sr) + pd.re, flip(li + si, s) + pd.im, 0);
    } else if constexpr (Formula == kFormulaTricorn) {
        return add_cut(sc_make(lr, neg_(li), 0), add_cut(sc_make(sr, neg_(si), 0), pd));
    } else {
        return add_cut(sc_make(lr, li, 0), sc_make(sr, si, 0));
    }
}

// A fold of the burning ship: a part of Z + d has crossed zero.
__device__ __forceinline__ bool folds(double z, double d) {
    return (hi_of(z) ^ hi_of(d)) < 0 && (bits_of(d) & 0x7fffffffffffffffull) >= (bits_of(z) & 0x7fffffffffffffffull);
}

// AlternateLinearBlaLevels::lookup (renderer.cpp:8536-8567).
// The delta's squared norm is formed only where the exponents leave its
// order against the two-step block's radius open.
__device__ __noinline__ const AltStep* alt_search(const AltParams& p, int offset, Sc d, const Fe pn, int top) {
    sc_normalize(d);
    const Nrm dnorm = sc_norm2(d);
    const Fe dn = fe_make(dnorm.m, dnorm.e);
    if (!fe_finite(dn)) return nullptr;
    if ((offset >> 1) < p.alt_index.count[1]) {
        const Fe r2 = ld_fe(&p.alt[p.alt_index.offset[1] + (offset >> 1)].r2);
        if (fe_finite(r2) && fe_cmp(dn, r2) >= 0) return nullptr;
    }
    for (int level = top; level >= 1; --level) {
        if ((offset & ((1 << level) - 1)) != 0) continue;
        const int index = offset >> level;
        if (index >= p.alt_index.count[level]) continue;
        const AltStep* s = p.alt + p.alt_index.offset[level] + index;
        const Fe r2 = ld_fe(&s->r2);
        if (__ldg(&s->len) > 1 && fe_finite(r2) && fe_cmp(dn, r2) < 0 && fe_cmp(pn, p.alt_input_radius2) <= 0) return s;
    }
    return nullptr;
}

__device__ __forceinline__ const AltStep* alt_lookup(const AltParams& p, int start, const Sc& d, const Fe& pn,
                                                     int max_length) {
    if (p.alt_index.levels == 0 || start < p.alt_start || max_length <= 0 || !sc_finite(d) || !fe_finite(pn)) {
        return nullptr;
    }
    const int offset = start - p.alt_start;
    if (offset < 0 || offset >= p.alt_index.count[0]) return nullptr;
    int top = 31 - __clz(max_length);
    top = top < p.alt_index.levels - 1 ? top : p.alt_index.levels - 1;
    // Only blocks of two or more steps are taken, and they start at even
    // offsets.  At one start the radii never grow with the level (a merge
    // keeps at most its first half's radius, times 1 - 2^-40; an unpaired
    // entry is copied), so a delta outside the two-step block's finite
    // radius is outside every longer block's too: one load settles the
    // common case of a delta too large for any block, with the same result
    // as the full top-down search.
    if (top < 1 || (offset & 1) != 0) return nullptr;
    if ((offset >> 1) < p.alt_index.count[1]) {
        const Fe r2 = ld_fe(&p.alt[p.alt_index.offset[1] + (offset >> 1)].r2);
        // With E the exponent of d's larger part (which is at least 2^(E - 1)),
        // |d|^2 >= 2^(2E - 2), and r2 < 2^r2.e.
        const int top_exponent = imax(bexp(d.re), bexp(d.im));
        if (fe_finite(r2) && is_normal(top_exponent) && 2LL * (static_cast<long long>(d.e) + top_exponent - 1022) - 2 >= r2.e) {
            return nullptr;
        }
    }
    return alt_search(p, offset, d, pn, top);
}

__device__ __noinline__ Sc apply_alt(const AltStep* s, const Sc d, const Sc c) {
    const Fe dr = fe_from(d.re, d.e), di = fe_from(d.im, d.e);
    const Fe cr = fe_from(c.re, c.e), ci = fe_from(c.im, c.e);
    Fe k[8];
    for (int j = 0; j < 8; ++j) k[j] = ld_fe(&s->c[j]);
    const Fe rr = fe_add(fe_add(fe_mul(k[0], dr), fe_mul(k[1], di)), fe_add(fe_mul(k[4], cr), fe_mul(k[5], ci)));
    const Fe ri = fe_add(fe_add(fe_mul(k[2], dr), fe_mul(k[3], di)), fe_add(fe_mul(k[6], cr), fe_mul(k[7], ci)));
    return sc_from_fe(rr, ri);
}

// One pixel's state between steps, so a lane can park it and carry on
// later (the lane-refill queue below) or run it to the end at once.  delta,
// total and pd are raw values where their range allows (raw_double.h).  The
// total Z + delta is kept only once the orbit has ended (`past`): before
// that it is formed where something reads it.
template <bool WithPlanes>
struct AltLane {
    long long index;
    Sc dc, pd, delta, total, tortoise;
    Fe pn;
    Jac jac;
    int ref, it, power, length, hits;
    unsigned ticks;
    bool ready, past;
};

__device__ __forceinline__ void alt_store(const AltParams& p, long long index, float out, std::uint32_t count) {
    p.out[index] = out;
    if (p.counts) p.counts[index] = count;
}

__device__ __noinline__ Sc alt_total(const AltParams& p, int ref, Sc delta) {
    sc_normalize(delta);
    return sc_add(ld_sc(&p.orbit[ref].z), delta);
}

__device__ __forceinline__ int raw_iteration(int formula, int n) {
    return formula == kFormulaJulia ? n : (n - 1 > 0 ? n - 1 : 0);
}

// Outputs of a pixel that escaped with `norm` at `total`; `prior` is the
// total one step earlier (planes only).
template <bool WithPlanes, int Formula>
__device__ __noinline__ void alt_finish(const AltParams& p, long long index, int it, const Nrm norm, Sc total, Sc prior,
                                        const Jac jac) {
    if constexpr (WithPlanes) {
        const Planes planes{p.p_iter, p.p_phase, p.p_dex, p.p_dey, p.p_t1, p.p_t2};
        planes.escape(index, raw_iteration(Formula, it), normal_form(total), sc_norm2(normal_form(prior)),
                      jac_normal(jac), p.pixel_spacing);
    }
    alt_store(p, index, smooth_escape(it, norm, p.output_bias), static_cast<std::uint32_t>(it));
}

// The escape test after a perturbation step to s.ref.  Returns true when the
// pixel escaped.
template <bool WithPlanes, int Formula>
__device__ __forceinline__ bool alt_escaped(const AltParams& p, const AltLane<WithPlanes>& s, const Sc& prior) {
    if (alt_inside(p, s.ref, s.delta)) return false;
    const Fe margin = alt_margin(p, s.ref, s.delta);
    const Nrm norm = nrm_from_margin(margin, p.escape_mode);
    if (!fe_positive(margin) && !nrm_outside(norm, p.escape_mode)) return false;
    alt_finish<WithPlanes, Formula>(p, s.index, s.it, norm, WithPlanes ? alt_total(p, s.ref, s.delta) : sc_zero(), prior,
                                    s.jac);
    return true;
}

// Start pixel `index`: coordinates, Julia series jump, first escape test.
// Returns true when the pixel is finished (its outputs written).
template <bool WithPlanes, int Formula>
__device__ __noinline__ bool alt_begin(const AltParams& p, long long index, AltLane<WithPlanes>& s) {
    constexpr bool julia = Formula == kFormulaJulia;
    const int py = static_cast<int>(index / p.width);
    const int px = static_cast<int>(index - static_cast<long long>(py) * p.width);
    const Planes planes{p.p_iter, p.p_phase, p.p_dex, p.p_dey, p.p_t1, p.p_t2};
    if constexpr (WithPlanes) planes.clear(index, p.max_iter);
    const double xf = pixel_offset(px, p.width, p.coordinate_mode) / static_cast<double>(p.width);
    const double yf = -pixel_offset(py, p.height, p.coordinate_mode) / static_cast<double>(p.height);
    s.index = index;
    s.dc = p.points ? sc_make(p.points[index].re, p.points[index].im, p.points[index].e)
                    : sc_from_fe(fe_mul(p.view_width, xf), fe_mul(p.view_height, yf));
    s.pd = julia ? sc_zero() : s.dc;
    const Nrm pnorm = sc_norm2(s.pd);
    s.pn = fe_make(pnorm.m, pnorm.e);
    s.delta = s.dc;
    s.jac = jac_identity();
    s.ref = julia ? 0 : 1;
    s.it = julia ? 0 : 1;
    if (p.series_on && nrm_cmp(sc_norm2(s.dc), p.series_r2) <= 0) {
        Sc value = ld_sc(&p.series[p.series_terms - 1]);
        Sc poly = sc_zero();
        for (int k = p.series_terms - 1; k > 1; --k) {
            if constexpr (WithPlanes) poly = sc_add(sc_mul(poly, s.dc), value);
            value = sc_add(sc_mul(value, s.dc), ld_sc(&p.series[k - 1]));
        }
        s.delta = sc_mul(value, s.dc);
        if constexpr (WithPlanes) s.jac = jac_holomorphic(sc_add(sc_mul(poly, s.dc), value));
        s.ref = p.series_iteration;
        s.it = p.series_iteration;
    }
    s.ticks = 0;
    if (!alt_inside(p, s.ref, s.delta)) {
        const Nrm norm = nrm_from_margin(alt_margin(p, s.ref, s.delta), p.escape_mode);
        if (nrm_outside(norm, p.escape_mode)) {
            alt_finish<WithPlanes, Formula>(p, index, s.it, norm, WithPlanes ? alt_total(p, s.ref, s.delta) : sc_zero(),
                                            sc_zero(), s.jac);
            return true;
        }
    }
    s.pd = to_raw(s.pd);
    s.delta = to_raw(s.delta);
    s.jac = jac_pack(s.jac);
    s.past = false;
    s.total = sc_zero();
    s.tortoise = sc_zero();
    s.power = 1;
    s.length = 0;
    s.hits = 0;
    s.ready = false;
    return false;
}

// Formula steps past the orbit's end (up to `turns`).  Returns true when the
// pixel is finished.
template <bool WithPlanes, int Formula>
__device__ __forceinline__ bool alt_past(const AltParams& p, AltLane<WithPlanes>& s, unsigned long long deadline,
                                         int turns) {
    constexpr bool julia = Formula == kFormulaJulia;
    if (!s.past) {
        s.total = to_raw(alt_total(p, s.ref, s.delta));
        s.past = true;
    }
    const Sc parameter = to_raw(julia ? p.parameter : sc_add(p.parameter, s.dc));
    const float estimate_bound = static_cast<float>(p.escape_mode == 1 ? 1.0e8 : 4.0) * (1.0f - 0x1p-14f);
    for (int k = 0; k < turns && s.it < p.max_iter; ++k) {
        if (k > 0 && deadline && ((s.ticks++ & 255U) == 0U) && global_ns() >= deadline) {
            alt_store(p, s.index, nan_f(), 0u);
            return true;
        }
        const Sc prior = s.total;
        // Raw step: 3 products and 3 sums.  Squares of parts in range are
        // normal; a sum that cancels is exact.
        const bool raw = raw_value(prior) && parameter.e == 0;
        if constexpr (WithPlanes) jac_advance<Formula>(prior, raw, s.jac);
        ++s.it;
        bool maybe_out = true;
        if (raw) {
            const double cross = add_exp(prior.re * prior.im, 1);
            const bool negate = Formula == kFormulaTricorn
                || (Formula == kFormulaBurningShip && (hi_of(prior.re) ^ hi_of(prior.im)) < 0);
            const Sc square = sc_make(prior.re * prior.re - prior.im * prior.im, flip(cross, negate), 0);
            s.total = add_cut(square, parameter);
            const float tx = float_of(s.total.re, 0), ty = float_of(s.total.im, 0);
            maybe_out = !(tx * tx + ty * ty < estimate_bound);
        } else {
            s.total = to_raw(formula_step<Formula>(prior, parameter));
        }
        if (maybe_out) {
            const Nrm norm = sc_norm2(normal_form(s.total));
            if (nrm_outside(norm, p.escape_mode)) {
                alt_finish<WithPlanes, Formula>(p, s.index, s.it, norm, s.total, prior, s.jac);
                return true;
            }
        }
    }
    return false;
}

// One turn of the per-pixel loop: formula steps past the orbit's end, a BLA
// block (or its exact replay), or one exact perturbation step with the
// escape and cycle tests.  Returns true when the pixel is finished.
template <bool WithPlanes, int Formula>
__device__ __forceinline__ bool alt_advance(const AltParams& p, AltLane<WithPlanes>& s, unsigned long long deadline,
                                            int max_block) {
    constexpr bool julia = Formula == kFormulaJulia;
    const long long index = s.index;
    if (s.it >= p.max_iter) {
        const Planes planes{p.p_iter, p.p_phase, p.p_dex, p.p_dey, p.p_t1, p.p_t2};
        if constexpr (WithPlanes) planes.clear(index, p.max_iter);
        alt_store(p, index, static_cast<float>(static_cast<double>(p.max_iter) - p.output_bias),
                  static_cast<std::uint32_t>(p.max_iter));
        return true;
    }
    if (deadline && ((s.ticks++ & 255U) == 0U) && global_ns() >= deadline) {
        alt_store(p, index, nan_f(), 0u);
        return true;
    }
    if (s.ref + 1 >= p.orbit_size) return alt_past<WithPlanes, Formula>(p, s, deadline, kAltPastTurns);
    const int remaining = p.max_iter - s.it;
    const AltStep* step = !p.disable_bla
        ? alt_lookup(p, s.ref, s.delta, s.pn, max_block < remaining ? max_block : remaining)
        : nullptr;
    int len = step != nullptr ? __ldg(&step->len) : 1;
    if (step != nullptr && s.ref + len < p.orbit_size) {
        const int end = s.ref + len;
        const Sc cand = apply_alt(step, s.delta, s.pd);
        const Fe cmargin = alt_margin(p, end, cand);
        const Nrm cnorm = nrm_from_margin(cmargin, p.escape_mode);
        const bool bad = !sc_finite(cand) || !fe_finite(cmargin) || !sc_finite(alt_total(p, end, cand))
            || fe_positive(cmargin) || nrm_cmp(cnorm, nrm_make(0.75, 2)) >= 0;
        if (!bad) {
            s.delta = to_raw(cand);
            if constexpr (WithPlanes) s.jac = jac_pack(jac_bla(step, s.jac, !julia));
            s.ref = end;
            s.it += len;
            return false;
        }
    } else {
        step = nullptr;
        len = 1;
    }
    // Exact steps: one, or the refused block's replay (whose steps have no
    // cycle test of their own).
    for (int k = 0; k < len && s.it < p.max_iter; ++k) {
        const OrbitRec* r = p.orbit + s.ref;
        const double2 z = __ldg(reinterpret_cast<const double2*>(&r->zd_re));
        const bool raw = __ldg(&r->raw) != 0 && raw_value(s.delta) && (julia || raw_value(s.pd));
        Sc prior = sc_zero();
        if constexpr (WithPlanes) {
            prior = raw ? add_cut(sc_make(z.x, z.y, 0), s.delta) : alt_total(p, s.ref, s.delta);
            jac_advance<Formula>(prior, raw, s.jac);
        }
        if (raw && !(Formula == kFormulaBurningShip && (folds(z.x, s.delta.re) || folds(z.y, s.delta.im)))) {
            s.delta = alt_step_raw<Formula>(z.x, z.y, s.delta, s.pd);
        } else {
            s.delta = to_raw(alt_step<Formula>(p, s.ref, s.delta, s.pd));
        }
        ++s.ref;
        ++s.it;
        if (!sc_finite(s.delta)) {
            alt_store(p, index, p.strict ? nan_f() : static_cast<float>(static_cast<double>(s.it) - p.output_bias),
                      p.strict ? 0u : static_cast<std::uint32_t>(s.it));
            return true;
        }
        if (alt_escaped<WithPlanes, Formula>(p, s, prior)) return true;
    }
    if (step != nullptr) return false;
    // Bounded cycle confirmed three times (non-strict renders only).
    if (!p.cycle || s.it < 2048 || (s.it & 31) != 0) return false;
    const Nrm total_norm = nrm_from_margin(alt_margin(p, s.ref, s.delta), p.escape_mode);
    if (nrm_cmp(total_norm, nrm_make(0.75, 2)) < 0) {
        const Sc total = alt_total(p, s.ref, s.delta);
        if (!s.ready) {
            s.tortoise = total;
            s.power = 1;
            s.length = 0;
            s.hits = 0;
            s.ready = true;
        } else {
            const Nrm dist = sc_norm2(sc_sub(total, s.tortoise));
            const int scale_e = total_norm.e > 0 ? total_norm.e : 0;
            if (is_zero(dist.m) || dist.e <= scale_e - 78) {
                if (++s.hits >= 3) {
                    const Planes planes{p.p_iter, p.p_phase, p.p_dex, p.p_dey, p.p_t1, p.p_t2};
                    if constexpr (WithPlanes) planes.clear(index, p.max_iter);
                    alt_store(p, index, static_cast<float>(static_cast<double>(p.max_iter) - p.output_bias),
                              static_cast<std::uint32_t>(p.max_iter));
                    return true;
                }
            } else {
                s.hits = 0;
            }
            if (++s.length >= s.power) {
                s.tortoise = total;
                s.power = s.power * 2 < (1 << 20) ? s.power * 2 : (1 << 20);
                s.length = 0;
            }
        }
    }
    return false;
}

__device__ __forceinline__ int alt_max_block(const AltParams& p) {
    return p.max_lin_len < 2 ? 2 : (p.max_lin_len > kMaxSafeLinearBlaLength ? kMaxSafeLinearBlaLength : p.max_lin_len);
}

__device__ __forceinline__ unsigned long long alt_deadline(const AltParams& p) {
    return p.deadline_base ? *p.deadline_base + p.budget_ns : 0ull;
}

// One thread per pixel (point lists).
template <bool WithPlanes, int Formula>
__global__ void __launch_bounds__(128) alt_kernel(const AltParams p) {
    const long long pixels = static_cast<long long>(p.width) * p.height;
    const long long index = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (index >= pixels) return;
    const unsigned long long deadline = alt_deadline(p);
    const int max_block = alt_max_block(p);
    AltLane<WithPlanes> begun;
    bool done = alt_begin<WithPlanes, Formula>(p, index, begun);
    AltLane<WithPlanes> s = begun;  // in registers: `begun` lives in memory for the call
    while (!done) done = alt_advance<WithPlanes, Formula>(p, s, deadline, max_block);
}

// Lane-refill queue for Julia fields.  GB300 issues an FP64 warp
// instruction at the same cost whatever the number of active lanes, and a
// Julia view (the dynamic plane, crossed by the Julia set) mixes a few very
// long orbits with many short ones: 99 % of pixels under 100 iterations,
// some at the cap, so a warp that keeps a lane per pixel runs mostly empty.
// Persistent warps instead keep every lane busy: each lane holds one
// pixel's state, the warp runs kAltRound turns of the loop, and lanes whose
// pixel finished take new ones (claimed for the whole warp with one atomic
// on the launch's counter) once at least kAltRefill of them wait, or when
// none has work left.  Parameter-plane views (burning ship, tricorn) have
// escape times close together; there lanes that start together stay on the
// same branch of the loop, and one thread per pixel is faster (measured:
// 1.47 s against 2.23 s for a 3840x2160 burning-ship field at 1e94).
constexpr int kAltRound = 16;
constexpr int kAltRefill = 8;

template <bool WithPlanes>
__global__ void __launch_bounds__(128) alt_queue_kernel(const AltParams p, unsigned long long* counter) {
    constexpr unsigned kFull = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31u;
    const long long pixels = static_cast<long long>(p.width) * p.height;
    const unsigned long long deadline = alt_deadline(p);
    const int max_block = alt_max_block(p);
    AltLane<WithPlanes> s;
    bool have = false;
    bool drained = false;
    while (true) {
        if (!drained) {
            unsigned need = __ballot_sync(kFull, !have);
            while (__popc(need) >= kAltRefill) {
                const unsigned n = static_cast<unsigned>(__popc(need));
                unsigned long long base = 0;
                if (lane == 0) base = atomicAdd(counter, static_cast<unsigned long long>(n));
                base = __shfl_sync(kFull, base, 0);
                if (!have) {
                    const long long index = static_cast<long long>(base) + __popc(need & ((1u << lane) - 1u));
                    if (index < pixels) {
                        AltLane<WithPlanes> begun;
                        have = !alt_begin<WithPlanes, kFormulaJulia>(p, index, begun);
                        s = begun;
                    }
                }
                if (static_cast<long long>(base) + n >= pixels) {
                    drained = true;
                    break;
                }
                need = __ballot_sync(kFull, !have);
            }
        }
        if (!__any_sync(kFull, have)) {
            if (drained) break;
            continue;
        }
        // One copy of the loop body: unrolled, the turns would multiply the
        // kernel's code and miss in the instruction cache.
#pragma unroll 1
        for (int k = 0; k < kAltRound; ++k) {
            if (have && alt_advance<WithPlanes, kFormulaJulia>(p, s, deadline, max_block)) have = false;
        }
    }
}

template <bool WithPlanes>
int alt_queue_blocks() {
    static int blocks = 0;
    if (blocks == 0) {
        int per_sm = 0, sms = 0, device = 0;
        cudaGetDevice(&device);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, alt_queue_kernel<WithPlanes>, 128, 0);
        blocks = (per_sm > 0 ? per_sm : 1) * (sms > 0 ? sms : 1);
    }
    return blocks;
}

}  // namespace

cudaError_t launch_plain_alternate(const AltParams& p, bool planes, bool stats, unsigned long long* queue_counter,
                                   cudaStream_t stream) {
    (void)stats;
    const long long pixels = static_cast<long long>(p.width) * p.height;
    if (queue_counter != nullptr && p.points == nullptr && p.formula == kFormulaJulia) {
        const cudaError_t cleared = cudaMemsetAsync(queue_counter, 0, sizeof(unsigned long long), stream);
        if (cleared != cudaSuccess) return cleared;
        // A field smaller than the persistent grid needs no more warps than pixels / 32.
        const long long needed = (pixels + 127) / 128;
        if (planes) {
            const long long grid = std::min<long long>(alt_queue_blocks<true>(), needed);
            alt_queue_kernel<true><<<static_cast<unsigned>(grid), 128, 0, stream>>>(p, queue_counter);
        } else {
            const long long grid = std::min<long long>(alt_queue_blocks<false>(), needed);
            alt_queue_kernel<false><<<static_cast<unsigned>(grid), 128, 0, stream>>>(p, queue_counter);
        }
        return cudaGetLastError();
    }
    const unsigned grid = static_cast<unsigned>((pixels + 127) / 128);
    const auto launch = [&](auto formula) {
        if (planes) {
            alt_kernel<true, formula.value><<<grid, 128, 0, stream>>>(p);
        } else {
            alt_kernel<false, formula.value><<<grid, 128, 0, stream>>>(p);
        }
    };
    if (p.formula == kFormulaJulia) launch(std::integral_constant<int, kFormulaJulia>{});
    else if (p.formula == kFormulaBurningShip) launch(std::integral_constant<int, kFormulaBurningShip>{});
    else launch(std::integral_constant<int, kFormulaTricorn>{});
    return cudaGetLastError();
}

}  // namespace fgb
