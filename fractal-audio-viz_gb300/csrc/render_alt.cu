// Plain form for julia / burning-ship / tricorn: FP64-mantissa perturbation
// with the formula-aware real 2x2 linear BLA, in a persistent lane-refill
// queue.
//
// Restates render_alternate_reference_impl and alternate_delta_step
// (renderer.cpp:11933-12448): the image series for Julia, the signed escape
// margin built on the MPFR margin of each reference step, block acceptance
// only when the endpoint stays inside (else an exact replay), the Burning
// Ship axis-crossing step in FloatExp components, the exact scaled formula
// step once the reference orbit ends, and the Jacobian carried for the
// analytic-DE plane.  Compiled with --fmad=false like the Mandelbrot plain
// form, so results match the reference release build bit for bit.
#define FX_OUTLINE 1
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "cycle_turn.h"
#include "device.h"
#include "int_mul.h"

namespace fgb {
namespace {

using namespace fx;

constexpr int kAltRound = 16;  // raw steps per round
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

// Render planes: the derivative pair, and the other four or none (a batch
// asks for the pair only).
struct Planes {
    std::int64_t* iter;
    double *phase, *dex, *dey, *t1, *t2;
    __device__ void clear(long long i, int max_iter) const {
        dex[i] = dey[i] = 0.0;
        if (iter == nullptr) return;
        iter[i] = max_iter;
        phase[i] = t1[i] = t2[i] = 0.0;
    }
    __device__ void escape(long long i, int raw, const Sc& total, const Nrm& test2, const Jac& j,
                           const Fe& spacing) const {
        double ox = 0.0, oy = 0.0;
        if (de_matrix(total, j, spacing, ox, oy)) {
            dex[i] = ox;
            dey[i] = oy;
        } else {
            dex[i] = 0.0;
            dey[i] = 0.0;
        }
        if (iter == nullptr) return;
        iter[i] = raw;
        const double re = sc_re_d(total), im = sc_im_d(total);
        double ph = 0.0;
        if (is_finite(re) && is_finite(im)) {
            ph = atan2(im, re) / kTwoPi;
            ph -= floor(ph);
            if (!is_finite(ph)) ph = 0.0;
        }
        phase[i] = ph;
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
// `bound` is R^2, or 3 for a block's endpoint (refused from there on).
__device__ __forceinline__ bool alt_below(const AltParams& p, int i, const Sc& d, float bound) {
    const float2 z = __ldg(reinterpret_cast<const float2*>(&p.orbit[i].zf_re));
    const int e = imax(imin(d.e, 64), -4096);
    const float dx = float_of(d.re, e), dy = float_of(d.im, e);
    const float tx = z.x + dx, ty = z.y + dy;
    return tx * tx + ty * ty < bound * (1.0f - 0x1p-14f) && dx * dx + dy * dy < bound * 16.0f;
}

__device__ __forceinline__ bool alt_inside(const AltParams& p, int i, const Sc& d) {
    return alt_below(p, i, d, p.escape_mode == 1 ? 1.0e8f : 4.0f);
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

// The Jacobian as a raw value: four doubles times 2^k.
struct RawJac {
    double xa, xb, ya, yb;
    int k;
};

__device__ __forceinline__ bool jac_part(double v) {
    return static_cast<unsigned>(bexp(v) - kRawLow) <= kJacSpan || is_zero(v);
}

// jac_step on the values themselves: total raw (a part may have cancelled to
// zero), entries on one exponent k.  The parameter plane's +1 is 2^-k in the
// entries' unit; below 2^-600 of it, it cannot move a sum that is above
// 2^-463.  Returns false, with nothing changed, where the ranges do not fit.
template <int Formula>
__device__ __forceinline__ bool jac_step_raw(const Sc& total, RawJac& j) {
    constexpr bool parameter_plane = Formula != kFormulaJulia;
    if (!(j.k >= -400 && jac_part(j.xa) && jac_part(j.xb) && jac_part(j.ya) && jac_part(j.yb))) return false;
    const double tr = twice_raw(total.re), ti = twice_raw(total.im);
    // Rows of M (jac_step): real part 2 (tr, -ti); imaginary part 2 (ti, tr),
    // negated for the tricorn and where the burning ship's signs differ.
    bool negate = Formula == kFormulaTricorn;
    if constexpr (Formula == kFormulaBurningShip) {
        negate = (hi_of(tr) < 0 && !is_zero(tr)) != (hi_of(ti) < 0 && !is_zero(ti));
    }
    const double m01 = neg_(ti), m10 = flip(ti, negate), m11 = flip(tr, negate);
    double xa = tr * j.xa + m01 * j.ya, yb = m10 * j.xb + m11 * j.yb;
    const double xb = tr * j.xb + m01 * j.yb, ya = m10 * j.xa + m11 * j.ya;
    if constexpr (parameter_plane) {
        if (j.k <= 600) {
            const double one = from_hilo((1023 - j.k) << 20, 0);
            xa = xa + one;
            yb = yb + one;
        } else if (bexp(xa) < 560 || bexp(yb) < 560) {
            return false;
        }
    }
    j.xa = xa;
    j.xb = xb;
    j.ya = ya;
    j.yb = yb;
    if (imax(imax(bexp(xa), bexp(xb)), imax(bexp(ya), bexp(yb))) > 1023 + 300) {
        const auto low = [](double v) { return is_zero(v) ? 2046 : bexp(v); };
        if (imin(imin(low(xa), low(xb)), imin(low(ya), low(yb))) - 300 >= kRawLow) {
            const auto down = [](double v) { return is_zero(v) ? v : add_exp(v, -300); };
            j = RawJac{down(xa), down(xb), down(ya), down(yb), j.k + 300};
        }
    }
    return true;
}

// alt_step on raw values: 7 products and 5 to 7 sums.  For the burning ship
// the signs of |Z| cancel to one sign on the imaginary part, and a step
// where a part of Z + d crosses zero (`fold`: 18 % of a 1e40 view's steps)
// runs the same products and sums on Z + d and the record's constant, so
// folding lanes do not leave the others.
template <int Formula>
__device__ __forceinline__ Sc alt_step_raw(const double2& z, const Sc& d, const Sc& pd, bool fold, const Sc& total,
                                           const double2& constant) {
    const double z2r = twice_raw(z.x), z2i = twice_raw(z.y);
    double lr = z2r * d.re - z2i * d.im;
    double li = z2r * d.im + z2i * d.re;
    if constexpr (Formula == kFormulaBurningShip) {
        const double u = choose(fold, total.re, d.re), v = choose(fold, total.im, d.im);
        const double sr = u * u - v * v;
        const double si = twice_raw(u * v);
        const bool s = !fold && (hi_of(z.x) ^ hi_of(z.y)) < 0;
        const double tr = choose(fold, constant.x, lr) + choose(fold, pd.re, sr);
        const double ti = choose(fold, constant.y, li) + choose(fold, pd.im, si);
        return sc_make(tr + choose(fold, sr, pd.re), flip(ti, s) + choose(fold, fabs_(si), pd.im), 0);
    }
    const double sr = d.re * d.re - d.im * d.im;
    const double si = twice_raw(d.re * d.im);
    if constexpr (Formula == kFormulaTricorn) {
        return add_cut(sc_make(lr, neg_(li), 0), add_cut(sc_make(sr, neg_(si), 0), pd));
    }
    return add_cut(sc_make(lr, li, 0), sc_make(sr, si, 0));
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

// Whether alt_search certainly finds no block for delta d at `offset`: no
// block of two steps starts at an odd offset, and with E the exponent of d's
// larger part (which is at least 2^(E - 1)) |d|^2 >= 2^(2E - 2), while
// r2 < 2^r2.e.
__device__ __forceinline__ bool no_block(const AltParams& p, int offset, const Sc& d) {
    if (offset < 0 || offset >= p.alt_index.count[0] || (offset & 1) != 0) return true;
    if ((offset >> 1) >= p.alt_index.count[1]) return false;
    const AltStep* s = p.alt + p.alt_index.offset[1] + (offset >> 1);
    const int high = __ldg(reinterpret_cast<const int*>(&s->r2.m) + 1);
    const int e = __ldg(&s->r2.e);
    const int top = imax(bexp(d.re), bexp(d.im));
    return (high & 0x7ff00000) != 0x7ff00000 && is_normal(top)
        && 2LL * (static_cast<long long>(d.e) + top - 1022) - 2 >= e;
}

__device__ const AltStep* alt_lookup(const AltParams& p, int start, const Sc& d, const Fe& pn, int max_length) {
    if (p.alt_index.levels == 0 || max_length <= 0 || !sc_finite(d) || !fe_finite(pn)) return nullptr;
    int top = 31 - __clz(max_length);
    top = top < p.alt_index.levels - 1 ? top : p.alt_index.levels - 1;
    if (top < 1 || no_block(p, start - p.alt_start, d)) return nullptr;
    return alt_search(p, start - p.alt_start, d, pn, top);
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

// One pixel's state.  It lives in local memory: the raw loop below keeps
// the few values it needs in registers, everything else is touched only on
// the rare general turns.  delta and pd are raw values where their range
// allows (raw_double.h); total is kept once the orbit has ended (`past`).
template <bool WithPlanes>
struct AltLane {
    long long index;
    Sc dc, pd, delta, total, tortoise;
    Sc prior;   // total before the step whose escape test is pending, or of the escape
    Fe pn;
    Nrm norm;   // escape norm of a pixel that has escaped
    Jac jac;
    int ref, it, power, length, hits;
    unsigned ticks;
    bool ready, past, pending;
};

// A pixel between rounds, as it waits on a list: 128 bytes.  Only pixels
// without cycle state are listed.
struct alignas(128) AltSaved {
    long long index;
    Sc dc;
    Sc value;  // delta, or total past the orbit's end
    Jac jac;
    int ref;   // -1 past the orbit's end
    int it;
};
static_assert(sizeof(AltSaved) == 128, "one cache line");

enum AltOutcome { kAltContinue = 0, kAltDone, kAltEscaped };

__device__ __forceinline__ void alt_store(const AltParams& p, long long index, float out, std::uint32_t count) {
    p.out[index] = out;
    if (p.counts) p.counts[index] = count;
}

template <bool WithPlanes>
__device__ __forceinline__ AltOutcome alt_interior(const AltParams& p, long long index) {
    if constexpr (WithPlanes) Planes{p.p_iter, p.p_phase, p.p_dex, p.p_dey, p.p_t1, p.p_t2}.clear(index, p.max_iter);
    alt_store(p, index, static_cast<float>(static_cast<double>(p.max_iter) - p.output_bias),
              static_cast<std::uint32_t>(p.max_iter));
    return kAltDone;
}

__device__ __noinline__ Sc alt_total(const AltParams& p, int ref, Sc delta) {
    sc_normalize(delta);
    return sc_add(ld_sc(&p.orbit[ref].z), delta);
}

// What an escaped pixel leaves for its outputs, parked in shared memory until
// a warp has 32: the logarithms, hypot, atan2 and divisions are several
// hundred FP64 instructions, which cost the same for one lane as for all.
template <bool WithPlanes>
struct AltEnd {
    long long index;
    Nrm norm;
    int it;
};
template <>
struct AltEnd<true> {
    long long index;
    Nrm norm;
    Sc total;
    Nrm prior;
    Jac jac;
    int it;
};
constexpr int kAltPark = 64;  // fewer than 32 waiting, and up to 32 more

template <bool WithPlanes, int Formula>
__device__ __noinline__ void alt_finish(const AltParams& p, const AltEnd<WithPlanes>& e) {
    if constexpr (WithPlanes) {
        const Planes planes{p.p_iter, p.p_phase, p.p_dex, p.p_dey, p.p_t1, p.p_t2};
        const int raw = Formula == kFormulaJulia ? e.it : (e.it - 1 > 0 ? e.it - 1 : 0);
        planes.escape(e.index, raw, normal_form(e.total), e.prior, jac_normal(e.jac), p.pixel_spacing);
    }
    alt_store(p, e.index, smooth_escape(e.it, e.norm, p.output_bias), static_cast<std::uint32_t>(e.it));
}

// The escape test after a perturbation step to s.ref, s.prior being the
// total before it.
template <bool WithPlanes>
__device__ __noinline__ bool alt_escaped(const AltParams& p, AltLane<WithPlanes>& s) {
    if (alt_inside(p, s.ref, s.delta)) return false;
    const Fe margin = alt_margin(p, s.ref, s.delta);
    s.norm = nrm_from_margin(margin, p.escape_mode);
    if (!fe_positive(margin) && !nrm_outside(s.norm, p.escape_mode)) return false;
    if constexpr (WithPlanes) s.total = alt_total(p, s.ref, s.delta);
    return true;
}

template <bool WithPlanes>
__device__ __forceinline__ void alt_save(const AltLane<WithPlanes>& s, AltSaved& e) {
    e.index = s.index;
    e.dc = s.dc;
    e.value = s.past ? s.total : s.delta;
    if constexpr (WithPlanes) e.jac = s.jac;
    e.ref = s.past ? -1 : s.ref;
    e.it = s.it;
}

// What does not change from step to step, from the pixel's offset dc.
template <bool WithPlanes, int Formula>
__device__ __forceinline__ void alt_reset(AltLane<WithPlanes>& s, const Sc& dc) {
    constexpr bool julia = Formula == kFormulaJulia;
    const Nrm pnorm = julia ? nrm_make(0.0, 0) : sc_norm2(dc);
    s.dc = dc;
    s.pd = julia ? sc_zero() : to_raw(dc);
    s.pn = fe_make(pnorm.m, pnorm.e);
    s.total = s.tortoise = s.prior = sc_zero();
    s.ticks = 0;
    s.past = s.pending = s.ready = false;
    s.power = 1;
    s.length = 0;
    s.hits = 0;
}

template <bool WithPlanes, int Formula>
__device__ __noinline__ void alt_restore(const AltParams& p, const AltSaved& e, AltLane<WithPlanes>& s) {
    alt_reset<WithPlanes, Formula>(s, e.dc);
    s.index = e.index;
    s.past = e.ref < 0;
    s.delta = e.value;
    if (s.past) s.total = e.value;
    if constexpr (WithPlanes) s.jac = e.jac;
    s.ref = s.past ? p.orbit_size - 1 : e.ref;
    s.it = e.it;
}

// Start pixel `index`: coordinates, Julia series jump, first escape test.
template <bool WithPlanes, int Formula>
__device__ __noinline__ AltOutcome alt_begin(const AltParams& p, long long index, AltLane<WithPlanes>& s) {
    constexpr bool julia = Formula == kFormulaJulia;
    const int py = static_cast<int>(index / p.width);
    const int px = static_cast<int>(index - static_cast<long long>(py) * p.width);
    if constexpr (WithPlanes) Planes{p.p_iter, p.p_phase, p.p_dex, p.p_dey, p.p_t1, p.p_t2}.clear(index, p.max_iter);
    const double xf = pixel_offset(px, p.width, p.coordinate_mode) / static_cast<double>(p.width);
    const double yf = -pixel_offset(py, p.height, p.coordinate_mode) / static_cast<double>(p.height);
    const Sc dc = p.points ? sc_make(p.points[index].re, p.points[index].im, p.points[index].e)
                           : sc_from_fe(fe_mul(p.view_width, xf), fe_mul(p.view_height, yf));
    Sc delta = dc;
    Jac jac = jac_identity();
    int at = julia ? 0 : 1;
    if (p.series_on && nrm_cmp(sc_norm2(dc), p.series_r2) <= 0) {
        Sc value = ld_sc(&p.series[p.series_terms - 1]);
        Sc poly = sc_zero();
        for (int k = p.series_terms - 1; k > 1; --k) {
            if constexpr (WithPlanes) poly = sc_add(sc_mul(poly, dc), value);
            value = sc_add(sc_mul(value, dc), ld_sc(&p.series[k - 1]));
        }
        delta = sc_mul(value, dc);
        if constexpr (WithPlanes) jac = jac_holomorphic(sc_add(sc_mul(poly, dc), value));
        at = p.series_iteration;
    }
    alt_reset<WithPlanes, Formula>(s, dc);
    s.index = index;
    s.delta = to_raw(delta);
    s.jac = jac_pack(jac);
    s.ref = at;
    s.it = at;
    if (!alt_inside(p, at, s.delta)) {
        s.norm = nrm_from_margin(alt_margin(p, at, s.delta), p.escape_mode);
        if (nrm_outside(s.norm, p.escape_mode)) {
            if constexpr (WithPlanes) s.total = alt_total(p, at, s.delta);
            return kAltEscaped;
        }
    }
    return kAltContinue;
}

// Square of a value below 2^128 in magnitude, low to about 2^-19, from its
// high word.
__device__ __forceinline__ float square_estimate(double v) {
    const float f = __int_as_float(imax((hi_of(v) & 0x7fffffff) - (896 << 20), 0) << 3);
    return f * f;
}

// High words of magnitudes: they order values to 2^-20.
constexpr int kHighLow = kRawLow << 20;                                 // 2^-400
constexpr int kHighTop = (kRawLow + static_cast<int>(kRawSpan)) << 20;  // 2^10
constexpr int kHighJac = (1023 + 300) << 20;
__device__ __forceinline__ int high(double v) { return hi_of(v) & 0x7fffffff; }

// Up to `limit` exact steps on raw values, the hot loop: it stops before a
// step that needs the general turn (a block may apply, a value out of range,
// the orbit's end, the cap) and after one whose escape or cycle test the
// general turn must settle (`pending`).  Returns the steps taken.
//
// FP64 instructions per step: 14 (12 for Julia), with planes 16 more (the
// total and the Jacobian).  Long orbits run few to an SM, where a step costs
// its instructions' issue and latency, so the usual step (`plain`) has every
// test on high words: nonzero parts in range, no block as large as the
// delta, and exponents near enough that no shared-exponent sum drops an
// operand (2 Z d and d^2 differ by the exponents of 2 Z and d, to within 4).
// The other steps on raw values take the longer form, among them every step
// of a reference on an axis, whose orbit has zero parts.
template <bool WithPlanes, int Formula>
__device__ __forceinline__ int alt_raw_run(const AltParams& p, AltLane<WithPlanes>& s, int limit) {
    const Sc pd = s.pd;
    Sc d = s.delta;
    RawJac j{};
    bool fits = !s.past && !s.pending && d.e == 0 && pd.e == 0 && raw_or_zero(pd.re) && raw_or_zero(pd.im);
    if constexpr (WithPlanes) {
        j = RawJac{s.jac.xa.m, s.jac.xb.m, s.jac.ya.m, s.jac.yb.m, s.jac.xa.e};
        fits = fits && j.k == s.jac.xb.e && j.k == s.jac.ya.e && j.k == s.jac.yb.e;
    }
    if (!fits) return 0;
    const int first = s.ref;
    const int room = imin(imin(limit, p.max_iter - s.it), p.orbit_size - 1 - first);
    const bool blocks = !p.disable_bla && p.alt_index.levels > 1;
    // |d|^2 >= 2^(2E - 2) with E = top - 1022: no block from this top on.
    const int block_top = blocks ? imin(imax(p.block_top, -4000), 4000) : -4000;
    const int cycle_from = p.cycle ? 2048 : INT_MAX;
    const int pd_top = imax(bexp(pd.re), bexp(pd.im));
    const OrbitRec* r = p.orbit + first;
    double2 z = __ldg(reinterpret_cast<const double2*>(r));
    int4 head = __ldg(reinterpret_cast<const int4*>(&r->zf_re));
    const float bound = (p.escape_mode == 1 ? 1.0e8f : 4.0f) * (1.0f - 0x1p-14f);
    const float far = (p.escape_mode == 1 ? 1.0e8f : 4.0f) * 16.0f;
    Sc total = sc_make(z.x + d.re, z.y + d.im, 0);  // kept with planes only
    Sc prior = sc_zero();
    int k = 0;
    bool pending = false;
#pragma unroll 1
    while (k < room) {
        const int flags = head.z;
        if (!(flags & (kRawOrbit | kRawZero))) break;
        const int dr = high(d.re), di = high(d.im);
        const int most = imax(dr, di), top = most >> 20;
        bool plain = (flags & kRawOrbit) && imin(dr, di) >= kHighLow && most <= kHighTop && 2 * (top - 1023) >= block_top
            && static_cast<unsigned>(head.w + 1 - top + 55) <= 110u;
        if constexpr (WithPlanes) {
            const int a = high(j.xa), b = high(j.xb), c = high(j.ya), e = high(j.yb);
            plain = plain && imin(imin(a, b), imin(c, e)) >= kHighLow && imax(imax(a, b), imax(c, e)) <= kHighJac
                && imin(high(total.re), high(total.im)) >= kHighLow;
            if constexpr (Formula != kFormulaJulia) plain = plain && static_cast<unsigned>(j.k + 400) <= 1000u;
        }
        bool with_pd = true;
        if constexpr (Formula == kFormulaTricorn) {
            // d^2 and pd: near enough to add, or pd dropped.
            const int apart = 2 * top - 1023 - pd_top;
            with_pd = apart < 60;
            plain = plain && (apart > 65 || static_cast<unsigned>(apart + 55) <= 110u);
        }
        bool fold = false;
        double2 constant{0.0, 0.0};
        if constexpr (Formula == kFormulaBurningShip) {
            fold = folds(z.x, d.re) || folds(z.y, d.im);
            if (fold) {
                if (!(flags & kRawFold)) break;
                constant = make_double2(__ldg(&r->fold[0]), __ldg(&r->fold[1]));
            }
            if (!WithPlanes && fold) total = sc_make(z.x + d.re, z.y + d.im, 0);
            plain = plain && (!fold || imin(high(total.re), high(total.im)) >= kHighLow);
        }
        const double2 zn = __ldg(reinterpret_cast<const double2*>(r + 1));
        head = __ldg(reinterpret_cast<const int4*>(&r[1].zf_re));
        if (plain) {
            // Products on the integer pipe, sums in FP64 beside them
            // (int_mul.h).
            const double z2r = add_exp(z.x, 1), z2i = add_exp(z.y, 1);
            std::uint32_t low = ~0u;
            RawJac nj = j;
            Sc nd = d;
            if constexpr (WithPlanes) {
                const double tr = add_exp(total.re, 1), ti = add_exp(total.im, 1);
                const FactorA fr = factor_a(tr), fi = factor_a(ti);
                const FactorB fxa = factor_b(j.xa), fya = factor_b(j.ya);
                const double rxa = int_mul(fr, fxa, low), iya = int_mul(fi, fya, low);
                const double ixa = int_mul(fi, fxa, low), rya = int_mul(fr, fya, low);
                const FactorB fxb = factor_b(j.xb), fyb = factor_b(j.yb);
                const double rxb = int_mul(fr, fxb, low), iyb = int_mul(fi, fyb, low);
                const double ixb = int_mul(fi, fxb, low), ryb = int_mul(fr, fyb, low);
                int sign = Formula == kFormulaTricorn ? static_cast<int>(0x80000000u) : 0;
                if constexpr (Formula == kFormulaBurningShip) {
                    sign = (hi_of(tr) ^ hi_of(ti)) & static_cast<int>(0x80000000u);
                }
                double xa = rxa - iya, yb = ixb + ryb;
                const double xb = rxb - iyb, ya = ixa + rya;
                yb = from_hilo(hi_of(yb) ^ sign, lo_of(yb));
                if constexpr (Formula != kFormulaJulia) {
                    // The +1, 2^-k here, does not move a sum 60 binades above it.
                    if (imin(bexp(xa), bexp(yb)) <= 1023 - j.k + 60) {
                        const double one = from_hilo((1023 - j.k) << 20, 0);
                        xa = xa + one;
                        yb = yb + one;
                    }
                }
                nj.xa = xa;
                nj.xb = xb;
                nj.ya = from_hilo(hi_of(ya) ^ sign, lo_of(ya));
                nj.yb = yb;
            }
            const FactorA fr = factor_a(d.re), fi = factor_a(d.im);
            const FactorB gr = factor_b(z2r), gi = factor_b(z2i);
            const double rr = int_mul(fr, gr, low), ii = int_mul(fi, gi, low);
            const double ri = int_mul(fi, gr, low), ir = int_mul(fr, gi, low);
            if constexpr (Formula == kFormulaBurningShip) {
                const double u = choose(fold, total.re, d.re), v = choose(fold, total.im, d.im);
                const FactorA eu = factor_a(u), ev = factor_a(v);
                const FactorB hu = factor_b(u), hv = factor_b(v);
                const double uu = int_mul(eu, hu, low), vv = int_mul(ev, hv, low), uv = int_mul(eu, hv, low);
                const double lr = rr - ii, li = ri + ir;
                const double sr = uu - vv, si = add_exp(uv, 1);
                const bool flipped = !fold && (hi_of(z.x) ^ hi_of(z.y)) < 0;
                double xr = choose(fold, constant.x, lr) + choose(fold, pd.re, sr);
                double xi = choose(fold, constant.y, li) + choose(fold, pd.im, si);
                xi = flip(xi, flipped);
                // pd does not move a sum 60 binades above it.
                if (fold || imin(bexp(xr), bexp(xi)) <= pd_top + 60) {
                    xr = xr + choose(fold, sr, pd.re);
                    xi = xi + choose(fold, fabs_(si), pd.im);
                }
                nd.re = xr;
                nd.im = xi;
            } else {
                const FactorB hr = factor_b(d.re), hi = factor_b(d.im);
                const double uu = int_mul(fr, hr, low), vv = int_mul(fi, hi, low), uv = int_mul(fr, hi, low);
                const double lr = rr - ii, li = ri + ir;
                const double sr = uu - vv, si = add_exp(uv, 1);
                if constexpr (Formula == kFormulaTricorn) {
                    if (with_pd) {
                        // This sum may cancel, so the outer one is checked.
                        nd = add_cut(sc_make(lr, neg_(li), 0), sc_make(sr + pd.re, pd.im - si, 0));
                    } else {
                        nd.re = lr + sr;
                        nd.im = neg_(li + si);
                    }
                } else {
                    nd.re = lr + sr;
                    nd.im = li + si;
                }
            }
            // A product that may be a tie: the longer form multiplies in FP64.
            plain = low != 0u;
            if (plain) {
                if constexpr (WithPlanes) prior = total;
                j = nj;
                d = nd;
            }
        }
        if (!plain) {
            if (!raw_or_zero(d.re) || !raw_or_zero(d.im)) break;
            if (blocks && !no_block(p, first + k - p.alt_start, d)) break;
            if constexpr (WithPlanes) {
                prior = add_cut(sc_make(z.x, z.y, 0), d);
                if (!jac_step_raw<Formula>(prior, j)) break;
            }
            d = alt_step_raw<Formula>(z, d, pd, fold, total, constant);
        }
        ++k;
        ++r;
        z = zn;
        // alt_inside at the new index: with planes from the total, which the
        // next step reads; else from FP32 estimates of both terms.
        bool inside;
        if constexpr (WithPlanes) {
            total = sc_make(z.x + d.re, z.y + d.im, 0);
            inside = square_estimate(total.re) + square_estimate(total.im) < bound;
        } else {
            const float dx = float_of(d.re, 0), dy = float_of(d.im, 0);
            const float tx = __int_as_float(head.x) + dx, ty = __int_as_float(head.y) + dy;
            inside = tx * tx + ty * ty < bound && dx * dx + dy * dy < far;
        }
        const int it = s.it + k;
        if (!inside || (it >= cycle_from && (it & 31) == 0)) {
            pending = true;
            break;
        }
    }
    s.delta = d;
    s.ref = first + k;
    s.it += k;
    s.pending = pending;
    if constexpr (WithPlanes) {
        s.prior = prior;
        s.jac = Jac{fe_make(j.xa, j.k), fe_make(j.xb, j.k), fe_make(j.ya, j.k), fe_make(j.yb, j.k)};
    }
    return k;
}

// The bounded cycle, confirmed three times (non-strict renders only).
template <bool WithPlanes>
__device__ __noinline__ bool alt_cycle(const AltParams& p, AltLane<WithPlanes>& s) {
    const Nrm total_norm = nrm_from_margin(alt_margin(p, s.ref, s.delta), p.escape_mode);
    if (nrm_cmp(total_norm, nrm_make(0.75, 2)) >= 0) return false;
    const Sc total = alt_total(p, s.ref, s.delta);
    if (!s.ready) {
        s.tortoise = total;
        s.power = 1;
        s.length = 0;
        s.hits = 0;
        s.ready = true;
        return false;
    }
    const Nrm dist = sc_norm2(sc_sub(total, s.tortoise));
    const int scale_e = total_norm.e > 0 ? total_norm.e : 0;
    if (is_zero(dist.m) || dist.e <= scale_e - 78) {
        if (++s.hits >= 3) return true;
    } else {
        s.hits = 0;
    }
    if (++s.length >= s.power) {
        s.tortoise = total;
        s.power = s.power * 2 < (1 << 20) ? s.power * 2 : (1 << 20);
        s.length = 0;
    }
    return false;
}

// Formula steps past the orbit's end, up to kAltRound.
template <bool WithPlanes, int Formula>
__device__ __noinline__ AltOutcome alt_past(const AltParams& p, AltLane<WithPlanes>& s) {
    constexpr bool julia = Formula == kFormulaJulia;
    Sc total = s.past ? s.total : to_raw(alt_total(p, s.ref, s.delta));
    s.past = true;
    const Sc parameter = to_raw(julia ? p.parameter : sc_add(p.parameter, s.dc));
    const float bound = (p.escape_mode == 1 ? 1.0e8f : 4.0f) * (1.0f - 0x1p-14f);
    int it = s.it;
    AltOutcome outcome = kAltContinue;
#pragma unroll 1
    for (int k = 0; k < kAltRound && it < p.max_iter; ++k) {
        const Sc prior = total;
        // Raw step: 3 products and 3 sums.
        const bool raw = raw_value(prior) && parameter.e == 0;
        if constexpr (WithPlanes) {
            bool stepped = false;
            const Jac g = s.jac;
            if (raw && g.xa.e == g.xb.e && g.xa.e == g.ya.e && g.xa.e == g.yb.e) {
                RawJac j{g.xa.m, g.xb.m, g.ya.m, g.yb.m, g.xa.e};
                stepped = jac_step_raw<Formula>(prior, j);
                if (stepped) s.jac = Jac{fe_make(j.xa, j.k), fe_make(j.xb, j.k), fe_make(j.ya, j.k), fe_make(j.yb, j.k)};
            }
            if (!stepped) s.jac = jac_step_general(Formula, prior, g, !julia);
        }
        ++it;
        bool maybe_out = true;
        if (raw) {
            const bool negate = Formula == kFormulaTricorn
                || (Formula == kFormulaBurningShip && (hi_of(prior.re) ^ hi_of(prior.im)) < 0);
            total = add_cut(sc_make(prior.re * prior.re - prior.im * prior.im,
                                    flip(add_exp(prior.re * prior.im, 1), negate), 0), parameter);
            const float tx = float_of(total.re, 0), ty = float_of(total.im, 0);
            maybe_out = !(tx * tx + ty * ty < bound);
        } else {
            total = to_raw(formula_step<Formula>(prior, parameter));
        }
        if (maybe_out) {
            const Nrm norm = sc_norm2(normal_form(total));
            if (nrm_outside(norm, p.escape_mode)) {
                s.norm = norm;
                s.prior = prior;
                outcome = kAltEscaped;
                break;
            }
        }
    }
    s.total = total;
    s.it = it;
    return outcome;
}

// One general turn: a pending escape or cycle test, formula steps past the
// orbit's end, a BLA block (or its exact replay), or one exact step.
template <bool WithPlanes, int Formula>
__device__ __noinline__ AltOutcome alt_general(const AltParams& p, AltLane<WithPlanes>& s, int max_block) {
    constexpr bool julia = Formula == kFormulaJulia;
    const AltStep* step = nullptr;
    if (!s.pending) {
        if (s.it >= p.max_iter) return alt_interior<WithPlanes>(p, s.index);
        if (s.ref + 1 >= p.orbit_size) return alt_past<WithPlanes, Formula>(p, s);
        const int remaining = p.max_iter - s.it;
        if (!p.disable_bla) {
            step = alt_lookup(p, s.ref, s.delta, s.pn, max_block < remaining ? max_block : remaining);
        }
        int len = step != nullptr ? __ldg(&step->len) : 1;
        if (step != nullptr && s.ref + len < p.orbit_size) {
            const int end = s.ref + len;
            const Sc cand = apply_alt(step, s.delta, s.pd);
            // Accepted where the endpoint stays inside (|Z + d|^2 < 3; the
            // total is finite when the delta is).
            bool good = sc_finite(cand);
            if (good && !alt_below(p, end, cand, 3.0f)) {
                const Fe cmargin = alt_margin(p, end, cand);
                good = fe_finite(cmargin) && !fe_positive(cmargin)
                    && nrm_cmp(nrm_from_margin(cmargin, p.escape_mode), nrm_make(0.75, 2)) < 0;
            }
            if (good) {
                s.delta = to_raw(cand);
                if constexpr (WithPlanes) s.jac = jac_pack(jac_bla(step, s.jac, !julia));
                s.ref = end;
                s.it += len;
                return kAltContinue;
            }
        } else {
            step = nullptr;
            len = 1;
        }
        // Exact steps: one, or the refused block's replay (whose steps have
        // no cycle test of their own).
        for (int k = 0; k < len && s.it < p.max_iter; ++k) {
            if constexpr (WithPlanes) {
                s.prior = alt_total(p, s.ref, s.delta);
                s.jac = jac_step_general(Formula, s.prior, s.jac, !julia);
            }
            s.delta = to_raw(alt_step<Formula>(p, s.ref, s.delta, s.pd));
            ++s.ref;
            ++s.it;
            if (!sc_finite(s.delta)) {
                alt_store(p, s.index,
                          p.strict ? nan_f() : static_cast<float>(static_cast<double>(s.it) - p.output_bias),
                          p.strict ? 0u : static_cast<std::uint32_t>(s.it));
                return kAltDone;
            }
            if (alt_escaped<WithPlanes>(p, s)) return kAltEscaped;
        }
        if (step != nullptr) return kAltContinue;
    } else {
        s.pending = false;
        if (alt_escaped<WithPlanes>(p, s)) return kAltEscaped;
    }
    if (cycle_turn(p.cycle != 0, s.it) && alt_cycle<WithPlanes>(p, s)) {
        return alt_interior<WithPlanes>(p, s.index);
    }
    return kAltContinue;
}

__device__ __forceinline__ int alt_max_block(const AltParams& p) {
    return p.max_lin_len < 2 ? 2 : (p.max_lin_len > kMaxSafeLinearBlaLength ? kMaxSafeLinearBlaLength : p.max_lin_len);
}

__device__ __forceinline__ unsigned long long alt_deadline(const AltParams& p) {
    return p.deadline_base ? *p.deadline_base + p.budget_ns : 0ull;
}

// The lane-refill queue.  GB300 issues an FP64 warp instruction at the same
// cost whatever the number of active lanes, and neighbouring pixels run for
// different times: a lane per pixel left 8 of 32 lanes active on average on a
// burning-ship view at 1e40 and 7 on a Julia view at 1e24.  So persistent
// warps keep every lane busy: each lane holds one pixel, the warp runs rounds
// of kAltRound raw steps and a general turn for the lanes that stopped, and
// lanes whose pixel finished take new ones once at least kAltRefill of them
// wait.  A general turn is some 2000 instructions of mostly integer work, so
// it is shared too: lanes that need one wait until kAltRefill do, and 32
// neighbouring pixels are started together (one claim), run through their
// first blocks, which neighbours take in step, and kept on the warp's list
// of ready pixels.  Run by the lanes just refilled, the starts and blocks
// took 80 % of the instructions.
//
// In a field of several launches (alt_launch), once no pixel is left to take, a
// warp that has run kAltPatience rounds with fewer than kAltLeave active lanes
// leaves: it spills them to a list that the next launch takes as its input, so
// the few long orbits (10 % of a Julia view past 500 steps, 1 % to the cap) run
// 32 to a warp instead of one in each.  Lifetimes are close to exponential
// whatever their scale, so a rule on lanes suits every view where a budget of
// steps suits one; the patience lets pixels that all end soon end where they
// are (a burning-ship view's, 8.4 ms without it and 5.8 ms with it).  A list
// short enough to give every SM sub-partition one warp gains nothing from
// another launch and runs to its end.
constexpr int kAltRefill = 8;
constexpr int kAltPhases = 8;
constexpr int kAltLeave = 20;
constexpr int kAltPatience = 24;  // rounds: 384 steps
constexpr int kAltShort = 32 * 4 * 152;      // pixels: one full warp per SM sub-partition
constexpr int kAltBusyWarps = 8 * 152;       // warps that keep the FP64 pipe busy
constexpr long long kAltPhasePixels = 131072; // smaller fields run in one launch (alt_launch)

// Registers: the parameter-plane formulas, whose general turns wait for
// instructions, gain from four blocks (1280x720 with planes: 10.0 against
// 10.6 ms); the long Julia orbits of the last launch from none spilled
// (43.8 against 49.1 ms).
template <bool WithPlanes, int Formula>
__global__ void __launch_bounds__(128, Formula == kFormulaJulia ? 3 : 4) alt_queue_kernel(const __grid_constant__ AltParams p, unsigned long long* claim,
                                                        const AltSaved* source,
                                                        const unsigned long long* source_count,
                                                        AltSaved* spill, unsigned long long* spill_count,
                                                        unsigned long long spill_capacity, int leave,
                                                        AltSaved* ready_lists) {
    constexpr unsigned kFull = 0xffffffffu;
    __shared__ AltEnd<WithPlanes> parks[4][kAltPark];
    AltEnd<WithPlanes>* park = parks[threadIdx.x >> 5];
    const unsigned lane = threadIdx.x & 31u;
    const unsigned below = (1u << lane) - 1u;
    unsigned long long items = static_cast<unsigned long long>(p.width) * static_cast<unsigned long long>(p.height);
    if (source != nullptr) {
        items = *source_count;
        if (items > spill_capacity) items = spill_capacity;
        // Warps beyond the busy ones (taken round the blocks) do not start.
        const unsigned long long rank = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
        const unsigned long long warps = (items + 31) / 32;
        if (rank >= (warps < kAltBusyWarps ? warps : static_cast<unsigned long long>(kAltBusyWarps))) return;
        if (items <= kAltShort) leave = 0;
    }
    const unsigned long long deadline = alt_deadline(p);
    const int max_block = alt_max_block(p);
    AltLane<WithPlanes> s;
    bool have = false;
    bool keep = false;  // the list was full: run on
    bool wait = false;  // the lane's pixel needs a general turn
    bool drained = false;
    int parked = 0;
    int ready = 0;  // pixels on the warp's list
    int lean = 0;   // rounds with few lanes
    AltSaved* list = ready_lists + static_cast<std::size_t>(blockIdx.x * 4 + (threadIdx.x >> 5)) * kAltPark;
    // Park the escaped among the warp's lanes `l`; finish 32 when they are there.
    const auto park_escaped = [&](bool escaped, const AltLane<WithPlanes>& l) {
        const unsigned ended = __ballot_sync(kFull, escaped);
        if (ended == 0u) return;
        if (escaped) {
            AltEnd<WithPlanes>& e = park[parked + __popc(ended & below)];
            e.index = l.index;
            e.norm = l.norm;
            e.it = l.it;
            if constexpr (WithPlanes) {
                e.total = l.total;
                e.prior = sc_norm2(normal_form(l.prior));
                e.jac = l.jac;
            }
        }
        parked += __popc(ended);
        __syncwarp();
        if (parked >= 32) {
            parked -= 32;
            alt_finish<WithPlanes, Formula>(p, park[parked + static_cast<int>(lane)]);
            __syncwarp();
        }
    };
    while (true) {
        AltOutcome outcome = kAltContinue;
        const unsigned need = __ballot_sync(kFull, !have);
        const int n = __popc(need);
        if (n >= kAltRefill && !(drained && ready == 0)) {
            const int rank = __popc(need & below);
            if (source != nullptr) {
                unsigned long long base = 0;
                if (lane == 0) base = atomicAdd(claim, static_cast<unsigned long long>(n));
                base = __shfl_sync(kFull, base, 0);
                if (!have && base + rank < items) {
                    alt_restore<WithPlanes, Formula>(p, source[base + rank], s);
                    have = true;
                }
                drained = base + n >= items;
            } else {
                if (ready < n && !drained) {
                    unsigned long long base = 0;
                    if (lane == 0) base = atomicAdd(claim, 32ull);
                    base = __shfl_sync(kFull, base, 0);
                    AltLane<WithPlanes> t;
                    AltOutcome started = kAltDone;
                    if (base + lane < items) {
                        started = alt_begin<WithPlanes, Formula>(p, static_cast<long long>(base + lane), t);
                        while (started == kAltContinue) {
                            // The first turn and every 16th look at the clock:
                            // blocks alone may take a pixel to the cap.
                            if (deadline && (t.ticks++ & 15u) == 0u && t.it < p.max_iter && global_ns() >= deadline) {
                                alt_store(p, t.index, nan_f(), 0u);
                                started = kAltDone;
                                break;
                            }
                            if (p.disable_bla || p.alt_index.levels <= 1 || !turn_before_listing(p.cycle != 0, t.it)
                                || no_block(p, t.ref - p.alt_start, t.delta)) {
                                break;
                            }
                            started = alt_general<WithPlanes, Formula>(p, t, max_block);
                        }
                    }
                    drained = base + 32 >= items;
                    __syncwarp();
                    park_escaped(started == kAltEscaped, t);
                    const unsigned kept = __ballot_sync(kFull, started == kAltContinue);
                    if (started == kAltContinue) alt_save(t, list[ready + __popc(kept & below)]);
                    ready += __popc(kept);
                    __syncwarp();
                }
                if (!have && rank < ready) {
                    alt_restore<WithPlanes, Formula>(p, list[ready - 1 - rank], s);
                    have = true;
                }
                ready -= n < ready ? n : ready;
                __syncwarp();
            }
            if ((need >> lane) & 1u) {
                keep = false;
                wait = false;
            }
        }
        if (!__any_sync(kFull, have)) {
            if (drained && ready == 0) break;
            continue;
        }
        if (have && !wait) {
            wait = alt_raw_run<WithPlanes, Formula>(p, s, kAltRound) < kAltRound || s.pending;
        }
        const int waiting = __popc(__ballot_sync(kFull, have && wait));
        if (waiting >= kAltRefill || !__any_sync(kFull, have && !wait)) {
            if (have && wait) outcome = alt_general<WithPlanes, Formula>(p, s, max_block);
            wait = false;
        }
        if (have && outcome == kAltContinue && deadline && (s.ticks++ & 15u) == 0u && global_ns() >= deadline) {
            alt_store(p, s.index, nan_f(), 0u);
            outcome = kAltDone;
        }
        park_escaped(outcome == kAltEscaped, s);
        if (outcome != kAltContinue) have = false;
        if (leave > 0 && drained && ready == 0) {
            const unsigned left = __ballot_sync(kFull, have);
            const unsigned mask = __ballot_sync(kFull, have && !wait && !keep && !s.ready);
            if (__popc(left) < leave) ++lean;
            if (lean > kAltPatience && mask != 0u) {
                unsigned long long base = 0;
                if (lane == 0) base = atomicAdd(spill_count, static_cast<unsigned long long>(__popc(mask)));
                base = __shfl_sync(kFull, base, 0);
                const unsigned long long slot = base + static_cast<unsigned>(__popc(mask & below));
                if ((mask >> lane) & 1u) {
                    if (slot < spill_capacity) {
                        alt_save(s, spill[slot]);
                        have = false;
                    } else {
                        keep = true;
                    }
                }
            }
        }
    }
    if (static_cast<int>(lane) < parked) alt_finish<WithPlanes, Formula>(p, park[lane]);
}

template <bool WithPlanes, int Formula>
int alt_queue_blocks() {
    static int blocks = 0;
    if (blocks == 0) {
        int per_sm = 0, sms = 0, device = 0;
        cudaGetDevice(&device);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, alt_queue_kernel<WithPlanes, Formula>, 128, 0);
        blocks = (per_sm > 0 ? per_sm : 1) * (sms > 0 ? sms : 1);
    }
    return blocks;
}

// The launches of one field: `queue.counters` holds the claim counters and
// spill counts (kAltQueueCounters words), `queue.spill` two lists.
//
// Up to kAltPhasePixels one launch does everything.  The later ones cost 4 us
// each, which a field of short orbits does not get back (400x225 at 1e12: 95
// us with eight, 66 with one, 84 as one thread per pixel), and a field of long
// ones has little to regroup while the first launch's lanes (77,824) hold most
// of its pixels: 320x180 at 1e24 took 3.6 ms with eight and 2.3 with one for
// one Julia set, with planes 2.9 and 3.9 for another.
template <bool WithPlanes, int Formula>
cudaError_t alt_launch(const AltParams& p, const AltQueue& queue, cudaStream_t stream) {
    const long long pixels = static_cast<long long>(p.width) * p.height;
    const int phases = pixels > kAltPhasePixels && queue.spill != nullptr && queue.capacity > 0 ? kAltPhases : 1;
    const cudaError_t cleared =
        cudaMemsetAsync(queue.counters, 0, sizeof(unsigned long long) * kAltQueueCounters, stream);
    if (cleared != cudaSuccess) return cleared;
    auto* lists = static_cast<AltSaved*>(queue.spill);
    const long long resident = alt_queue_blocks<WithPlanes, Formula>();
    for (int phase = 0; phase < phases; ++phase) {
        // A field smaller than the persistent grid needs no more warps than
        // pixels / 32.
        const long long blocks = phase == 0 ? resident : std::min<long long>(resident, kAltBusyWarps / 4);
        const unsigned grid = static_cast<unsigned>(std::min<long long>(blocks, (pixels + 127) / 128));
        alt_queue_kernel<WithPlanes, Formula><<<grid, 128, 0, stream>>>(
            p, queue.counters + phase, phase == 0 ? nullptr : lists + ((phase - 1) & 1) * queue.capacity,
            phase == 0 ? nullptr : queue.counters + kAltPhases + phase - 1, lists + (phase & 1) * queue.capacity,
            queue.counters + kAltPhases + phase, static_cast<unsigned long long>(queue.capacity),
            phase + 1 < phases ? kAltLeave : 0, static_cast<AltSaved*>(queue.ready));
    }
    return cudaGetLastError();
}

}  // namespace

std::size_t alt_spill_entry_bytes() { return sizeof(AltSaved); }

// More entries than the lanes of a launch; none where one launch does.
long long alt_spill_capacity(long long pixels) {
    return pixels > kAltPhasePixels ? std::min<long long>(pixels, 1ll << 18) : 0;
}

// One list of kAltPark pixels per warp of the largest grid for the field.
std::size_t alt_ready_bytes(long long pixels) {
    const long long blocks = std::max({alt_queue_blocks<true, kFormulaJulia>(), alt_queue_blocks<false, kFormulaJulia>(),
                                 alt_queue_blocks<true, kFormulaBurningShip>(),
                                 alt_queue_blocks<false, kFormulaBurningShip>(),
                                 alt_queue_blocks<true, kFormulaTricorn>(), alt_queue_blocks<false, kFormulaTricorn>()});
    return static_cast<std::size_t>(std::min(blocks, (pixels + 127) / 128)) * 4 * kAltPark * sizeof(AltSaved);
}

cudaError_t launch_plain_alternate(const AltParams& p, bool planes, const AltQueue& queue, cudaStream_t stream) {
    static_assert(2 * kAltPhases <= kAltQueueCounters, "claim counters and spill counts");
    const auto launch = [&](auto formula) {
        return planes ? alt_launch<true, formula.value>(p, queue, stream)
                      : alt_launch<false, formula.value>(p, queue, stream);
    };
    if (p.formula == kFormulaJulia) return launch(std::integral_constant<int, kFormulaJulia>{});
    if (p.formula == kFormulaBurningShip) return launch(std::integral_constant<int, kFormulaBurningShip>{});
    return launch(std::integral_constant<int, kFormulaTricorn>{});
}

}  // namespace fgb
