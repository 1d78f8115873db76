// Direct (shallow) field render in plain double: a persistent lane-refill
// queue over a batch of fields.
//
// Restates render_direct_scalar_formula and render_direct_with_planes_formula
// (renderer.cpp:10054-10135, 10281-10438): cardioid/bulb culling for the
// Mandelbrot set, z^2 + c for the four formulas with the same operation
// order as the reference (the alternate maps keep separate products, which
// this --fmad=false translation unit guarantees for every formula), escape at
// |z|^2 > R^2 and smooth value n + 1 - log(log|z|)/log 2.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "device.h"
#include "int_mul.h"

namespace fgb {
namespace {

using namespace fx;

constexpr double kLogTwoD = 0.6931471805599453094;  // log(2.0) as a double
constexpr double kTwoPi = 6.283185307179586476925286766559005768;

template <int Formula>
__device__ __forceinline__ void step(double zr, double zi, double pr, double pi, double& nr, double& ni) {
    if constexpr (Formula == kFormulaBurningShip) {
        const double ar = fabs_(zr);
        const double ai = fabs_(zi);
        const double rs = ar * ar;
        const double is = ai * ai;
        const double cross = 2.0 * ar * ai;
        const double diff = rs - is;
        ni = cross + pi;
        nr = diff + pr;
    } else if constexpr (Formula == kFormulaTricorn) {
        const double rs = zr * zr;
        const double is = zi * zi;
        const double cross = -2.0 * zr * zi;
        const double diff = rs - is;
        ni = cross + pi;
        nr = diff + pr;
    } else {
        // Mandelbrot and Julia share the map; only the start point differs.
        nr = zr * zr - zi * zi + pr;
        ni = 2.0 * zr * zi + pi;
    }
}

__device__ bool direct_de(double zr, double zi, double dr, double di, const Fe& spacing, double& out_re,
                          double& out_im) {
    const Sc total = sc_from_fe(fe_from(zr, 0), fe_from(zi, 0));
    const Sc derivative = sc_from_fe(fe_from(dr, 0), fe_from(di, 0));
    const double mag = hypot(total.re, total.im);
    if (!(mag > 0.0) || !is_finite(mag)) return false;
    const double log_mag = log(mag) + static_cast<double>(total.e) * 0.693147180559945309417232121458176568;
    if (!(log_mag > 0.0) || !is_finite(log_mag)) return false;
    const double ur = total.re / mag;
    const double ui = total.im / mag;
    const Sc unit = sc_from_fe(fe_from(ur, 0), fe_from(ui, 0));
    const Sc spacing_c = sc_from_fe(spacing, fe_zero());
    const Sc den = sc_mul(unit, sc_mul(sc_conj(derivative), spacing_c));
    const double den2 = den.re * den.re + den.im * den.im;
    if (!(den2 > 0.0) || !is_finite(den2)) return false;
    Sc r = sc_make(mag * log_mag * den.re / den2, -mag * log_mag * den.im / den2,
                   sat_exp(static_cast<long long>(total.e) - den.e));
    sc_normalize(r);
    out_re = sc_re_d(r);
    out_im = sc_im_d(r);
    return is_finite(out_re) && is_finite(out_im);
}

// The cross term of a step in FP64, as the reference orders it; out of line,
// for the few operands the integer product does not take.
template <int Formula>
__device__ __noinline__ double cross_general(double zr, double zi) {
    if constexpr (Formula == kFormulaBurningShip) return 2.0 * fabs_(zr) * fabs_(zi);
    if constexpr (Formula == kFormulaTricorn) return -2.0 * zr * zi;
    return 2.0 * zr * zi;
}
__device__ __noinline__ double square_general(double v) { return v * v; }

// Parts whose products with each other stay normal: 2^-500 to 2^500.
__device__ __forceinline__ bool product_range(double v) {
    return static_cast<unsigned>((hi_of(v) & 0x7fffffff) - (523 << 20)) < (1000u << 20);
}

// (2 zr) zi (signs as the formula has them) on the integer pipe: the exact
// product rounded once, doubled by its exponent, which is the reference's
// (2 zr) zi bit for bit in this range.  A zero factor gives the signed zero
// of the product.  Returns false where the value is not to be used.
//
// Beside the FP32 queue, which needs the issue slots (85 % taken) and leaves
// the FP64 pipe alone, the product is an FP64 one (`Integer` false): the 1e100
// atlas step took 16.8 ms with integer products in its direct levels.
template <int Formula, bool Integer>
__device__ __forceinline__ bool cross_product(double zr, double zi, double& cross) {
    if constexpr (!Integer) {
        const double product = Formula == kFormulaBurningShip ? fabs_(zr) * fabs_(zi) : zr * zi;
        const bool zero = is_zero(zr) || is_zero(zi);
        const bool fits = static_cast<unsigned>(bexp(product) - 2) < 2044u;
        cross = fits ? add_exp(product, 1) : product;
        if constexpr (Formula == kFormulaTricorn) cross = neg_(cross);
        return fits || zero;
    }
    FactorA a = factor_a(zr);
    FactorB b = factor_b(zi);
    if constexpr (Formula == kFormulaBurningShip) {
        a.x &= 0x7ff00000;
        b.x &= 0x7ff00000;
    } else if constexpr (Formula == kFormulaTricorn) {
        a.x ^= static_cast<int>(0x80000000u);
    }
    std::uint32_t low = ~0u;
    const int sign = (a.x ^ b.x) & static_cast<int>(0x80000000u);
    a.x += 1 << 20;
    cross = int_mul(a, b, low);
    if (low == 0u) cross = int_mul_even(a, b);
    const bool zero = is_zero(zr) || is_zero(zi);
    if (zero) cross = from_hilo(sign, 0);
    return zero ? is_finite(zr) && is_finite(zi) : product_range(zr) && product_range(zi);
}

template <bool Integer>
__device__ __forceinline__ bool square_product(double v, double& square) {
    if constexpr (!Integer) {
        square = v * v;
        return true;
    }
    std::uint32_t low = ~0u;
    FactorA a = factor_a(v);
    const FactorB b = factor_b(v);
    square = int_mul(a, b, low);
    if (low == 0u) square = int_mul_even(a, b);
    if (is_zero(v)) square = 0.0;
    return is_zero(v) || product_range(v);
}

__device__ __forceinline__ unsigned long long dbits(double v) {
    return static_cast<unsigned long long>(__double_as_longlong(v));
}

// The reference's escape test m2 > R^2 with m2 = RN(a + b), a = zr*zr and
// b = zi*zi (so a, b >= +0), decided on the bit patterns without an FP64
// instruction: a lone term above R^2 (or infinite / NaN) escapes, two terms
// at most R^2/2 cannot, and in between the exact sum is compared with the
// rounding midpoint above R^2 in integer units of half an ulp of R^2 (ties
// to even, as the FP64 add rounds).  R^2 is a normal double above 2.
__device__ __forceinline__ bool sum_exceeds(unsigned long long a, unsigned long long b, unsigned long long r2) {
    constexpr unsigned long long kMant = (1ull << 52) - 1;
    constexpr unsigned long long kMag = 0x7fffffffffffffffull;
    a &= kMag;
    b &= kMag;
    if (a < b) {
        const unsigned long long t = a;
        a = b;
        b = t;
    }
    if (a > r2) return true;
    if (a <= r2 - (1ull << 52)) return false;
    const int er = static_cast<int>(r2 >> 52);
    const unsigned long long mr = (r2 & kMant) | (1ull << 52);
    const int ea = static_cast<int>(a >> 52);
    const unsigned long long big = ((a & kMant) | (1ull << 52)) << (ea - er + 1);
    int eb = static_cast<int>(b >> 52);
    unsigned long long mb = b & kMant;
    if (eb == 0) {
        eb = 1;
    } else {
        mb |= 1ull << 52;
    }
    const int shift = eb - er + 1;
    unsigned long long small;
    bool below = false;  // bits of b under the unit
    if (shift >= 0) {
        small = mb << shift;
    } else if (shift > -64) {
        small = mb >> -shift;
        below = (mb & ((1ull << -shift) - 1)) != 0;
    } else {
        small = 0;
        below = mb != 0;
    }
    const unsigned long long sum = big + small;
    const unsigned long long midpoint = 2 * mr + 1;
    if (sum != midpoint) return sum > midpoint;
    return below || (mr & 1) != 0;
}

// Per-lane state of one pixel in flight.
struct Lane {
    double zr, zi;      // z_n
    double rs, is;      // zr*zr, zi*zi of z_n (the escape test's products)
    double pr, pi;      // additive parameter
    double dr, di;      // derivative (planes with DE only)
    double test1, test2;
    double escape2;
    unsigned long long saved_r, saved_i;  // cycle probe (Brent): z at the last power of two
    unsigned long long mark_r, mark_i;    // and z at the last multiple of 64 steps
    int it;             // completed steps
    int check_at;
    int max_iter;
    int stop_at;        // spill when `it` reaches this (phase budget)
    int field;
    int local;          // pixel index inside the field
};

// Step at which a fresh pixel is spilled (the cap when spilling is off).
__device__ __forceinline__ int budget_stop(const DirectBatch& b, int max_iter) {
    if (b.budget <= 0 || b.spill_capacity <= 0) return max_iter;
    return b.budget < max_iter ? b.budget : max_iter;
}

// direct_run for an orbit on the real axis (a row of every view centred there
// with an odd height, the period-2 point of a Julia set with a real constant):
// one square and one sum a step.  The imaginary part stays a zero, negative
// where the cross term and the parameter's zero both are.  As general steps,
// one a round, these pixels held up a 400x225 whole-set view: 6.5 ms, 3.0 ms
// here.
template <int Formula>
__device__ __forceinline__ int direct_run_real(Lane& l, int room, unsigned saved, unsigned mark) {
    const unsigned long long r2 = dbits(l.escape2);
    const int added = hi_of(l.pi);
    double zr = l.zr, rs = l.rs;
    int sign = hi_of(l.zi);
    int k = 0;
#pragma unroll 1
    for (; k < room; ++k) {
        const double nr = rs + l.pr;
        const int hr = hi_of(nr) & 0x7fffffff;
        const double nrs = int_mul_even(factor_a(nr), factor_b(nr));
        if (hr < (523 << 20) || hr >= (1523 << 20) || lo_of(nr) == saved || lo_of(nr) == mark || dbits(nrs) > r2) break;
        int cross = sign ^ hi_of(zr);
        if constexpr (Formula == kFormulaBurningShip) cross = 0;
        if constexpr (Formula == kFormulaTricorn) cross = ~cross;
        sign = cross & added;
        zr = nr;
        rs = nrs;
    }
    l.zr = zr;
    l.zi = from_hilo(sign & static_cast<int>(0x80000000u), 0);
    l.rs = rs;
    l.is = 0.0;
    l.it += k;
    return k;
}

// Up to `limit` steps of a spilled pixel on the integer and FP64 pipes, each
// with its tests on single words: it stops before a step that escapes, may
// close a cycle or moves the cycle marks (multiples of 64; spilled pixels are
// past 64 steps), or whose parts are out of range, which the general step
// then repeats.  Returns the steps taken.  Spilled pixels give each
// sub-partition few warps, where a step costs its instructions: 110 here
// against 250.
template <int Formula>
__device__ __forceinline__ int direct_run(Lane& l, int limit) {
    const int room = min(min(limit, l.max_iter - 1 - l.it), 63 - (l.it & 63));
    if (room <= 0 || !product_range(l.zr)) return 0;
    const unsigned saved = lo_of(__longlong_as_double(static_cast<long long>(l.saved_r)));
    const unsigned mark = lo_of(__longlong_as_double(static_cast<long long>(l.mark_r)));
    if (is_zero(l.zi) && is_zero(l.pi)) return direct_run_real<Formula>(l, room, saved, mark);
    if (!product_range(l.zi)) return 0;
    const int bound = hi_of(l.escape2) - (1 << 20);  // both squares below R^2 / 2 cannot escape
    double zr = l.zr, zi = l.zi, rs = l.rs, is = l.is;
    FactorA fr = factor_a(zr);
    FactorB gi = factor_b(zi);
    int k = 0;
#pragma unroll 1
    for (; k < room; ++k) {
        FactorA f = fr;
        FactorB g = gi;
        if constexpr (Formula == kFormulaBurningShip) {
            f.x &= 0x7ff00000;
            g.x &= 0x7ff00000;
        } else if constexpr (Formula == kFormulaTricorn) {
            f.x ^= static_cast<int>(0x80000000u);
        }
        f.x += 1 << 20;
        std::uint32_t low = ~0u;
        double cross = int_mul(f, g, low);
        if (low == 0u) cross = int_mul_even(f, g);
        const double nr = (rs - is) + l.pr;
        const double ni = cross + l.pi;
        const int hr = hi_of(nr) & 0x7fffffff, hi = hi_of(ni) & 0x7fffffff;
        fr = factor_a(nr);
        gi = factor_b(ni);
        const FactorB gr = factor_b(nr);
        const FactorA fi = factor_a(ni);
        low = ~0u;
        double nrs = int_mul(fr, gr, low), nis = int_mul(fi, gi, low);
        if (low == 0u) {
            nrs = int_mul_even(fr, gr);
            nis = int_mul_even(fi, gi);
        }
        if (min(hr, hi) < (523 << 20) || max(hr, hi) >= (1523 << 20) || lo_of(nr) == saved || lo_of(nr) == mark) break;
        if (max(hi_of(nrs), hi_of(nis)) >= bound && sum_exceeds(dbits(nrs), dbits(nis), dbits(l.escape2))) break;
        zr = nr;
        zi = ni;
        rs = nrs;
        is = nis;
    }
    l.zr = zr;
    l.zi = zi;
    l.rs = rs;
    l.is = is;
    l.it += k;
    return k;
}

template <bool Planes>
__device__ void write_inside(const DirectParams& p, int local) {
    p.out[local] = static_cast<float>(static_cast<double>(p.max_iter) - p.output_bias);
    if (p.counts) p.counts[local] = static_cast<std::uint32_t>(p.max_iter);
    if constexpr (Planes) {
        p.p_dex[local] = 0.0;
        p.p_dey[local] = 0.0;
        if (p.p_iter == nullptr) return;  // the derivative pair alone
        p.p_iter[local] = p.max_iter;
        p.p_phase[local] = 0.0;
        p.p_t1[local] = 0.0;
        p.p_t2[local] = 0.0;
    }
}

// Smooth escape value n + 1 - log(log|z|)/log 2 (renderer.cpp:10108-10116).
__device__ float smooth_value(const DirectParams& p, int iteration, double m2) {
    const double safe2 = escape_r2_d(p.escape_mode) + 1.0e-7;
    const double safe = is_finite(m2) ? dmax(m2, safe2) : 1.7976931348623157e308;
    const double magnitude = sqrt(safe);
    return static_cast<float>((static_cast<double>(iteration + 1) - log(log(magnitude)) / kLogTwoD) - p.output_bias);
}

template <int Formula>
__device__ void write_escape_planes(const DirectParams& p, const Lane& l, double m2) {
    constexpr bool has_de = Formula == kFormulaMandelbrot || Formula == kFormulaJulia;
    const int local = l.local;
    p.out[local] = smooth_value(p, l.it, m2);
    if (p.counts) p.counts[local] = static_cast<std::uint32_t>(l.it + 1);
    double de_re = 0.0, de_im = 0.0;
    if (has_de && p.need_de && is_finite(l.zr) && is_finite(l.zi) && is_finite(l.dr) && is_finite(l.di)) {
        if (!direct_de(l.zr, l.zi, l.dr, l.di, fe_from(p.pixel_spacing, 0), de_re, de_im)) {
            de_re = 0.0;
            de_im = 0.0;
        }
    }
    p.p_dex[local] = de_re;
    p.p_dey[local] = de_im;
    if (p.p_iter == nullptr) return;
    p.p_iter[local] = l.it;
    double phase = 0.0;
    if (p.need_phase && is_finite(l.zr) && is_finite(l.zi)) {
        phase = atan2(l.zi, l.zr) / kTwoPi;
        phase -= floor(phase);
    }
    p.p_phase[local] = phase;
    p.p_t1[local] = l.test1;
    p.p_t2[local] = l.test2;
}

// Warp-private staging in shared memory.  Pixel starts and escapes happen
// on single lanes at scattered times; doing their FP64 work (the
// cardioid/bulb test, the smooth value's logs) there would issue a full warp
// instruction for one lane each time.  Instead the warp classifies 32 new
// pixels at once into a start stack and parks escaped pixels until 32 are
// waiting, then finishes them with every lane busy (ballot + popc compaction).
struct StartSlot {
    double cx, cy;
    int field, local;
};
struct ParkSlot {
    double rs, is;  // the escaping step's squares (|z|^2 = rs + is)
    int it, field, local, pad;
};
constexpr int kStage = 64;
struct WarpStage {
    StartSlot start[kStage];
    ParkSlot park[kStage];
};

// Warp-uniform queue state (every lane holds the same values).
struct WarpQueue {
    long long next, end;  // claimed pixel range not yet classified
    int field;            // field of `next` (search hint)
    int starts;           // pixels waiting in the start stack
    int parked;           // escapes waiting in the park buffer
    bool drained;         // the batch counter ran out
};

// Classify up to 32 pixels of the warp's claimed range (claiming a new chunk
// when it is empty): interior-culled pixels are written at once, the others
// pushed on the start stack with their coordinates.
template <int Formula, bool Planes>
__device__ void classify(const DirectBatch& b, WarpQueue& q, WarpStage& st, unsigned long long* claim,
                         unsigned lane, unsigned below, long long total) {
    constexpr unsigned kFull = 0xffffffffu;
    if (q.next >= q.end) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(claim, static_cast<unsigned long long>(b.chunk));
        base = __shfl_sync(kFull, base, 0);
        if (static_cast<long long>(base) >= total) {
            q.drained = true;
            return;
        }
        q.next = static_cast<long long>(base);
        q.end = q.next + b.chunk < total ? q.next + b.chunk : total;
    }
    const long long avail = q.end - q.next;
    const int n = avail < 32 ? static_cast<int>(avail) : 32;
    const long long g = q.next + lane;
    bool keep = false;
    double cx = 0.0, cy = 0.0;
    int f = q.field, local = 0;
    if (static_cast<int>(lane) < n) {
        while (g >= b.first[f + 1]) ++f;
        const DirectParams& p = b.field[f];
        local = static_cast<int>(g - b.first[f]);
        const int py = local / p.width;
        const int px = local - py * p.width;
        const double* coords = b.coords + b.coord_offset[f];
        cx = coords[px];
        cy = coords[p.width + py];
        keep = true;
        if constexpr (Formula == kFormulaMandelbrot) {
            if (b.interior_test[f]) {
                // renderer.cpp:10060-10066
                const double qq = (cx - 0.25) * (cx - 0.25) + cy * cy;
                const bool cardioid = qq * (qq + cx - 0.25) <= 0.25 * cy * cy;
                const bool bulb = (cx + 1.0) * (cx + 1.0) + cy * cy <= 0.0625;
                if (cardioid || bulb) keep = false;
            }
        }
        if (p.max_iter <= 0) keep = false;
        if (!keep) write_inside<Planes>(p, local);
    }
    q.field = __shfl_sync(kFull, f, n - 1);
    q.next += n;
    const unsigned kept = __ballot_sync(kFull, keep);
    if (keep) {
        StartSlot& slot = st.start[q.starts + __popc(kept & below)];
        slot.cx = cx;
        slot.cy = cy;
        slot.field = f;
        slot.local = local;
    }
    q.starts += __popc(kept);
    __syncwarp();
}

template <int Formula>
__device__ void begin_pixel(const DirectBatch& b, const StartSlot& slot, Lane& l) {
    constexpr bool julia = Formula == kFormulaJulia;
    const DirectParams& p = b.field[slot.field];
    l.field = slot.field;
    l.local = slot.local;
    l.zr = julia ? slot.cx : 0.0;
    l.zi = julia ? slot.cy : 0.0;
    l.rs = l.zr * l.zr;
    l.is = l.zi * l.zi;
    l.pr = julia ? p.julia_re : slot.cx;
    l.pi = julia ? p.julia_im : slot.cy;
    l.dr = julia ? 1.0 : 0.0;
    l.di = 0.0;
    l.test1 = 0.0;
    l.test2 = 0.0;
    l.escape2 = escape_r2_d(p.escape_mode);
    l.saved_r = dbits(l.zr);
    l.saved_i = dbits(l.zi);
    l.mark_r = l.saved_r;
    l.mark_i = l.saved_i;
    l.it = 0;
    l.check_at = 1;
    l.max_iter = p.max_iter;
    l.stop_at = budget_stop(b, p.max_iter);
}

// Resume a spilled pixel.
template <int Formula>
__device__ void resume_pixel(const DirectBatch& b, const DirectSpill& e, Lane& l) {
    constexpr bool julia = Formula == kFormulaJulia;
    const int field = __ldcg(&e.field);
    const int local = __ldcg(&e.local);
    const DirectParams& p = b.field[field];
    l.field = field;
    l.local = local;
    l.zr = __ldcg(&e.zr);
    l.zi = __ldcg(&e.zi);
    l.rs = l.zr * l.zr;
    l.is = l.zi * l.zi;
    if (julia) {
        l.pr = p.julia_re;
        l.pi = p.julia_im;
    } else {
        const int py = local / p.width;
        const int px = local - py * p.width;
        const double* coords = b.coords + b.coord_offset[field];
        l.pr = coords[px];
        l.pi = coords[p.width + py];
    }
    l.dr = __ldcg(&e.dr);
    l.di = __ldcg(&e.di);
    l.test1 = __ldcg(&e.test1);
    l.test2 = __ldcg(&e.test2);
    l.escape2 = escape_r2_d(p.escape_mode);
    l.saved_r = __ldcg(&e.saved_r);
    l.saved_i = __ldcg(&e.saved_i);
    l.mark_r = __ldcg(&e.mark_r);
    l.mark_i = __ldcg(&e.mark_i);
    l.it = __ldcg(&e.it);
    l.check_at = __ldcg(&e.check_at);
    l.max_iter = p.max_iter;
    l.stop_at = p.max_iter;  // resumed pixels run to their end
}

// The smooth value with the logarithms in FP32 (the floatexp form's direct
// levels): the same formula, within a few float ulps of the FP64 value, at
// no FP64 cost.  Non-finite |z|^2 keeps the FP64 path.
__device__ float smooth_value_fast(const DirectParams& p, int iteration, double m2) {
    if (!is_finite(m2)) return smooth_value(p, iteration, m2);
    const double safe2 = escape_r2_d(p.escape_mode) + 1.0e-7;
    const float safe = static_cast<float>(dbits(m2) > dbits(safe2) ? m2 : safe2);
    const float log_mag = 0.5f * logf(safe);
    return (static_cast<float>(iteration + 1) - log2f(log_mag)) - static_cast<float>(p.output_bias);
}

__device__ void finish_parked(const DirectBatch& b, const ParkSlot& e) {
    const DirectParams& p = b.field[e.field];
    const double m2 = e.rs + e.is;
    p.out[e.local] = b.fast_smooth ? smooth_value_fast(p, e.it, m2) : smooth_value(p, e.it, m2);
    if (p.counts) p.counts[e.local] = static_cast<std::uint32_t>(e.it + 1);
}

// Direct field render over a batch of fields with lane refill.
//
// Restates render_direct_scalar_formula / render_direct_with_planes_formula
// (renderer.cpp:10054-10135, 10281-10438) pixel for pixel: the same
// coordinates, cardioid/bulb culling, the map z^2 + c with the reference's
// operation order (this translation unit is built without FMA contraction),
// escape at |z|^2 > R^2 and the smooth value.  Two rewrites leave every
// output bit unchanged:
//   * the squares zr*zr and zi*zi of the escape test are the next step's
//     squares, and 2 zr zi is formed as the product zr*zi with its exponent
//     raised by one; the three products run on the integer pipe (int_mul.h)
//     beside the three FP64 sums;
//   * an orbit that returns bit for bit to an earlier z repeats forever and
//     can never escape, so it is settled as interior at once (interior
//     outputs do not depend on z); z is kept at every power of two (Brent's
//     probe, any period) and at every multiple of 64 steps (short periods
//     found within ~64 steps of the orbit settling).
// FP64 is the bottleneck on this part (one warp instruction takes an SM
// sub-partition 80 cycles, whatever its active lanes), so a warp never waits
// on a finished lane: each warp claims chunks of pixels from a device counter
// over all fields of the batch and refills idle lanes every step from its
// start stack; escapes are parked and finished 32 at a time.  A pixel past
// b.budget steps goes to a list that later launches (`Resume`) take 32 to a
// warp.  Resumed by whichever warp had idle lanes, while others still ran
// fresh pixels, the long orbits of a 1920x1080 whole-set view were spread
// over all warps, a few lanes in each (16.4 ms; 3.3 ms now, most of it the
// latency of the orbits that run to the cap).
//
// The launch of fresh pixels is capped at 64 registers (a few spills): beside
// the FP32 queue on one SM, a block then takes as many registers as an
// FP32-queue block, so two of each kind fit where 80-register blocks left
// room for fewer.
constexpr int kRefill = 8;                // idle lanes before a resuming warp takes more
constexpr int kLeave = 20;                // active lanes below which it gives its pixels back ...
constexpr int kPatience = 16;             // ... after so many rounds,
constexpr int kShortList = 32 * 4 * 152;  // unless the list gives a warp to each sub-partition at most
constexpr long long kOneResume = 262144;  // pixels of a batch up to which one launch resumes
constexpr int kResumeBlocks = 2;          // per SM: two warps for each sub-partition

template <int Formula, bool Planes, bool Resume, bool Integer>
__global__ void __launch_bounds__(128, Resume ? 4 : 8) direct_queue_kernel(const __grid_constant__ DirectBatch b,
                                                                           int launch) {
    constexpr unsigned kFull = 0xffffffffu;
    __shared__ WarpStage stages[4];
    WarpStage& st = stages[threadIdx.x >> 5];
    const unsigned lane_id = threadIdx.x & 31u;
    const unsigned below = (1u << lane_id) - 1u;
    unsigned long long* claim = b.counter + kClaimFresh;
    const unsigned long long generation = *(b.counter + kGeneration);
    const long long total = b.first[b.count];
    // This launch's input list (Resume) and the list it spills to.
    DirectSpill* const made_list = b.spill + (launch & 1) * b.spill_capacity;
    const DirectSpill* const list = b.spill + ((launch + 1) & 1) * b.spill_capacity;
    unsigned long long* const made = b.counter + kSpillMade + launch;
    unsigned long long items = 0;
    int leave = 0;
    if constexpr (Resume) {
        items = *(b.counter + kSpillMade + launch - 1);
        if (items > static_cast<unsigned long long>(b.spill_capacity)) {
            items = static_cast<unsigned long long>(b.spill_capacity);
        }
        const unsigned long long rank = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
        if (rank >= (items + 31) / 32) return;
        leave = launch + 1 < b.launches && items > kShortList ? kLeave : 0;
    }
    WarpQueue q{0, 0, 0, 0, 0, false};
    bool active = false;
    int lean = 0;  // rounds with few lanes (Resume)
    unsigned long long executed = 0;  // steps this lane computed for a pixel
    Lane l;
    l.field = 0;
    l.zr = l.zi = l.rs = l.is = l.pr = l.pi = 0.0;
    l.dr = l.di = l.test1 = l.test2 = 0.0;
    l.escape2 = 4.0;
    l.saved_r = l.saved_i = 0;
    l.it = 0;
    l.check_at = 1;
    l.max_iter = 0;
    l.stop_at = 0;
    l.local = 0;

    while (true) {
        const unsigned idle = __ballot_sync(kFull, !active);
        const int need = __popc(idle);
        const int rank = __popc(idle & below);
        if constexpr (Resume) {
            if (need >= kRefill && !q.drained) {
                unsigned long long base = 0;
                if (lane_id == 0) {
                    base = atomicAdd(b.counter + kSpillTaken + launch, static_cast<unsigned long long>(need));
                }
                base = __shfl_sync(kFull, base, 0);
                if (!active && base + rank < items) {
                    // Written by the launch before, whose mark it must carry;
                    // the wait for it is bounded.
                    const DirectSpill& e = list[base + rank];
                    bool ready = false;
                    for (int spin = 0; spin < b.spin_limit; ++spin) {
                        if (*reinterpret_cast<const volatile unsigned long long*>(&e.ready)
                            == spill_mark(generation, launch - 1)) {
                            ready = true;
                            break;
                        }
                    }
                    if (ready) {
                        resume_pixel<Formula>(b, e, l);
                        active = true;
                    } else {
                        atomicExch(b.counter + kQueueError, 1ull);
                    }
                }
                q.drained = base + need >= items;
            }
        } else if (need != 0) {
            while (q.starts < need && !q.drained) classify<Formula, Planes>(b, q, st, claim, lane_id, below, total);
            if (!active && rank < q.starts) {
                begin_pixel<Formula>(b, st.start[q.starts - 1 - rank], l);
                active = true;
            }
            q.starts -= need < q.starts ? need : q.starts;
            __syncwarp();
        }
        if (__ballot_sync(kFull, active) == 0u) {
            if (Resume && !q.drained) continue;  // every entry taken was unpublished
            // Drained: finish what is parked (fewer than 32) and stop.
            if constexpr (!Planes) {
                if (static_cast<int>(lane_id) < q.parked) finish_parked(b, st.park[lane_id]);
            }
            for (int o = 16; o > 0; o >>= 1) executed += __shfl_xor_sync(kFull, executed, o);
            if (lane_id == 0) atomicAdd(b.counter + kStepsExecuted, executed);
            break;
        }

        // Up to `steps` steps before the next refill: every lane computes
        // each step (an idle or settled lane on stale values that it then
        // discards: the FP64 pipe costs the same per warp instruction), and a
        // lane stops updating at its first event (escape, interior, budget).
        constexpr bool has_de = Formula == kFormulaMandelbrot || Formula == kFormulaJulia;
        bool running = active;
        bool escaped = false, inside = false, spill = false;
        double rs_at_escape = 0.0, is_at_escape = 0.0;
        int steps = Resume ? b.long_steps : b.steps;
        if constexpr (Resume && Integer && !(Planes && has_de)) {
            if (active) {
                const int taken = direct_run<Formula>(l, steps);
                executed += static_cast<unsigned>(taken);
                running = taken < steps;
                // The escaping step, a general one, moves it to test2.
                if (Planes && taken > 0) l.test1 = l.rs + l.is;
            }
            steps = 1;
        }
        for (int s = 0; s < steps; ++s) {
            if (!__any_sync(kFull, running)) break;
            executed += running ? 1u : 0u;
            if constexpr (Planes && has_de) {
                if (running && b.field[l.field].need_de) {
                    // d' = 2 z d + 1 (parameter plane) or 2 z d (Julia) on the
                    // pre-step z (renderer.cpp:336-338).
                    const double add_re = Formula == kFormulaJulia ? 0.0 : 1.0;
                    const double ndr = 2.0 * l.zr * l.dr - 2.0 * l.zi * l.di + add_re;
                    const double ndi = 2.0 * l.zr * l.di + 2.0 * l.zi * l.dr + 0.0;
                    l.dr = ndr;
                    l.di = ndi;
                }
            }
            double cross;
            const bool crossed = cross_product<Formula, Integer>(l.zr, l.zi, cross);
            if (__any_sync(kFull, running && !crossed)) {
                if (!crossed) cross = cross_general<Formula>(l.zr, l.zi);
            }
            const double nr = (l.rs - l.is) + l.pr;
            const double ni = cross + l.pi;
            double rs, is;
            const bool squared_r = square_product<Integer>(nr, rs), squared_i = square_product<Integer>(ni, is);
            if (__any_sync(kFull, running && !(squared_r && squared_i))) {
                if (!squared_r) rs = square_general(nr);
                if (!squared_i) is = square_general(ni);
            }
            if (!running) continue;
            l.zr = nr;
            l.zi = ni;
            l.rs = rs;
            l.is = is;
            if constexpr (Planes) {
                l.test2 = l.test1;
                l.test1 = rs + is;
            }
            if (sum_exceeds(dbits(rs), dbits(is), dbits(l.escape2))) {
                escaped = true;
                rs_at_escape = rs;
                is_at_escape = is;
                running = false;
                continue;
            }
            ++l.it;
            const unsigned long long br = dbits(l.zr), bi = dbits(l.zi);
            if ((br == l.saved_r && bi == l.saved_i) || (br == l.mark_r && bi == l.mark_i) || l.it >= l.max_iter) {
                inside = true;
                running = false;
                continue;
            }
            if (l.it == l.check_at) {
                l.saved_r = br;
                l.saved_i = bi;
                l.check_at = l.check_at < (1 << 30) ? l.check_at << 1 : l.check_at;
            }
            if ((l.it & 63) == 0) {
                l.mark_r = br;
                l.mark_i = bi;
            }
            if (!Resume && l.it >= l.stop_at) {
                spill = true;
                running = false;
            }
        }
        if constexpr (Resume) {
            if (leave > 0 && q.drained) {
                const bool going = active && !escaped && !inside;
                if (__popc(__ballot_sync(kFull, going)) < leave) ++lean;
                spill = lean > kPatience && going && l.stop_at == l.max_iter;
            }
        }
        if (inside) {
            write_inside<Planes>(b.field[l.field], l.local);
            active = false;
        }
        const unsigned spilling = __ballot_sync(kFull, spill);
        if (spilling != 0u) {
            // Hand the lanes to the spill list (one reservation per warp, the
            // entry's mark written last); a full list lets them
            // run on here.
            const int leader = __ffs(spilling) - 1;
            unsigned long long base = 0;
            if (static_cast<int>(lane_id) == leader) {
                base = atomicAdd(made, static_cast<unsigned long long>(__popc(spilling)));
            }
            base = __shfl_sync(kFull, base, leader);
            if (spill) {
                const long long slot = static_cast<long long>(base) + __popc(spilling & below);
                if (slot < b.spill_capacity) {
                    DirectSpill& e = made_list[slot];
                    e.zr = l.zr;
                    e.zi = l.zi;
                    e.dr = l.dr;
                    e.di = l.di;
                    e.test1 = l.test1;
                    e.test2 = l.test2;
                    e.saved_r = l.saved_r;
                    e.saved_i = l.saved_i;
                    e.mark_r = l.mark_r;
                    e.mark_i = l.mark_i;
                    e.it = l.it;
                    e.check_at = l.check_at;
                    e.field = l.field;
                    e.local = l.local;
                    __threadfence();
                    if (!b.withhold_publish) *reinterpret_cast<volatile unsigned long long*>(&e.ready) = spill_mark(generation, launch);
                    active = false;
                } else {
                    l.stop_at = Resume ? l.max_iter + 1 : l.max_iter;  // (never offered again)
                }
            }
        }
        if constexpr (Planes) {
            if (escaped) {
                write_escape_planes<Formula>(b.field[l.field], l, rs_at_escape + is_at_escape);
                active = false;
            }
        } else {
            const unsigned esc = __ballot_sync(kFull, escaped);
            if (esc != 0u) {
                if (escaped) {
                    ParkSlot& slot = st.park[q.parked + __popc(esc & below)];
                    slot.rs = rs_at_escape;
                    slot.is = is_at_escape;
                    slot.it = l.it;
                    slot.field = l.field;
                    slot.local = l.local;
                    active = false;
                }
                q.parked += __popc(esc);
                __syncwarp();
                if (q.parked >= 32) {
                    finish_parked(b, st.park[q.parked - 32 + static_cast<int>(lane_id)]);
                    q.parked -= 32;
                    __syncwarp();
                }
            }
        }
    }
}

// Per-field coordinate tables (renderer.cpp:10185-10196): cx per column and
// cy per row, each centre + offset * span / size in double; also zeroes the
// batch's claim counter.
__global__ void direct_coords_kernel(const __grid_constant__ DirectBatch b) {
    const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < kGeneration) b.counter[i] = 0ull;
    if (i == kGeneration) b.counter[i] += 1ull;  // new marks for this batch's spill entries
    for (int f = 0; f < b.count; ++f) {
        const DirectParams& p = b.field[f];
        const long long span = static_cast<long long>(p.width) + p.height;
        const long long start = b.coord_offset[f];
        if (i < start || i >= start + span) continue;
        const int k = static_cast<int>(i - start);
        double value;
        if (k < p.width) {
            const double x_origin = p.coordinate_mode == 1 ? static_cast<double>(p.width / 2)
                                                           : static_cast<double>(p.width - 1) / 2.0;
            const double x_offset = (static_cast<double>(k) - x_origin) * p.width_span / static_cast<double>(p.width);
            value = p.center_re + x_offset;
        } else {
            const int py = k - p.width;
            const double y_origin = p.coordinate_mode == 1 ? static_cast<double>(p.height / 2)
                                                           : static_cast<double>(p.height - 1) / 2.0;
            const double y_offset =
                -(static_cast<double>(py) - y_origin) * p.height_span / static_cast<double>(p.height);
            value = p.center_im + y_offset;
        }
        b.coords[i] = value;
    }
}

template <int Formula, bool Planes, bool Integer>
cudaError_t launch_queue(const DirectBatch& b, int sms, int blocks_per_sm, cudaStream_t s) {
    static int per_sm = 0;
    if (per_sm == 0) {
        int blocks = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, direct_queue_kernel<Formula, Planes, false, Integer>, 128, 0);
        per_sm = blocks > 0 ? blocks : 1;
    }
    const long long pixels = b.first[b.count];
    const int use = blocks_per_sm > 0 && blocks_per_sm < per_sm ? blocks_per_sm : per_sm;
    long long grid = static_cast<long long>(sms) * use;
    const long long needed = (pixels + 127) / 128;
    if (grid > needed) grid = needed;
    if (grid < 1) grid = 1;
    direct_queue_kernel<Formula, Planes, false, Integer><<<static_cast<unsigned>(grid), 128, 0, s>>>(b, 0);
    const long long resume = std::min<long long>(static_cast<long long>(sms) * kResumeBlocks, needed);
    // A resumed step with the derivative's eight FP64 products gains nothing
    // from three more on the integer pipe, which only lengthen its chain: 64x36
    // with planes at 1e0, cap 4000, 4.2 ms with them and 3.4 without.
    constexpr bool derivative = Planes && (Formula == kFormulaMandelbrot || Formula == kFormulaJulia);
    for (int launch = 1; launch < b.launches; ++launch) {
        direct_queue_kernel<Formula, Planes, true, Integer && !derivative><<<static_cast<unsigned>(resume), 128, 0, s>>>(b, launch);
    }
    return cudaGetLastError();
}

template <bool Planes, bool Integer>
cudaError_t launch_formula(const DirectBatch& b, int formula, int sms, int blocks_per_sm, cudaStream_t s) {
    switch (formula) {
        case kFormulaMandelbrot: return launch_queue<kFormulaMandelbrot, Planes, Integer>(b, sms, blocks_per_sm, s);
        case kFormulaJulia: return launch_queue<kFormulaJulia, Planes, Integer>(b, sms, blocks_per_sm, s);
        case kFormulaBurningShip: return launch_queue<kFormulaBurningShip, Planes, Integer>(b, sms, blocks_per_sm, s);
        default: return launch_queue<kFormulaTricorn, Planes, Integer>(b, sms, blocks_per_sm, s);
    }
}

__device__ __forceinline__ std::uint8_t palette_byte(double v) {
    return static_cast<std::uint8_t>(v < 0.0 ? 0.0 : (255.0 < v ? 255.0 : v));
}

__device__ __forceinline__ double unit(double v) { return v < 0.0 ? 0.0 : (1.0 < v ? 1.0 : v); }

// aurora_palette_for (renderer.cpp:4841-4923): the palette's entries with the
// reference's double operations in its order (this translation unit has no
// FMA contraction), so its bytes are the reference's.  A music-driven frame
// has new controls each time: on the host the 65,536 entries took 1.2 ms of
// such a frame, here 13 us of FP64, and nothing waits for an upload.
__global__ void __launch_bounds__(128) aurora_lut_kernel(const float2* __restrict__ waves, int size,
                                                         const __grid_constant__ AuroraPalette p,
                                                         std::uint8_t* __restrict__ lut) {
    const int i = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x);
    if (i >= size) return;
    const float2 w = waves[i];
    const double c = w.x, s = w.y;
    double r = (0.5 - 0.5 * (c * p.rc + s * p.rs)) * 140.0;
    double g = (0.5 - 0.5 * (c * p.gc + s * p.gs)) * 140.0;
    double b = (0.5 - 0.5 * (c * p.bc + s * p.bs)) * 140.0;
    if (p.accented) {
        // The waves projected through the accents before the hue rotation.
        const double wr = unit(static_cast<double>(palette_byte(r)) / 140.0);
        const double wg = unit(static_cast<double>(palette_byte(g)) / 140.0);
        const double wb = unit(static_cast<double>(palette_byte(b)) / 140.0);
        r = (wr * static_cast<double>(p.accents[0]) + wg * static_cast<double>(p.accents[3])
             + wb * static_cast<double>(p.accents[6])) / 1.8;
        g = (wr * static_cast<double>(p.accents[1]) + wg * static_cast<double>(p.accents[4])
             + wb * static_cast<double>(p.accents[7])) / 1.8;
        b = (wr * static_cast<double>(p.accents[2]) + wg * static_cast<double>(p.accents[5])
             + wb * static_cast<double>(p.accents[8])) / 1.8;
    }
    if (p.rotate) {
        // Chroma rotation in YIQ (renderer.cpp:4815-4833).
        const double y = 0.299 * r + 0.587 * g + 0.114 * b;
        const double ii = 0.596 * r - 0.275 * g - 0.321 * b;
        const double q = 0.212 * r - 0.523 * g + 0.311 * b;
        const double ri = ii * p.hue_cos - q * p.hue_sin;
        const double rq = ii * p.hue_sin + q * p.hue_cos;
        r = y + 0.956 * ri + 0.621 * rq;
        g = y - 0.272 * ri - 0.647 * rq;
        b = y - 1.106 * ri + 1.703 * rq;
    }
    lut[3 * i] = palette_byte(r);
    lut[3 * i + 1] = palette_byte(g);
    lut[3 * i + 2] = palette_byte(b);
}

// Aurora palette lookup (write_colour_pixel, renderer.cpp:5210-5237): the
// palette index is smooth * ((size-1)/max_iter), the reference's double
// product of two floats, truncated and clamped; interior and non-finite
// pixels take the interior colour.  Four pixels per thread: 16 B of field in, 12 B of RGB out.
__global__ void __launch_bounds__(256) aurora_kernel(const float* __restrict__ field,
                                                     std::uint8_t* __restrict__ rgb, long long pixels,
                                                     const std::uint8_t* __restrict__ lut, int lut_size,
                                                     float index_scale, int max_iter, int vector_ok,
                                                     std::uint32_t interior) {
    const float limit = static_cast<float>(max_iter);
    const long long quads = vector_ok ? pixels / 4 : 0;
    const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
    auto colour = [&](float smooth, std::uint8_t* dst) {
        if (!isfinite(smooth) || smooth >= limit) {
            dst[0] = static_cast<std::uint8_t>(interior);
            dst[1] = static_cast<std::uint8_t>(interior >> 8);
            dst[2] = static_cast<std::uint8_t>(interior >> 16);
            return;
        }
        // trunc(double(smooth) * double(index_scale)), clamped: the product
        // of two floats is exact as p + e (FMA two-product), so it is
        // compared and truncated without FP64 (smooth is finite here).
        const float p = smooth * index_scale;
        const float e = __fmaf_rn(smooth, index_scale, -p);
        const float last_f = static_cast<float>(lut_size - 1);
        int k;
        if (p > last_f || (p == last_f && e >= 0.0f)) {
            k = lut_size - 1;
        } else if (!(p > 0.0f)) {
            k = 0;
        } else {
            const float f = floorf(p);
            k = static_cast<int>(f) - (p == f && e < 0.0f ? 1 : 0);
        }
        dst[0] = __ldg(lut + 3 * k);
        dst[1] = __ldg(lut + 3 * k + 1);
        dst[2] = __ldg(lut + 3 * k + 2);
    };
    for (long long q = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; q < quads; q += stride) {
        const float4 v = __ldcs(reinterpret_cast<const float4*>(field) + q);
        std::uint8_t out[12];
        colour(v.x, out);
        colour(v.y, out + 3);
        colour(v.z, out + 6);
        colour(v.w, out + 9);
        std::uint32_t w0 = out[0] | (out[1] << 8) | (out[2] << 16) | (static_cast<std::uint32_t>(out[3]) << 24);
        std::uint32_t w1 = out[4] | (out[5] << 8) | (out[6] << 16) | (static_cast<std::uint32_t>(out[7]) << 24);
        std::uint32_t w2 = out[8] | (out[9] << 8) | (out[10] << 16) | (static_cast<std::uint32_t>(out[11]) << 24);
        uint3 packed = make_uint3(w0, w1, w2);
        // 12-byte store: the RGB buffer of a 4-pixel group starts at 12*q,
        // which is 4-byte aligned.
        std::uint32_t* dst = reinterpret_cast<std::uint32_t*>(rgb + 12 * q);
        __stcs(dst, packed.x);
        __stcs(dst + 1, packed.y);
        __stcs(dst + 2, packed.z);
    }
    // Tail pixels (count not divisible by four).
    const long long tail_start = quads * 4;
    for (long long i = tail_start + static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < pixels;
         i += stride) {
        colour(field[i], rgb + 3 * i);
    }
}

__global__ void stamp_time_kernel(unsigned long long* slot) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    *slot = t;
}

}  // namespace

cudaError_t launch_stamp_time(unsigned long long* slot, cudaStream_t stream) {
    stamp_time_kernel<<<1, 1, 0, stream>>>(slot);
    return cudaGetLastError();
}

cudaError_t direct_queue_attributes(cudaFuncAttributes* attributes) {
    return cudaFuncGetAttributes(attributes, direct_queue_kernel<kFormulaMandelbrot, false, false, false>);
}

int direct_queue_occupancy() {
    int blocks = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, direct_queue_kernel<kFormulaMandelbrot, false, false, false>, 128, 0);
    return blocks > 0 ? blocks : 1;
}

std::size_t direct_scratch_bytes(const DirectParams* fields, int count, long long spill_entries) {
    std::size_t doubles = 0;
    for (int f = 0; f < count; ++f) doubles += static_cast<std::size_t>(fields[f].width) + fields[f].height;
    std::size_t bytes = 256 + doubles * sizeof(double);
    if (spill_entries > 0) {
        bytes = (bytes + 255) / 256 * 256;
        bytes += 2 * static_cast<std::size_t>(spill_entries) * sizeof(DirectSpill);
    }
    return bytes;
}

// Interior culling can matter only where the view reaches the cardioid's or
// the period-2 bulb's bounding box (with a wide margin).
static bool view_meets_interior(const DirectParams& p) {
    const double half_w = 0.5 * p.width_span + 0.05, half_h = 0.5 * p.height_span + 0.05;
    const double x0 = p.center_re - half_w, x1 = p.center_re + half_w;
    const double y0 = p.center_im - half_h, y1 = p.center_im + half_h;
    const bool cardioid = x1 >= -0.80 && x0 <= 0.40 && y1 >= -0.70 && y0 <= 0.70;
    const bool bulb = x1 >= -1.30 && x0 <= -0.70 && y1 >= -0.30 && y0 <= 0.30;
    return cardioid || bulb;
}

// Launches of a batch: one for fresh pixels and up to three for spilled ones.
// None of those finds anything where no cap exceeds the budget, and each costs
// 3 us and twice that of the calling thread: 257x256 around nothing that
// spills took 61 us with three, 55 with one.  One also serves the batches of
// up to kOneResume pixels that do spill better: it keeps its 38,912 lanes full
// from the list (640x360 at 1e5.7: 4.1 ms, with three 6.5 ms).
static int direct_launches(const DirectBatch& b, long long pixels) {
    if (b.spill_capacity <= 0) return 1;
    int longest = 0;
    for (int f = 0; f < b.count; ++f) longest = std::max(longest, b.field[f].max_iter);
    if (longest <= b.budget) return 1;
    return pixels > kOneResume ? kDirectLaunches : 2;
}

namespace {
constexpr int kDefaultSpinLimit = 1 << 22;
thread_local int fault_spin_limit = kDefaultSpinLimit;
thread_local int fault_withhold_publish = 0;
}  // namespace

void set_direct_fault_injection(int spin_limit, int withhold_publish) {
    fault_spin_limit = spin_limit > 0 ? spin_limit : kDefaultSpinLimit;
    fault_withhold_publish = withhold_publish ? 1 : 0;
}

cudaError_t launch_direct_batch(const DirectParams* fields, int count, void* scratch, const QueueShape& shape,
                                long long spill_entries, cudaStream_t stream, bool fast_smooth, bool beside_fp32) {
    if (count < 1 || count > kMaxDirectFields || !scratch) return cudaErrorInvalidValue;
    DirectBatch b{};
    b.spin_limit = fault_spin_limit;
    b.withhold_publish = fault_withhold_publish;
    b.count = count;
    b.fast_smooth = fast_smooth ? 1 : 0;
    b.counter = static_cast<unsigned long long*>(scratch);
    b.coords = reinterpret_cast<double*>(static_cast<char*>(scratch) + 256);
    b.chunk = shape.chunk > 0 ? shape.chunk : 64;
    const int formula = fields[0].formula;
    const bool planes = fields[0].p_dex != nullptr;
    long long pixels = 0, coords = 0;
    for (int f = 0; f < count; ++f) {
        if (fields[f].formula != formula || (fields[f].p_dex != nullptr) != planes) return cudaErrorInvalidValue;
        b.field[f] = fields[f];
        b.first[f] = pixels;
        b.coord_offset[f] = static_cast<int>(coords);
        b.interior_test[f] = formula == kFormulaMandelbrot && view_meets_interior(fields[f]) ? 1 : 0;
        pixels += static_cast<long long>(fields[f].width) * fields[f].height;
        coords += static_cast<long long>(fields[f].width) + fields[f].height;
    }
    b.first[count] = pixels;
    if (spill_entries > 0) {
        const std::size_t head = (256 + static_cast<std::size_t>(coords) * sizeof(double) + 255) / 256 * 256;
        b.spill = reinterpret_cast<DirectSpill*>(static_cast<char*>(scratch) + head);
        b.spill_capacity = spill_entries;
        b.budget = 256;
    }
    b.launches = direct_launches(b, pixels);
    b.steps = shape.steps > 0 ? shape.steps : 2;
    b.long_steps = 16;
    int device = 0, sms = 152;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    direct_coords_kernel<<<static_cast<unsigned>((coords + 255) / 256), 256, 0, stream>>>(b);
    cudaError_t status = cudaGetLastError();
    if (status != cudaSuccess) return status;
    if (planes) return launch_formula<true, true>(b, formula, sms, shape.blocks_per_sm, stream);
    return beside_fp32 ? launch_formula<false, false>(b, formula, sms, shape.blocks_per_sm, stream)
                       : launch_formula<false, true>(b, formula, sms, shape.blocks_per_sm, stream);
}

cudaError_t launch_aurora_lut(const float2* waves, int size, const AuroraPalette& palette, std::uint8_t* lut,
                              cudaStream_t stream) {
    aurora_lut_kernel<<<static_cast<unsigned>((size + 127) / 128), 128, 0, stream>>>(waves, size, palette, lut);
    return cudaGetLastError();
}

cudaError_t launch_aurora(const float* field, std::uint8_t* rgb, long long pixels, const std::uint8_t* lut,
                          int lut_size, float index_scale, int max_iter, cudaStream_t stream,
                          std::uint32_t interior) {
    int device = 0, sms = 152;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    // The palette (up to 192 KiB) is read through L1: neighbouring pixels
    // take neighbouring entries.
    const long long quads = (pixels + 3) / 4;
    const int threads = 256;
    long long blocks = (quads + threads - 1) / threads;
    const long long cap = static_cast<long long>(sms) * 8;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    const int vector_ok = (reinterpret_cast<std::uintptr_t>(field) % 16 == 0)
        && (reinterpret_cast<std::uintptr_t>(rgb) % 4 == 0);
    aurora_kernel<<<static_cast<unsigned>(blocks), threads, 0, stream>>>(field, rgb, pixels, lut, lut_size,
                                                                              index_scale, max_iter, vector_ok,
                                                                              interior);
    return cudaGetLastError();
}

}  // namespace fgb
