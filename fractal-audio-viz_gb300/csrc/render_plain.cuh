// Plain form (included by render_plain_*.cu, one kernel variant each): FP64-mantissa / int32-exponent perturbation of one deep
// Mandelbrot field per launch, one thread per pixel.
//
// The per-pixel procedure restates render_bla_impl (renderer.cpp:12673-13583)
// and render_scaled_double_tail (:12451-12669): image-series jump, glitch
// sentinel, escape with signed margin, Brent cycle test (non-strict only),
// Zhuoran rebasing with the 64-rebase exact fallback, map_end direct
// continuation, cubic / linear / deep-linear BLA lookup with endpoint replay,
// plain-double tail, and the exact step d' = 2 Z d + d^2 + dc.  This file is
// compiled with --fmad=false so every double operation rounds exactly as the
// reference release build does; the derivative (analytic DE) is carried only
// when the caller asked for render planes, because nothing else reads it.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "device.h"
#include "pixel_fraction.h"
#include "raw_series.h"

namespace fgb {
namespace plain {
namespace {

using namespace fx;

constexpr double kTwoPi = 6.283185307179586476925286766559005768;
constexpr double kLogTwo = 0.693147180559945309417232121458176568;

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ float encode(double value, double bias) {
    return static_cast<float>(value - bias);
}

__device__ __forceinline__ float nan_f() { return __int_as_float(0x7fc00000); }

// Local copies of the counters in the reference's RenderStats order.
struct Counters {
    unsigned long long v[kStatsSlots];
};

enum Slot {
    kPixels = 0, kLogical, kBlaBlocks, kLinearBlocks, kCubicBlocks, kExactSteps, kReplaySteps,
    kBlaRetries, kCycleInside, kDoubleTailPixels, kBlaDisabledPixels, kTailSteps, kMaxTailSteps,
    kTailRebases, kTailRebaseFallbacks, kMaxPixelIterations, kSeriesPixels, kSeriesJumps,
    kGlitchCount, kUnresolvedPixels, kDeadlineAborts, kSecondaryReferences, kRenderNs, kHist0
};

template <bool Stats>
struct StatSink {
    Counters c;
    __device__ void init() {
        if constexpr (Stats) {
#pragma unroll
            for (int i = 0; i < kStatsSlots; ++i) c.v[i] = 0;
        }
    }
    __device__ void add(int slot, unsigned long long n = 1) {
        if constexpr (Stats) c.v[slot] += n;
    }
    __device__ void max(int slot, unsigned long long n) {
        if constexpr (Stats) c.v[slot] = c.v[slot] > n ? c.v[slot] : n;
    }
    __device__ void bla_length(int length) {
        if constexpr (Stats) {
            if (length <= 0) return;
            int bucket = 0;
            unsigned int value = static_cast<unsigned int>(length);
            while (value > 1U && bucket < 15) {
                value >>= 1U;
                ++bucket;
            }
            c.v[kHist0 + bucket] += 1;
        }
    }
    // Warp-aggregate then one atomic per warp and slot.
    __device__ void flush(unsigned long long* out) {
        if constexpr (Stats) {
            const unsigned mask = __activemask();
            const int lane = threadIdx.x & 31;
            const int leader = __ffs(mask) - 1;
            for (int i = 0; i < kStatsSlots; ++i) {
                unsigned long long value = c.v[i];
                const bool is_max = i == kMaxTailSteps || i == kMaxPixelIterations;
                for (int offset = 16; offset > 0; offset >>= 1) {
                    const unsigned long long other = __shfl_down_sync(mask, value, offset);
                    const bool valid = (lane + offset) < 32 && ((mask >> (lane + offset)) & 1u);
                    if (valid) value = is_max ? (value > other ? value : other) : value + other;
                }
                // Lanes below the leader are not in the mask; the leader holds
                // the sum of every active lane above it.
                if (lane == leader) {
                    if (is_max) {
                        atomicMax(out + i, value);
                    } else if (value) {
                        atomicAdd(out + i, value);
                    }
                }
            }
        }
    }
};

// ------------------------------------------------------------ planes
__device__ double plane_phase(const Sc& v) {
    const double re = sc_re_d(v);
    const double im = sc_im_d(v);
    if (!is_finite(re) || !is_finite(im)) return 0.0;
    double phase = atan2(im, re) / kTwoPi;
    phase -= floor(phase);
    return is_finite(phase) ? phase : 0.0;
}

// render_plane_de (renderer.cpp:7844-7890).
__device__ bool plane_de(const Sc& total, const Sc& derivative, const Fe& spacing, double& out_re,
                         double& out_im) {
    const double mag = hypot(total.re, total.im);
    if (!(mag > 0.0) || !is_finite(mag)) return false;
    const double log_mag = log(mag) + static_cast<double>(total.e) * kLogTwo;
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

// Render planes: the derivative pair, and the other four or none (a batch
// asks for the pair only).
struct PlaneOut {
    std::int64_t* iter;
    double* phase;
    double* dex;
    double* dey;
    double* t1;
    double* t2;

    __device__ void clear(long long i, int max_iter) const {
        dex[i] = 0.0;
        dey[i] = 0.0;
        if (iter == nullptr) return;
        iter[i] = max_iter;
        phase[i] = 0.0;
        t1[i] = 0.0;
        t2[i] = 0.0;
    }
    __device__ void escape(long long i, int raw, const Sc& total, const Nrm& test1, const Nrm& test2,
                           const Sc& derivative, const Fe& spacing) const {
        double de_re = 0.0, de_im = 0.0;
        if (plane_de(total, derivative, spacing, de_re, de_im)) {
            dex[i] = de_re;
            dey[i] = de_im;
        } else {
            dex[i] = 0.0;
            dey[i] = 0.0;
        }
        if (iter == nullptr) return;
        iter[i] = raw;
        phase[i] = plane_phase(total);
        t1[i] = nrm_to_d(test1);
        t2[i] = nrm_to_d(test2);
    }
};

__device__ __forceinline__ int kalles_raw(int iteration) { return iteration - 1 > 0 ? iteration - 1 : 0; }

// smooth_escape_value (renderer.cpp:8170-8181), evaluated in double.
__device__ float smooth_escape(int iteration, const Nrm& norm, double bias) {
    if (is_zero(norm.m)) return encode(static_cast<double>(iteration), bias);
    const double log_mag = 0.5 * (log(norm.m) + static_cast<double>(norm.e) * kLogTwo);
    if (!(log_mag > 0.0) || !is_finite(log_mag)) return encode(static_cast<double>(iteration), bias);
    return encode(static_cast<double>(iteration) - log(log_mag) / kLogTwo, bias);
}

// ------------------------------------------------------------ BLA lookup
__device__ const CubicStep* lookup_cubic(const PlainParams& p, int start, const Fe& dn, int max_length) {
    if (start <= 0 || max_length <= 0 || !fe_finite(dn)) return nullptr;
    const int levels = p.cubic_index.levels;
    const int base = levels ? p.cubic_index.count[0] : 0;
    if (start > base) return nullptr;
    int highest = 31 - __clz(max_length);
    highest = highest < levels - 1 ? highest : levels - 1;
    const int offset = start - 1;
    for (int level = highest; level >= 0; --level) {
        if ((offset & ((1 << level) - 1)) != 0) continue;
        const int index = offset >> level;
        if (index >= p.cubic_index.count[level]) continue;
        const CubicStep* c = p.cubic + p.cubic_index.offset[level] + index;
        const int len = __ldg(&c->len);
        const Fe r2 = fe_make(__ldg(&c->r2.m), __ldg(&c->r2.e));
        if (len > 1 && fe_finite(r2) && fe_cmp(dn, r2) < 0) return c;
    }
    return nullptr;
}

__device__ const LinearStep* lookup_linear(const PlainParams& p, int start, const Fe& dn, int max_length) {
    if (start <= 0 || max_length <= 0 || !fe_finite(dn)) return nullptr;
    const int levels = p.linear_index.levels;
    const int base = levels ? p.linear_index.count[0] : 0;
    if (start > base) return nullptr;
    int highest = 31 - __clz(max_length);
    highest = highest < levels - 1 ? highest : levels - 1;
    const int offset = start - 1;
    for (int level = highest; level >= 0; --level) {
        if ((offset & ((1 << level) - 1)) != 0) continue;
        const int index = offset >> level;
        if (index >= p.linear_index.count[level]) continue;
        const LinearStep* c = p.linear + p.linear_index.offset[level] + index;
        const int len = __ldg(&c->len);
        const Fe r2 = fe_make(__ldg(&c->r2.m), __ldg(&c->r2.e));
        if (len > 1 && fe_finite(r2) && fe_cmp(dn, r2) < 0) return c;
    }
    return nullptr;
}

__device__ __forceinline__ Sc ld_sc(const Sc* s) { return sc_make(__ldg(&s->re), __ldg(&s->im), __ldg(&s->e)); }

// apply_bla_series (renderer.cpp:8686-8730).
__device__ Sc apply_cubic(const CubicStep* step, const Sc& d, const Sc& c, int order) {
    const Sc k0 = ld_sc(&step->c[0]);
    const Sc k1 = ld_sc(&step->c[1]);
    if (order <= 1) return sc_add(sc_mul(k0, d), sc_mul(k1, c));
    const Sc k2 = ld_sc(&step->c[2]);
    const Sc k3 = ld_sc(&step->c[3]);
    const Sc k4 = ld_sc(&step->c[4]);
    if (order == 2) {
        const Sc d_inner = sc_add(sc_mul(k2, d), sc_mul(k3, c));
        const Sc c_inner = sc_add(k1, sc_mul(k4, c));
        return sc_add(sc_mul(d, sc_add(k0, d_inner)), sc_mul(c, c_inner));
    }
    const Sc k5 = ld_sc(&step->c[5]);
    const Sc k6 = ld_sc(&step->c[6]);
    const Sc k7 = ld_sc(&step->c[7]);
    const Sc k8 = ld_sc(&step->c[8]);
    const Sc d_cubic = sc_add(sc_add(sc_mul(k5, d), sc_mul(k6, c)), k2);
    const Sc c_cubic = sc_add(k3, sc_mul(k7, c));
    const Sc d_inner = sc_add(k0, sc_add(sc_mul(d, d_cubic), sc_mul(c, c_cubic)));
    const Sc c_inner = sc_add(k1, sc_mul(c, sc_add(k4, sc_mul(k8, c))));
    return sc_add(sc_mul(d, d_inner), sc_mul(c, c_inner));
}

// apply_bla_series_derivative (renderer.cpp:8732-8795).
__device__ __noinline__ Sc apply_cubic_derivative(const CubicStep* step, const Sc& d, const Sc& c, const Sc& dd,
                                     int order) {
    const Sc k0 = ld_sc(&step->c[0]);
    const Sc k1 = ld_sc(&step->c[1]);
    if (order <= 1) return sc_add(sc_mul(k0, dd), k1);
    Sc pd = k0;
    Sc pc = k1;
    const Sc k2 = ld_sc(&step->c[2]);
    const Sc k3 = ld_sc(&step->c[3]);
    const Sc k4 = ld_sc(&step->c[4]);
    pd = sc_add(pd, sc_add(sc_twice(sc_mul(k2, d)), sc_mul(k3, c)));
    pc = sc_add(pc, sc_add(sc_mul(k3, d), sc_twice(sc_mul(k4, c))));
    if (order >= 3) {
        const Sc k5 = ld_sc(&step->c[5]);
        const Sc k6 = ld_sc(&step->c[6]);
        const Sc k7 = ld_sc(&step->c[7]);
        const Sc k8 = ld_sc(&step->c[8]);
        const Sc d2 = sc_mul(d, d);
        const Sc c2 = sc_mul(c, c);
        pd = sc_add(pd, sc_add(sc_mul(sc_add(sc_twice(sc_mul(k5, d)), sc_mul(k5, d)), d),
                               sc_add(sc_twice(sc_mul(k6, sc_mul(d, c))), sc_mul(k7, c2))));
        pc = sc_add(pc, sc_add(sc_mul(k6, d2),
                               sc_add(sc_twice(sc_mul(k7, sc_mul(d, c))),
                                      sc_mul(sc_add(sc_twice(sc_mul(k8, c)), sc_mul(k8, c)), c))));
    }
    return sc_add(sc_mul(pd, dd), pc);
}

struct OrbitView {
    const OrbitRec* r;
    __device__ Sc z(int i) const { return ld_sc(&r[i].z); }
    __device__ double zd_re(int i) const { return __ldg(&r[i].zd_re); }
    __device__ double zd_im(int i) const { return __ldg(&r[i].zd_im); }
    __device__ Fe glitch(int i) const { return fe_make(__ldg(&r[i].glitch.m), __ldg(&r[i].glitch.e)); }
    // Signed escape margin |Z_i + d|^2 - R^2 (renderer.cpp:8374-8390) with
    // the reference-only terms read from the record.
    __device__ Fe margin(int i, const Sc& d) const {
        const Fe pr = fe_make(__ldg(&r[i].parts.re.m), __ldg(&r[i].parts.re.e));
        const Fe pi = fe_make(__ldg(&r[i].parts.im.m), __ldg(&r[i].parts.im.e));
        const Fe m0 = fe_make(__ldg(&r[i].margin.m), __ldg(&r[i].margin.e));
        const Fe dr = fe_from(d.re, d.e);
        const Fe di = fe_from(d.im, d.e);
        const Fe cross = fe_twice(fe_add(fe_mul(pr, dr), fe_mul(pi, di)), false);
        return fe_add(fe_add(m0, cross), fe_add(fe_sqr(dr), fe_sqr(di)));
    }
};

// How a pixel left its loops.  The logarithms of an escape are evaluated once
// per warp after them: inside, each lane's own escape step ran them again.
enum Exit { kExitNone, kExitNorm, kExitTail, kExitRecord };

// High words of magnitudes: they order values to 2^-20.
constexpr int kHighLow = kRawLow << 20;                                 // 2^-400
constexpr int kHighTop = (kRawLow + static_cast<int>(kRawSpan)) << 20;  // 2^10
constexpr int kHighUnit = (1023 - 300) << 20;
__device__ __forceinline__ int high(double v) { return hi_of(v) & 0x7fffffff; }
__device__ __forceinline__ bool same(const Sc& a, const Sc& b) {
    return bits_of(a.re) == bits_of(b.re) && bits_of(a.im) == bits_of(b.im) && a.e == b.e;
}
// a < b for values >= +0.
__device__ __forceinline__ bool below(double a, double b) { return bits_of(a) < bits_of(b); }

__device__ __forceinline__ double2 ld_zd(const OrbitRec* r) { return __ldg(reinterpret_cast<const double2*>(r)); }
__device__ __forceinline__ int4 ld_head(const OrbitRec* r) { return __ldg(reinterpret_cast<const int4*>(&r->zf_re)); }

// derivative <- 2 total derivative + 1 on plain values, where the + 1 does not
// move it (60 binades below) and the parts are in range; else false.
__device__ __forceinline__ bool derivative_run(double re, double im, const Sc& v, Sc& out) {
    const int low = imin(imin(high(re), high(im)) - kHighLow, imin(high(v.re), high(v.im)) - kHighUnit);
    if (low < 0 || imax(high(re), high(im)) > kHighTop || static_cast<unsigned>(v.e) >= 1u << 28) return false;
    const FactorA tr = factor_a(re), ti = factor_a(im);
    const FactorB vr = factor_b(v.re), vi = factor_b(v.im);
    const double xr = int_mul_even(tr, vr) - int_mul_even(ti, vi);
    const double xi = int_mul_even(ti, vr) + int_mul_even(tr, vi);
    const int shift = imax(bexp(xr), bexp(xi)) - 1022;
    out = sc_make(add_exp(xr, -shift), add_exp(xi, -shift), v.e + shift + 1);
    return imin(bexp(xr), bexp(xi)) >= 100 && out.e > 60;
}

// Up to `room` steps total <- total^2 + parameter on plain doubles whose
// tests an FP32 estimate settles (tail_run's bound on it): 4 FP64
// instructions each, 2 more with planes.  `open` as in tail_run.
template <bool Planes>
__device__ __forceinline__ int exact_run(const PlainParams& p, const Sc& parameter, int iteration, int room,
                                         int cycle_min, Sc& total, Sc& prior, Sc& derivative, bool& open) {
    const float bound = (p.escape_mode == 1 ? 1.0e8f : 4.0f) * (1.0f - 0x1p-14f);
    int made = 0;
    while (made < room) {
        const int hr = high(total.re), hi = high(total.im);
        if (imin(hr, hi) < kHighLow || imax(hr, hi) > kHighTop) break;
        if constexpr (Planes) {
            Sc next;
            if (!derivative_run(total.re, total.im, derivative, next)) break;
            derivative = next;
            prior = total;
        }
        const FactorA fr = factor_a(total.re), fi = factor_a(total.im);
        const FactorB gr = factor_b(total.re), gi = factor_b(total.im);
        const double rr = int_mul_even(fr, gr), ii = int_mul_even(fi, gi), ri = int_mul_even(fr, gi);
        total = add_cut(sc_make(rr - ii, add_exp(ri, 1), 0), parameter);
        ++made;
        const float x = float_of(total.re, 0), y = float_of(total.im, 0);
        const int it = iteration + made;
        if (!(x * x + y * y < bound) || (p.cycle && it >= cycle_min && (it & 31) == 0)) {
            open = true;
            break;
        }
    }
    return made;
}

// How many general steps follow before a run that took none is tried again:
// none after its first failure, then one, two, up to 32.  A pixel exactly on an
// axis has a zero part at every step, and entering the run in vain each time
// lengthened them all: a 200x113 field around -1.62 at 1e12, one row of it on
// the axis, took 6.0 ms (9.2 with thread-per-pixel FP64 tests) and 4.8 this way.
struct Rest {
    int left = 0, next = 0;
    __device__ bool over() { return left == 0 || left-- == 0; }
    __device__ void tell(int made) {
        left = made == 0 ? next : 0;
        next = made == 0 ? imin(imax(2 * next, 1), 32) : 0;
    }
};

// Exact scaled recurrence from the reconstructed total once the pixel has
// left the compact reference (renderer.cpp:13053-13146 and 13155-13250).
// kExitNorm with the last total, its norm and the one before for a value that
// the caller finishes.
template <bool Planes, bool Stats>
__device__ __forceinline__ Exit exact_continuation(const PlainParams& p, const OrbitView& orbit, const Sc& dc, Sc& total,
                                   Nrm& total_norm, Nrm& prior, Sc& derivative, int& iteration, StatSink<Stats>& st,
                                   unsigned& ticks, unsigned long long deadline_ns, float& out_value,
                                   std::uint32_t& out_count, bool& deadline) {
    const Sc parameter = sc_add(orbit.z(1), dc);
    const Sc plain_parameter = to_raw(parameter);
    const bool plain = plain_parameter.e == 0 && raw_or_zero(plain_parameter.re) && raw_or_zero(plain_parameter.im);
    Sc tortoise = sc_zero();
    int power = 1, length = 0;
    bool ready = false;
    const int cycle_min = p.strict_cycle ? 2048 : 512;
    const int cycle_margin = p.strict_cycle ? 78 : 60;
    out_value = encode(static_cast<double>(p.max_iter), p.output_bias);
    out_count = static_cast<std::uint32_t>(p.max_iter);
    Rest rest;
    while (iteration < p.max_iter) {
        if (deadline_ns && (ticks & 255U) == 0U && global_ns() >= deadline_ns) {
            out_value = nan_f();
            out_count = 0;
            deadline = true;
            st.add(kDeadlineAborts);
            st.add(kUnresolvedPixels);
            return kExitNone;
        }
        prior = total_norm;
        int made = 0;
        bool open = false;
        if (plain && rest.over()) {
            total = to_raw(total);
            Sc before = sc_zero();
            const int room = imin(p.max_iter - iteration, deadline_ns ? 256 - static_cast<int>(ticks & 255U) : INT_MAX);
            if (total.e == 0) {
                made = exact_run<Planes>(p, plain_parameter, iteration, room, cycle_min, total, before, derivative, open);
            }
            if constexpr (Planes) {
                if (made > 1) prior = sc_norm2(normal_form(before));
            }
            total = normal_form(total);
            rest.tell(made);
        }
        if (made == 0) {
            if constexpr (Planes) derivative = sc_add(sc_twice(sc_mul(total, derivative)), sc_one());
            total = sc_add(sc_sqr(total), parameter);
            made = 1;
            open = true;
        }
        ticks += static_cast<unsigned>(made);
        iteration += made;
        st.add(kLogical, static_cast<unsigned long long>(made));
        st.add(kExactSteps, static_cast<unsigned long long>(made));
        total_norm = sc_norm2(total);
        if (!open) continue;
        if (nrm_outside(total_norm, p.escape_mode)) {
            out_count = static_cast<std::uint32_t>(iteration);
            return kExitNorm;
        }
        if (p.cycle) {
            if (iteration >= cycle_min && (iteration & 31) == 0 && nrm_cmp(total_norm, nrm_make(0.75, 2)) < 0) {
                if (!ready) {
                    tortoise = total;
                    power = 1;
                    length = 0;
                    ready = true;
                } else {
                    const Nrm dist = sc_norm2(sc_sub(total, tortoise));
                    const int scale_e = total_norm.e > 0 ? total_norm.e : 0;
                    if (is_zero(dist.m) || dist.e <= scale_e - cycle_margin) return kExitNone;
                    if (++length >= power) {
                        tortoise = total;
                        power = power * 2 < (1 << 20) ? power * 2 : (1 << 20);
                        length = 0;
                    }
                }
            }
        }
    }
    return kExitNone;
}

// State of the double tail that its hot loop advances.
template <bool Planes>
struct Tail {
    double dr, di;
    Sc derivative;
    double prior_re, prior_im;  // Z + d before the last step
    int ref, steps, rebases;    // steps since the last rebase
    bool ready;                 // a cycle reference is set
};

// Up to `room` tail steps whose tests FP32 estimates settle, rebases
// included, products on the integer pipe (int_mul.h).  It stops before a step
// it does not cover (a value out of range, the orbit's end) and after one
// whose tests the caller must settle (`open`).  Returns the steps taken.
//
// A step is 5 FP64 instructions, 7 while dc reaches the sum, and 4 more with
// planes, where the same step written out is 28 (38 with planes); the integer
// instructions beside them take about as long.  |Z + d|^2 and |d|^2 are known
// from FP32 to 2^-17 of the larger: R^2 is passed only above (1 - 2^-14) R^2
// or with |d| > 4 R, and one is the smaller for certain when the estimates
// differ by 2^-8 (the larger not below 2^-100).
//
// `Axis`: the reference lies on an axis and its orbit has zero parts, which
// the integer products do not take; its products with Z run in FP64.  A kernel
// of its own: a branch in the usual loop cost it 1 %, a second loop beside it
// 1 to 3 %.
template <bool Planes, bool Axis>
__device__ __forceinline__ int tail_run(const PlainParams& p, double dc_re, double dc_im, int room, Tail<Planes>& t,
                                        bool& open) {
    constexpr int kMaxRebases = 64;
    double dr = t.dr, di = t.di;
    int at = t.ref, made = 0;
    double2 z = ld_zd(p.orbit + at);
    int4 head = ld_head(p.orbit + at);
    const float bound = (p.escape_mode == 1 ? 1.0e8f : 4.0f) * (1.0f - 0x1p-14f);
    const float far = (p.escape_mode == 1 ? 1.0e8f : 4.0f) * 16.0f;
    const int dc_top = imax(bexp(dc_re), bexp(dc_im));
    double total_re = 0.0, total_im = 0.0;
    if constexpr (Planes) {
        total_re = z.x + dr;
        total_im = z.y + di;
    }
    while (made < room && at + 1 < p.orbit_size) {
        const bool origin = is_zero(z.x) && is_zero(z.y);  // after a rebase
        if (!origin && !(head.z & (Axis ? kRawOrbit | kRawZero : kRawOrbit))) break;
        const int hr = high(dr), hi = high(di);
        if (imin(hr, hi) < kHighLow || imax(hr, hi) > kHighTop) break;
        const OrbitRec* const next = p.orbit + at + 1;
        const double2 zn = ld_zd(next);
        const int4 hn = ld_head(next);
        Sc derivative = sc_zero();
        if constexpr (Planes) {
            if (!derivative_run(total_re, total_im, t.derivative, derivative)) break;
        }
        const FactorA fr = factor_a(dr), fi = factor_a(di);
        double lr, li;
        if constexpr (Axis) {
            const double z2r = twice_raw(z.x), z2i = twice_raw(z.y);
            lr = z2r * dr - z2i * di;
            li = z2r * di + z2i * dr;
        } else {
            const FactorB zr = factor_b(add_exp(z.x, 1)), zi = factor_b(add_exp(z.y, 1));
            const double rr = int_mul_even(fr, zr), ii = int_mul_even(fi, zi);
            const double ri = int_mul_even(fi, zr), ir = int_mul_even(fr, zi);
            lr = rr - ii;
            li = ri + ir;
        }
        const FactorB gr = factor_b(dr), gi = factor_b(di);
        const double uu = int_mul_even(fr, gr), vv = int_mul_even(fi, gi), uv = int_mul_even(fr, gi);
        const double sr = uu - vv, si = add_exp(uv, 1);
        double xr = lr + sr, xi = li + si;
        xr = choose(origin, sr, xr);
        xi = choose(origin, si, xi);
        // dc does not move a sum 60 binades above it.
        if (imin(bexp(xr), bexp(xi)) <= dc_top + 60) {
            xr = xr + dc_re;
            xi = xi + dc_im;
        }
        dr = xr;
        di = xi;
        ++at;
        ++made;
        if constexpr (Planes) {
            t.derivative = derivative;
            t.prior_re = total_re;
            t.prior_im = total_im;
            total_re = zn.x + dr;
            total_im = zn.y + di;
        }
        const float dx = float_of(dr, 0), dy = float_of(di, 0);
        const float tx = __int_as_float(hn.x) + dx, ty = __int_as_float(hn.y) + dy;
        const float m = tx * tx + ty * ty, dm = dx * dx + dy * dy;
        const int steps = t.steps + 1;
        const bool keep = m > dm * (1.0f + 0x1p-8f) && m > 0x1p-100f;
        const bool move = m * (1.0f + 0x1p-8f) < dm && dm > 0x1p-100f && t.rebases < kMaxRebases;
        if (!(m < bound && dm < far) || !(keep || move) || (p.cycle && steps >= 64 && (steps & 31) == 0)) {
            open = true;
            break;
        }
        t.steps = steps;
        z = zn;
        head = hn;
        if (move) {
            if constexpr (Planes) {
                dr = total_re;
                di = total_im;
            } else {
                dr = zn.x + dr;
                di = zn.y + di;
            }
            at = 0;
            t.steps = 0;
            t.ready = false;
            ++t.rebases;
            z = ld_zd(p.orbit);
            head = ld_head(p.orbit);
            if constexpr (Planes) {
                total_re = z.x + dr;
                total_im = z.y + di;
            }
        }
    }
    t.dr = dr;
    t.di = di;
    t.ref = at;
    return made;
}

// render_scaled_double_tail (renderer.cpp:12451-12669). Returns kExitTail,
// with |Z + d|^2 in `exit_mag2`, for a value that the caller finishes.
template <bool Planes, bool Stats, bool Axis>
__device__ __forceinline__ Exit double_tail(const PlainParams& p, const OrbitView& orbit, long long index, const Sc& dc,
                            int& iteration, int& ref, const Sc& delta_in, Sc& derivative,
                            const Nrm& initial_norm, StatSink<Stats>& st, unsigned& ticks,
                            unsigned long long deadline_ns, float& out_value, std::uint32_t& out_count, bool& deadline,
                            bool& unresolved, const PlaneOut& planes, double& exit_mag2,
                            Sc& exit_total, Nrm& exit_previous) {
    const int kMaxTailRebases = 64;
    const int kMaxTailSteps = 65536;
    const double dc_re = sc_re_d(dc);
    const double dc_im = scale2(dc.im, dc.e);
    const double escape2 = escape_r2_d(p.escape_mode);
    Tail<Planes> t{};
    t.dr = sc_re_d(delta_in);
    t.di = scale2(delta_in.im, delta_in.e);
    t.ref = ref;
    t.derivative = derivative;
    out_value = encode(static_cast<double>(p.max_iter), p.output_bias);
    out_count = static_cast<std::uint32_t>(p.max_iter);
    double tort_re = 0.0, tort_im = 0.0;
    int power = 1, length = 0, tail_iterations = 0;
    Nrm previous = initial_norm;
    const bool strict = p.strict != 0;
    Exit exit = kExitNone;
    bool ended = false;
    Rest rest;
    while (iteration < p.max_iter && t.ref >= 0 && t.ref + 1 < p.orbit_size) {
        if (deadline_ns && (ticks & 255U) == 0U && global_ns() >= deadline_ns) {
            out_value = nan_f();
            out_count = 0;
            deadline = true;
            unresolved = true;
            st.add(kDeadlineAborts);
            st.add(kUnresolvedPixels);
            ended = true;
            break;
        }
        int room = imin(p.max_iter - iteration, kMaxTailSteps - tail_iterations);
        if (deadline_ns) room = imin(room, 256 - static_cast<int>(ticks & 255U));
        bool open = false;
        const int moved = t.rebases;
        int made = 0;
        if (rest.over()) {
            made = tail_run<Planes, Axis>(p, dc_re, dc_im, room, t, open);
            rest.tell(made);
        }
        st.add(kTailRebases, static_cast<unsigned long long>(t.rebases - moved));
        if (made > 0) {
            ticks += static_cast<unsigned>(made);
            iteration += made;
            tail_iterations += made;
            st.add(kLogical, static_cast<unsigned long long>(made));
            st.add(kExactSteps, static_cast<unsigned long long>(made));
            if constexpr (Planes) {
                if (!open) {
                    const double re = orbit.zd_re(t.ref) + t.dr, im = orbit.zd_im(t.ref) + t.di;
                    previous = nrm_from_d(re * re + im * im);
                } else if (made > 1) {
                    previous = nrm_from_d(t.prior_re * t.prior_re + t.prior_im * t.prior_im);
                }
            }
            if (!open) continue;
        } else {
            ++ticks;
            const double dr = t.dr, di = t.di;
            const double zr = orbit.zd_re(t.ref);
            const double zi = orbit.zd_im(t.ref);
            if constexpr (Planes) {
                Sc prior = sc_make(zr + dr, zi + di, 0);
                sc_normalize(prior);
                t.derivative = sc_add(sc_twice(sc_mul(prior, t.derivative)), sc_one());
            }
            const double lin_re = 2.0 * (zr * dr - zi * di);
            const double lin_im = 2.0 * (zr * di + zi * dr);
            const double sq_re = dr * dr - di * di;
            const double sq_im = 2.0 * dr * di;
            t.dr = lin_re + sq_re + dc_re;
            t.di = lin_im + sq_im + dc_im;
            ++t.ref;
            ++iteration;
            if (++tail_iterations > kMaxTailSteps) {
                st.add(kTailRebaseFallbacks);
                st.add(kUnresolvedPixels);
                unresolved = true;
                out_value = strict ? nan_f() : encode(static_cast<double>(iteration), p.output_bias);
                out_count = strict ? 0u : static_cast<std::uint32_t>(iteration);
                ended = true;
                break;
            }
            st.add(kLogical);
            st.add(kExactSteps);
        }
        // The tests of the step just taken, exactly.
        const double tr = orbit.zd_re(t.ref) + t.dr;
        const double ti = orbit.zd_im(t.ref) + t.di;
        const double mag2 = tr * tr + ti * ti;
        if (!is_finite(mag2)) {
            unresolved = true;
            st.add(kGlitchCount);
            st.add(kUnresolvedPixels);
            out_value = strict ? nan_f() : encode(static_cast<double>(iteration), p.output_bias);
            out_count = strict ? 0u : static_cast<std::uint32_t>(iteration);
            ended = true;
            break;
        }
        if (below(escape2, mag2)) {
            out_count = static_cast<std::uint32_t>(iteration);
            exit = kExitTail;
            exit_mag2 = mag2;
            if constexpr (Planes) {
                exit_total = sc_make(tr, ti, 0);
                exit_previous = previous;
            }
            ended = true;
            break;
        }
        if constexpr (Planes) previous = nrm_from_d(mag2);
        const double dmag2 = t.dr * t.dr + t.di * t.di;
        ++t.steps;
        if (p.cycle) {
            if (t.steps >= 64 && (t.steps & 31) == 0) {
                if (!t.ready) {
                    tort_re = tr;
                    tort_im = ti;
                    power = 1;
                    length = 0;
                    t.ready = true;
                } else {
                    const double cr = tr - tort_re;
                    const double ci = ti - tort_im;
                    const double dist2 = cr * cr + ci * ci;
                    const int cycle_min = p.strict_cycle ? 2048 : 512;
                    const double tol = p.strict_cycle ? 1.0e-24 : 1.0e-18;
                    if (iteration >= cycle_min && mag2 < 3.0 && dist2 <= tol * dmax(1.0, mag2)) {
                        if constexpr (Planes) planes.clear(index, p.max_iter);
                        ended = true;
                        break;
                    }
                    if (++length >= power) {
                        tort_re = tr;
                        tort_im = ti;
                        power = power * 2 < (1 << 20) ? power * 2 : (1 << 20);
                        length = 0;
                    }
                }
            }
        }
        if (below(mag2, dmag2)) {
            t.dr = tr;
            t.di = ti;
            t.ref = 0;
            t.steps = 0;
            t.ready = false;
            st.add(kTailRebases);
            if (++t.rebases > kMaxTailRebases) {
                st.add(kTailRebaseFallbacks);
                st.add(kUnresolvedPixels);
                unresolved = true;
                out_value = strict ? nan_f() : encode(static_cast<double>(iteration), p.output_bias);
                out_count = strict ? 0u : static_cast<std::uint32_t>(iteration);
                if constexpr (Planes) planes.clear(index, p.max_iter);
                ended = true;
                break;
            }
        }
    }
    derivative = t.derivative;
    if (!ended && iteration < p.max_iter) {
        unresolved = true;
        st.add(kUnresolvedPixels);
        out_value = strict ? nan_f() : encode(static_cast<double>(iteration), p.output_bias);
        out_count = strict ? 0u : static_cast<std::uint32_t>(iteration);
        if constexpr (Planes) planes.clear(index, p.max_iter);
    }
    return exit;
}

// The FP64 pipe bounds it, with the integer instructions beside it issuing in
// 40 % of the cycles.  640x360 at 1e30: 202 us (0.92 ms with products in FP64,
// every test exact and the logarithms at each lane's own escape), 247 us where
// pixels repeat a rebase (1.73 ms).  Blocks of 64 threads and the larger
// operations out of line were 2 to 8 % slower, integer products in the general
// operations too 7 %.
template <bool Planes, bool Stats, bool Axis>
__global__ void __launch_bounds__(128) plain_mandelbrot_kernel(const PlainParams p) {
    const long long total_pixels = static_cast<long long>(p.width) * p.height;
    const long long index = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (index >= total_pixels) return;
    const int py = static_cast<int>(index / p.width);
    const int px = static_cast<int>(index - static_cast<long long>(py) * p.width);
    const OrbitView orbit{p.orbit};
    const PlaneOut planes{p.p_iter, p.p_phase, p.p_dex, p.p_dey, p.p_t1, p.p_t2};
    StatSink<Stats> st;
    st.init();
    st.add(kPixels);

    // Pixel offsets (renderer.cpp:12764-12783): the view span times the
    // signed pixel-centre fraction, both in FloatExp.
    // A point render takes dc from its list (renderer.cpp:12838-12842).
    const double x_fraction = pixel_fraction(px, p.width, p.coordinate_mode);
    const double y_fraction = neg_(pixel_fraction(py, p.height, p.coordinate_mode));
    const Sc dc = p.points ? sc_make(p.points[index].re, p.points[index].im, p.points[index].e)
                           : sc_from_fe(fe_mul(p.view_width, x_fraction), fe_mul(p.view_height, y_fraction));
    const unsigned long long deadline_ns = p.deadline_base ? *p.deadline_base + p.budget_ns : 0ull;
    if constexpr (Planes) planes.clear(index, p.max_iter);
    Sc delta = dc;
    Sc derivative = sc_one();
    int ref = 1;
    int iteration = 1;
    if (p.series_on && nrm_cmp(sc_norm2(dc), p.series_r2) <= 0) {
        Sc value, poly;
        series_sum<Planes>([&](int k) { return ld_sc(&p.series[k]); }, p.series_terms, dc, value, poly);
        if constexpr (Planes) derivative = sc_add(sc_mul(poly, dc), value);
        delta = sc_mul(value, dc);
        ref = p.series_iteration;
        iteration = p.series_iteration;
        st.add(kSeriesPixels);
        st.add(kSeriesJumps, static_cast<unsigned long long>(iteration));
    }

    float out_value = 0.0f;
    std::uint32_t out_count = 0;
    bool escaped = false;
    bool have_total = false;
    Sc total = sc_zero();
    Nrm total_norm = nrm_make(0.0, 0);
    Nrm prev_total_norm = nrm_make(0.0, 0);
    Fe margin = fe_zero();
    Sc tortoise = sc_zero();
    int power = 1, length = 0;
    bool ready = false;
    bool pixel_disable_bla = false;
    int rebases = 0;
    unsigned ticks = 0;
    bool timed_out = false;
    bool unresolved = false;
    const int cycle_min = p.strict_cycle ? 2048 : 512;
    const int cycle_margin = p.strict_cycle ? 78 : 60;
    bool beyond = false;  // left the reference: exact steps finish the pixel
    Exit exit = kExitNone;
    double exit_mag2 = 0.0;
    Sc exit_total = sc_zero();
    Nrm exit_norm = nrm_make(0.0, 0), exit_previous = nrm_make(0.0, 0);

    while (iteration < p.max_iter) {
        if (deadline_ns && ((ticks++ & 255U) == 0U) && global_ns() >= deadline_ns) {
            out_value = nan_f();
            out_count = 0;
            timed_out = true;
            unresolved = true;
            st.add(kDeadlineAborts);
            st.add(kUnresolvedPixels);
            break;
        }
        if (ref < 0 || ref >= p.orbit_size) {
            out_value = encode(static_cast<double>(iteration), p.output_bias);
            out_count = static_cast<std::uint32_t>(iteration);
            exit = kExitRecord;
            exit_total = total;
            exit_norm = total_norm;
            exit_previous = prev_total_norm;
            escaped = true;
            break;
        }
        if (!have_total) {
            total = sc_add(orbit.z(ref), delta);
            margin = orbit.margin(ref, delta);
            total_norm = nrm_from_margin(margin, p.escape_mode);
        }
        have_total = false;
        // Glitch sentinel (renderer.cpp:12938-12988).
        const Fe glitch = orbit.glitch(ref);
        if (!is_zero(glitch.m) && fe_cmp(fe_make(total_norm.m, total_norm.e), glitch) < 0) {
            st.add(kGlitchCount);
            if (p.exact_flags) {
                // Strict point renders repair the pixel exactly (MPFR, on
                // the host) before any rebase (renderer.cpp:12944-12966).
                p.exact_flags[index] = 1;
                out_value = nan_f();
                out_count = 0;
                escaped = true;  // finished by the repair, as in the reference
                break;
            }
            if (p.allow_recovery && sc_finite(total) && ++rebases <= 64) {
                delta = total;
                ref = 0;
                have_total = false;
                continue;
            }
            out_value = nan_f();
            out_count = 0;
            unresolved = true;
            st.add(kUnresolvedPixels);
            break;
        }
        if (nrm_outside(total_norm, p.escape_mode) || fe_positive(margin)) {
            out_count = static_cast<std::uint32_t>(iteration);
            exit = kExitNorm;
            exit_total = total;
            exit_norm = total_norm;
            exit_previous = prev_total_norm;
            escaped = true;
            break;
        }
        const bool cycle_turn = p.cycle && iteration >= cycle_min && (iteration & 31) == 0;
        if (cycle_turn) {
            if (nrm_cmp(total_norm, nrm_make(0.75, 2)) < 0) {
                if (!ready) {
                    tortoise = total;
                    power = 1;
                    length = 0;
                    ready = true;
                } else {
                    const Nrm dist = sc_norm2(sc_sub(total, tortoise));
                    const int scale_e = total_norm.e > 0 ? total_norm.e : 0;
                    if (is_zero(dist.m) || dist.e <= scale_e - cycle_margin) {
                        st.add(kCycleInside);
                        out_value = encode(static_cast<double>(p.max_iter), p.output_bias);
                        out_count = static_cast<std::uint32_t>(p.max_iter);
                        escaped = true;
                        break;
                    }
                    if (++length >= power) {
                        tortoise = total;
                        power = power * 2 < (1 << 20) ? power * 2 : (1 << 20);
                        length = 0;
                    }
                }
            }
        }
        // Rebase when |Z + d| < |d| (renderer.cpp:13047-13153).
        const Nrm delta_norm = sc_norm2(delta);
        if (nrm_cmp(total_norm, delta_norm) < 0) {
            // At index 0 the total is the delta: where the two norms, rounded
            // differently, compare less there, the same turn repeats to the
            // limit.  64 turns of 23 FP64 instructions doubled a field's time
            // when one pixel in ten met them.
            const bool repeats = ref == 0 && same(delta, total) && deadline_ns == 0 && !cycle_turn;
            if (++rebases > 64 || repeats) {
                beyond = true;
                break;
            }
            delta = total;
            ref = 0;
            continue;
        }
        if (p.map_end > 1 && ref >= p.map_end) {
            beyond = true;
            break;
        }
        const Fe dn = fe_make(delta_norm.m, delta_norm.e);
        const int remaining = p.max_iter - iteration;
        const int order = p.approx_order >= 3 && delta_norm.e < -115 ? (delta_norm.e < -160 ? 1 : 2)
                                                                     : p.approx_order;
        const LinearStep* lin = nullptr;
        const CubicStep* cub = nullptr;
        const bool bla_allowed = !p.disable_bla && !pixel_disable_bla;
        if (bla_allowed) {
            if (order <= 1) {
                lin = lookup_linear(p, ref, dn, p.max_lin_len < remaining ? p.max_lin_len : remaining);
            } else {
                cub = lookup_cubic(p, ref, dn, p.max_bla_len < remaining ? p.max_bla_len : remaining);
            }
        }
        const int map_length = lin ? __ldg(&lin->len) : (cub ? __ldg(&cub->len) : 0);
        if (bla_allowed && (map_length <= 0 || ref + map_length > p.max_iter) && delta_norm.e > -90) {
            st.add(kDoubleTailPixels);
            const int tail_start = iteration;
            exit = double_tail<Planes, Stats, Axis>(p, orbit, index, dc, iteration, ref, delta, derivative, total_norm, st,
                                              ticks, deadline_ns, out_value, out_count, timed_out, unresolved,
                                              planes, exit_mag2, exit_total, exit_previous);
            if (timed_out || unresolved) break;
            const unsigned long long steps = iteration > tail_start ? iteration - tail_start : 0;
            st.add(kTailSteps, steps);
            st.max(kMaxTailSteps, steps);
            escaped = true;
            break;
        }
        if (map_length > 0 && ref + map_length <= p.max_iter) {
            st.add(kBlaBlocks);
            st.add(lin ? kLinearBlocks : kCubicBlocks);
            st.add(kSeriesJumps);
            st.bla_length(map_length);
            const Sc prev_delta = delta;
            const Sc prev_derivative = derivative;
            const int prev_ref = ref;
            const int prev_iteration = iteration;
            if (lin) {
                const Sc a = ld_sc(&lin->a);
                const Sc b = ld_sc(&lin->b);
                delta = sc_add(sc_mul(a, prev_delta), sc_mul(b, dc));
                if constexpr (Planes) derivative = sc_add(sc_mul(a, prev_derivative), b);
            } else {
                delta = apply_cubic(cub, prev_delta, dc, order);
                if constexpr (Planes) derivative = apply_cubic_derivative(cub, prev_delta, dc, prev_derivative, order);
            }
            ref += map_length;
            iteration += map_length;
            const Sc endpoint = sc_add(orbit.z(ref), delta);
            const Fe end_margin = orbit.margin(ref, delta);
            const Nrm endpoint_norm = nrm_from_margin(end_margin, p.escape_mode);
            if (!sc_finite(delta) || !sc_finite(endpoint)) {
                delta = prev_delta;
                derivative = prev_derivative;
                ref = prev_ref;
                iteration = prev_iteration;
                st.add(kBlaRetries);
                if (!pixel_disable_bla) st.add(kBlaDisabledPixels);
                pixel_disable_bla = true;
                have_total = false;
                continue;
            }
            if (nrm_cmp(endpoint_norm, nrm_make(0.75, 2)) >= 0) {
                // Replay the block one exact step at a time near escape.
                delta = prev_delta;
                derivative = prev_derivative;
                ref = prev_ref;
                iteration = prev_iteration;
                Sc replay_total = sc_zero();
                Nrm replay_norm = nrm_make(0.0, 0);
                Fe replay_margin = fe_zero();
                bool retry = false;
                for (int k = 0; k < map_length && iteration < p.max_iter; ++k) {
                    if (deadline_ns && ((ticks++ & 255U) == 0U) && global_ns() >= deadline_ns) {
                        out_value = nan_f();
                        out_count = 0;
                        timed_out = true;
                        unresolved = true;
                        st.add(kDeadlineAborts);
                        st.add(kUnresolvedPixels);
                        break;
                    }
                    const Sc z = orbit.z(ref);
                    if constexpr (Planes) {
                        const Sc prior = sc_add(z, delta);
                        derivative = sc_add(sc_twice(sc_mul(prior, derivative)), sc_one());
                    }
                    delta = sc_add(sc_twice(sc_mul(z, delta)), sc_add(sc_sqr(delta), dc));
                    ++ref;
                    ++iteration;
                    st.add(kReplaySteps);
                    st.add(kLogical);
                    replay_total = sc_add(orbit.z(ref), delta);
                    replay_margin = orbit.margin(ref, delta);
                    replay_norm = nrm_from_margin(replay_margin, p.escape_mode);
                    if (!sc_finite(delta) || !sc_finite(replay_total)) {
                        retry = true;
                        break;
                    }
                    if (nrm_outside(replay_norm, p.escape_mode) || fe_positive(replay_margin)) {
                        out_count = static_cast<std::uint32_t>(iteration);
                        exit = kExitNorm;
                        exit_total = replay_total;
                        exit_norm = replay_norm;
                        exit_previous = total_norm;
                        escaped = true;
                        break;
                    }
                }
                if (timed_out || escaped) break;
                if (retry) {
                    delta = prev_delta;
                    derivative = prev_derivative;
                    ref = prev_ref;
                    iteration = prev_iteration;
                    st.add(kBlaRetries);
                    if (!pixel_disable_bla) st.add(kBlaDisabledPixels);
                    pixel_disable_bla = true;
                    have_total = false;
                    continue;
                }
                total = replay_total;
                total_norm = replay_norm;
                margin = replay_margin;
                prev_total_norm = total_norm;
                have_total = true;
            } else {
                total = endpoint;
                total_norm = endpoint_norm;
                margin = end_margin;
                prev_total_norm = total_norm;
                have_total = true;
                st.add(kLogical, static_cast<unsigned long long>(map_length));
            }
            continue;
        }
        // One exact perturbation step.
        const Sc z = orbit.z(ref);
        const Nrm prior_norm = total_norm;
        if constexpr (Planes) {
            const Sc prior = sc_add(z, delta);
            derivative = sc_add(sc_twice(sc_mul(prior, derivative)), sc_one());
        }
        delta = sc_add(sc_twice(sc_mul(z, delta)), sc_add(sc_sqr(delta), dc));
        ++ref;
        ++iteration;
        prev_total_norm = prior_norm;
        st.add(kLogical);
        st.add(kExactSteps);
    }
    if (beyond) {
        exit = exact_continuation<Planes, Stats>(p, orbit, dc, total, total_norm, exit_previous, derivative, iteration,
                                                 st, ticks, deadline_ns, out_value, out_count, timed_out);
        exit_total = total;
        exit_norm = total_norm;
        if (timed_out) unresolved = true;
        escaped = !timed_out;
    }
    if (exit == kExitNorm) out_value = smooth_escape(iteration, exit_norm, p.output_bias);
    if (exit == kExitTail) {
        const double magnitude = sqrt(dmax(exit_mag2, escape_r2_d(p.escape_mode) + 1.0e-7));
        out_value = static_cast<float>((static_cast<double>(iteration) - log(log(magnitude)) / kLogTwo)
                                       - p.output_bias);
        if constexpr (Planes) {
            sc_normalize(exit_total);
            exit_norm = nrm_from_d(exit_mag2);
        }
    }
    if constexpr (Planes) {
        if (exit != kExitNone) planes.escape(index, kalles_raw(iteration), exit_total, exit_norm, exit_previous,
                                             derivative, p.pixel_spacing);
    }
    if (!escaped && !timed_out && !unresolved) {
        out_value = encode(static_cast<double>(p.max_iter), p.output_bias);
        out_count = static_cast<std::uint32_t>(p.max_iter);
    }
    st.max(kMaxPixelIterations, static_cast<unsigned long long>(iteration > 0 ? iteration : 0));
    p.out[index] = out_value;
    if (p.counts) p.counts[index] = out_count;
    st.flush(p.stats);
}

}  // namespace
}  // namespace plain

template <bool Planes, bool Stats>
cudaError_t launch_plain_variant(const PlainParams& p, cudaStream_t stream) {
    const long long pixels = static_cast<long long>(p.width) * p.height;
    const dim3 block(128);
    const dim3 grid(static_cast<unsigned>((pixels + 127) / 128));
    if (p.axis) {
        plain::plain_mandelbrot_kernel<Planes, Stats, true><<<grid, block, 0, stream>>>(p);
    } else {
        plain::plain_mandelbrot_kernel<Planes, Stats, false><<<grid, block, 0, stream>>>(p);
    }
    return cudaGetLastError();
}

}  // namespace fgb
