// The FP64 interval push, included by kpt_push.cu into both of its builds
// (strict and contracted arithmetic).
//
// What bounds it.  GB300 issues one FP64 warp instruction (add, multiply,
// FMA, compare or conversion alike) per 64 cycles and SM sub-partition,
// however many of its lanes are active and whatever else the warp could
// issue meanwhile; a division costs about 9 such slots, a square root 9, the
// project pow about 100.  One warp per sub-partition fills the pipe, and the
// time of an interval is the number of FP64 warp instructions on the busiest
// sub-partition.  The code below is therefore organised around that count,
// with the same operations on the same operands (strict arithmetic equals the
// lane-by-lane evaluation bit for bit, contracted arithmetic but for last bits
// of single particles, where the compiler fuses another product):
//
//  * Warp-collective work.  The table interpolation (17 operations per
//    component) and the divisions, square roots and powers of a substep are
//    spread over all 32 lanes as (particle, item) tasks that travel through
//    the warp's shared memory: n particles cost ceil(n K / 32) rounds instead
//    of K, so the warps of a small population, and those of the tail, whose
//    lanes are mostly idle, finish a substep in a third of the instructions.
//    A full warp takes the same rounds as before.
//  * Divisions by a known divisor (interval length, p0, cell width, 3) are
//    one multiplication and two FMAs with the rounded reciprocal (Markstein
//    1990; Brisebarre, Muller, Raina 2004), 3 slots instead of 9.
//  * Comparisons, finiteness tests, the cell index and the uniform draws run
//    on the integer pipes.
//  * A power's logarithm is taken once per base, not once per exponent
//    (strict arithmetic), and the step limiters that cannot win are not
//    divided out.
//
// Before and after are measured at push_f64_kernel.
#pragma once

#include "kpt_f64.cuh"

namespace kpt {
namespace {

// --------------------------------------------------------- warp-wide tasks
// Shared memory of one warp: task operands and results, the published
// stencils (kF64Stencil doubles per particle, aliasing the tasks) and the
// rows of sampled components (odd stride: the owners' reads are free of bank
// conflicts).
constexpr int kF64Bases = 4;       // distinct bases of a substep's powers
constexpr int kF64Stencil = 7;     // 4 corner weights, 2 time weights, point
constexpr int kF64TaskDoubles = 32 * (2 * kF64Bases + kF64Powers);
__host__ __device__ constexpr int f64_row(bool focused) { return focused ? 21 : 17; }
__host__ __device__ constexpr size_t f64_warp_doubles(bool focused) {
    return kF64TaskDoubles + 32u * f64_row(focused);
}
static_assert(32 * kF64Stencil <= kF64TaskDoubles, "stencils fit in the task area");

struct WarpTasks {
    double* buf;
    unsigned mask;  // the lanes with a particle
    int n;          // how many
    int rank;       // this lane's position among them (valid if it has one)
    bool mine;
};

// out[k] = f(in[k]) for the K operand pairs of every particle lane.
template <int K, typename F>
__device__ __forceinline__ void warp_map(const WarpTasks& w, const double2 (&in)[K],
                                         double (&out)[K], F f) {
    double2* buf = reinterpret_cast<double2*>(w.buf);
    if (w.mine) {
#pragma unroll
        for (int k = 0; k < K; ++k) buf[k * w.n + w.rank] = in[k];
    }
    __syncwarp();
#pragma unroll 1
    for (int t = static_cast<int>(threadIdx.x & 31u); t < K * w.n; t += 32) {
        const double2 v = buf[t];
        buf[t].x = f(v.x, v.y);
    }
    __syncwarp();
    if (w.mine) {
#pragma unroll
        for (int k = 0; k < K; ++k) out[k] = buf[k * w.n + w.rank].x;
    }
    __syncwarp();
}

struct DivTask {
    __device__ __forceinline__ double operator()(double a, double b) const { return a / b; }
};
struct SqrtTask {
    __device__ __forceinline__ double operator()(double a, double) const { return ::sqrt(a); }
};

// out[e] = base[plan.base[e]] ^ plan.exponent[e] for every particle lane.
template <int NB>
__device__ __forceinline__ void warp_pows(const WarpTasks& w, const PowPlan& plan,
                                          const double (&base)[NB], double (&out)[kF64Powers]) {
    static_assert(NB <= kF64Bases, "task area");
    double2* logs = reinterpret_cast<double2*>(w.buf);
    double* res = w.buf + 32 * 2 * kF64Bases;
    const int lane = static_cast<int>(threadIdx.x & 31u);
    // a payload no logarithm's low part has: "no logarithm here, x is the base"
    const double marker = __longlong_as_double(0x7ff8000000000001ll);
    if (w.mine) {
#pragma unroll
        for (int k = 0; k < NB; ++k) logs[k * w.n + w.rank] = make_double2(base[k], marker);
    }
    __syncwarp();
    const int powers = plan.powers;
#if KPT_PUSH_PART == 1
    // x^y = exp(y ln x) in kpt_pow's own steps for a positive, finite, normal
    // x other than 1, the logarithm shared by the base's exponents; every
    // other base (and a launch with a non-finite exponent) goes through
    // kpt_pow as a whole.
    if (plan.shared_logs != 0) {
#pragma unroll 1
        for (int t = lane; t < NB * w.n; t += 32) {
            const double x = logs[t].x;
            const unsigned hi = static_cast<unsigned>(__double2hiint(x));
            if (hi - 0x00100000u < 0x7ff00000u - 0x00100000u &&
                f64_bits(x) != 0x3ff0000000000000ll) {
                double2 l;
                kpt_pow_log(x, &l.x, &l.y);
                logs[t] = l;
            }
        }
        __syncwarp();
    }
#endif
#pragma unroll 1
    for (int t = lane; t < powers * w.n; t += 32) {
        const int e = t / w.n;
        const double y = plan.exponent[e];
        const double2 l = logs[plan.base[e] * w.n + (t - e * w.n)];
#if KPT_PUSH_PART == 1
        if (f64_bits(l.y) == f64_bits(marker)) {
            res[t] = kpt_pow(l.x, y);
        } else if (f64_zero(y)) {
            res[t] = 1.0;
        } else {
            const double t_hi = __dmul_rn(y, l.x);
            res[t] = kpt_pow_exp(t_hi, __fma_rn(y, l.y, __fma_rn(y, l.x, -t_hi)));
        }
#else
        res[t] = ::pow(l.x, y);
#endif
    }
    __syncwarp();
    if (w.mine) {
#pragma unroll
        for (int e = 0; e < kF64Powers; ++e) out[e] = e < powers ? res[e * w.n + w.rank] : 1.0;
    }
    __syncwarp();
}

// --------------------------------------------------------------- state
struct StateF64 {
    double x, y, p, t, diag_dt, mu;
    int steps;
    int status;
    uint32_t index;
};

template <bool FOCUSED>
__device__ __forceinline__ void load(StateF64& st, const PushParams& P, uint32_t index) {
    const ParticleArrays& a = P.parts;
    st.index = index;
    st.x = a.x[index];
    st.y = a.y[index];
    st.p = a.p[index];
    st.t = a.t[index];
    st.diag_dt = a.step_dt[index];
    st.mu = FOCUSED ? clamp_mu(a.mu[index], P.s.mu_max) : 0.0;
    st.steps = 0;
    st.status = 0;
}

template <bool FOCUSED>
__device__ __forceinline__ void store(StateF64& st, const PushParams& P) {
    const ParticleArrays& a = P.parts;
    const DeviceSettings& s = P.s;
    if (st.steps >= s.max_steps && st.t < P.interval_end) st.status = 2;
    const uint32_t i = st.index;
    a.x[i] = wrap_driver(st.x, s.x_lower, s.x_upper, s.x_width);
    a.y[i] = wrap_driver(st.y, s.y_lower, s.y_upper, s.y_width);
    a.p[i] = st.p;
    a.t[i] = st.t;
    a.step_dt[i] = st.diag_dt;
    if (FOCUSED) a.mu[i] = st.mu;
    a.status[i] = st.status;
}

__device__ __forceinline__ bool live(const StateF64& st, const PushParams& P) {
    return st.t < P.interval_end && st.steps < P.s.max_steps;
}

// --------------------------------------------------------------- sampling
// wrap_driver; a coordinate inside [lower, upper) is its own wrap.
__device__ __forceinline__ double wrap_f64(double v, const F64AxisKeys& k, double lower,
                                           double upper, double width) {
    const long long key = f64_key(f64_bits(v));
    return key >= k.lower && key < k.upper ? v : wrap_driver(v, lower, upper, width);
}

// axis_stencil of grid_wrap(q): the lower cell, whether the upper one
// differs, and the upper weight.  k.floor_zero bounds the coordinates whose
// wrap count floor((q - lower) inv_width) is surely 0; on a uniform axis the
// logical index (q - start) / step - 1/2 of a coordinate in the domain lies
// in [-1/2, n - 1/2].
__device__ __forceinline__ void axis_stencil_f64(const Axis& a, const F64AxisKeys& k, double q,
                                                 int& lo, int& span, double& w) {
    const long long key = f64_key(f64_bits(q));
    const bool inside = key >= k.lower && key < k.floor_zero;
    const double c = inside ? q : grid_wrap(a, q);
    const long long ckey = f64_key(f64_bits(c));
    if (!(ckey >= k.lower && ckey < k.upper)) {  // not a number, or an end of the axis
        int hi;
        axis_stencil(a, c, lo, hi, w);
        span = hi - lo;
        return;
    }
    double logical;
    if (!a.stored) {
        logical = __dsub_rn(div_known(__dsub_rn(c, a.start), a.step, k.rcp_step), 0.5);
    } else {
        // cell_grid_index on a stored axis, the interval search on the keys
        const double* x = a.centers;  // logical -2 .. n + 1
        int b = 0;
        if (a.bucket_count > 0) {
            b = static_cast<int>((c - a.bucket_origin) * a.bucket_scale);
            b = b < 0 ? 0 : (b >= a.bucket_count ? a.bucket_count - 1 : b);
            b = __ldg(a.buckets + b);
        } else {
            b = -2;
        }
        const long long* bits = reinterpret_cast<const long long*>(x);
        while (b > -2 && ckey < f64_key(__ldg(bits + b + 2))) --b;
        while (b < a.n && ckey >= f64_key(__ldg(bits + b + 3))) ++b;
        const double left = __ldg(x + b + 2);
        const double right = __ldg(x + b + 3);
        const double lb = b >= 0 ? f64_of_int(b) : -f64_of_int(-b);
        logical = __dadd_rn(lb, __ddiv_rn(__dsub_rn(c, left), __dsub_rn(right, left)));
    }
    if (!f64_floor(logical, lo) || lo < -1 || lo >= a.n + 1) {  // outside the cells
        int hi;
        axis_stencil(a, c, lo, hi, w);
        span = hi - lo;
        return;
    }
    span = 1;
    w = __dsub_rn(logical, lo < 0 ? -1.0 : f64_of_int(lo));
}

constexpr int kF64PointBits = 62;  // of a published stencil's point; spans above

// The first part of a substep, warp-collective: count it, wrap the position,
// publish the stencil, interpolate the tables component by component over
// all lanes (task t = particle t / C, component t % C: neighbouring lanes
// read neighbouring doubles of a table row), rows[rank][component].
template <bool FOCUSED>
__device__ __forceinline__ void sample_f64(StateF64& st, const PushParams& P,
                                           const WarpTasks& w, double* rows) {
    constexpr int C = FOCUSED ? 21 : 16;
    constexpr int STRIDE = FOCUSED ? 22 : 16;
    constexpr int ROW = f64_row(FOCUSED);
    const DeviceSettings& s = P.s;
    const F64Consts& k = P.f64;
    if (w.mine) {
        ++st.steps;
        st.x = wrap_f64(st.x, k.axis[0], s.x_lower, s.x_upper, s.x_width);
        st.y = wrap_f64(st.y, k.axis[1], s.y_lower, s.y_upper, s.y_width);
        const double rt = div_known(__dsub_rn(st.t, P.interval_start), s.mhd_dt, k.rcp_mhd_dt);
        int lo0, lo1, span0, span1;
        double w0, w1;
        axis_stencil_f64(P.grid.axis[0], k.axis[0], __dadd_rn(st.x, s.shift_x), lo0, span0, w0);
        axis_stencil_f64(P.grid.axis[1], k.axis[1], __dadd_rn(st.y, s.shift_y), lo1, span1, w1);
        const double a0 = 1.0 - w0;
        const double a1 = 1.0 - w1;
        double* sc = w.buf + w.rank * kF64Stencil;
        sc[0] = a0 * a1;
        sc[1] = w0 * a1;
        sc[2] = a0 * w1;
        sc[3] = w0 * w1;
        // the time weight clamped to [0, 1]
        double uw = rt;
        if (!f64_nan(rt) && !f64_zero(rt)) {
            uw = f64_bits(rt) < 0 ? 0.0 : (f64_bits(rt) > 0x3ff0000000000000ll ? 1.0 : rt);
        }
        sc[4] = 1.0 - uw;
        sc[5] = uw;
        const unsigned long long pt =
            static_cast<unsigned long long>(lo0 + 2) +
            static_cast<unsigned long long>(lo1 + 2) * static_cast<unsigned long long>(P.grid.ex);
        sc[6] = __longlong_as_double(static_cast<long long>(
            pt | (static_cast<unsigned long long>(span0) << kF64PointBits) |
            (static_cast<unsigned long long>(span1) << (kF64PointBits + 1))));
    }
    __syncwarp();
    const double* __restrict__ lower = static_cast<const double*>(P.lower);
    const double* __restrict__ upper = static_cast<const double*>(P.upper);
    const size_t ex = static_cast<size_t>(P.grid.ex);
    const bool use_time = s.time_interpolation != 0;
    const int tasks = w.n * C;
    int t = static_cast<int>(threadIdx.x & 31u);
    // the next round's loads are in flight during a round's arithmetic
    double v[8], next[8];
    int q = 0, comp = 0;
    auto fetch = [&](int task, double (&dst)[8]) {
        const int particle = task / C;
        const int c = task - particle * C;
        const unsigned long long word = static_cast<unsigned long long>(
            f64_bits(w.buf[particle * kF64Stencil + 6]));
        const size_t pt = static_cast<size_t>(word & ((1ull << kF64PointBits) - 1ull));
        const size_t d0 = static_cast<size_t>((word >> kF64PointBits) & 1ull);
        const size_t d1 = static_cast<size_t>(word >> (kF64PointBits + 1)) * ex;
        const size_t at[4] = {pt, pt + d0, pt + d1, pt + d0 + d1};
#pragma unroll
        for (int corner = 0; corner < 4; ++corner) {
            dst[corner] = __ldg(lower + at[corner] * STRIDE + c);
        }
        if (use_time) {
#pragma unroll
            for (int corner = 0; corner < 4; ++corner) {
                dst[4 + corner] = __ldg(upper + at[corner] * STRIDE + c);
            }
        }
    };
    if (t < tasks) fetch(t, next);
#pragma unroll 1
    for (; t < tasks; t += 32) {
#pragma unroll
        for (int m = 0; m < 8; ++m) v[m] = next[m];
        if (t + 32 < tasks) fetch(t + 32, next);
        q = t / C;
        comp = t - q * C;
        const double* sc = w.buf + q * kF64Stencil;
        double out = sc[0] * v[0];
#pragma unroll
        for (int corner = 1; corner < 4; ++corner) out = out + sc[corner] * v[corner];
        if (use_time) {
            double up = sc[0] * v[4];
#pragma unroll
            for (int corner = 1; corner < 4; ++corner) up = up + sc[corner] * v[4 + corner];
            out = sc[4] * out + sc[5] * up;
        }
        rows[q * ROW + comp] = out;
    }
    __syncwarp();
}

// ---------------------------------------------------------------- physics
// Step limiters in the reference's order, for operands the reduced form below
// does not cover (src/main.cpp:1243-1257, :1596-1650).
template <bool FOCUSED>
__device__ __noinline__ double step_limit_general(double dx, double dy, double skpara,
                                                  double skperp, double dx_dt, double dy_dt,
                                                  double dp_dt, double dmu_dt, double duu,
                                                  double p) {
    const double scale = skperp > 0.0 ? skperp : skpara;
    const double diffusion = FOCUSED ? scale : skpara;
    double dt = min_positive(square(0.5 * dx / diffusion), square(0.5 * dy / diffusion));
    dt = min_positive(dt, square(scale / dx_dt));
    dt = min_positive(dt, square(scale / dy_dt));
    dt = min_positive(dt, 0.1 * p / fabs(dp_dt));
    if (FOCUSED) {
        dt = min_positive(dt, 0.1 / fabs(dmu_dt));
        dt = min_positive(dt, 2.0 * duu / square(dmu_dt));
    }
    return dt;
}

// Physics, step size, noise and state update of one substep from the sampled
// components c (src/main.cpp:1167-1303 Parker, :1421-1730 focused), as
// physics / increments / advance_mixed evaluate them in FP32, warp-collective:
// every lane calls it, lanes without a particle only take tasks.  The
// expressions keep the reference's operand order.  served: the learned
// closure's values (SURR).  Returns whether the particle goes on.
template <bool FOCUSED, bool SURR>
__device__ __forceinline__ bool advance_f64(StateF64& st, const PushParams& P, const double* c,
                                            const WarpTasks& w, const Served* served) {
    const DeviceSettings& set = P.s;
    const Consts<double>& s = P.kd;
    const F64Consts& k = P.f64;
    const bool mine = w.mine;
    const double p = st.p;
    double vx, vy, bx, by, bz, b, dvx_dx, dvy_dy, dbx_dx, dbx_dy, dby_dx, dby_dy, dbz_dx, dbz_dy,
        db_dx, db_dy;
    double dvx_dy = 0, dvy_dx = 0, dvz_dx = 0, dvz_dy = 0;
    if (FOCUSED) {
        vx = c[0]; vy = c[1]; bx = c[3]; by = c[4]; bz = c[5]; b = c[6];
        dvx_dx = c[7]; dvx_dy = c[8]; dvy_dx = c[9]; dvy_dy = c[10]; dvz_dx = c[11];
        dvz_dy = c[12]; dbx_dx = c[13]; dbx_dy = c[14]; dby_dx = c[15]; dby_dy = c[16];
        dbz_dx = c[17]; dbz_dy = c[18]; db_dx = c[19]; db_dy = c[20];
    } else {
        vx = c[0]; vy = c[1]; bx = c[2]; by = c[3]; bz = c[4]; b = c[5]; dvx_dx = c[6];
        dvy_dy = c[7]; dbx_dx = c[8]; dbx_dy = c[9]; dby_dx = c[10]; dby_dy = c[11];
        dbz_dx = c[12]; dbz_dy = c[13]; db_dx = c[14]; db_dy = c[15];
    }
    bool ok = f64_finite(p) && f64_positive(p) && f64_finite(b) && f64_positive(b);

    // quotients and roots that need no power
    const double p0 = s.p0;
    const double gamma = s.gamma_turb;
    double pitch_mu = 0.0, mu2 = 0.0, bv_gradv = 0.0, speed = 0.0;
    double ib, drift1, drift2;
    {
        const double2 in[3] = {make_double2(1.0, b), make_double2(k.drift1_p0, p),
                               make_double2(k.drift2_p0_p0, p * p)};
        double out[3];
        warp_map<3>(w, in, out, DivTask());
        ib = out[0];
        drift1 = out[1];
        drift2 = out[2];
    }
    const double ib2 = ib * ib;
    const double ib3 = ib2 * ib;
    const double p_over_p0 = div_known(p, p0, k.rcp_p0);
    double drift_denominator, lorentz = 0.0;
    if (FOCUSED) {
        pitch_mu = f64_clamp(st.mu, s.mu_max);
        mu2 = pitch_mu * pitch_mu;
        speed = div_known(s.particle_v0 * p, p0, k.rcp_p0);
        bv_gradv = (bx * (vx * dvx_dx + vy * dvx_dy) + by * (vx * dvy_dx + vy * dvy_dy) +
                    bz * (vx * dvz_dx + vy * dvz_dy)) *
                   ib;
    }
    // the learned closure serves kappa, D and D' (SURR); lanes it does not
    // serve take the plain ones
    const bool need = !SURR || __any_sync(0xffffffffu, mine && !served->use);
    const bool plain_qlt = FOCUSED && s.closure != 0 && need;
    if (plain_qlt) {
        const double2 in[2] = {make_double2(square(drift1) + square(drift2), 0.0),
                               make_double2(1.0 + p * p, 0.0)};
        double out[2];
        warp_map<2>(w, in, out, SqrtTask());
        drift_denominator = out[0];
        lorentz = out[1];
    } else {
        const double2 in[1] = {make_double2(square(drift1) + square(drift2), 0.0)};
        double out[1];
        warp_map<1>(w, in, out, SqrtTask());
        drift_denominator = out[0];
    }
    double vdp, pitch_bv = 0.0, two_bv = 0.0, omega = 0.0;
    if (FOCUSED) {
        const double2 in[4] = {make_double2(k.inv_charge, drift_denominator),
                               make_double2(pitch_mu * bv_gradv, speed),
                               make_double2(2.0 * bv_gradv, speed),
                               make_double2(s.qlt_omega0 * b, lorentz)};
        double out[4];
        if (plain_qlt) {
            warp_map<4>(w, in, out, DivTask());
            omega = out[3];
        } else {
            const double2 in3[3] = {in[0], in[1], in[2]};
            double out3[3];
            warp_map<3>(w, in3, out3, DivTask());
            out[0] = out3[0];
            out[1] = out3[1];
            out[2] = out3[2];
        }
        vdp = out[0];
        pitch_bv = out[1];
        two_bv = out[2];
    } else {
        vdp = k.inv_charge / drift_denominator;
    }

    // powers: those of kappa (b, p / p0), then the closure's
    double pw[kF64Powers];
    double reg = 0.0, xi = 0.0;
    if (need) {
        if (plain_qlt) {
            reg = fabs(pitch_mu) + s.qlt_h0;
            xi = omega * s.qlt_lc / speed;
            const double base[4] = {b, p_over_p0, reg, xi};
            warp_pows<4>(w, P.pows, base, pw);
        } else if (FOCUSED) {
            const double base[3] = {b, p_over_p0, fabs(pitch_mu)};
            warp_pows<3>(w, P.pows, base, pw);
        } else {
            const double base[2] = {b, p_over_p0};
            warp_pows<2>(w, P.pows, base, pw);
        }
    }
    double kpara;
    if (SURR && served->use) {
        kpara = served->kpara;
    } else {
        double knorm_para = 1.0;
        if (s.magnetic_dependency == 1) knorm_para *= pw[0];
        double knorm = knorm_para;
        if (s.momentum_dependency == 1) knorm *= pw[1];
        kpara = s.kpara0 * knorm;
    }
    const double kperp = kpara * s.kperp_over_kpara;
    ok = ok && f64_finite(kpara) && f64_positive(kpara) && f64_finite(kperp) && !f64_negative(kperp);
    double skpara = 0.0, skperp, skpara_perp = 0.0;
    if (FOCUSED) {
        const double2 in[1] = {make_double2(2.0 * kperp, 0.0)};
        double out[1];
        warp_map<1>(w, in, out, SqrtTask());
        skperp = out[0];
        if (mine && !f64_positive(skperp)) skpara = ::sqrt(2.0 * kpara);
    } else {
        const double2 in[3] = {make_double2(2.0 * kpara, 0.0), make_double2(2.0 * kperp, 0.0),
                               make_double2(2.0 * (kpara - kperp), 0.0)};
        double out[3];
        warp_map<3>(w, in, out, SqrtTask());
        skpara = out[0];
        skperp = out[1];
        skpara_perp = out[2];
    }
    const double kpp = FOCUSED ? -kperp : kpara - kperp;

    double dkdx = 0.0;
    double dkdy = 0.0;
    if (s.magnetic_dependency == 1) {
        const double magnetic_exponent = gamma - 2.0;
        dkdx = db_dx * ib * magnetic_exponent;
        dkdy = db_dy * ib * magnetic_exponent;
    }
    const double dkxx_dx = kperp * dkdx + kpp * dkdx * bx * bx * ib2 +
                           2.0 * kpp * bx * (dbx_dx * b - bx * db_dx) * ib3;
    const double dkyy_dy = kperp * dkdy + kpp * dkdy * by * by * ib2 +
                           2.0 * kpp * by * (dby_dy * b - by * db_dy) * ib3;
    const double dkxy_dx = kpp * dkdx * bx * by * ib2 +
                           kpp * ((dbx_dx * by + bx * dby_dx) * ib2 - 2.0 * bx * by * db_dx * ib3);
    const double dkxy_dy = kpp * dkdy * bx * by * ib2 +
                           kpp * ((dbx_dy * by + bx * dby_dy) * ib2 - 2.0 * bx * by * db_dy * ib3);

    double dx_dt, dy_dt, dp_dt;
    double dmu_dt = 0.0, duu = 0.0;
    if (FOCUSED) {
        const double muf1 = 0.5 * (1.0 - mu2);
        const double muf2 = 0.5 * (3.0 * mu2 - 1.0);
        const double kx = bx * dbx_dx + by * dbx_dy;
        const double ky = bx * dby_dx + by * dby_dy;
        const double kz = bx * dbz_dx + by * dbz_dy;
        const double bdot_curvb = bx * dbz_dy - by * dbz_dx + bz * (dby_dx - dbx_dy);
        const double vdx = vdp * (muf1 * (-bz * db_dy) * ib2 + mu2 * (by * kz - bz * ky) * ib3 +
                                  muf1 * bx * bdot_curvb * ib3);
        const double vdy = vdp * (muf1 * (bz * db_dx) * ib2 + mu2 * (bz * kx - bx * kz) * ib3 +
                                  muf1 * by * bdot_curvb * ib3);
        ok = ok && f64_finite(speed) && f64_positive(speed);
        const double v_parallel_over_b = speed * pitch_mu * ib;
        dx_dt = vx + vdx + v_parallel_over_b * bx + dkxx_dx + dkxy_dy;
        dy_dt = vy + vdy + v_parallel_over_b * by + dkxy_dx + dkyy_dy;

        const double divv = dvx_dx + dvy_dy;
        const double bb_gradv = (bx * (bx * dvx_dx + by * dvx_dy) +
                                 by * (bx * dvy_dx + by * dvy_dy) +
                                 bz * (bx * dvz_dx + by * dvz_dy)) *
                                ib2;
        const double acc_rate = -(muf1 * divv + muf2 * bb_gradv + pitch_bv);
        dp_dt = p * acc_rate;

        const double div_bnorm = -(bx * db_dx + by * db_dy) * ib2;
        dmu_dt = speed * div_bnorm + pitch_mu * divv - 3.0 * pitch_mu * bb_gradv - two_bv;
        dmu_dt *= 0.5 * (1.0 - mu2);
        double duu_du = 0.0;
        if (SURR && served->use) {
            duu = served->duu;
            duu_du = served->duu_du;
        } else if (s.closure != 0) {
            // slab QLT (LegencyModel.hpp:557-645): Omega = Omega_0 |B| / gamma
            const double one_minus_mu2 = 1.0 - pitch_mu * pitch_mu;
            if (f64_positive(one_minus_mu2)) {
                const double gk = s.qlt_gk;
                const double reg_gk1 = pw[2];
                const double denominator = pw[3] + pw[4];
                const double prefactor = (0.25 * 3.141592653589793238462643383279502884) * omega *
                                         s.qlt_sigma2 * s.qlt_norm;
                duu = prefactor * one_minus_mu2 * xi * reg_gk1 / denominator;
                if (!f64_zero(duu) && !f64_zero(pitch_mu)) {
                    const double sign_mu = f64_positive(pitch_mu) ? 1.0 : -1.0;
                    const double shape =
                        sign_mu * ((gk - 1.0) / reg - gk * reg_gk1 / denominator);
                    const double endpoint = -2.0 * pitch_mu / one_minus_mu2;
                    duu_du = duu * (endpoint + shape);
                }
            }
        } else {
            // the driver's reduced closure (src/main.cpp:1551-1589)
            const double dtmp = pw[2] + s.h0;
            const double duu0 = s.duu0;
            duu = duu0 * (1.0 - mu2) * dtmp;
            if (f64_positive(pitch_mu)) {
                duu_du = duu0 * (-2.0 * pitch_mu * dtmp + (1.0 - mu2) * pw[3]);
            } else if (f64_negative(pitch_mu)) {
                duu_du = duu0 * (-2.0 * pitch_mu * dtmp - (1.0 - mu2) * pw[3]);
            }
            double duu_norm = 1.0;
            if (s.magnetic_dependency == 1) duu_norm *= pw[4];
            if (s.momentum_dependency == 1) duu_norm *= pw[5];
            duu *= duu_norm;
            duu_du *= duu_norm;
        }
        dmu_dt += duu_du;
        ok = ok && f64_finite(dmu_dt) && f64_finite(duu) && !f64_negative(duu);
    } else {
        const double vdx = vdp * (dbz_dy * ib2 - 2.0 * bz * db_dy * ib3);
        const double vdy = vdp * (-dbz_dx * ib2 + 2.0 * bz * db_dx * ib3);
        dx_dt = vx + vdx + dkxx_dx + dkxy_dy;
        dy_dt = vy + vdy + dkxy_dx + dkyy_dy;
        const double divv = dvx_dx + dvy_dy;
        dp_dt = div_known(-p * divv, 3.0, k.rcp_3);
    }

    // Step limiters.  For finite non-zero rates the minimum over both axes is
    // the quotient of the smaller cell, or of the larger rate (division,
    // squaring and the minimum are monotone under rounding); with a single
    // permitted step (dt_min = dt_max) no quotient is needed.
    double dt = set.dt_min;
    bool moves = !f64_zero(dx_dt) && !f64_zero(dy_dt) && !f64_zero(dp_dt);
    const double scale = f64_positive(skperp) ? skperp : skpara;
    if (FOCUSED) moves = moves && !f64_zero(dmu_dt) && f64_positive(scale);
    bool reduced = f64_moderate(dx_dt) && f64_moderate(dy_dt) && f64_moderate(dp_dt) &&
                   f64_moderate(scale) && f64_moderate(FOCUSED ? scale : skpara);
    if (FOCUSED) {
        reduced = reduced && f64_moderate(dmu_dt) && (f64_moderate(duu) || f64_zero(duu));
    }
    if (k.single_step == 0) {
        const double rate = f64_bits(fabs(dx_dt)) > f64_bits(fabs(dy_dt)) ? dx_dt : dy_dt;
        double limit;
        if (FOCUSED) {
            const double2 in[5] = {make_double2(k.half_cell, scale), make_double2(scale, rate),
                                   make_double2(0.1 * p, fabs(dp_dt)),
                                   make_double2(0.1, fabs(dmu_dt)),
                                   make_double2(2.0 * duu, square(dmu_dt))};
            double out[5];
            warp_map<5>(w, in, out, DivTask());
            limit = square(out[0]);
            const double bound[4] = {square(out[1]), out[2], out[3], out[4]};
#pragma unroll
            for (int m = 0; m < 4; ++m) limit = f64_below(bound[m], limit) ? bound[m] : limit;
        } else {
            const double2 in[3] = {make_double2(k.half_cell, skpara), make_double2(scale, rate),
                                   make_double2(0.1 * p, fabs(dp_dt))};
            double out[3];
            warp_map<3>(w, in, out, DivTask());
            limit = square(out[0]);
            const double bound[2] = {square(out[1]), out[2]};
#pragma unroll
            for (int m = 0; m < 2; ++m) limit = f64_below(bound[m], limit) ? bound[m] : limit;
        }
        if (moves) dt = limit;
    }
    if (mine && ok && moves && !reduced) {
        dt = step_limit_general<FOCUSED>(s.dx, s.dy, skpara, skperp, dx_dt, dy_dt, dp_dt, dmu_dt,
                                         duu, p);
    }
    const bool number = !f64_nan(dt);
    if (number) {
        if (f64_below(dt, set.dt_min)) dt = set.dt_min;
        if (f64_below(set.dt_max, dt)) dt = set.dt_max;
    }
    if (ok) st.diag_dt = dt;
    const double remaining = __dsub_rn(P.interval_end, st.t);
    if (number && f64_below(remaining, dt)) dt = remaining;
    ok = ok && number && f64_finite(dt) && f64_positive(dt);

    // displacements and the new pitch cosine (src/main.cpp:1280-1291,
    // :1660-1702)
    const uint32_t block = 2u * static_cast<uint32_t>(st.steps - 1);
    const uint4 r0 = philox4x32_10(make_uint4(block, st.index, P.frame, kTagPush), P.key);
    const uint4 r1 = philox4x32_10(make_uint4(block + 1u, st.index, P.frame, kTagPush), P.key);
    auto noise = [](uint32_t lo, uint32_t hi) {
        return __dadd_rn(-kSqrt3, __dmul_rn(kSqrt3 + kSqrt3, u01_f64_int(lo, hi)));
    };
    const double ran1 = noise(r0.x, r0.y);
    const double ran2 = noise(r0.z, r0.w);
    double delta_x, delta_y;
    if (FOCUSED) {
        const double bxn = bx * ib;
        const double byn = by * ib;
        const double bzn = bz * ib;
        const double2 in[3] = {make_double2(dt, 0.0), make_double2(2.0 * duu, 0.0),
                               make_double2(bxn * bxn + byn * byn, 0.0)};
        double out[3];
        warp_map<3>(w, in, out, SqrtTask());
        const double sdt = out[0];
        const double bxy_norm = out[2];
        double stochastic_x = 0.0;
        double stochastic_y = 0.0;
        if (f64_positive(bxy_norm) && !f64_nan(bxy_norm)) {
            const double ibxy_norm = 1.0 / bxy_norm;
            // (-by, +bx) on ran2 as written in src/main.cpp:1682-1687.
            stochastic_x = skperp * ibxy_norm * sdt * (-bxn * bzn * ran1 - by * ran2);
            stochastic_y = skperp * ibxy_norm * sdt * (-byn * bzn * ran1 + bx * ran2);
        }
        delta_x = dx_dt * dt + stochastic_x;
        delta_y = dy_dt * dt + stochastic_y;
        const double pitch_random = noise(r1.z, r1.w);
        const double mu =
            f64_clamp(pitch_mu + dmu_dt * dt + pitch_random * out[1] * sdt, s.mu_max);
        if (ok) st.mu = mu;
    } else {
        const double ran3 = noise(r1.x, r1.y);
        const double sdt = ::sqrt(dt);
        delta_x = dx_dt * dt + ran1 * skperp * sdt + ran3 * skpara_perp * sdt * bx * ib;
        delta_y = dy_dt * dt + ran2 * skperp * sdt + ran3 * skpara_perp * sdt * by * ib;
    }
    if (!mine) return false;
    if (!ok) {
        st.status = 2;
        return false;
    }
    st.x = __dadd_rn(st.x, delta_x);
    st.y = __dadd_rn(st.y, delta_y);
    st.p = __dadd_rn(st.p, dp_dt * dt);
    st.t = __dadd_rn(st.t, dt);
    if (!f64_nan(st.p) && f64_below(st.p, k.p_floor)) st.p = k.p_floor;
    if (!f64_finite(st.x) || !f64_finite(st.y) || !f64_finite(st.p) || !f64_finite(st.t)) {
        st.status = 2;
        return false;
    }
    return f64_key(f64_bits(st.t)) < k.end_key && st.steps < set.max_steps;
}

// ----------------------------------------------------------------- kernel
// The FP64 focused substep with the learned closure (mma.sync engine): the
// table is sampled and the physics evaluated in FP64, the network serves
// D_mumu, dD_mumu/dmu and kappa_parallel in place of the plain closure's
// powers.  The served values are FP32 whichever closure gives them, so the
// lanes outside the training box, and the judged and blended ones, take the
// plain closure in FP32 too.
template <bool FP16, int H>
__device__ __forceinline__ Served serve_f64(const StateF64& st, const PushParams& P, bool have,
                                            double b64, const uint2* smem, BlockTally& tally) {
    const SurrogateDevice& sg = P.sg;
    const SurrogateBox& box = sg.box;
    float f[kMlpIn] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    bool use = false;
    const double mu = f64_clamp(st.mu, P.kd.mu_max);
    const float b = static_cast<float>(b64);
    const float p = static_cast<float>(st.p);
    const float amu = fabsf(static_cast<float>(mu));
    if (have && sg.constants_in_box && amu >= box.mu_cut && b > 0.0f && p > 0.0f) {
        const float lm = __logf(amu);
        const float lp = __logf(p);
        const float lb = __logf(b);
        use = lm <= box.in_hi[0] && lp >= box.in_lo[1] && lp <= box.in_hi[1] &&
              lb >= box.in_lo[2] && lb <= box.in_hi[2];
        if (use) {
            f[0] = lm * box.in_scale[0] + box.in_offset[0];
            f[1] = lp * box.in_scale[1] + box.in_offset[1];
            f[2] = lb * box.in_scale[2] + box.in_offset[2];
            f[3] = sg.f3;
            f[4] = sg.f4;
        }
    }
    float y[kMlpOut];
    __syncwarp();
    mlp_warp<FP16, H>(smem, f, y);
    Served served{};
    if (have) {
        served = serve_closure(P, use, static_cast<float>(mu), b, p, st.steps, y, tally);
    }
    return served;
}

// Persistent warps with lane refill.  A warp holds at most P.f64.lane_cap
// particles: its first ones are fixed by its place (warps of different SMs
// first), the rest come from the device cursor.  The cap spreads a
// population smaller than the lanes of one warp per sub-partition over all
// of those (a warp's FP64 instructions cost the same for one lane as for 32,
// and the shared tasks make thin warps cheaper).  P.f64.simple: no refill, a
// warp takes 32 particles at a time and finishes them (the schedule
// alternative).
// Blocks of 128 threads an SM's registers hold.  The contracted build keeps
// all its values in registers (188): which products fuse into FMAs is the
// assembler's choice, and at 128 registers it chose otherwise.
#if KPT_PUSH_PART == 1
constexpr int kF64Blocks = 4;
#else
constexpr int kF64Blocks = 2;
#endif
template <bool FOCUSED, int SURR = 0>
__global__ void __launch_bounds__(128, kF64Blocks) push_f64_kernel(const PushParams P) {
    const unsigned full = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31u;
    const unsigned lanes_below = (1u << lane) - 1u;
    extern __shared__ __align__(16) unsigned char f64_smem[];
    const uint2* network = reinterpret_cast<const uint2*>(f64_smem);
    __shared__ BlockTally tally;
    tally_init(tally);
    if (SURR) {
        load_surrogate_block<surr_hidden(SURR)>(P.sg.block, reinterpret_cast<uint2*>(f64_smem));
    }
    double* mem = reinterpret_cast<double*>(
                      f64_smem + (SURR ? (mlp_smem_bytes(surr_hidden(SURR)) + 15) / 16 * 16 : 0)) +
                  (threadIdx.x >> 5) * f64_warp_doubles(FOCUSED);
    double* rows = mem + kF64TaskDoubles;
    const unsigned cap = P.f64.lane_cap;
    const uint64_t warps = static_cast<uint64_t>(gridDim.x) * (blockDim.x >> 5);
    const uint64_t placed = warps * cap;  // particles placed by position
    uint64_t next = (static_cast<uint64_t>(threadIdx.x >> 5) * gridDim.x + blockIdx.x) * cap;
    bool first = true;
    StateF64 st{};
    bool have = false;
    bool exhausted = false;
    for (;;) {
        const unsigned idle = __ballot_sync(full, !have);
        const unsigned held = 32u - __popc(idle);
        if (!exhausted && held < cap && (held == 0u || P.f64.simple == 0)) {
            const unsigned want = cap - held;
            uint64_t base = next;
            if (P.f64.simple != 0) {
                next += placed;
                exhausted = next >= P.count;
            } else if (first) {
                exhausted = placed >= P.count;
            } else {
                unsigned got = 0;
                if (lane == 0u) got = atomicAdd(&P.counters->next_particle, want);
                base = placed + __shfl_sync(full, got, 0);
                exhausted = base + want >= P.count;
            }
            first = false;
            const unsigned place = __popc(idle & lanes_below);
            if (!have && place < want) {
                const uint64_t slot = base + place;
                if (slot < P.count) {
                    const uint32_t idx = P.order != nullptr ? __ldg(P.order + slot)
                                                            : static_cast<uint32_t>(slot);
                    if (P.parts.status[idx] == 0) {
                        load<FOCUSED>(st, P, idx);
                        have = true;
                        if (!live(st, P)) {
                            store<FOCUSED>(st, P);
                            tally_finish(tally, st.steps, st.status);
                            have = false;
                        }
                    }
                }
            }
        }
        WarpTasks w;
        w.buf = mem;
        w.mask = __ballot_sync(full, have);
        w.n = __popc(w.mask);
        w.rank = __popc(w.mask & lanes_below);
        w.mine = have;
        if (w.n == 0) {
            if (exhausted) {
                break;
            }
            continue;
        }
        sample_f64<FOCUSED>(st, P, w, rows);
        // lanes without a particle read the first row (their values are not used)
        const double* c = rows + (have ? w.rank : 0) * f64_row(FOCUSED);
        bool more;
        if constexpr (SURR) {
            const Served served = serve_f64<surr_fp16(SURR), surr_hidden(SURR)>(
                st, P, have, c[6], network, tally);
            more = advance_f64<FOCUSED, true>(st, P, c, w, &served);
        } else {
            more = advance_f64<FOCUSED, false>(st, P, c, w, nullptr);
        }
        if (have && !more) {
            store<FOCUSED>(st, P);
            tally_finish(tally, st.steps, st.status);
            have = false;
        }
    }
    tally_flush(tally, P.counters, SURR ? P.sg.judge : nullptr);
}

// Reciprocals, keys and the plan of powers of one launch.
F64Consts make_f64_consts(const PushLaunch& L) {
    const DeviceSettings& s = L.settings;
    F64Consts k{};
    auto key = [](double v) {
        long long bits;
        std::memcpy(&bits, &v, sizeof(bits));
        // a threshold of either zero is the lower one's key: -0 >= +0 holds
        return v == 0.0 ? -1ll : f64_key(bits);
    };
    for (int d = 0; d < 2; ++d) {
        const Axis& a = L.grid.axis[d];
        k.axis[d].lower = key(a.lower);
        k.axis[d].upper = key(a.upper);
        // below lower + (1 - 2^-40) width the wrap count's product rounds
        // below 1
        const double safe = a.lower + (1.0 - 9.094947017729282e-13) * a.width;
        k.axis[d].floor_zero = safe < a.upper ? key(safe) : key(a.lower);
        k.axis[d].rcp_step = a.stored ? 1.0 : 1.0 / a.step;
    }
    k.rcp_mhd_dt = 1.0 / s.mhd_dt;
    k.rcp_p0 = 1.0 / s.p0;
    k.rcp_3 = 1.0 / 3.0;
    k.drift1_p0 = s.drift_param1 * s.p0;
    k.drift2_p0_p0 = s.drift_param2 * s.p0;
    k.drift2_p0_p0 = k.drift2_p0_p0 * s.p0;
    k.inv_charge = 1.0 / (L.focused ? s.charge : 3.0 * s.charge);
    k.half_cell = 0.5 * (s.dx < s.dy ? s.dx : s.dy);
    k.p_floor = 0.25 * s.p0;
    k.end_key = key(L.interval_end);
    k.single_step = s.dt_min == s.dt_max ? 1 : 0;
    k.lane_cap = 32;
    return k;
}

PowPlan make_pow_plan(const PushLaunch& L) {
    const DeviceSettings& s = L.settings;
    PowPlan plan{};
    auto add = [&plan](int base, double exponent) {
        plan.base[plan.powers] = base;
        plan.exponent[plan.powers] = exponent;
        ++plan.powers;
    };
    const double g = s.gamma_turb;
    add(0, g - 2.0);     // kappa: |B|, p / p0
    add(1, s.pindex);
    if (L.focused && s.closure != 0) {
        add(2, s.qlt_gk - 1.0);  // slab QLT: |mu| + h0, xi
        add(2, s.qlt_gk);
        add(3, s.qlt_gk);
    } else if (L.focused) {
        add(2, g - 1.0);  // the driver's closure: |mu|, |B|, p / p0
        add(2, g - 2.0);
        add(0, 2.0 - g);
        add(1, g - 1.0);
    }
    plan.shared_logs = 1;
    for (int e = 0; e < plan.powers; ++e) {
        if (!std::isfinite(plan.exponent[e])) plan.shared_logs = 0;
    }
    return plan;
}

template <bool FOCUSED, int SURR = 0>
cudaError_t launch_push_f64(const PushLaunch& L, cudaStream_t stream) {
    PushParams P = make_push_params(L);
    const int threads = 128;
    const size_t smem = (SURR ? (mlp_smem_bytes(surr_hidden(SURR)) + 15) / 16 * 16 : 0) +
                        (threads / 32) * f64_warp_doubles(FOCUSED) * sizeof(double);
    cudaError_t err = cudaFuncSetAttribute(push_f64_kernel<FOCUSED, SURR>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           static_cast<int>(smem));
    if (err != cudaSuccess) return err;
    const uint64_t sm = static_cast<uint64_t>(L.sm_count);
    const uint64_t lanes = sm * threads;  // those of one block per SM
    const int per_sm = f64_blocks_per_sm(L.count, L.settings.dt_min == L.settings.dt_max, lanes,
                                         kF64Blocks, L.blocks_per_sm);
    const uint64_t warps = sm * per_sm * (threads / 32);
    const uint64_t cap = (L.count + warps - 1) / warps;
    P.f64.simple = L.schedule == kScheduleSimple ? 1 : 0;
    P.f64.lane_cap = P.f64.simple || cap > 32 ? 32u : static_cast<unsigned>(cap);
    push_f64_kernel<FOCUSED, SURR>
        <<<static_cast<unsigned>(sm) * per_sm, threads, smem, stream>>>(P);
    return cudaGetLastError();
}

}  // namespace
}  // namespace kpt
