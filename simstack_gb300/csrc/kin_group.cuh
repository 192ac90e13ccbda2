// Lane-group kernels: G = 8, 16 or 32 lanes integrate one cell (4, 2 or 1 cells per warp), for
// any mechanism within the KinMech capacities whose tables group_tab.h could lay out.
//
// What bounds them and why they exist. One lane per cell (kin_kernels.cuh) runs ~4,000 FP64
// instructions per step attempt one after the other. On sm_103a an FP64 warp instruction holds
// its scheduler's FP64 unit for 64 cycles, whatever its active lanes and whatever the
// instruction-level parallelism (19 cycles per SM with all four schedulers busy), so an attempt
// takes 134 us from one cell to 32 per warp, and a small batch or the tail of a large one leaves
// most of the chip idle for its length. With the cell's work spread over G lanes the same attempt
// is ~600 (G = 32) to ~1,200 (G = 8, four cells at once) FP64 instructions: the shorter chain where
// latency counts, at fewer cells per instruction than the lane kernels where throughput does.
// The rule that chooses between them is in group.h (group_rule, group_most).
//
// Warps are independent: a warp claims cells from the work queue (or the suspension list) for
// its 32 / G groups, and its groups take each attempt together. A cell's vectors and dense LU
// live in the warp's shared memory, the step's row quantities in the registers of the lane that
// owns the row (row i: lane i % G, register i / G); the mechanism's schedule (group_tab.h) is
// staged into shared memory once per CTA by a TMA bulk copy with a bounded wait. Every element
// sees the lane kernels' operations in the lane kernels' order, so results keep their bits in
// every precision.

#pragma once
#include "group_tab.h"
#include "kin_device.cuh"

namespace sgb {

// FP64 comparisons on the integer pipe (a DSETP costs an FP64 slot): IEEE semantics, NaN false, -0 == +0.
__device__ __forceinline__ long long fp64_key(double a) {
    const long long x = __double_as_longlong(a);
    return x < 0 ? (long long)(0x8000000000000000ull - (unsigned long long)x) : x;
}
__device__ __forceinline__ bool fp64_nan(double a) {
    return ((unsigned long long)__double_as_longlong(a) << 1) > 0xffe0000000000000ull;
}
__device__ __forceinline__ bool g_lt(double a, double b) { return !fp64_nan(a) && !fp64_nan(b) && fp64_key(a) < fp64_key(b); }
__device__ __forceinline__ bool g_le(double a, double b) { return !fp64_nan(a) && !fp64_nan(b) && fp64_key(a) <= fp64_key(b); }
__device__ __forceinline__ bool g_lt(float a, float b) { return a < b; }
__device__ __forceinline__ bool g_le(float a, float b) { return a <= b; }
template <class T> __device__ __forceinline__ T g_min(T a, T b) { return g_lt(a, b) ? a : b; }
template <class T> __device__ __forceinline__ T g_max(T a, T b) { return g_lt(b, a) ? a : b; }
__device__ __forceinline__ float g_abs(float a) { return a < 0.0f ? -a : a; }
__device__ __forceinline__ double g_abs(double a) {   // vabs: -a where a < 0 (so -0 and NaN stay)
    const unsigned long long x = (unsigned long long)__double_as_longlong(a);
    return (x >> 63) && (x << 1) && !fp64_nan(a) ? __longlong_as_double((long long)(x ^ 0x8000000000000000ull)) : a;
}
__device__ __forceinline__ bool g_finite(double a) {
    return ((unsigned long long)__double_as_longlong(a) << 1) < 0xffe0000000000000ull;
}
__device__ __forceinline__ bool g_finite(float a) { return is_finite_lane(a); }
__device__ __forceinline__ bool g_zero(double a) { return ((unsigned long long)__double_as_longlong(a) << 1) == 0; }
__device__ __forceinline__ bool g_one(double a) { return __double_as_longlong(a) == 0x3ff0000000000000ll; }

// step_factor / cbrt_clamped (kin_device.cuh) with the comparisons above
template <class T> __device__ __forceinline__ T g_step_factor(T err, uint32_t order) {
    const T e = g_min(g_max(err, (T)1e-4), (T)1e4);
    T root;
    if (order == 2) root = vsqrt(e);
    else if (order == 4) root = vsqrt(vsqrt(e));
    else {   // e is within cbrt_clamped's limits already
        const T r4 = vsqrt(vsqrt(e));
        const T r16 = vsqrt(vsqrt(r4));
        const T r64 = vsqrt(vsqrt(r16));
        T g = r4 * r16 * r64;
        const T two = (T)2.0, third = (T)(1.0 / 3.0);
        g = (two * g + e / (g * g)) * third;
        g = (two * g + e / (g * g)) * third;
        root = g;
    }
    const T fac = (T)0.9 / root;
    return g_min(g_max(fac, (T)0.2), (T)6.0);
}

// The coefficient in a term word: the top 16 bits of a double or a float.
__device__ __forceinline__ double term_coef(uint32_t w, double) { return __hiloint2double((int)(w & 0xffff0000u), 0); }
__device__ __forceinline__ float term_coef(uint32_t w, float) { return __uint_as_float(w & 0xffff0000u); }

// Stage coefficient a (point) or c of the lane's type.
template <class T, class M> __device__ __forceinline__ T coef(const DevArgs &A, int i, bool point) {
    if constexpr (sizeof(T) == 4) return point ? M::a_df(A, i).hi : M::c_df(A, i).hi;   // hi: the FP32 rounding
    else return point ? M::a(A, i) : M::c(A, i);
}
__device__ __forceinline__ bool g_zero(float a) { return a == 0.0f; }

// What the three precisions share: the staged schedule, the cell's controller state and the
// segment machinery (Lane::seg_start, seg_finish, settle of kin_device.cuh). T: the type of t and h.
template <class T, int G, int NM>
struct GroupBase {
    static constexpr int NQ = (NM + G - 1) / G;   // rows per lane at most (NM: the kernel's largest n)
    static constexpr bool kExact = NM == kGroupExact;   // n is NM: strides and columns are constants
    const uint32_t *w;                  // staged image
    uint32_t n, R, ld, l;
    T t, h, seg_end, applied, duration, period, first, count;
    T h_min, h_max, h_start, inv_n;
    uint32_t steps, rejects, pulses, iterations, transitions;
    int phase;
    bool failed, pending, reject_last, reject_more;
    double failed_in;

    __device__ __forceinline__ const GroupHead &head() const { return *(const GroupHead *)w; }
    __device__ __forceinline__ void bind_image(const DevArgs &A, const uint32_t *image, uint32_t lane) {
        w = image;
        n = kExact ? (uint32_t)NM : head().n;
        R = head().R;
        ld = kExact ? (uint32_t)NM | 1u : head().ld;
        l = lane;
        h_min = (T)A.ctl.h_min;
        h_max = (T)A.ctl.h_max;
        h_start = (T)A.ctl.h_start;
        inv_n = (T)(1.0 / (double)n);
    }
    __device__ __forceinline__ bool row_ok(int q) const { return (uint32_t)q * G + l < n; }
    __device__ __forceinline__ uint32_t row(int q) const { return (uint32_t)q * G + l; }
    __device__ __forceinline__ bool round_on(int q) const { return (uint32_t)q * G < n; }   // same for the whole warp

    __device__ __forceinline__ void load_scalars(const DevArgs &A, uint32_t i) {
        h = (T)A.h[i];
        period = (T)A.period[i];
        first = (T)A.pulse_first[i];
        count = (T)A.pulse_count[i];
        duration = (T)A.duration;
        steps = rejects = pulses = 0;
        failed_in = A.failed[i];
        failed = (T)failed_in > (T)0.0;
        t = (T)0.0;
        applied = (T)0.0;
        transitions = 0;
        phase = kPhaseSegStart;
    }
    // The controller state of the group whose first lane is `from`, held by another group shape.
    template <class O> __device__ __forceinline__ void take_scalars(const O &o, int from) {
        auto get = [from](auto v) { return __shfl_sync(0xffffffffu, v, from); };
        t = get(o.t);
        h = get(o.h);
        seg_end = get(o.seg_end);
        applied = get(o.applied);
        steps = get(o.steps);
        rejects = get(o.rejects);
        pulses = get(o.pulses);
        iterations = get(o.iterations);
        transitions = get(o.transitions);
        failed = get((int)o.failed) != 0;
        failed_in = get(o.failed_in);
        pending = get((int)o.pending) != 0;
        reject_last = get((int)o.reject_last) != 0;
        reject_more = get((int)o.reject_more) != 0;
        phase = kPhaseStepping;
    }
    __device__ __forceinline__ void restore_scalars(const SuspendRec &r) {
        t = (T)r.t;
        h = (T)r.h;
        seg_end = (T)r.seg_end;
        applied = (T)r.applied;
        pending = (r.flags & 1u) != 0;
        reject_last = (r.flags & 2u) != 0;
        reject_more = (r.flags & 4u) != 0;
        iterations = r.iterations;
        transitions = r.transitions;
        phase = kPhaseStepping;
    }
    // failed holds 1 once a lane fails here, else what the block had (sticky)
    __device__ __forceinline__ void store_scalars(const DevArgs &A, uint32_t i) const {
        if (l != 0) return;
        A.h[i] = (double)h;
        A.failed[i] = failed && !((T)failed_in > (T)0.0) ? 1.0 : (double)(T)failed_in;
        A.steps[i] += counter(steps);
        A.rejects[i] += counter(rejects);
        A.pulses[i] += counter(pulses);
    }
    // the lane kernels count in T: an f32 counter stops at 2^24
    __device__ __forceinline__ static double counter(uint32_t c) { return (double)(sizeof(T) == 4 ? min(c, 1u << 24) : c); }
    __device__ __forceinline__ void seg_start() {
        pending = g_lt(applied, count);
        const T next_pulse = sgb_fma(applied, period, first);
        seg_end = pending ? g_min(next_pulse, duration) : duration;
        const bool active = g_lt(t, seg_end) && !failed;
        reject_last = false;
        reject_more = false;
        h = g_lt((T)0.0, h) ? h : h_start;
        iterations = 0;
        phase = active ? kPhaseStepping : kPhaseSegFinish;
    }
    // true: a pulse is due (the caller adds it to its rows)
    __device__ __forceinline__ bool seg_finish() {
        const bool alive = !failed;
        const bool hit = pending && alive && g_le(seg_end, t);
        if (hit) {
            applied = applied + (T)1.0;
            ++pulses;
            h = h_start;
        }
        const bool done = (g_le(duration, t) && g_le(count, applied)) || !alive;
        phase = done ? kPhaseDone : kPhaseSegStart;
        return hit;
    }
    template <class AddPulse> __device__ __forceinline__ bool settle(const DevArgs &A, AddPulse add_pulse) {
        for (;;) {
            if (++transitions > (1u << 24)) {
                failed = true;
                failed_in = 0.0;
                phase = kPhaseDone;
            }
            switch (phase) {
                case kPhaseSegStart: seg_start(); break;
                case kPhaseSegFinish:
                    if (seg_finish()) add_pulse();
                    break;
                case kPhaseStepping:
                    if (++iterations > A.ctl.max_steps) {
                        failed = true;
                        failed_in = 0.0;
                        phase = kPhaseSegFinish;
                        break;
                    }
                    return true;
                default: return false;
            }
        }
    }
    // The controller after an attempt of size hs with error norm err and factor fac
    // (kin_solver.h:281-311); returns whether the step is accepted.
    __device__ __forceinline__ bool control(const DevArgs &A, bool last, T hs, T h_wanted, T err, T fac, bool commit) {
        const T one = (T)1.0;
        bool ok = g_le(err, one) || g_le(hs, h_min);
        if (A.ctl.fixed_step) {
            ok = true;
            fac = one;
        }
        if (!commit) return false;
        if (ok) t = last ? seg_end : t + hs;
        T h_acc = hs * fac;
        const T h_grown = h_acc;
        h_acc = reject_last ? g_min(h_acc, hs) : h_acc;
        h_acc = (last && g_le(one, fac)) ? g_max(h_acc, h_wanted) : h_acc;
        T h_rej = reject_more ? hs * (T)0.1 : g_min(h_grown, hs);
        if (A.ctl.fixed_step) {
            h_acc = h_wanted;
            h_rej = h_wanted;
        }
        h = ok ? h_acc : h_rej;
        reject_more = !ok && reject_last;
        reject_last = !ok;
        steps += ok ? 1u : 0u;
        rejects += ok ? 0u : 1u;
        if (!(g_lt(t, seg_end) && !failed)) phase = kPhaseSegFinish;
        return ok;
    }
    // The step size of this attempt (kin_solver.h:211-216).
    __device__ __forceinline__ T step_size(bool *last, T *h_wanted) const {
        const T remaining = seg_end - t;
        T h_cap = remaining;
        if (g_lt((T)0.0, h_max)) h_cap = g_min(h_cap, h_max);
        *h_wanted = g_max(h, h_min);
        *last = g_le(remaining, *h_wanted);
        return *last ? remaining : g_min(*h_wanted, h_cap);
    }

    // ---- phases on the cell's shared memory; Cf: the arithmetic of J, LU and solves ----

    template <class V> __device__ __forceinline__ static const V &at(const V *base, uint32_t bytes) {
        return *(const V *)((const char *)base + bytes);
    }
    template <class V> __device__ __forceinline__ static V &at(V *base, uint32_t bytes) { return *(V *)((char *)base + bytes); }

    // acc = fma(coef, base[offset], acc) over `len` term words of this lane, G words apart, the next
    // batch's words on their way while a batch is summed
    template <class V> __device__ __forceinline__ static V gather(V acc, const uint32_t *term, uint32_t len, const V *base) {
        uint32_t v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = term[u * G];
        uint32_t e = 0;
        for (; e + 4 <= len; e += 4) {
            V x[4];
            uint32_t c[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                x[u] = at(base, v[u] & 0x7fffu);
                c[u] = v[u];
                v[u] = term[(e + 4 + u) * G];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) acc = sgb_fma(term_coef(c[u], (V)0), x[u], acc);
        }
#pragma unroll
        for (int u = 0; u < 3; ++u)
            if (e + u < len) acc = sgb_fma(term_coef(v[u], (V)0), at(base, v[u] & 0x7fffu), acc);
        return acc;
    }
    // a = -J from the products d (zero at the fill-in)
    template <class Cf> __device__ __forceinline__ void neg_jac(const Cf *d, Cf *a) const {
        const uint32_t *z = w + head().zero, nz = head().nzero;
        for (uint32_t e = l; e < nz; e += G) at(a, z[e]) = (Cf)0.0;
        const uint32_t rounds = head().jrounds, *jr = w + head().jround, *dst = w + head().jdst;
        for (uint32_t q = 0; q < rounds; ++q) {
            const uint32_t to = dst[q * G + l];
            const Cf acc = gather<Cf>((Cf)0.0, w + jr[2 * q] + l, jr[2 * q + 1], d);
            if (to != kGroupNone) at(a, to) = acc;
        }
    }
    // a -> L\U of I ghinv - J in place, the diagonal holding 1/U(k,k). Everything a pivot needs but its
    // reciprocal is loaded ahead of it. FP32: a task forms its own multiplier (a product is cheaper
    // than an exchange); FP64: the multipliers are formed once per row and read back (a product holds
    // the FP64 unit 64 cycles).
    template <class Cf> __device__ __forceinline__ void factor(Cf ghinv, Cf *a) const {
        const uint4 *pv = (const uint4 *)(w + head().pivot);
        uint4 p = pv[0];
#pragma unroll 1
        for (uint32_t k = 0; k < n; ++k) {   // p: rows, row count, tasks, task count (counts: multiples of G)
            const uint4 next = pv[k + 1 < n ? k + 1 : k];
            switch (p.w / G) {   // rounds of tasks: the same for the whole warp
                case 0: pivot<0>(p, k, ghinv, a); break;
                case 1: pivot<1>(p, k, ghinv, a); break;
                case 2: pivot<2>(p, k, ghinv, a); break;
                case 3: pivot<3>(p, k, ghinv, a); break;
                default: pivot<4>(p, k, ghinv, a);
            }
            p = next;
            __syncwarp();
        }
    }
    // One pivot, its first C rounds of tasks loaded ahead of the reciprocal.
    template <int C, class Cf> __device__ __forceinline__ void pivot(const uint4 p, uint32_t k, Cf ghinv, Cf *a) const {
        constexpr uint32_t sz = (uint32_t)sizeof(Cf);
        constexpr bool kOwn = sizeof(Cf) == 4;
        constexpr int CC = C > 0 ? C : 1;
        const uint32_t colk = k * sz, rowk = k * ld * sz;
        uint32_t v[CC], r0 = 0;
        Cf m[CC], u[CC], x[CC], raw = (Cf)0.0;
        const bool any = C > 0 || p.y != 0;
        if (any) r0 = w[p.x + l];
#pragma unroll
        for (int c = 0; c < C; ++c) v[c] = w[p.z + l + c * G];
        const Cf diag = at(a, rowk + colk);
        if (any) raw = at(a, r0 + colk);
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const uint32_t ij = v[c] & 0xffffu, i0 = v[c] >> 16;
            if (kOwn) m[c] = at(a, i0 + colk);
            u[c] = at(a, rowk + ij - i0);
            x[c] = at(a, ij);
        }
        const Cf inv = (Cf)1.0 / (diag + ghinv);
        if (kOwn) __syncwarp();   // every lane has read the raw column
        if (any) at(a, r0 + colk) = raw * inv;
        for (uint32_t e = l + G; e < p.y; e += G) {
            const uint32_t r = w[p.x + e];
            at(a, r + colk) = at(a, r + colk) * inv;
        }
        if (!kOwn) __syncwarp();   // the multipliers are in place, and every lane has read a[k][k]
        if (l == 0) at(a, rowk + colk) = inv;
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const Cf lm = kOwn ? m[c] * inv : at(a, (v[c] >> 16) + colk);
            at(a, v[c] & 0xffffu) = sgb_fma(-lm, u[c], x[c]);
        }
        if constexpr (C == 4) {
            if (p.w > 4 * G) {
                if (kOwn) __syncwarp();
                for (uint32_t e = l + 4 * G; e < p.w; e += 2 * G) {   // two rounds at a time
                    const bool two = e - l + G < p.w;
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        if (c && !two) break;
                        v[c] = w[p.z + e + c * G];
                        const uint32_t ij = v[c] & 0xffffu, i0 = v[c] >> 16;
                        m[c] = at(a, i0 + colk);
                        u[c] = at(a, rowk + ij - i0);
                        x[c] = at(a, ij);
                    }
                    at(a, v[0] & 0xffffu) = sgb_fma(-m[0], u[0], x[0]);
                    if (two) at(a, v[1] & 0xffffu) = sgb_fma(-m[1], u[1], x[1]);
                }
            }
        }
    }

    // The own rows' patterns (columns below / above the diagonal) and, in FP32, their LU coefficients,
    // which the solves of a step then read from registers.
    template <class Cf> struct Rows {
        static constexpr bool kRegs = sizeof(Cf) == 4;   // FP64: the loop measured faster (the FP64 unit is the cost)
        uint32_t lo[NQ], hi[NQ];
        Cf c[kRegs ? NQ : 1][kRegs ? NM : 1];
    };
    template <class Cf> __device__ __forceinline__ void load_masks(Rows<Cf> &r) const {
        const uint32_t *mask = w + head().mask;
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            r.lo[q] = row_ok(q) ? mask[2 * row(q)] : 0u;
            r.hi[q] = row_ok(q) ? mask[2 * row(q) + 1] : 0u;
        }
    }
    template <class Cf> __device__ __forceinline__ void load_rows(const Cf *a, Rows<Cf> &r) const {
        if constexpr (Rows<Cf>::kRegs) {
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const Cf *mine = a + (row_ok(q) ? row(q) * ld : 0u);
#pragma unroll
                for (int k = 0; k < NM; ++k) r.c[q][k] = mine[min((uint32_t)k, n - 1)];
            }
        }
    }
    // x = (LU)^-1 x, rows in registers. FP32: the columns are unrolled (columns past n change nothing: no
    // row has them in its pattern), so that a step is a shuffle, the updates and little else: a lone
    // warp pays ~4 cycles for every instruction it issues (a step attempt of the shipped mechanism at
    // G = 32: 18.7k cycles of solves as a loop over shared memory, 9.9k this way).
    template <class Cf> __device__ __forceinline__ void solve(const Cf *a, const Rows<Cf> &r, Cf *xs, Cf (&x)[NQ]) const {
        if constexpr (Rows<Cf>::kRegs) {
#pragma unroll
            for (int k = 0; k + 1 < NM; ++k) {
                const Cf xk = __shfl_sync(0xffffffffu, x[k / G], k % G, G);
#pragma unroll
                for (int q = 0; q < NQ; ++q)
                    if ((q + 1) * G - 1 > k && ((r.lo[q] >> k) & 1u)) x[q] = sgb_fma(-r.c[q][k], xk, x[q]);
            }
#pragma unroll
            for (int k = NM - 1; k >= 0; --k) {
                if (l == (uint32_t)(k % G)) x[k / G] = x[k / G] * r.c[k / G][k];   // the owner: times 1/U(k,k)
                const Cf xk = __shfl_sync(0xffffffffu, x[k / G], k % G, G);
#pragma unroll
                for (int q = 0; q < NQ; ++q)
                    if (q * G < k && ((r.hi[q] >> k) & 1u)) x[q] = sgb_fma(-r.c[q][k], xk, x[q]);
            }
        } else if constexpr (kExact && NQ == 1) {
            solve_unrolled(a, r, xs, x);
        } else {
            solve_columns(a, r, xs, x);
        }
    }
    // FP64 with the columns unrolled: addresses are constants and the pattern bits predicates, which leaves a
    // load, the FMA and the hand-over through xs per column (64 cells x 1 s at 32 lanes per cell 13.95 ->
    // 13.32 ms; with several rows per lane, 4,096 cells at 8 lanes 23.2 -> 24.3, the loop stays).
    template <class Cf> __device__ __forceinline__ void solve_unrolled(const Cf *a, const Rows<Cf> &r, Cf *xs, Cf (&x)[NQ]) const {
        const Cf *mine[NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            mine[q] = a + (row_ok(q) ? row(q) * ld : 0u);
            if (row_ok(q)) xs[row(q)] = x[q];
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k + 1 < NM; ++k) {
            const Cf xk = xs[k];
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                if ((q + 1) * G - 1 <= k) continue;
                const Cf c = mine[q][k];
                if ((r.lo[q] >> k) & 1u) x[q] = sgb_fma(-c, xk, x[q]);
                if (row(q) > (uint32_t)k && row_ok(q)) xs[row(q)] = x[q];
            }
            __syncwarp();
        }
#pragma unroll
        for (int k = NM - 1; k >= 0; --k) {
            const Cf xk = xs[k] * a[k * (int)ld + k];   // every lane forms it: one exchange fewer per column
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                if (q * G > k) continue;
                const Cf c = mine[q][k];
                if ((r.hi[q] >> k) & 1u) x[q] = sgb_fma(-c, xk, x[q]);
                if (row(q) == (uint32_t)k) x[q] = xk;
                if (row(q) < (uint32_t)k) xs[row(q)] = x[q];
            }
            __syncwarp();
        }
    }
    // Column by column, solved elements published in xs, coefficients read one column ahead.
    template <class Cf> __device__ __forceinline__ void solve_columns(const Cf *a, const Rows<Cf> &r, Cf *xs, Cf (&x)[NQ]) const {
        Cf c[NQ];
        uint32_t r0[NQ];   // the row's start (row 0 stands in for one past the end)
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            r0[q] = row_ok(q) ? row(q) * ld : 0u;
            c[q] = a[r0[q]];
            if (row_ok(q)) xs[row(q)] = x[q];
        }
        __syncwarp();
#pragma unroll 1
        for (uint32_t k = 0; k + 1 < n; ++k) {
            const Cf xk = xs[k];
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const Cf cn = a[r0[q] + k + 1];
                if (round_on(q) && (uint32_t)(q + 1) * G - 1u > k) {   // same for the whole warp
                    const Cf v = sgb_fma(-c[q], xk, x[q]);
                    x[q] = (r.lo[q] >> k) & 1u ? v : x[q];
                    if (row_ok(q)) xs[row(q)] = x[q];   // rows <= k rewrite what they hold
                }
                c[q] = cn;
            }
            __syncwarp();
        }
        Cf inv = a[(n - 1) * ld + n - 1];
#pragma unroll
        for (int q = 0; q < NQ; ++q) c[q] = a[r0[q] + n - 1];
#pragma unroll 1
        for (uint32_t k = n; k-- > 0;) {
            const Cf xk = xs[k] * inv;   // every lane forms it: one exchange fewer per column
            const uint32_t kn = k ? k - 1 : 0;
            inv = a[kn * ld + kn];
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const Cf cn = a[r0[q] + kn];
                if ((uint32_t)q * G <= k) {   // same for the whole warp
                    const Cf v = sgb_fma(-c[q], xk, x[q]);
                    x[q] = row(q) == k ? xk : (r.hi[q] >> k) & 1u ? v : x[q];
                    if (row(q) < k) xs[row(q)] = x[q];
                }
                c[q] = cn;
            }
            __syncwarp();
        }
    }
};

// FP64 lanes (PREC 0) and f32 Delta lanes (PREC 1): Lane<Ops, M, PREC> over G lanes.
template <class M, int PREC, int G, int NM>
struct GroupLane : GroupBase<typename Pick<PREC == 1, float, double>::type, G, NM> {
    typedef typename Pick<PREC == 1, float, double>::type T;
    typedef GroupBase<T, G, NM> B;
    typedef T LuT;
    using B::NQ;
    using B::n;
    using B::R;
    using B::l;
    using B::w;
    using B::head;
    using B::row;
    using B::row_ok;
    using B::round_on;
    static constexpr bool kDelta = PREC == 1;
    static constexpr int S = M::kStages;

    T y[NQ], base[kDelta ? NQ : 1], rtol, atol;
    T *a, *d, *ks, *rate, *ys, *fs, *xs, *qs, *src, *K;   // K: [stage][species], read and written by the row's lane

    __device__ __forceinline__ void bind(const DevArgs &A, unsigned char *cell) {
        rtol = (T)A.ctl.rtol;
        atol = (T)A.ctl.atol;
        a = (T *)cell;
        d = a + (n + 1) * this->ld;
        ks = d + head().pairs + 1;
        rate = ks + R;
        ys = rate + R + 1;
        fs = ys + n;
        xs = fs + n;
        qs = xs + n;
        src = qs + n;
        K = src + n;
        if (l == 0) d[head().pairs] = rate[R] = (T)0.0;   // what a lane without a term adds -0 times
    }
    __device__ __forceinline__ void load(const DevArgs &A, uint32_t i) {
        const uint32_t p = A.padded;
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            if (!row_ok(q)) continue;
            const double v = A.y[(size_t)row(q) * p + i];
            if constexpr (kDelta) {
                base[q] = (T)v;
                y[q] = (T)0.0;
            } else {
                y[q] = (T)v;
            }
            src[row(q)] = (T)A.src[(size_t)row(q) * p + i];
        }
        for (uint32_t r = l; r < R; r += G) ks[r] = (T)A.k[(size_t)r * p + i];
        this->load_scalars(A, i);
    }
    __device__ __forceinline__ void restore(const DevArgs &, uint32_t, const SuspendRec &r) { this->restore_scalars(r); }
    __device__ __forceinline__ void put_state(void *out) const {
#pragma unroll
        for (int q = 0; q < NQ; ++q)
            if (row_ok(q)) ((T *)out)[row(q)] = y[q];
    }
    __device__ __forceinline__ void get_state(const void *in) {
#pragma unroll
        for (int q = 0; q < NQ; ++q)
            if (row_ok(q)) y[q] = ((const T *)in)[row(q)];
    }
    __device__ __forceinline__ void store(const DevArgs &A, uint32_t i) {
        const uint32_t p = A.padded;
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            if (!row_ok(q)) continue;
            double *dst = A.y + (size_t)row(q) * p + i;
            if constexpr (kDelta) {
                double v = *dst + (double)y[q];
                if (A.ctl.clamp_negative) v = v > 0.0 ? v : 0.0;
                *dst = v;
            } else {
                *dst = (double)y[q];
            }
        }
        this->store_scalars(A, i);
    }
    __device__ __forceinline__ bool settle(const DevArgs &A, uint32_t cell) {
        return B::settle(A, [&]() {
#pragma unroll
            for (int q = 0; q < NQ; ++q)
                if (row_ok(q)) y[q] = y[q] + (T)A.pulse[(size_t)row(q) * A.padded + cell];
        });
    }
    // The step's rates k_r y y y at ys, and with kPairs the Jacobian's products; four of a lane's
    // elements at a time, so that their loads overlap.
    template <bool kPairs> __device__ __forceinline__ void products(const uint32_t *list, uint32_t count, T *out) const {
        for (uint32_t e = l; e < count; e += 4 * G) {
            uint32_t v[4];
            T x[4], y0[4], y1[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = e + u * G < count ? list[e + u * G] : 0u;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                x[u] = ks[v[u] & 0xffu];
                y0[u] = ys[(v[u] >> 8) & 63u];
                y1[u] = ys[(v[u] >> 14) & 63u];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t c = v[u] >> 26;
                if (c > 0) x[u] = x[u] * y0[u];
                if (c > 1) x[u] = x[u] * y1[u];
                if (!kPairs && c > 2) x[u] = x[u] * ys[(v[u] >> 20) & 63u];
                if (e + u * G < count) out[kPairs ? e + u * G : v[u] & 0xffu] = x[u];
            }
        }
    }
    // f at ys (published) into f, the own rows
    __device__ __forceinline__ void rhs(T (&f)[NQ]) {
        products<false>(w + head().rx, R, rate);
        __syncwarp();
        const uint32_t *fr = w + head().fround, *order = w + head().forder;
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            if (!round_on(q)) continue;
            const uint32_t s = order[q * G + l];
            const T acc = B::template gather<T>(s != kGroupNone ? src[s] : (T)0.0, w + fr[2 * q] + l, fr[2 * q + 1], rate);
            if (s != kGroupNone) fs[s] = acc;
        }
        __syncwarp();
#pragma unroll
        for (int q = 0; q < NQ; ++q) f[q] = row_ok(q) ? fs[row(q)] : (T)0.0;
    }
    __device__ __forceinline__ void publish(const T (&v)[NQ]) {   // the point f and J are evaluated at
#pragma unroll
        for (int q = 0; q < NQ; ++q)
            if (row_ok(q)) ys[row(q)] = kDelta ? base[kDelta ? q : 0] + v[q] : v[q];
        __syncwarp();
    }

    __device__ __forceinline__ void attempt(const DevArgs &A, bool commit) {
        const T one = (T)1.0;
        bool last;
        T h_wanted;
        const T hs = this->step_size(&last, &h_wanted);
        const T hinv = one / hs;
        // 1 / (gamma h): for gamma = 1/2 and a step whose reciprocal is normal, 2 (1 / h) exactly
        const bool half = !kDelta && M::gamma0(A) == 0.5 && g_lt((T)1e-300, hs) && g_lt(hs, (T)1e300);
        const T ghinv = half ? (T)2.0 * hinv : one / (hs * (T)M::gamma0(A));
        T f[NQ], yt[NQ], x[NQ];
        typename B::template Rows<LuT> rows;
        this->load_masks(rows);
        bool f_at_y = false;
        // one copy of the stage body (and one call of each phase): an attempt's code stays in the
        // instruction caches, which a lone warp feels more than the loop's arithmetic
#pragma unroll 1
        for (int st = 0; st < S; ++st) {
            if (st >= M::stages(A)) break;
            const int packed = st * (st - 1) / 2;
            bool eval = st == 0;
#pragma unroll
            for (int q = 0; q < NQ; ++q) yt[q] = y[q];
            if (st > 0 && M::new_f(A, st)) {
                bool moved = false;
#pragma unroll 1
                for (int j = 0; j < st; ++j) {
                    const T ac = coef<T, M>(A, packed + j, true);
                    if (g_zero(ac)) continue;
                    moved = true;
#pragma unroll
                    for (int q = 0; q < NQ; ++q)
                        if (row_ok(q)) yt[q] = sgb_fma(ac, K[j * n + row(q)], yt[q]);
                }
                eval = moved || !f_at_y;
                f_at_y = !moved;
            }
            if (eval) {   // same for the whole warp, as everything about the stages is
                publish(yt);
                if (st == 0) products<true>(w + head().pr, head().pairs, d);
                rhs(f);   // its barriers also publish the products
            }
            if (st == 0) {
                f_at_y = true;
                this->template neg_jac<T>(d, a);
                __syncwarp();
                this->template factor<T>(ghinv, a);
                this->load_rows(a, rows);
            }
#pragma unroll
            for (int q = 0; q < NQ; ++q) x[q] = f[q];
#pragma unroll 1
            for (int j = 0; j < st; ++j) {
                const T c = coef<T, M>(A, packed + j, false);
                if (g_zero(c)) continue;
                const T hc = c * hinv;
#pragma unroll
                for (int q = 0; q < NQ; ++q)
                    if (row_ok(q)) x[q] = sgb_fma(hc, K[j * n + row(q)], x[q]);
            }
            this->template solve<T>(a, rows, xs, x);
#pragma unroll
            for (int q = 0; q < NQ; ++q)
                if (row_ok(q)) K[st * n + row(q)] = x[q];
        }
        // y_new and the weighted RMS error (kin_solver.h:263-280)
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            if (!round_on(q)) continue;
            T ynew = y[q], yerr = (T)0.0;
            bool first_e = true;
#pragma unroll
            for (int st = 0; st < S; ++st) {
                if (st >= M::stages(A)) break;
                const double mc = M::m(A, st), ec = M::e(A, st);
                const T kv = row_ok(q) ? K[st * n + row(q)] : (T)0.0;
                if (!g_zero(mc)) ynew = sgb_fma((T)mc, kv, ynew);
                if (!g_zero(ec)) {
                    yerr = (first_e && g_one(ec)) ? sgb_first_pos(kv) : sgb_fma((T)ec, kv, yerr);
                    first_e = false;
                }
            }
            T scale;
            if constexpr (kDelta) scale = sgb_fma(rtol, g_max(g_abs(base[q] + y[q]), g_abs(base[q] + ynew)), atol);
            else scale = sgb_fma(rtol, g_max(g_abs(y[q]), g_abs(ynew)), atol);
            yt[q] = ynew;
            if (row_ok(q)) qs[row(q)] = yerr / scale;
        }
        __syncwarp();
        T err = (T)0.0;
        for (uint32_t s = 0; s < n; ++s) err = sgb_fma(qs[s], qs[s], err);
        err = vsqrt(err * this->inv_n);
        if (!g_finite(err)) err = (T)1e10;
        const T fac = g_step_factor(err, M::order(A));
        if (this->control(A, last, hs, h_wanted, err, fac, commit)) {
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                T v = yt[q];
                if (A.ctl.clamp_negative) v = kDelta ? g_max(v, -base[kDelta ? q : 0]) : g_max(v, (T)0.0);
                y[q] = v;
            }
        }
    }
};

// Mixed lanes with refined stages (mixed variant 2): LaneIr over G lanes -- double-float state,
// right-hand sides, stage vectors and error norm; FP32 -J, LU and solves; one double-float
// refinement sweep per stage. The products k_r prod_{q != p} y_q of the residual are formed once
// per attempt (the lane kernel re-forms them in every stage: the same operations).
template <class M, int G, int NM>
struct GroupIr : GroupBase<double, G, NM> {
    typedef GroupBase<double, G, NM> B;
    typedef float LuT;
    using B::NQ;
    using B::n;
    using B::R;
    using B::l;
    using B::w;
    using B::head;
    using B::row;
    using B::row_ok;
    using B::round_on;
    static constexpr int S = M::kStages;

    Df y[NQ], rtol, atol;
    Df *ks, *rate, *prod, *ys, *fs, *qs, *src, *K;   // K: [stage][species], read and written by the row's lane
    float *a, *d, *xs;

    __device__ __forceinline__ void bind(const DevArgs &A, unsigned char *cell) {
        rtol = df_from(A.ctl.rtol);
        atol = df_from(A.ctl.atol);
        ks = (Df *)cell;
        rate = ks + R;
        prod = rate + R + 1;
        ys = prod + head().pairs;
        fs = ys + n;
        qs = fs + n;
        src = qs + n;
        K = src + n;
        a = (float *)(K + 4 * n);
        d = a + (n + 1) * this->ld;
        xs = d + head().pairs + 1;
        if (l == 0) d[head().pairs] = 0.0f;
    }
    __device__ __forceinline__ void load(const DevArgs &A, uint32_t i) {
        const uint32_t p = A.padded;
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            if (!row_ok(q)) continue;
            y[q] = df_from(A.y[(size_t)row(q) * p + i]);
            src[row(q)] = df_from(A.src[(size_t)row(q) * p + i]);
        }
        for (uint32_t r = l; r < R; r += G) ks[r] = df_from(A.k[(size_t)r * p + i]);
        this->load_scalars(A, i);
    }
    __device__ __forceinline__ void put_state(void *out) const {
#pragma unroll
        for (int q = 0; q < NQ; ++q)
            if (row_ok(q)) ((Df *)out)[row(q)] = y[q];
    }
    __device__ __forceinline__ void get_state(const void *in) {
#pragma unroll
        for (int q = 0; q < NQ; ++q)
            if (row_ok(q)) y[q] = ((const Df *)in)[row(q)];
    }
    // a parked mixed cell keeps its state as the float pairs themselves in its y slots
    __device__ __forceinline__ void restore(const DevArgs &A, uint32_t i, const SuspendRec &r) {
#pragma unroll
        for (int q = 0; q < NQ; ++q)
            if (row_ok(q)) y[q] = ((const Df *)A.y)[(size_t)row(q) * A.padded + i];
        this->restore_scalars(r);
    }
    __device__ __forceinline__ void store(const DevArgs &A, uint32_t i) {
#pragma unroll
        for (int q = 0; q < NQ; ++q)
            if (row_ok(q)) A.y[(size_t)row(q) * A.padded + i] = df_to(y[q]);
        this->store_scalars(A, i);
    }
    __device__ __forceinline__ bool settle(const DevArgs &A, uint32_t cell) {
        return B::settle(A, [&]() {
#pragma unroll
            for (int q = 0; q < NQ; ++q)
                if (row_ok(q)) y[q] = df_add(y[q], df_from(A.pulse[(size_t)row(q) * A.padded + cell]));
        });
    }
    // acc += coef * v, lazily normalised (kin_table.cuh lazy_term)
    __device__ __forceinline__ Df add_term(Df acc, Df v, float c, bool odd) const {
        if (odd && c != 1.0f && c != -1.0f && c != 2.0f && c != -2.0f && c != 4.0f && c != -4.0f)
            return df_acc(acc, df_mul_u(v, Df{c, 0.0f}));
        return df_acc(acc, df_scale(v, c));   // c = 1: the value itself
    }
    // acc += the terms of one species over `rate`; skip: terms of reactions without reactants are left out
    __device__ __forceinline__ Df gather_df(Df acc, const uint32_t *term, uint32_t len, bool skip, bool odd) const {
        uint32_t v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = term[u * G];
        for (uint32_t e = 0; e < len; e += 4) {
            Df x[4];
            uint32_t c[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                c[u] = e + u < len ? v[u] : kGroupNoTerm;   // past the list: no term, and nothing read by its word
                x[u] = B::at(rate, c[u] & 0x7fffu);
                v[u] = term[(e + 4 + u) * G];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const Df s = add_term(acc, x[u], term_coef(c[u], 0.0f), odd);
                const bool on = (c[u] & 0xffff0000u) != kGroupNoTerm && !(skip && (c[u] & kGroupNoReactant));
                acc.hi = on ? s.hi : acc.hi;
                acc.lo = on ? s.lo : acc.lo;
            }
        }
        return acc;
    }
    // f(ys) in lazily normalised double-float (fun_dfl)
    __device__ __forceinline__ void rhs(Df (&f)[NQ]) {
        const uint32_t *rx = w + head().rx;
        for (uint32_t e = l; e < R; e += G) {
            const uint32_t v = rx[e], c = v >> 26, r = v & 0xffu;
            Df x = ks[r];
            if (c > 0) x = df_mul_u(x, ys[(v >> 8) & 63u]);
            if (c > 1) x = df_mul_u(x, ys[(v >> 14) & 63u]);
            if (c > 2) x = df_mul_u(x, ys[(v >> 20) & 63u]);
            rate[r] = x;
        }
        __syncwarp();
        const bool odd = head().odd_coef != 0;
        const uint32_t *fr = w + head().fround, *order = w + head().forder;
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            if (!round_on(q)) continue;
            const uint32_t s = order[q * G + l];
            const Df acc = gather_df(s != kGroupNone ? src[s] : Df{0.0f, 0.0f}, w + fr[2 * q] + l, fr[2 * q + 1], false, odd);
            if (s != kGroupNone) fs[s] = df_norm(acc);
        }
        __syncwarp();
#pragma unroll
        for (int q = 0; q < NQ; ++q) f[q] = row_ok(q) ? fs[row(q)] : Df{0.0f, 0.0f};
    }
    // the residual's products k_r prod y at ys in double-float, and the FP32 Jacobian's at the FP32
    // rounding of ys
    __device__ __forceinline__ void products() {
        const uint32_t *pr = w + head().pr, np = head().pairs;
        for (uint32_t e = l; e < np; e += G) {
            const uint32_t v = pr[e], c = v >> 26;
            Df x = ks[v & 0xffu];
            const Df s0 = ys[(v >> 8) & 63u], s1 = ys[(v >> 14) & 63u];
            float x32 = x.hi;
            if (c > 0) {
                x = df_mul_u(x, s0);
                x32 = x32 * s0.hi;
            }
            if (c > 1) {
                x = df_mul_u(x, s1);
                x32 = x32 * s1.hi;
            }
            prod[e] = x;
            d[e] = x32;
        }
    }
    // r = b - ghinv x + J(y) x in lazily normalised double-float (residual_df); x published in xs,
    // b in fs; out: the FP32 rounding of the own rows' r
    __device__ __forceinline__ void residual(const Df gd, float (&r)[NQ]) {
        const uint32_t *rr = w + head().rr, *pf = w + head().pfirst, *pi = w + head().pidx;
        for (uint32_t e = l; e < R; e += G) {
            const uint32_t v = rr[e], c = v >> 18, q0 = pf[e];
            Df dr{0.0f, 0.0f};
            for (uint32_t p = 0; p < c; ++p) {
                const Df tm = df_mul_fu(prod[pi[q0 + p]], xs[(v >> (6 * p)) & 63u]);
                dr = p == 0 ? tm : df_acc(dr, tm);
            }
            rate[e] = dr;
        }
        __syncwarp();
        const bool odd = head().odd_coef != 0;
        const uint32_t *fr = w + head().fround, *order = w + head().forder;
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            if (!round_on(q)) continue;
            const uint32_t s = order[q * G + l];
            Df acc = s != kGroupNone ? df_acc(fs[s], df_neg(df_mul_fu(gd, xs[s]))) : Df{0.0f, 0.0f};
            acc = gather_df(acc, w + fr[2 * q] + l, fr[2 * q + 1], true, odd);
            if (s != kGroupNone) qs[s].hi = acc.hi + acc.lo;
        }
        __syncwarp();
#pragma unroll
        for (int q = 0; q < NQ; ++q) r[q] = row_ok(q) ? qs[row(q)].hi : 0.0f;
    }
    __device__ __forceinline__ void publish(const Df (&v)[NQ]) {
#pragma unroll
        for (int q = 0; q < NQ; ++q)
            if (row_ok(q)) ys[row(q)] = v[q];
        __syncwarp();
    }

    __device__ __forceinline__ void attempt(const DevArgs &A, bool commit) {
        bool last;
        double h_wanted;
        const double hs = this->step_size(&last, &h_wanted);
        const double hinv = 1.0 / hs;
        const double ghinv = M::gamma0(A) == 0.5 ? 2.0 * hinv : 1.0 / (hs * M::gamma0(A));
        const Df gd = df_from(ghinv), hd = df_from(hinv);
        Df f[NQ], yt[NQ], b[NQ];
        float x[NQ], x2[NQ];
        typename B::template Rows<LuT> rows;
        this->load_masks(rows);
        bool f_at_y = false;
#pragma unroll 1   // one copy of the stage body, as in GroupLane
        for (int st = 0; st < S; ++st) {
            if (st >= M::stages(A)) break;
            const int packed = st * (st - 1) / 2;
            bool eval = st == 0;
#pragma unroll
            for (int q = 0; q < NQ; ++q) yt[q] = y[q];
            if (st > 0 && M::new_f(A, st)) {
                bool moved = false;
#pragma unroll 1
                for (int j = 0; j < st; ++j) {
                    const Df ac = M::a_df(A, packed + j);
                    if (ac.hi == 0.0f) continue;
                    moved = true;
#pragma unroll
                    for (int q = 0; q < NQ; ++q)
                        if (row_ok(q)) yt[q] = df_acc(yt[q], df_times_coef_df_u(K[j * n + row(q)], ac));
                }
                if (moved) {
#pragma unroll
                    for (int q = 0; q < NQ; ++q) yt[q] = df_norm(yt[q]);
                }
                eval = moved || !f_at_y;
                f_at_y = !moved;
            }
            if (eval) {
                publish(yt);
                if (st == 0) products();
                rhs(f);
            }
            if (st == 0) {
                f_at_y = true;
                this->template neg_jac<float>(d, a);
                __syncwarp();
                this->template factor<float>((float)ghinv, a);
                this->load_rows(a, rows);
            }
#pragma unroll
            for (int q = 0; q < NQ; ++q) b[q] = f[q];
#pragma unroll 1
            for (int j = 0; j < st; ++j) {
                const Df c = M::c_df(A, packed + j);
                if (c.hi == 0.0f) continue;
                const Df ch = df_mul(c, hd);   // c / h in double-float
#pragma unroll
                for (int q = 0; q < NQ; ++q)
                    if (row_ok(q)) b[q] = df_acc(b[q], df_mul_u(ch, K[j * n + row(q)]));
            }
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                b[q] = df_norm(b[q]);
                x2[q] = b[q].hi;
                if (row_ok(q)) fs[row(q)] = b[q];   // this stage's f has been read
            }
#pragma unroll 1
            for (int pass = 0; pass < 2; ++pass) {   // x = W32^-1 b, then x2 = W32^-1 (b - W x)
                if (pass) residual(gd, x2);
                this->template solve<float>(a, rows, xs, x2);
                if (pass) break;
#pragma unroll
                for (int q = 0; q < NQ; ++q) {
                    x[q] = x2[q];
                    if (row_ok(q)) xs[row(q)] = x[q];
                }
                __syncwarp();
            }
#pragma unroll
            for (int q = 0; q < NQ; ++q)
                if (row_ok(q)) K[st * n + row(q)] = df_two_sum(x[q], x2[q]);
        }
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            if (!round_on(q)) continue;
            Df yn = y[q], ye{0.0f, 0.0f};
            bool first_e = true;
#pragma unroll
            for (int st = 0; st < S; ++st) {
                if (st >= M::stages(A)) break;
                const double mc = M::m(A, st), ec = M::e(A, st);
                const Df kv = row_ok(q) ? K[st * n + row(q)] : Df{0.0f, 0.0f};
                if (!g_zero(mc)) yn = df_acc(yn, df_times_coef_u(kv, mc));
                if (!g_zero(ec)) {
                    ye = first_e ? df_times_coef_u(kv, ec) : df_acc(ye, df_times_coef_u(kv, ec));
                    first_e = false;
                }
            }
            yn = df_norm(yn);
            if (!first_e) ye = df_norm(ye);
            const Df ay = df_abs(y[q]), an = df_abs(yn);
            const Df scale = df_add(df_mul(rtol, df_less(ay, an) ? an : ay), atol);
            const float inv = 1.0f / scale.hi;
            const float q1 = ye.hi * inv;
            const float q2 = df_add(ye, df_neg(df_mul_f(scale, q1))).hi * inv;
            const Df qv = df_two_sum(q1, q2);
            yt[q] = yn;
            if (row_ok(q)) qs[row(q)] = df_mul(qv, qv);
        }
        __syncwarp();
        Df err2{0.0f, 0.0f};
        for (uint32_t s = 0; s < n; ++s) err2 = df_add(err2, qs[s]);
        double err = sqrt(df_to(err2) * this->inv_n);
        if (!g_finite(err)) err = 1e10;
        const double fac = step_factor_mixed(err, M::order(A));
        if (this->control(A, last, hs, h_wanted, err, fac, commit)) {
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                Df v = yt[q];
                if (A.ctl.clamp_negative && (v.hi < 0.0f || (v.hi == 0.0f && v.lo < 0.0f))) v = Df{0.0f, 0.0f};
                y[q] = v;
            }
        }
        __syncwarp();   // qs is read before the next attempt writes it
    }
};

// The lanes of the group that lane `from` opens.
template <int G> __device__ __forceinline__ uint32_t gmask_of(int from) {
    return G == 32 ? 0xffffffffu : ((1u << (G & 31)) - 1u) << from;
}

template <class M, int PREC, int G, int NM> struct GroupOf { typedef GroupLane<M, PREC, G, NM> type; };
template <class M, int G, int NM> struct GroupOf<M, 4, G, NM> { typedef GroupIr<M, G, NM> type; };

// Two images (the group shape's, and the 32-lane one a warp falls back to) and the shared-memory
// layout after them: warps x warp_bytes, each a hand-over slot for one state, then the cells.
struct GroupArgs {
    const void *image, *image32;
    uint32_t bytes, bytes32, cell_bytes, warp_bytes;
};
constexpr uint32_t kGroupStateBytes = KIN_MAX_SPECIES * 8;

// Persistent over cells: the groups of a warp claim cells from the queue (A.resume: from the
// suspension list) and take each attempt together; a group without a cell computes on what it last had
// and keeps nothing. When a warp is down to one cell and nothing is left to claim, all 32 lanes
// take that cell over (G = 8: 62 -> 34 us per FP64 attempt of the shipped mechanism), which is what
// the end of a batch and its stiffest cells wait for: a warp holding a cell past A.budget attempts
// stops claiming, so that it gets there soon, and when there are fewer cells than warps each
// warp claims one only.
template <class M, int PREC, int G, int NM>
__global__ void __launch_bounds__(PREC == 0 ? 256 : 128, 1) kin_group_kernel(const __grid_constant__ DevArgs A, const __grid_constant__ GroupArgs S) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t bar;
    constexpr uint32_t kCells = 32 / G;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        mbar_arrive_expect_tx(&bar, S.bytes + (kCells > 1 ? S.bytes32 : 0u));
        tma_bulk_g2s(smem, S.image, S.bytes, &bar);
        if (kCells > 1) tma_bulk_g2s(smem + S.bytes, S.image32, S.bytes32, &bar);
    }
    const bool staged = mbar_wait(&bar, 0, A.wait_polls);
    if (!staged) mbar_wait(&bar, 0);   // let the copies land before the CTA exits
    if (__syncthreads_or(!staged)) {
        if (threadIdx.x == 0) atomicExch(A.error_flag, 1u);
        return;
    }
    const uint32_t lane = threadIdx.x & 31u, sub = lane / G, l = lane % G;
    const uint32_t gmask = G == 32 ? 0xffffffffu : ((1u << (G & 31)) - 1u) << (sub * G);
    unsigned char *state = smem + S.bytes + (kCells > 1 ? S.bytes32 : 0u) + (size_t)(threadIdx.x >> 5) * S.warp_bytes;
    unsigned char *cells = state + kGroupStateBytes;
    typename GroupOf<M, PREC, G, NM>::type C;
    C.bind_image(A, (const uint32_t *)smem, l);
    C.bind(A, cells + (size_t)sub * S.cell_bytes);
    const uint32_t parked = A.resume ? min(*(volatile uint32_t *)A.suspend_count, A.suspend_cap) : 0u;
    const uint32_t limit = A.resume ? parked : A.lanes;
    if (limit == 0) return;
    // groups of this warp that claim: all, unless the cells would not go round the warps
    const uint32_t warps = gridDim.x * (blockDim.x >> 5), share = (limit + warps - 1) / warps;
    C.load(A, 0);   // defined values for a group that never gets a cell
    bool have = false, dry = sub >= share;
    uint32_t cell = 0, attempts = 0;
    for (;;) {
        bool need = false;
        const bool hold = kCells > 1 && A.budget && __any_sync(0xffffffffu, have && attempts >= A.budget);
        for (;;) {   // the same for every lane of a group
            if (!have) {
                if (dry || hold) break;
                uint32_t at = 0;
                if (l == 0) at = atomicAdd(A.cursor, 1u);
                at = __shfl_sync(gmask, at, 0, G);
                if (at >= limit) {
                    dry = true;
                    break;
                }
                if (A.resume) {
                    const SuspendRec r = A.suspend[at];
                    cell = r.cell;
                    C.load(A, cell);
                    C.restore(A, cell, r);
                } else {
                    cell = at;
                    C.load(A, cell);
                }
                have = true;
                attempts = 0;
            }
            if (C.settle(A, cell)) {
                need = true;
                ++attempts;
                break;
            }
            C.store(A, cell);
            have = false;
        }
        const uint32_t busy = __ballot_sync(0xffffffffu, need);
        if (!busy) {
            if (hold) continue;   // the held cell is done: claim again
            break;
        }
        if constexpr (kCells > 1) {
            const int from = __ffs((int)busy) - 1;
            if (busy == gmask_of<G>(from) && __all_sync(0xffffffffu, need || dry || hold)) {
                if (need) C.put_state(state);
                __syncwarp();
                typename GroupOf<M, PREC, 32, NM>::type D;
                D.bind_image(A, (const uint32_t *)(smem + S.bytes), lane);
                D.bind(A, cells);
                const uint32_t one = __shfl_sync(0xffffffffu, cell, from);
                D.load(A, one);
                D.take_scalars(C, from);
                D.get_state(state);
                do {
                    D.attempt(A, true);
                } while (D.settle(A, one));
                D.store(A, one);
                __syncwarp();
                C.bind(A, cells + (size_t)sub * S.cell_bytes);
                C.load(A, 0);
                have = false;
                continue;
            }
        }
        C.attempt(A, need);
    }
}

}   // namespace sgb
