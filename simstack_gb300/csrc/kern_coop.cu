// Cooperative kernels for large mechanisms: one CTA integrates one cell at a
// time (persistent CTAs take cells from a work queue), its threads splitting
// every phase of the Rosenbrock step -- rates per reaction, RHS and Jacobian
// per species and entry from products formed once, elimination in panels of
// four (FP64) or eight (FP32) pivots with a thread per row, solves with a thread per
// row in blocks of columns. The step control is the reference's
// (src/sim/kinetics/kin_solver.h:189-345): every thread runs the scalar
// controller on the same values, so its decisions are uniform across the CTA.
//
// Precision 0: FP64 throughout, the same bits as the reference's solver (each
// element sees the reference's operations in the reference's order; see
// coop.h). The dense LU lives in per-CTA global scratch (L2-resident), or in
// shared memory when it fits in 64 KB; the pattern bitmask, vectors and rates
// live in shared memory.
// Precision 2 (mixed): FP64 RHS, Jacobian, residual, state and control; the
// LU and the triangular solves in FP32 with the dense LU in shared memory;
// each stage solve refined with FP64 residual sweeps.

#include <cuda_runtime.h>
#include <string.h>

#include <vector>

#include "../../include/simstack_gpu.h"
#include "coop.h"
#include "kin_device.cuh"
#include "mech.h"

namespace sgb {

namespace {

constexpr uint32_t kCoopMaxSpecies = 256;   // register cache of a pivot row: 8 columns per lane
constexpr size_t kCoopSmemLuF64Max = 64 * 1024;   // FP64 LUs up to this size live in shared memory (n <= ~90)
constexpr uint32_t kCoopMaxCols = kCoopMaxSpecies / 32;

struct CoopTab {
    const CoopMech *h;
    const uint16_t *reac;
    const uint2 *pair, *fgrp, *fterm, *jgrp, *jdst, *jterm;
    const uint32_t *fdst, *jrow;
    const uint16_t *jcol;

    // at: where the image's byte 0 lies, or would (the lists may be staged elsewhere than the header)
    __device__ __forceinline__ void init(const CoopMech *head, const unsigned char *at) {
        h = head;
        reac = (const uint16_t *)(at + h->off_reac);
        pair = (const uint2 *)(at + h->off_pair);
        fgrp = (const uint2 *)(at + h->off_fgrp);
        fdst = (const uint32_t *)(at + h->off_fdst);
        fterm = (const uint2 *)(at + h->off_fterm);
        jgrp = (const uint2 *)(at + h->off_jgrp);
        jdst = (const uint2 *)(at + h->off_jdst);
        jterm = (const uint2 *)(at + h->off_jterm);
        jrow = (const uint32_t *)(at + h->off_jrow);
        jcol = (const uint16_t *)(at + h->off_jcol);
    }
};

// Build-time phase timing (-DSGB_COOP_PROFILE): thread 0 of every CTA adds the
// clock cycles of each phase to g_coop_phase_cycles (rhs, Jacobian, factor,
// solves, refinement residual, total attempt).
#ifdef SGB_COOP_PROFILE
__device__ unsigned long long g_coop_phase_cycles[8];
#define SGB_PHASE(i, stmt)                                                      \
    do {                                                                        \
        const long long _t0 = clock64();                                       \
        stmt;                                                                   \
        if (tid == 0) atomicAdd(&g_coop_phase_cycles[i], (unsigned long long)(clock64() - _t0)); \
    } while (0)
#else
#define SGB_PHASE(i, stmt) stmt
#endif

// Species from which the elimination runs in panels (a thread per row: CTAs of at least n threads);
// below, and in smaller CTAs, pivot by pivot. FP64 steps with panels, to those with pivots: 6 species 0.96, 17 0.88, 24 0.84,
// 32 0.80, 39 0.78 (a CTA of a warp: 17 species 0.65, 24 0.51). Mixed steps of 40 species: 0.82.
constexpr uint32_t kCoopPanelMin = 40, kCoopPanelMinF64 = 4;

// Shared-memory doubles before the mixed path's FP32 arrays.
__host__ __device__ inline uint32_t coop_smem_doubles(uint32_t n, uint32_t R) { return 11u * n + 2u * R + 8u; }

// Default budget up to which the term lists join shared memory: none. Measured on the 200-species
// FP64 case, staging them (149 KB of shared memory per CTA) made the step 1.31x slower, because the
// smaller L1 then caches less of the global-memory LU; callers may enable it per precision.
constexpr uint32_t kCoopSmemBudget = 0;

// Shared memory of one CTA: doubles, x32 (256 floats), pattern (n x 8 words), lcnt (n u16,
// padded), then the LU (mixed always, n x ld floats; FP64 when it fits kCoopSmemLuF64Max), then
// -- when they fit the budget -- the RHS / Jacobian term lists (image bytes [off_reac, off_pat)).
struct CoopSmemLayout {
    size_t lu, lu_bytes, terms, terms_bytes, total;
};
__host__ __device__ inline CoopSmemLayout coop_layout(int prec, const CoopMech &h, uint32_t budget) {
    CoopSmemLayout L;
    L.lu = (size_t)coop_smem_doubles(h.n, h.R) * 8 + kCoopMaxSpecies * 4 + (size_t)h.n * 32 + ((h.n + 7) / 8) * 16;
    const size_t lu64 = (size_t)h.n * h.ld * sizeof(double);
    L.lu_bytes = prec == 2 ? (size_t)h.n * h.ld * 4 : (lu64 <= kCoopSmemLuF64Max ? lu64 : 0);
    L.terms = (L.lu + L.lu_bytes + 15) / 16 * 16;
    const size_t tb = (size_t)h.off_pat - h.off_reac;
    L.terms_bytes = L.terms + tb <= budget ? tb : 0;
    L.total = L.terms + L.terms_bytes;
    return L;
}

// Whether the Jacobian's products fit the shared-memory vectors that are free while it is formed, and the
// CTA's scratch before them: the FP64 LU, or the mixed path's Jacobian entries.
__host__ __device__ inline bool coop_products_fit(const CoopMech &h) { return h.pairs <= 8u * h.n + h.R; }
__host__ __device__ inline size_t coop_scratch_base(int prec, const CoopMech &h) {
    return prec == 2 ? (size_t)h.nj : (size_t)h.n * h.ld;
}

template <int PREC>
struct CoopCell {
    typedef typename Pick<PREC == 0, double, float>::type Cf;   // LU and solve arithmetic
    static constexpr bool kMixed = PREC == 2;
    typedef RuntimeCoef M;

    CoopTab tb;
    uint32_t n, R, ld, nj, tid, NT, lane, warp, W;
    double *y, *ytmp, *fcn, *src, *qv, *rb, *xv, *K, *kr, *rate, *red;
    float *x32;
    Cf *a;          // dense LU [n][ld]
    bool lu_global;         // eliminate with loads before stores (the LU lives in global scratch: FP64, large)
    const uint32_t *pat;    // shared: filled pattern, 8 words per row
    const uint16_t *lcnt;   // shared: rows below the diagonal per column
    double *js;     // mixed: Jacobian entries (a = -J) in FP64
    double *prod;   // the Jacobian's products
    // replicated scalar state (kin_solver.h:189-345)
    double t, h, seg_end, applied, duration, period, first, count, steps, rejects, pulses, failed;
    uint32_t iterations, transitions;
    int phase;
    bool pending, reject_last, reject_more;
    bool on_pattern;        // mixed: this attempt touches the pattern's elements alone

    __device__ __forceinline__ void sync() const { __syncthreads(); }
    __device__ __forceinline__ bool bit(uint32_t i, uint32_t j) const { return (pat[i * 8u + (j >> 5)] >> (j & 31u)) & 1u; }

    __device__ void load(const DevArgs &A, uint32_t cell) {
        const uint32_t p = A.padded;
        for (uint32_t s = tid; s < n; s += NT) {
            y[s] = A.y[(size_t)s * p + cell];
            src[s] = A.src[(size_t)s * p + cell];
        }
        for (uint32_t r = tid; r < R; r += NT) kr[r] = A.k[(size_t)r * p + cell];
        h = A.h[cell];
        period = A.period[cell];
        first = A.pulse_first[cell];
        count = A.pulse_count[cell];
        duration = A.duration;
        steps = rejects = pulses = 0.0;
        failed = A.failed[cell];
        t = 0.0;
        applied = 0.0;
        transitions = 0;
        phase = kPhaseSegStart;
        sync();
    }

    // A parked cell: its scalar state from the record (load() read y, k, src and failed).
    __device__ void restore(const SuspendRec &r) {
        t = r.t;
        h = r.h;
        seg_end = r.seg_end;
        applied = r.applied;
        pending = (r.flags & 1u) != 0;
        reject_last = (r.flags & 2u) != 0;
        reject_more = (r.flags & 4u) != 0;
        iterations = r.iterations;
        transitions = r.transitions;
        phase = kPhaseStepping;
    }

    __device__ void store(const DevArgs &A, uint32_t cell) {
        const uint32_t p = A.padded;
        for (uint32_t s = tid; s < n; s += NT) A.y[(size_t)s * p + cell] = y[s];
        if (tid == 0) {
            A.h[cell] = h;
            A.failed[cell] = failed;
            A.steps[cell] += steps;
            A.rejects[cell] += rejects;
            A.pulses[cell] += pulses;
        }
        sync();
    }

    __device__ void seg_start(const DevArgs &A) {
        pending = applied < count;
        double next_pulse = sgb_fma(applied, period, first);
        seg_end = pending ? vmin(next_pulse, duration) : duration;
        bool active = t < seg_end && !(failed > 0.0);
        reject_last = false;
        reject_more = false;
        h = h > 0.0 ? h : A.ctl.h_start;
        iterations = 0;
        phase = active ? kPhaseStepping : kPhaseSegFinish;
    }

    __device__ void seg_finish(const DevArgs &A, uint32_t cell) {
        bool alive = !(failed > 0.0);
        bool hit = pending && alive && t >= seg_end;
        if (hit) {
            const uint32_t p = A.padded;
            for (uint32_t s = tid; s < n; s += NT) y[s] = y[s] + A.pulse[(size_t)s * p + cell];
            sync();
            applied = applied + 1.0;
            pulses = pulses + 1.0;
            h = A.ctl.h_start;
        }
        bool done = (t >= duration && applied >= count) || !alive;
        phase = done ? kPhaseDone : kPhaseSegStart;
    }

    // As the lane kernels' settle: transitions until a step attempt is due (true) or the cell is done.
    __device__ bool settle(const DevArgs &A, uint32_t cell) {
        for (;;) {
            if (++transitions > (1u << 24)) {
                failed = 1.0;
                phase = kPhaseDone;
            }
            switch (phase) {
                case kPhaseSegStart: seg_start(A); break;
                case kPhaseSegFinish: seg_finish(A, cell); break;
                case kPhaseStepping:
                    if (++iterations > A.ctl.max_steps) {
                        failed = 1.0;
                        phase = kPhaseSegFinish;
                        break;
                    }
                    return true;
                default: return false;
            }
        }
    }

    // acc = fma(coef, from[index], acc) over this lane's list of a group (coop.h), four terms at a time so
    // that their loads overlap.
    __device__ __forceinline__ double gather(double acc, const uint2 *term, uint32_t len, const double *from) const {
        for (uint32_t k = 0; k < len; k += 4) {
            uint2 t[4];
            double v[4];
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q) t[q] = k + q < len ? term[(k + q) * 32u] : make_uint2(~0u, 0u);
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q) v[q] = t[q].x != ~0u ? from[t[q].x] : 0.0;
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q)
                if (t[q].x != ~0u) acc = sgb_fma(__hiloint2double((int)t[q].y, 0), v[q], acc);
        }
        return acc;
    }

    // fcn = f(yy): rates per reaction, then each species' terms in reaction order.
    __device__ void rhs(const double *yy) {
        const uint2 *words = (const uint2 *)tb.reac;   // count, s0 | s1 << 16 in 16-bit fields
        for (uint32_t r0 = tid; r0 < R; r0 += 4 * NT) {
            uint2 w[4];
            double v[4];
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q) {
                const uint32_t r = r0 + q * NT;
                w[q] = r < R ? words[r] : make_uint2(0u, 0u);
                v[q] = r < R ? kr[r] : 0.0;
            }
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q) {
                const uint32_t c = w[q].x & 0xffffu;
                if (c > 0) v[q] = v[q] * yy[w[q].x >> 16];
                if (c > 1) v[q] = v[q] * yy[w[q].y & 0xffffu];
                if (c > 2) v[q] = v[q] * yy[w[q].y >> 16];
                if (r0 + q * NT < R) rate[r0 + q * NT] = v[q];
            }
        }
        sync();
        for (uint32_t g = warp; g < (n + 31) / 32; g += W) {
            const uint2 range = tb.fgrp[g];
            const uint32_t s = tb.fdst[g * 32 + lane];
            const double f = gather(s != ~0u ? src[s] : 0.0, tb.fterm + range.x + lane, range.y, rate);
            if (s != ~0u) fcn[s] = f;
        }
        sync();
    }

    // a = -J at yy (zero elsewhere); mixed: the FP64 entries also kept in js. The products
    // k_r prod_{q != p} y_q are formed once per (reaction, reactant) in `prod` (the panel buffers and the
    // rates' array, or the CTA's scratch where they do not fit) and summed per entry in (r, p, e)
    // order, entries of like length to a warp (200 species: 230k -> 40k cycles FP64, 130k -> 20k mixed,
    // where every term formed its own product behind four dependent table reads).
    __device__ void neg_jac(const double *yy) {
        if (kMixed || !lu_global) {
            uint2 *z = (uint2 *)a;   // 8-byte aligned
            const uint32_t words = n * ld * (uint32_t)sizeof(Cf) / 8u;
            for (uint32_t q = tid; q < words; q += NT) z[q] = make_uint2(0u, 0u);
            if (tid == 0 && sizeof(Cf) == 4 && ((n * ld) & 1u)) a[n * ld - 1] = (Cf)0.0;
        } else {
            double2 *z = (double2 *)a;
            for (uint32_t q = tid; q < n * ld / 2; q += NT) z[q] = make_double2(0.0, 0.0);
            if (tid == 0 && ((n * ld) & 1u)) a[n * ld - 1] = (Cf)0.0;
        }
        const uint32_t pairs = tb.h->pairs;
        for (uint32_t q0 = tid; q0 < pairs; q0 += 4 * NT) {
            uint2 w[4];
            double v[4];
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q) w[q] = q0 + q * NT < pairs ? tb.pair[q0 + q * NT] : make_uint2(0u, 0u);
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q) v[q] = R ? kr[w[q].x & 0xffffffu] : 0.0;
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q) {
                const uint32_t c = w[q].x >> 24;
                if (c > 0) v[q] = v[q] * yy[w[q].y & 0xffffu];
                if (c > 1) v[q] = v[q] * yy[w[q].y >> 16];
                if (q0 + q * NT < pairs) prod[q0 + q * NT] = v[q];
            }
        }
        sync();
        for (uint32_t g = warp; g < (nj + 31) / 32; g += W) {
            const uint2 range = tb.jgrp[g], to = tb.jdst[g * 32 + lane];
            const double acc = gather(0.0, tb.jterm + range.x + lane, range.y, prod);
            if (to.x == ~0u) continue;
            if constexpr (kMixed) js[to.y] = acc;
            a[to.x] = (Cf)acc;
        }
        sync();
    }

    // In place: a -> L\U of (I ghinv - J), diagonal holding 1/U(k,k); pivot by
    // pivot (kin_solver.h:97-113 applies the same updates row by row). Rows and
    // columns are walked densely; the pattern bits select the elements the
    // reference updates. The warp that updates row i also forms its multiplier
    // l(i,k) = a[i][k] * (1/U(k,k)) and stores it once the row is done, so a pivot
    // needs one barrier (FP32) or two (FP64: the shared inverse).
    __device__ void factor(Cf ghinv) {
        if (n >= (kMixed ? kCoopPanelMin : kCoopPanelMinF64) && NT >= n && !(kMixed && on_pattern)) {
            if constexpr (kMixed) factor_panels_f32(ghinv);
            else factor_panels<4>(ghinv);
            return;
        }
        for (uint32_t k = 0; k < n; ++k) {
            const uint32_t nl = lcnt[k];
            Cf inv;
            if constexpr (kMixed) {
                // FP32: every thread divides (cheap on the FP32 pipe); the inverted diagonal is
                // stored after the pivot's closing barrier, once every thread has read a[k][k]
                if (nl == 0) {   // nothing below the pivot: the next pivot reads none of this pivot's writes
                    if (tid == 0) a[(size_t)k * ld + k] = (Cf)1.0 / (a[(size_t)k * ld + k] + ghinv);
                    continue;
                }
                inv = (Cf)1.0 / (a[(size_t)k * ld + k] + ghinv);
            } else {
                // FP64: 1/U(k,k) once (a division costs many FP64 instructions per warp), shared through red[4]
                Cf *inv_s = (Cf *)(red + 4);
                if (tid == 0) {
                    const Cf v = (Cf)1.0 / (a[(size_t)k * ld + k] + ghinv);
                    a[(size_t)k * ld + k] = v;
                    *inv_s = v;
                }
                if (nl == 0) continue;
                sync();
                inv = *inv_s;
            }
            // pivot row k (final) cached per lane: columns k+1+lane+32c in the pattern
            const uint32_t width = n - 1 - k, chunks = (width + 31) / 32;
            Cf pv[kCoopMaxCols];
            uint32_t live = 0;
#pragma unroll
            for (uint32_t c = 0; c < kCoopMaxCols; ++c) {
                const uint32_t j = k + 1 + lane + 32u * c;
                const bool on = c < chunks && j < n && bit(k, j);
                pv[c] = (Cf)0.0;
                if (on) {
                    pv[c] = a[(size_t)k * ld + j];
                    live |= 1u << c;
                }
            }
            if (lu_global) {
                // global-memory LU: the row's elements first, then the updates, so the loads issue
                // back to back instead of each waiting behind the previous element's store
                for (uint32_t i = k + 1 + warp; i < n; i += W) {
                    if (!bit(i, k)) continue;   // same for the whole warp
                    Cf *row = a + (size_t)i * ld;
                    const Cf l = row[k] * inv;
                    Cf v[kCoopMaxCols];
#pragma unroll
                    for (uint32_t c = 0; c < kCoopMaxCols; ++c) {
                        const uint32_t j = k + 1 + lane + 32u * c;
                        v[c] = (Cf)0.0;
                        if ((live >> c) & 1u) v[c] = row[j];
                    }
#pragma unroll
                    for (uint32_t c = 0; c < kCoopMaxCols; ++c) {
                        const uint32_t j = k + 1 + lane + 32u * c;
                        if ((live >> c) & 1u) row[j] = sgb_fma(-l, pv[c], v[c]);
                    }
                    __syncwarp();   // every lane has read a[i][k]
                    if (lane == 0) row[k] = l;
                }
            } else {
                for (uint32_t i = k + 1 + warp; i < n; i += W) {
                    if (!bit(i, k)) continue;
                    Cf *row = a + (size_t)i * ld;
                    const Cf l = row[k] * inv;
#pragma unroll
                    for (uint32_t c = 0; c < kCoopMaxCols; ++c) {
                        const uint32_t j = k + 1 + lane + 32u * c;
                        if ((live >> c) & 1u) row[j] = sgb_fma(-l, pv[c], row[j]);
                    }
                    __syncwarp();
                    if (lane == 0) row[k] = l;
                }
            }
            sync();
            if constexpr (kMixed) {   // every thread has read a[k][k]
                if (tid == 0) a[(size_t)k * ld + k] = inv;
            }
        }
        sync();
    }

    // B pivots per pass (k .. k+B-1), one thread per row in the panel:
    //   panel     thread i holds row i's B block entries; pivot by pivot the pivot row's thread takes
    //             1/U and publishes its entries, and every row below forms its multiplier and takes the
    //             update of the block's later columns
    //   U rows    one thread per column right of the block: the block's rows take each other's
    //             updates (loaded ahead of the panel)
    //   trailing  a warp per row, 32 columns at a time with the block's U entries in registers: every
    //             element is loaded and stored once and takes the block's updates in ascending order
    // Every element receives the operations of the pivot-by-pivot order, in that order. What this buys
    // over a pivot (FP32) or two (FP64) per pass: a row's multiplier is one instruction per 32 rows and not
    // one per row (FP64: a third of the instructions of the unit that bounds it), and the trailing
    // elements make 1/B of the trips to shared memory (FP32) or L2 (FP64). The buffers are the
    // stage vectors K (multipliers) and the four vectors after them (U rows), free until the
    // stages begin, so B is 4 in FP64 and 8 in FP32; the pattern words use x32. Measured on 200 species /
    // 1,200 reactions, cycles per factorisation: FP64 one CTA per SM 3.05M -> 1.85M, two (per pair of
    // cells) 2.62M, most of it FP64 instructions at the rate of their unit; FP32 550k -> 357k.
    template <uint32_t B>
    __device__ void factor_panels(Cf ghinv) {
        static_assert(B * sizeof(Cf) <= 32, "panel buffers: 32 bytes per row in K, and as much for the U rows");
        Cf *inv_s = (Cf *)(red + 4);
        Cf *Lp = (Cf *)K;        // [row][B]
        Cf *Up = (Cf *)ytmp;     // [B][column]
        uint16_t *live = (uint16_t *)x32, *rows_on = live + kCoopMaxSpecies;   // pattern bits per column / row of the block
        for (uint32_t k = 0; k < n; k += B) {
            const uint32_t nb = n - k < B ? n - k : B, j0 = k + nb;
            const uint32_t mine = (1u << nb) - 1u;
            // row tid of the panel
            const bool row_in = tid >= k && tid < n;
            uint32_t bm = 0;
            Cf pa[B];
            if (row_in) {
                bm = (pat[tid * 8u + (k >> 5)] >> (k & 31u)) & mine;   // k is a multiple of B: one word
#pragma unroll
                for (uint32_t p = 0; p < B; ++p) pa[p] = p < nb ? a[(size_t)tid * ld + k + p] : (Cf)0.0;
            }
            // column j0 + tid of the U rows, loaded ahead
            const uint32_t j = j0 + tid;
            uint32_t lv = 0;
            Cf ux[B];
            if (j < n) {
#pragma unroll
                for (uint32_t p = 0; p < B; ++p) {
                    ux[p] = (Cf)0.0;
                    if (p < nb && bit(k + p, j)) {
                        lv |= 1u << p;
                        ux[p] = a[(size_t)(k + p) * ld + j];
                    }
                }
            }
#pragma unroll
            for (uint32_t p = 0; p < B; ++p) {
                if (p >= nb) break;
                const uint32_t kp = k + p;
                if (tid == kp) {
                    const Cf v = (Cf)1.0 / (pa[p] + ghinv);
#pragma unroll
                    for (uint32_t q = 0; q < B; ++q) Lp[kp * B + q] = pa[q];
                    inv_s[p & 3u] = v;
                    pa[p] = v;
                }
                sync();
                if (tid > kp && row_in && ((bm >> p) & 1u)) {
                    const Cf l = pa[p] * inv_s[p & 3u];
                    pa[p] = l;
                    const uint32_t on = (pat[kp * 8u + (k >> 5)] >> (k & 31u)) & mine;   // row kp's columns in the block
#pragma unroll
                    for (uint32_t q = p + 1; q < B; ++q)
                        if ((on >> q) & 1u) pa[q] = sgb_fma(-l, Lp[kp * B + q], pa[q]);
                }
            }
            if (row_in) {
#pragma unroll
                for (uint32_t p = 0; p < B; ++p)
                    if (p < nb) a[(size_t)tid * ld + k + p] = pa[p];
                if (tid >= j0) {
#pragma unroll
                    for (uint32_t p = 0; p < B; ++p) Lp[tid * B + p] = pa[p];
                    rows_on[tid] = (uint16_t)bm;
                }
            }
            if (j0 >= n) break;
            if (j < n) {
#pragma unroll
                for (uint32_t p = 1; p < B; ++p) {
                    const uint32_t lo = (pat[(k + p) * 8u + (k >> 5)] >> (k & 31u)) & lv;
#pragma unroll
                    for (uint32_t q = 0; q < p; ++q)
                        if ((lo >> q) & 1u) ux[p] = sgb_fma(-Lp[(k + p) * B + q], ux[q], ux[p]);
                }
#pragma unroll
                for (uint32_t p = 0; p < B; ++p) {
                    if ((lv >> p) & 1u) a[(size_t)(k + p) * ld + j] = ux[p];
                    Up[p * n + j] = ux[p];
                }
                live[j] = (uint16_t)lv;
            }
            sync();
            for (uint32_t c = j0; c < n; c += 32) {
                if (n - c <= 16) {   // the last columns: two or four rows to a warp
                    trailing_rest<B>(Lp, Up, live, rows_on, c, j0, n - c <= 8 ? 8u : 16u);
                    break;
                }
                const uint32_t jc = c + lane;
                const bool on = jc < n;
                const uint32_t lc = on ? live[jc] : 0u;
                const uint32_t any = __reduce_or_sync(0xffffffffu, lc);
                if (!any) continue;
                const bool full = __all_sync(0xffffffffu, !on || lc == mine);
                Cf u[B];
#pragma unroll
                for (uint32_t p = 0; p < B; ++p) u[p] = on ? Up[p * n + jc] : (Cf)0.0;
                for (uint32_t i = j0 + warp; i < n; i += 4 * W) {   // four rows at a time: their loads overlap
                    uint32_t b[4];
                    Cf v[4];
#pragma unroll
                    for (uint32_t r = 0; r < 4; ++r) {   // b: the same for the whole warp
                        const uint32_t ii = i + r * W;
                        b[r] = ii < n ? rows_on[ii] & any : 0u;
                        v[r] = (Cf)0.0;
                        if (b[r] && on) v[r] = a[(size_t)ii * ld + jc];
                    }
#pragma unroll
                    for (uint32_t r = 0; r < 4; ++r) {
                        if (!b[r]) continue;
                        const uint32_t ii = i + r * W;
                        const Cf *lp = Lp + ii * B;
                        if (full && b[r] == mine) {
#pragma unroll
                            for (uint32_t p = 0; p < B; ++p) v[r] = sgb_fma(-lp[p], u[p], v[r]);
                            if (on) a[(size_t)ii * ld + jc] = v[r];
                        } else {
                            const uint32_t m = b[r] & lc;
#pragma unroll
                            for (uint32_t p = 0; p < B; ++p)
                                if ((m >> p) & 1u) v[r] = sgb_fma(-lp[p], u[p], v[r]);
                            if (m) a[(size_t)ii * ld + jc] = v[r];
                        }
                    }
                }
            }
            sync();
        }
        sync();
    }

    // The trailing update's last `width` (8 or 16) columns or fewer: a row's FMA there would use a quarter or half
    // of the lanes for the FP64 unit's same 64 cycles, so a warp takes 32 / width rows side by side
    // (200 species, two cells per SM: 2.77M -> 2.62M cycles per factorisation).
    template <uint32_t B>
    __device__ __forceinline__ void trailing_rest(const Cf *Lp, const Cf *Up, const uint16_t *live, const uint16_t *rows_on, uint32_t c,
                                                  uint32_t j0, uint32_t width) {
        const uint32_t jc = c + (lane & (width - 1)), rows = 32 / width, step = W * rows;
        const uint32_t lc = jc < n ? live[jc] : 0u;
        if (!__any_sync(0xffffffffu, lc != 0)) return;
        Cf u[B];
#pragma unroll
        for (uint32_t p = 0; p < B; ++p) u[p] = jc < n ? Up[p * n + jc] : (Cf)0.0;
        for (uint32_t i0 = j0 + warp * rows; i0 < n; i0 += 2 * step) {   // two rows per lane: their loads overlap
            uint32_t m[2];
            Cf v[2];
#pragma unroll
            for (uint32_t r = 0; r < 2; ++r) {
                const uint32_t ii = i0 + lane / width + r * step;
                m[r] = ii < n ? rows_on[ii] & lc : 0u;
                v[r] = m[r] ? a[(size_t)ii * ld + jc] : (Cf)0.0;
            }
#pragma unroll
            for (uint32_t r = 0; r < 2; ++r) {
                const uint32_t ii = i0 + lane / width + r * step;
                if (!m[r]) continue;
                const Cf *lp = Lp + ii * B;
#pragma unroll
                for (uint32_t p = 0; p < B; ++p)
                    if ((m[r] >> p) & 1u) v[r] = sgb_fma(-lp[p], u[p], v[r]);
                a[(size_t)ii * ld + jc] = v[r];
            }
        }
    }

    // factor_panels in FP32, B = 8, without pattern tests: an element off the pattern is zero and stays
    // zero, and a product with it changes no finite value (the others: attempt()). The block's rows lie in one warp, which
    // factors them by shuffle (a reciprocal, one shuffle per entry), so a panel needs two barriers and
    // not one per pivot; trailing rows are walked 64 columns at a time, the multipliers of a row
    // (two 16-byte broadcasts) serving sixteen FMAs per lane. 357k cycles per factorisation of 200
    // species with the FP64 panels' pattern tests and barriers, 175k so.
    static __device__ __forceinline__ void load8(float (&out)[8], const float *from) {   // 16-byte aligned
        const float4 lo = ((const float4 *)from)[0], hi = ((const float4 *)from)[1];
        out[0] = lo.x; out[1] = lo.y; out[2] = lo.z; out[3] = lo.w;
        out[4] = hi.x; out[5] = hi.y; out[6] = hi.z; out[7] = hi.w;
    }
    __device__ void factor_panels_f32(float ghinv) {
        constexpr uint32_t B = 8;
        float *A32 = (float *)a, *Lp = (float *)K, *Up = (float *)ytmp;
        for (uint32_t k = 0; k < n; k += B) {
            const uint32_t nb = n - k < B ? n - k : B, j0 = k + nb, j = j0 + tid, w0 = k >> 5, base = k & 31u;
            const bool row_in = tid >= k && tid < n;
            float pa[B], ux[B];
#pragma unroll
            for (uint32_t p = 0; p < B; ++p) {
                pa[p] = row_in && p < nb ? A32[(size_t)tid * ld + k + p] : 0.0f;
                ux[p] = j < n && p < nb ? A32[(size_t)(k + p) * ld + j] : 0.0f;
            }
            if (warp == w0) {
#pragma unroll
                for (uint32_t p = 0; p < B; ++p) {
                    if (p >= nb) break;
                    const float inv = 1.0f / (__shfl_sync(0xffffffffu, pa[p], base + p) + ghinv);
                    const float l = pa[p] * inv;
#pragma unroll
                    for (uint32_t q = p + 1; q < B; ++q) {
                        const float u = __shfl_sync(0xffffffffu, pa[q], base + p);
                        if (lane > base + p) pa[q] = sgb_fma(-l, u, pa[q]);
                    }
                    pa[p] = lane > base + p ? l : lane == base + p ? inv : pa[p];
                }
                if (lane >= base && lane < base + nb) {
#pragma unroll
                    for (uint32_t p = 0; p < B; ++p) Lp[tid * B + p] = pa[p];
                }
            }
            sync();
            if (row_in && warp > w0) {
#pragma unroll
                for (uint32_t p = 0; p < B; ++p) {
                    if (p >= nb) break;
                    float up[B];
                    load8(up, Lp + (k + p) * B);
                    const float l = pa[p] * up[p];
                    pa[p] = l;
#pragma unroll
                    for (uint32_t q = p + 1; q < B; ++q) pa[q] = sgb_fma(-l, up[q], pa[q]);
                }
            }
            if (row_in) {
#pragma unroll
                for (uint32_t p = 0; p < B; ++p)
                    if (p < nb) A32[(size_t)tid * ld + k + p] = pa[p];
                if (tid >= j0) {
#pragma unroll
                    for (uint32_t p = 0; p < B; ++p) Lp[tid * B + p] = pa[p];
                }
            }
            if (j0 >= n) break;
            if (j < n) {
#pragma unroll
                for (uint32_t p = 1; p < B; ++p)
#pragma unroll
                    for (uint32_t q = 0; q < p; ++q) ux[p] = sgb_fma(-Lp[(k + p) * B + q], ux[q], ux[p]);
#pragma unroll
                for (uint32_t p = 0; p < B; ++p) {
                    A32[(size_t)(k + p) * ld + j] = ux[p];
                    Up[p * n + j] = ux[p];
                }
            }
            sync();
            for (uint32_t c = j0; c < n; c += 64) {
                const uint32_t c0 = c + lane, c1 = c0 + 32;
                const bool on0 = c0 < n, on1 = c1 < n;
                float u0[B], u1[B];
                bool any = false;
#pragma unroll
                for (uint32_t p = 0; p < B; ++p) {
                    u0[p] = on0 ? Up[p * n + c0] : 0.0f;
                    u1[p] = on1 ? Up[p * n + c1] : 0.0f;
                    any = any || u0[p] != 0.0f || u1[p] != 0.0f;
                }
                if (!__any_sync(0xffffffffu, any)) continue;
                for (uint32_t i = j0 + warp; i < n; i += 4 * W) {   // four rows at a time
                    float v0[4], v1[4];
#pragma unroll
                    for (uint32_t r = 0; r < 4; ++r) {
                        const uint32_t ii = i + r * W;
                        if (ii >= n) break;   // the same for the whole warp
                        const float *q = A32 + ii * ld + c0;
                        v0[r] = on0 ? q[0] : 0.0f;
                        v1[r] = on1 ? q[32] : 0.0f;
                    }
#pragma unroll
                    for (uint32_t r = 0; r < 4; ++r) {
                        const uint32_t ii = i + r * W;
                        if (ii >= n) break;
                        float lp[B];
                        load8(lp, Lp + ii * B);
#pragma unroll
                        for (uint32_t p = 0; p < B; ++p) {
                            v0[r] = sgb_fma(-lp[p], u0[p], v0[r]);
                            v1[r] = sgb_fma(-lp[p], u1[p], v1[r]);
                        }
                        float *q = A32 + ii * ld + c0;
                        if (on0) q[0] = v0[r];
                        if (on1) q[32] = v1[r];
                    }
                }
            }
            sync();
        }
        sync();
    }

    // x = (LU)^-1 x in place. Forward (unit L) takes each row's columns ascending, backward (U,
    // diagonal holding 1/U(k,k)) descending, then the diagonal.
    template <class V>
    __device__ void solve(V *x) {
        // Few species: the FP32 solve of whole blocks costs more than the elements that there are (a step, by
        // elements / by blocks, to the solve before both: 3 species 0.95 / 1.29, 8 0.91 / 1.20, 17 0.94 / 1.06, 33 0.91 / 0.98,
        // 39 0.87 / 0.89).
        if (NT < n || (kMixed ? on_pattern || n < kCoopPanelMin : n < kCoopPanelMinF64)) {
            solve_plain(x);
            return;
        }
        const uint32_t warps = (n + 31) / 32;   // the warps that hold rows; the others wait at the end
        if (warp < warps) {
            if constexpr (kMixed) solve_rows_f32(a, n, ld, x, 32 * warps);
            else solve_rows(a, pat, n, ld, x, 32 * warps);
        }
        sync();
    }

    // A barrier among the CTA's first `threads` threads.
    static __device__ __forceinline__ void sync_rows(uint32_t threads) { asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory"); }

    // A thread per row, its x in a register, eight columns per barrier: the warp that holds those
    // rows solves them, passing each one on through shared memory (35 cycles; the two shuffles take
    // 64), while the rows past that warp take the eight before; every row has the next eight
    // columns' coefficients on their way meanwhile. What is left is the chain itself: an FMA
    // (FP64 64 cycles, backward a product before it) and the hand-over per column: 157k -> 86k
    // cycles per FP64 solve of 200 species (one CTA per SM).
    // (Calls of their own: inlined, the compiler spreads the registers of the whole step over them.)
    static __device__ __noinline__ void solve_rows(const Cf *a, const uint32_t *pat, uint32_t n, uint32_t ld, double *x,
                                                   uint32_t threads) {
        constexpr uint32_t B = 8;
        const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
        const uint32_t i = tid, blocks = (n + B - 1) / B;
        const bool mine = i < n;
        const Cf *row = a + (size_t)(mine ? i : 0) * ld;
        const uint32_t *prow = pat + (mine ? i : 0) * 8u;
        double xi = mine ? x[i] : 0.0;
        Cf c[B], next[B];
        auto load = [&](Cf (&r)[B], uint32_t k, bool need) {
#pragma unroll
            for (uint32_t q = 0; q < B; ++q) r[q] = need && k + q < n ? row[k + q] : (Cf)0.0;
        };
        auto bits = [&](uint32_t k) { return (prow[k >> 5] >> (k & 31u)) & 0xffu; };   // this row's pattern at columns k..k+7
        load(c, 0, mine);
        sync_rows(threads);   // x is read
        for (uint32_t s = 0; s < blocks; ++s) {
            const uint32_t k = s * B, w0 = k >> 5, base = k & 31u, on = bits(k);
            load(next, k + B, mine && i > k + B);
            if (warp == w0) {
#pragma unroll
                for (uint32_t q = 0; q < B; ++q) {
                    if (k + q >= n) break;
                    if (lane == base + q) x[k + q] = xi;
                    __syncwarp();
                    if (mine && lane > base + q && ((on >> q) & 1u)) xi = sgb_fma(-(double)c[q], x[k + q], xi);
                }
            }
            sync_rows(threads);
            if (warp > w0 && mine) {
#pragma unroll
                for (uint32_t q = 0; q < B; ++q)
                    if (k + q < n && ((on >> q) & 1u)) xi = sgb_fma(-(double)c[q], x[k + q], xi);
            }
#pragma unroll
            for (uint32_t q = 0; q < B; ++q) c[q] = next[q];
        }
        load(c, (blocks - 1) * B, mine);
        for (uint32_t s = blocks; s-- > 0;) {
            const uint32_t k = s * B, w0 = k >> 5, base = k & 31u, on = bits(k);
            load(next, s ? k - B : 0u, mine && s && i < k);
            if (warp == w0) {
#pragma unroll
                for (uint32_t q = B; q-- > 0;) {
                    if (k + q >= n) continue;
                    if (lane == base + q) x[k + q] = xi = xi * (double)c[q];   // all its updates are in
                    __syncwarp();
                    if (lane < base + q && ((on >> q) & 1u)) xi = sgb_fma(-(double)c[q], x[k + q], xi);
                }
            }
            sync_rows(threads);
            if (warp < w0) {
#pragma unroll
                for (uint32_t q = B; q-- > 0;)
                    if (k + q < n && ((on >> q) & 1u)) xi = sgb_fma(-(double)c[q], x[k + q], xi);
            }
#pragma unroll
            for (uint32_t q = 0; q < B; ++q) c[q] = next[q];
        }
    }
    // FP32, a barrier per 32 columns: a warp solves its 32 rows by shuffle (~30 cycles a column; the barriers of
    // eight-column blocks cost more than they spread) from coefficients it loaded once for both
    // directions, the rows past it have theirs on their way meanwhile. No pattern or bounds tests:
    // off the pattern the LU is zero, and so are the triangle and x of rows past the end (x has
    // room for whole blocks). 34k -> 24k cycles per solve of 200 species.
    static __device__ __noinline__ void solve_rows_f32(const Cf *a, uint32_t n, uint32_t ld, float *x, uint32_t threads) {
        constexpr uint32_t B = 32;
        const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
        const uint32_t blocks = threads / 32;
        const bool mine = tid < n;
        const float *row = (const float *)a + (size_t)(mine ? tid : 0) * ld;
        float xi = mine ? x[tid] : 0.0f;
        float cd[B], co[B];   // this row's coefficients in its own block, and in the one being applied
        auto load = [&](float (&r)[B], uint32_t k) {
            if (k + B <= n) {
#pragma unroll
                for (uint32_t q = 0; q < B; ++q) r[q] = row[k + q];
            } else {
#pragma unroll
                for (uint32_t q = 0; q < B; ++q) r[q] = k + q < n ? row[k + q] : 0.0f;
            }
        };
        auto apply = [&](uint32_t k, bool up) {   // the columns of block k, ascending or descending
            float xk[B];
#pragma unroll
            for (uint32_t q = 0; q < B; ++q) xk[q] = x[k + q];
            if (up) {
#pragma unroll
                for (uint32_t q = 0; q < B; ++q) xi = sgb_fma(-co[q], xk[q], xi);
            } else {
#pragma unroll
                for (uint32_t q = B; q-- > 0;) xi = sgb_fma(-co[q], xk[q], xi);
            }
            xi = mine ? xi : 0.0f;
        };
        load(cd, warp * B);
        float inv = 0.0f;   // 1/U(i,i)
#pragma unroll
        for (uint32_t q = 0; q < B; ++q) inv = lane == q ? cd[q] : inv;
        float ct[B];        // the own block's triangle, zero elsewhere: a step is a shuffle and an FMA
#pragma unroll
        for (uint32_t q = 0; q < B; ++q) ct[q] = mine && lane > q ? cd[q] : 0.0f;   // (past the end cd is row 0's)
        sync_rows(threads);   // x is read
        for (uint32_t b = 0; b < blocks; ++b) {
            if (warp == b) {
#pragma unroll
                for (uint32_t q = 0; q + 1 < B; ++q) xi = sgb_fma(-ct[q], __shfl_sync(0xffffffffu, xi, q), xi);
                xi = mine ? xi : 0.0f;
                x[tid] = xi;
            } else if (warp > b) {
                load(co, b * B);
            }
            sync_rows(threads);
            if (warp > b) apply(b * B, true);
        }
#pragma unroll
        for (uint32_t q = 0; q < B; ++q) ct[q] = lane < q ? cd[q] : 0.0f;
        for (uint32_t b = blocks; b-- > 0;) {
            if (warp == b) {
#pragma unroll
                for (uint32_t q = B; q-- > 0;) xi = sgb_fma(-ct[q], __shfl_sync(0xffffffffu, xi * inv, q), xi);
                xi = mine ? xi * inv : 0.0f;   // nothing changed a row after its own column
                x[tid] = xi;
            } else if (warp < b) {
                load(co, b * B);
            }
            sync_rows(threads);
            if (warp < b) apply(b * B, false);
        }
    }

    // In 32-column blocks, for CTAs of fewer threads than rows, few species and attempts on the pattern
    // alone: a warp solves the diagonal block with shuffles, then every row outside it takes the block's
    // updates.
    template <class V>
    __device__ void solve_plain(V *x) {
        const uint32_t nb = (n + 31) / 32;
        for (uint32_t b = 0; b < nb; ++b) {
            const uint32_t kb = b * 32;
            const uint32_t kend = kb + 32 < n ? kb + 32 : n;
            if (warp == 0) {
                const uint32_t i = kb + lane;
                V xi = i < n ? x[i] : (V)0.0;
                const Cf *row = a + (size_t)(i < n ? i : 0) * ld;
                // this row's pattern bits for the block's columns, below the diagonal only
                const uint32_t w = i < n ? pat[i * 8u + b] & ((1u << lane) - 1u) : 0u;
                const uint32_t kn = kend - kb;   // columns in this block (32, or fewer in the last)
#pragma unroll 8
                for (uint32_t kk = 0; kk < kn; ++kk) {
                    const V xk = __shfl_sync(0xffffffffu, xi, kk);
                    if ((w >> kk) & 1u) xi = sgb_fma(-(V)row[kb + kk], xk, xi);
                }
                if (i < n) x[i] = xi;
            }
            sync();
            for (uint32_t i = kend + tid; i < n; i += NT) {
                const Cf *row = a + (size_t)i * ld;
                const uint32_t w = pat[i * 8u + b];
                V xi = x[i];
                for (uint32_t k = kb; k < kend; ++k)
                    if ((w >> (k - kb)) & 1u) xi = sgb_fma(-(V)row[k], x[k], xi);
                x[i] = xi;
            }
            sync();
        }
        for (uint32_t b = nb; b-- > 0;) {
            const uint32_t kb = b * 32;
            const uint32_t kend = kb + 32 < n ? kb + 32 : n;
            if (warp == 0) {
                const uint32_t i = kb + lane;
                V xi = i < n ? x[i] : (V)0.0;
                const Cf *row = a + (size_t)(i < n ? i : 0) * ld;
                // this row's pattern bits for the block's columns, above the diagonal only (columns < n)
                const uint32_t w = i < n ? pat[i * 8u + b] & ~((2u << lane) - 1u) : 0u;
                const V d = i < n ? (V)row[i] : (V)0.0;   // 1/U(i,i)
#pragma unroll 8
                for (uint32_t kk = kend - kb; kk-- > 0;) {
                    if (lane == kk) xi = xi * d;   // row kb+kk: all its updates are in
                    const V xk = __shfl_sync(0xffffffffu, xi, kk);
                    if ((w >> kk) & 1u) xi = sgb_fma(-(V)row[kb + kk], xk, xi);
                }
                if (i < n) x[i] = xi;
            }
            sync();
            for (uint32_t i = tid; i < kb; i += NT) {
                const Cf *row = a + (size_t)i * ld;
                const uint32_t w = pat[i * 8u + b];
                V xi = x[i];
                for (uint32_t k = kend; k-- > kb;)
                    if ((w >> (k - kb)) & 1u) xi = sgb_fma(-(V)row[k], x[k], xi);
                x[i] = xi;
            }
            sync();
        }
    }

    // Mixed: out = W^-1 rb by the FP32 LU, then `sweeps` FP64-residual refinement sweeps.
    __device__ void solve_refined(const DevArgs &A, double ghinv, double *out) {
        float *xs = x32;
        for (uint32_t s = tid; s < n; s += NT) xs[s] = (float)rb[s];
        sync();
        SGB_PHASE(3, solve(xs));
        for (uint32_t s = tid; s < n; s += NT) out[s] = (double)xs[s];
        sync();
        for (uint32_t sw = 0; sw < A.ir_sweeps; ++sw) {
            for (uint32_t i = tid; i < n; i += NT) {
                double w = ghinv * out[i];
                const uint32_t end = tb.jrow[i + 1];
#pragma unroll 8
                for (uint32_t e = tb.jrow[i]; e < end; ++e) w = sgb_fma(js[e], out[tb.jcol[e]], w);
                xs[i] = (float)(rb[i] - w);
            }
            sync();
            SGB_PHASE(3, solve(xs));
            for (uint32_t s = tid; s < n; s += NT) out[s] = out[s] + (double)xs[s];
            sync();
        }
    }

    // One pass of kin_integrate's step loop (kin_solver.h:216-311); true: nothing is decided, and it is to be
    // made again with on_pattern. The mixed path's panels and solves multiply by the zeros off the
    // pattern, which changes no finite value, but an element of the LU or of a solution past FP32's range
    // makes NaNs of them, which reach species that it has nothing to do with. Either leaves some
    // stage value that is not finite.
    __device__ bool attempt(const DevArgs &A) {
        const double h_min = A.ctl.h_min, rtol = A.ctl.rtol, atol = A.ctl.atol;
        const double inv_n = 1.0 / (double)n;
        double remaining = seg_end - t;
        double h_cap = remaining;
        if (A.ctl.h_max > 0.0) h_cap = vmin(h_cap, A.ctl.h_max);
        double h_wanted = vmax(h, h_min);
        bool last = h_wanted >= remaining;
        double hs = last ? remaining : vmin(h_wanted, h_cap);

        if (tid == 0) {   // the step's two divisions once, shared through red[2..3] (rhs synchronises)
            red[2] = 1.0 / (hs * M::gamma0(A));
            red[3] = 1.0 / hs;
        }
        SGB_PHASE(0, rhs(y));
        SGB_PHASE(1, neg_jac(y));
        const double ghinv = red[2];
        SGB_PHASE(2, factor((Cf)ghinv));
        const double hinv = red[3];

        bool fcn_at_y = true;
        const int S = M::stages(A);
        for (int st = 0; st < S; ++st) {
            const int packed = st * (st - 1) / 2;
            double *Ks = K + (size_t)st * n;
            if (st > 0 && M::new_f(A, st)) {
                bool moved = false;
                for (int j = 0; j < st; ++j)
                    if (M::a(A, packed + j) != 0.0) moved = true;
                if (moved || !fcn_at_y) {
                    for (uint32_t s = tid; s < n; s += NT) {
                        double v = y[s];
                        for (int j = 0; j < st; ++j) {
                            const double av = M::a(A, packed + j);
                            if (av == 0.0) continue;
                            v = sgb_fma(av, K[(size_t)j * n + s], v);
                        }
                        ytmp[s] = v;
                    }
                    sync();
                    SGB_PHASE(0, rhs(ytmp));
                    fcn_at_y = !moved;
                }
            }
            for (uint32_t s = tid; s < n; s += NT) {
                double v = fcn[s];
                for (int j = 0; j < st; ++j) {
                    const double c = M::c(A, packed + j);
                    if (c == 0.0) continue;
                    v = sgb_fma(c * hinv, K[(size_t)j * n + s], v);
                }
                if constexpr (kMixed) rb[s] = v;
                else Ks[s] = v;
            }
            sync();
            if constexpr (kMixed) {
                solve_refined(A, ghinv, Ks);
            } else {
                SGB_PHASE(3, solve(Ks));
            }
        }

        // y_new into ytmp and the weighted RMS error (kin_solver.h:263-280)
        bool finite = true;
        for (uint32_t s = tid; s < n; s += NT) {
            double ynew = y[s], yerr = 0.0;
            for (int st = 0; st < S; ++st) {
                if (kMixed) finite = finite && (__double2hiint(K[(size_t)st * n + s]) & 0x7ff00000) != 0x7ff00000;
                const double mc = M::m(A, st), ec = M::e(A, st);
                if (mc != 0.0) ynew = sgb_fma(mc, K[(size_t)st * n + s], ynew);
                if (ec != 0.0) yerr = sgb_fma(ec, K[(size_t)st * n + s], yerr);
            }
            const double scale = sgb_fma(rtol, vmax(vabs(y[s]), vabs(ynew)), atol);
            qv[s] = yerr / scale;
            ytmp[s] = ynew;
        }
        if constexpr (kMixed) {
            if (__syncthreads_or(!finite) && !on_pattern && NT >= n) return true;
        } else {
            sync();
        }
        if (tid == 0) {   // error norm and step factor once, shared through red[0..1]
            double e = 0.0;
#pragma unroll 8
            for (uint32_t s = 0; s < n; ++s) e = sgb_fma(qv[s], qv[s], e);
            e = vsqrt(e * inv_n);
            if (!is_finite_lane(e)) e = 1e10;
            red[0] = e;
            red[1] = step_factor(e, M::order(A));
        }
        sync();
        const double err = red[0];
        double fac = red[1];
        bool ok = err <= 1.0 || hs <= h_min;
        if (A.ctl.fixed_step) {
            ok = true;
            fac = 1.0;
        }
        if (ok) {
            for (uint32_t s = tid; s < n; s += NT) {
                double ynew = ytmp[s];
                if (A.ctl.clamp_negative) ynew = vmax(ynew, 0.0);
                y[s] = ynew;
            }
            t = last ? seg_end : t + hs;
        }
        double h_acc = hs * fac;
        h_acc = reject_last ? vmin(h_acc, hs) : h_acc;
        h_acc = (last && fac >= 1.0) ? vmax(h_acc, h_wanted) : h_acc;
        double h_rej = reject_more ? hs * 0.1 : vmin(hs * fac, hs);
        if (A.ctl.fixed_step) {
            h_acc = h_wanted;
            h_rej = h_wanted;
        }
        h = ok ? h_acc : h_rej;
        reject_more = !ok && reject_last;
        reject_last = !ok;
        steps = steps + (ok ? 1.0 : 0.0);
        rejects = rejects + (ok ? 0.0 : 1.0);
        if (!(t < seg_end && !(failed > 0.0))) phase = kPhaseSegFinish;
        sync();
        return false;
    }
};

template <int PREC>
__global__ void __launch_bounds__(512, 1) kin_coop_kernel(const __grid_constant__ DevArgs A, double *scratch, uint64_t stride) {
    extern __shared__ __align__(16) double sm[];
    __shared__ uint32_t cell_s;
    CoopCell<PREC> C;
    C.tb.init((const CoopMech *)A.tables, (const unsigned char *)A.tables);
    C.n = C.tb.h->n;
    C.R = C.tb.h->R;
    C.ld = C.tb.h->ld;
    C.nj = C.tb.h->nj;
    C.tid = threadIdx.x;
    C.NT = blockDim.x;
    C.lane = threadIdx.x & 31u;
    C.warp = threadIdx.x >> 5;
    C.W = blockDim.x >> 5;
    const uint32_t n = C.n;
    C.K = sm;   // 4 stage vectors; with the four vectors after them the elimination's panel buffers
    C.ytmp = C.K + 4 * n;
    C.qv = C.ytmp + n;
    C.rb = C.qv + n;
    C.xv = C.rb + n;
    C.rate = C.xv + n;   // the products of a Jacobian take everything up to here and the rates
    C.y = C.rate + C.R;
    C.fcn = C.y + n;
    C.src = C.fcn + n;
    C.kr = C.src + n;
    C.red = C.kr + C.R;
    C.x32 = (float *)(sm + coop_smem_doubles(n, C.R));
    uint32_t *pat_s = (uint32_t *)(C.x32 + kCoopMaxSpecies);
    uint16_t *lcnt_s = (uint16_t *)(pat_s + (size_t)n * 8);
    {   // stage the pattern once per CTA
        const uint32_t *pg = (const uint32_t *)((const unsigned char *)A.tables + C.tb.h->off_pat);
        const uint16_t *lg = (const uint16_t *)((const unsigned char *)A.tables + C.tb.h->off_lcnt);
        for (uint32_t q = threadIdx.x; q < n * 8; q += blockDim.x) pat_s[q] = pg[q];
        for (uint32_t q = threadIdx.x; q < n; q += blockDim.x) lcnt_s[q] = lg[q];
    }
    C.pat = pat_s;
    C.lcnt = lcnt_s;
    const CoopSmemLayout lay = coop_layout(PREC, *C.tb.h, A.coop_smem_budget);
    unsigned char *smb = (unsigned char *)sm;
    double *g = scratch + (size_t)blockIdx.x * stride;
    if constexpr (PREC == 2) {
        C.a = (typename CoopCell<PREC>::Cf *)(smb + lay.lu);
        C.js = g;
    } else {   // FP64: small LUs in shared memory, large ones in per-CTA global scratch (L2)
        C.a = lay.lu_bytes ? (typename CoopCell<PREC>::Cf *)(smb + lay.lu) : (typename CoopCell<PREC>::Cf *)g;
        C.js = nullptr;
    }
    C.prod = coop_products_fit(*C.tb.h) ? C.K : g + coop_scratch_base(PREC, *C.tb.h);
    C.lu_global = PREC == 0 && lay.lu_bytes == 0;
    if (lay.terms_bytes) {   // the RHS / Jacobian term lists, once per CTA
        const CoopMech *h = C.tb.h;
        const uint4 *src = (const uint4 *)((const unsigned char *)A.tables + h->off_reac);
        uint4 *dst = (uint4 *)(smb + lay.terms);
        for (uint32_t q = threadIdx.x; q < lay.terms_bytes / 16; q += blockDim.x) dst[q] = src[q];
        C.tb.init(h, smb + lay.terms - h->off_reac);   // image offset o lives at terms - off_reac + o
    }
    __syncthreads();
    for (;;) {
        if (threadIdx.x == 0) cell_s = atomicAdd(A.cursor, 1u);
        __syncthreads();
        const uint32_t idx = cell_s;
        __syncthreads();
        uint32_t cell = idx;
        if (PREC == 0 && A.resume) {   // cells parked by a lane kernel of this launch
            if (idx >= min(*(volatile uint32_t *)A.suspend_count, A.suspend_cap)) break;
            const SuspendRec r = A.suspend[idx];
            cell = r.cell;
            C.load(A, cell);
            C.restore(r);
        } else {
            if (idx >= A.lanes) break;
            C.load(A, cell);
        }
        while (C.settle(A, cell)) {
            const long long t_attempt = clock64();
            C.on_pattern = false;
            while (C.attempt(A)) C.on_pattern = true;
#ifdef SGB_COOP_PROFILE
            if (threadIdx.x == 0) atomicAdd(&g_coop_phase_cycles[5], (unsigned long long)(clock64() - t_attempt));
#else
            (void)t_attempt;
#endif
        }
        C.store(A, cell);
    }
}

// Module state of the cooperative path.
struct CoopModule {
    bool ready = false;
    std::vector<uint8_t> image;
    CoopMech head;
    void *d_image = nullptr;
    uint32_t *d_header = nullptr;   // cursor (+0), error flag (+32 words)
    double *d_scratch = nullptr;
    size_t scratch_bytes = 0;
    KinMethod method;
    KinControl control;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    uint32_t ir_sweeps = 1;
    float last_ms = 0.0f;
    uint32_t block[3] = {256, 0, 512};    // threads per CTA by precision (0 FP64, 2 mixed)
    uint32_t ctas[3] = {2, 0, 1};         // resident CTAs per SM by precision
    uint32_t smem_budget[3] = {kCoopSmemBudget, 0, kCoopSmemBudget};
    int sms = 0;
};
CoopModule cm;
constexpr uint32_t kCoopMaxCtasPerSm = 2;   // scratch slots per SM

// Dynamic shared memory of a launch (the L1 / shared split is left to the driver: preferring L1
// measured no faster for the global-memory FP64 LU at one CTA per SM, and cost occupancy at two).
cudaError_t set_coop_attributes(void (*fn)(DevArgs, double *, uint64_t), int prec, const CoopMech &h, uint32_t budget) {
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)coop_layout(prec, h, budget).total);
}

size_t coop_smem_bytes(int prec, const CoopMech &h, uint32_t budget = kCoopSmemBudget) {
    return coop_layout(prec, h, budget).total;
}

size_t coop_scratch_doubles(int prec, const CoopMech &h) {
    const size_t d = coop_scratch_base(prec, h) + (coop_products_fit(h) ? 0u : h.pairs);
    return (d + 31) / 32 * 32;   // 256-byte aligned per CTA
}

}   // namespace

size_t coop_smem_bytes_for(int prec, const CoopMech &h) { return coop_smem_bytes(prec, h); }
size_t coop_scratch_doubles_for(int prec, const CoopMech &h) { return coop_scratch_doubles(prec, h); }

// The cooperative kernel on `A` (A.tables the coop image, A.cursor zeroed):
// lanes [0, A.lanes), or with A.resume (FP64) the cells a lane kernel parked;
// `scratch` holds grid slots of coop_scratch_doubles_for(prec) doubles.
cudaError_t coop_launch(int prec, const DevArgs &A0, const CoopMech &head, double *scratch, uint32_t grid,
                               uint32_t block, cudaStream_t s) {
    void (*fn)(DevArgs, double *, uint64_t) = prec == 0 ? kin_coop_kernel<0> : kin_coop_kernel<2>;
    DevArgs A = A0;
    if (!A.coop_smem_budget) A.coop_smem_budget = kCoopSmemBudget;
    const size_t smem = coop_smem_bytes(prec, head, A.coop_smem_budget);
    cudaError_t ce = set_coop_attributes(fn, prec, head, A.coop_smem_budget);
    if (ce != cudaSuccess) return ce;
    fn<<<grid, block, smem, s>>>(A, scratch, coop_scratch_doubles(prec, head));
    return cudaGetLastError();
}

}   // namespace sgb

using namespace sgb;

namespace sgb {
const Model *model_of(const KinModelHandle *h);
}

SGB_API int32_t gpu_kin_coop_set_mech(const KinModelHandle *model, const KinMethod *method, const KinControl *control) {
    if (!model || !method || !control || method->stages < 2 || method->stages > 4) return (int32_t)cudaErrorInvalidValue;
    const Model *m = model_of(model);
    if (!m || !m->finalized || m->n() > kCoopMaxSpecies) return (int32_t)cudaErrorInvalidValue;
    std::vector<uint8_t> img;
    if (!coop_image(*m, &img)) return (int32_t)cudaErrorInvalidValue;
    CoopMech h;
    memcpy(&h, img.data(), sizeof(h));
    int dev = 0, sms = 0, max_smem = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return (int32_t)e;
    if (coop_smem_bytes(0, h) > (size_t)max_smem) return (int32_t)cudaErrorInvalidValue;
    if (cm.d_image) cudaFree(cm.d_image);
    cm.d_image = nullptr;
    if (!cm.d_header) {
        e = cudaMalloc((void **)&cm.d_header, 256);
        if (e != cudaSuccess) return (int32_t)e;
    }
    e = cudaMalloc(&cm.d_image, img.size());
    if (e == cudaSuccess) e = cudaMemcpy(cm.d_image, img.data(), img.size(), cudaMemcpyHostToDevice);
    // scratch for the larger of the two precisions' needs, one slot per resident CTA (one CTA per SM)
    const size_t per = coop_scratch_doubles(0, h) > coop_scratch_doubles(2, h) ? coop_scratch_doubles(0, h)
                                                                              : coop_scratch_doubles(2, h);
    const size_t need = per * 8 * (size_t)sms * kCoopMaxCtasPerSm;
    if (e == cudaSuccess && need > cm.scratch_bytes) {
        if (cm.d_scratch) cudaFree(cm.d_scratch);
        cm.d_scratch = nullptr;
        cm.scratch_bytes = 0;
        e = cudaMalloc((void **)&cm.d_scratch, need);
        if (e == cudaSuccess) cm.scratch_bytes = need;
    }
    if (e == cudaSuccess && !cm.ev0) e = cudaEventCreate(&cm.ev0);
    if (e == cudaSuccess && !cm.ev1) e = cudaEventCreate(&cm.ev1);
    if (e != cudaSuccess) return (int32_t)e;
    cm.image.swap(img);
    cm.head = h;
    cm.sms = sms;
    cm.method = *method;
    cm.control = *control;
    cm.ready = true;
    return 0;
}

SGB_API int32_t gpu_kin_coop_advance(const GpuKinLaunch *L, float *kernel_ms) {
    if (!cm.ready || !L) return (int32_t)cudaErrorInvalidValue;
    if ((L->precision != 0 && L->precision != 2) || L->padded == 0 || L->lane_count > L->padded)
        return (int32_t)cudaErrorInvalidValue;
    if (!(L->duration >= 0.0) || L->duration > 1.0e300) return (int32_t)cudaErrorInvalidValue;
    if (!L->y || !L->h || !L->steps || !L->rejects || !L->pulses || !L->failed || !L->k || !L->src || !L->pulse ||
        !L->period || !L->pulse_first || !L->pulse_count)
        return (int32_t)cudaErrorInvalidValue;
    const int prec = (int)L->precision;
    int max_smem = 0;
    if (cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, 0) != cudaSuccess ||
        coop_smem_bytes(prec, cm.head, cm.smem_budget[prec]) > (size_t)max_smem)
        return (int32_t)cudaErrorInvalidValue;   // the mixed path's FP32 LU must fit one CTA's shared memory
    DevArgs A;
    memset(&A, 0, sizeof(A));
    A.y = L->y; A.h = L->h; A.steps = L->steps; A.rejects = L->rejects; A.pulses = L->pulses; A.failed = L->failed;
    A.k = L->k; A.src = L->src; A.pulse = L->pulse; A.period = L->period;
    A.pulse_first = L->pulse_first; A.pulse_count = L->pulse_count;
    A.padded = L->padded;
    A.lanes = L->lane_count ? L->lane_count : L->padded;
    A.duration = L->duration;
    A.ctl = cm.control;
    memcpy(A.ma, cm.method.a, sizeof(A.ma));
    memcpy(A.mc, cm.method.c, sizeof(A.mc));
    memcpy(A.mm, cm.method.m, sizeof(A.mm));
    memcpy(A.me, cm.method.e, sizeof(A.me));
    A.gamma0 = cm.method.gamma0;
    memcpy(A.new_f, cm.method.new_f, sizeof(A.new_f));
    A.stages = cm.method.stages;
    A.order = cm.method.order;
    A.ir_sweeps = cm.ir_sweeps;
    A.cursor = cm.d_header;
    A.error_flag = cm.d_header + 32;
    A.wait_polls = kSpinLimit;
    A.tables = cm.d_image;
    A.table_bytes = cm.head.bytes;
    if (A.lanes == 0 || A.duration == 0.0) {
        if (kernel_ms) *kernel_ms = 0.0f;
        return 0;
    }
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return (int32_t)e;
    void (*fn)(DevArgs, double *, uint64_t) = prec == 0 ? kin_coop_kernel<0> : kin_coop_kernel<2>;
    A.coop_smem_budget = cm.smem_budget[prec];
    const size_t smem = coop_smem_bytes(prec, cm.head, A.coop_smem_budget);
    e = set_coop_attributes(fn, prec, cm.head, A.coop_smem_budget);
    if (e != cudaSuccess) return (int32_t)e;
    int fit = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, fn, (int)cm.block[prec], smem);
    if (e != cudaSuccess) return (int32_t)e;
    const uint32_t per_sm = (uint32_t)(fit < 1 ? 1 : fit) < cm.ctas[prec] ? (uint32_t)(fit < 1 ? 1 : fit) : cm.ctas[prec];
    const uint32_t resident = per_sm * (uint32_t)sms;
    const uint32_t grid = resident < A.lanes ? resident : A.lanes;
    const uint64_t stride = coop_scratch_doubles(prec, cm.head);
    cudaStream_t s = (cudaStream_t)gpu_stream();
    e = cudaMemsetAsync(cm.d_header, 0, 256, s);
    if (e == cudaSuccess) e = cudaEventRecord(cm.ev0, s);
    if (e != cudaSuccess) return (int32_t)e;
    fn<<<grid, cm.block[prec], smem, s>>>(A, cm.d_scratch, stride);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaEventRecord(cm.ev1, s);
    if (e == cudaSuccess) e = cudaEventSynchronize(cm.ev1);
    if (e != cudaSuccess) return (int32_t)e;
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, cm.ev0, cm.ev1);
    cm.last_ms = ms;
    if (kernel_ms) *kernel_ms = ms;
    return 0;
}

// Counts of the cooperative path's mechanism image: n, R, nnz, Jacobian
// entries, L entries, U entries, LU updates, image bytes.
SGB_API int32_t gpu_kin_coop_info(uint64_t *out8) {
    if (!cm.ready || !out8) return (int32_t)cudaErrorInvalidValue;
    const CoopMech &h = cm.head;
    out8[0] = h.n; out8[1] = h.R; out8[2] = h.nnz; out8[3] = h.nj;
    out8[4] = h.l_entries; out8[5] = h.u_entries; out8[6] = h.lu_updates; out8[7] = h.bytes;
    return 0;
}

// Phase cycle counters of a -DSGB_COOP_PROFILE build (zeros otherwise); reading resets them.
SGB_API int32_t gpu_kin_coop_phase_cycles(uint64_t *out6) {
    if (!out6) return (int32_t)cudaErrorInvalidValue;
    memset(out6, 0, 6 * sizeof(uint64_t));
#ifdef SGB_COOP_PROFILE
    unsigned long long v[8];
    cudaError_t e = cudaMemcpyFromSymbol(v, g_coop_phase_cycles, sizeof(v));
    if (e != cudaSuccess) return (int32_t)e;
    for (int i = 0; i < 6; ++i) out6[i] = v[i];
    memset(v, 0, sizeof(v));
    e = cudaMemcpyToSymbol(g_coop_phase_cycles, v, sizeof(v));
    if (e != cudaSuccess) return (int32_t)e;
#endif
    return 0;
}

SGB_API int32_t gpu_kin_coop_set_smem_budget(uint32_t precision, uint32_t bytes) {
    if ((precision != 0 && precision != 2) || bytes > 227 * 1024) return (int32_t)cudaErrorInvalidValue;
    cm.smem_budget[precision] = bytes;
    return 0;
}

SGB_API int32_t gpu_kin_coop_set_shape(uint32_t precision, uint32_t block, uint32_t ctas_per_sm) {
    if ((precision != 0 && precision != 2) || block < 64 || block > 512 || (block & 31) || ctas_per_sm < 1 ||
        ctas_per_sm > kCoopMaxCtasPerSm)
        return (int32_t)cudaErrorInvalidValue;
    cm.block[precision] = block;
    cm.ctas[precision] = ctas_per_sm;
    return 0;
}

SGB_API int32_t gpu_kin_coop_set_refinement(uint32_t sweeps) {
    if (sweeps > 4) return (int32_t)cudaErrorInvalidValue;
    cm.ir_sweeps = sweeps;
    return 0;
}
