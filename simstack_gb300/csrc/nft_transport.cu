// The NFT film transport of one coupling window on the device (src/sim/nft.cpp:1028-1106,
// nft_transport): per channel (lane) and substep, flux-form upwind advection of the nine
// film fields in f32 deltas from the inlet, the linearised wall / radiant / latent heat
// update, O2 exchange toward saturation, and the plant sites' uptake booked as what was
// actually removed; then the window's outlet sums and film evaporation.
//
// Data: device copies of the reference's group arrays in the reference's byte layout
// (nft.cpp:134-203: groups of 8 channels, every per-cell quantity a [8] f32 lane array),
// packed group after group. Within a substep the reference sweeps outlet -> inlet so
// that every cell reads its upstream neighbour's value from before the substep; the cells
// of a substep are therefore independent, and each thread sweeps its own run of cells the
// same way (outlet end first). The one value a run needs from outside is the old state of
// the previous run's last cell.
//
// Two kernels. nft_resident_kernel (channels of up to 2,304 cells) holds a channel in the
// registers of a warp, or of several: each lane keeps a run of kRun cells (nine fields and
// four coefficients each) for the whole window and takes its upstream value by shuffle, so
// a substep touches no memory but the plant sites' shared-memory slots and needs no barrier
// while one warp holds the channel. It is bound by its own instruction issue (~30 per cell
// and ~56 per site and substep). nft_transport_kernel keeps the state in global memory (L1)
// and one CTA per group, the boundary values in shared memory with one barrier per substep:
// longer channels, windows of few substeps (resident_pays), and runs whose site slots do not fit. 512 channels x 240 cells x 253
// substeps: 990 us through memory (3.9 us per substep: load latency and the barrier), 184 us
// resident (0.73 us).
//
// Every element receives the reference's f32 operations in the reference's order, issued
// as explicit PTX (no contraction, no reassociation). The reference runs the transport
// with x86 FTZ/DAZ set (NftFlushDenormals, nft.cpp:1130-1136) on x86-64 hosts and IEEE
// elsewhere; flush_denormals selects the matching PTX forms (.ftz or not), so the result
// is bit-identical to the reference on either kind of host. Bounded: no waits; every
// loop has a fixed trip count.

#include <cuda_runtime.h>

#include "../../include/simstack_gpu.h"

namespace sgb {
cudaError_t module_mark_start();
cudaError_t module_finish(float *device_ms);
cudaStream_t module_stream();
}   // namespace sgb

using namespace sgb;

namespace {

constexpr uint32_t kLanes = 8;
constexpr uint32_t kFields = 9;
// group-array strides and field offsets, in floats (nft.cpp:134-178)
constexpr uint32_t kRow = kFields * kLanes;   // NftRow: f[9][8]
constexpr uint32_t kHot = 4 * kLanes;         // NftCellHot: c, kT, bT, ko
constexpr uint32_t kHotC = 0, kHotKT = 8, kHotBT = 16, kHotKO = 24;
constexpr uint32_t kCold = 80;                // NftCellCold: vol_L f64[8] (16 floats), inv_v, kw, kr, ge, ev, depth, phi, vel
constexpr uint32_t kColdKW = 24, kColdKR = 32, kColdGE = 40, kColdEV = 48;
constexpr uint32_t kSite = 288;               // NftSiteRow, 1,152 B
constexpr uint32_t kSiteDrop = 16, kSiteRemoved = 216;
constexpr uint32_t kFieldT = 0, kFieldDO = 1;
constexpr uint32_t kMaxRuns = 128;            // runs per channel: 8 x 128 = 1,024 threads

// f32 arithmetic with an explicit denormal mode: kFtz = the reference's x86 mode.
template <bool kFtz>
struct F32 {
    static __device__ __forceinline__ float add(float a, float b) {
        float r;
        if constexpr (kFtz) asm("add.rn.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
        else asm("add.rn.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
        return r;
    }
    static __device__ __forceinline__ float sub(float a, float b) {
        float r;
        if constexpr (kFtz) asm("sub.rn.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
        else asm("sub.rn.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
        return r;
    }
    static __device__ __forceinline__ float mul(float a, float b) {
        float r;
        if constexpr (kFtz) asm("mul.rn.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
        else asm("mul.rn.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
        return r;
    }
    // a * b + c, one rounding (lane_fmadd)
    static __device__ __forceinline__ float fma(float a, float b, float c) {
        float r;
        if constexpr (kFtz) asm("fma.rn.ftz.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
        else asm("fma.rn.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
        return r;
    }
    // c - a * b, one rounding (lane_fnmadd: the product's sign flipped, then fused)
    static __device__ __forceinline__ float fnma(float a, float b, float c) { return fma(-a, b, c); }
    // lane_max for f32: a > b ? a : b (the comparison sees the denormal mode)
    static __device__ __forceinline__ float max(float a, float b) {
        uint32_t gt;
        if constexpr (kFtz) asm("{ .reg .pred p; setp.gt.ftz.f32 p, %1, %2; selp.u32 %0, 1, 0, p; }" : "=r"(gt) : "f"(a), "f"(b));
        else asm("{ .reg .pred p; setp.gt.f32 p, %1, %2; selp.u32 %0, 1, 0, p; }" : "=r"(gt) : "f"(a), "f"(b));
        return gt ? a : b;
    }
};

// O2 saturation in fresh water at 1 atm, mg/L (nft.cpp:491-497): the f64 coefficients
// rounded to f32, Horner with fused steps.
template <bool kFtz>
__device__ __forceinline__ float do_sat(float T) {
    using F = F32<kFtz>;
    return F::fma(F::fma(F::fma((float)-0.000077774, T, (float)0.007991), T, (float)-0.41022), T, (float)14.652);
}

// The plant site on cell j, as the reference's sweep finds it: it counts sites down from
// the last site row (site_offset + (sites - 1) * stride) and only matches a row equal to
// the next one, so when that last row lies beyond the channel no site is ever applied.
__device__ __forceinline__ int site_on(uint32_t j, const GpuNftTransport &t) {
    if (t.sites_count == 0) return -1;
    const uint32_t last = t.site_offset + (t.sites_count - 1) * t.site_stride;
    if (last >= t.cells) return -1;
    if (t.site_stride == 0) return j == t.site_offset ? (int)t.sites_count - 1 : -1;
    if (j < t.site_offset || (j - t.site_offset) % t.site_stride) return -1;
    const uint32_t s = (j - t.site_offset) / t.site_stride;
    return s < t.sites_count ? (int)s : -1;
}

template <bool kFtz>
__global__ void __launch_bounds__(1024) nft_transport_kernel(const __grid_constant__ GpuNftTransport t, uint32_t run_len) {
    using F = F32<kFtz>;
    extern __shared__ float boundary[];   // [2][runs][9][8]: the old state of each run's last cell
    const uint32_t g = blockIdx.x;
    const uint32_t l = threadIdx.x & (kLanes - 1), q = threadIdx.x / kLanes;
    const uint32_t runs = blockDim.x / kLanes;
    const uint32_t cells = t.cells;
    const uint32_t j0 = q * run_len;
    const uint32_t j1 = min(cells, j0 + run_len);
    float *rows = t.rows + (size_t)g * cells * kRow + l;
    float *hot = t.hot + (size_t)g * cells * kHot + l;
    const float *cold = t.cold + (size_t)g * cells * kCold + l;
    float *sites = t.sites + (size_t)g * t.sites_count * kSite + l;

    // this window's heat coefficients, linear in the cell temperature delta (nft.cpp:1036-1047)
    const float tamb_rel = F::sub(t.T_amb, t.ref[kFieldT]);
    for (uint32_t j = j0; j < j1; ++j) {
        const float kw = cold[(size_t)j * kCold + kColdKW];
        const float ge = cold[(size_t)j * kCold + kColdGE];
        const float kr = cold[(size_t)j * kCold + kColdKR];
        hot[(size_t)j * kHot + kHotKT] = F::fma(ge, t.es_slope, kw);
        hot[(size_t)j * kHot + kHotBT] = F::fnma(ge, t.e0, F::fma(kw, tamb_rel, F::mul(kr, t.radiant)));
    }
    float floor_[kFields];
    for (uint32_t k = 0; k < kFields; ++k) floor_[k] = -t.ref[k];
    const float refT = t.ref[kFieldT], refDO = t.ref[kFieldDO];
    float out[kFields];
    for (uint32_t k = 0; k < kFields; ++k) out[k] = 0.0f;
    const bool owns_last = j0 < j1 && j1 == cells;

    for (uint32_t s = 0; s < t.substeps; ++s) {
        float *pub = boundary + ((s & 1) * runs + q) * kRow + l;
        float v[kFields];
        if (j0 < j1) {
            const float *last = rows + (size_t)(j1 - 1) * kRow;
            for (uint32_t k = 0; k < kFields; ++k) {
                v[k] = last[k * kLanes];
                pub[k * kLanes] = v[k];
            }
            if (owns_last)
                for (uint32_t k = 0; k < kFields; ++k) out[k] = F::add(out[k], v[k]);
        }
        __syncthreads();
        const float *upstream_run = boundary + ((s & 1) * runs + (q ? q - 1 : 0)) * kRow + l;
        for (uint32_t j = j1; j-- > j0;) {
            float *row = rows + (size_t)j * kRow;
            const float *h = hot + (size_t)j * kHot;
            const float c = h[kHotC];
            float x[kFields], up[kFields];
            if (j > 0) {
                if (j > j0) {
                    const float *u = row - kRow;
                    for (uint32_t k = 0; k < kFields; ++k) up[k] = u[k * kLanes];
                } else {
                    for (uint32_t k = 0; k < kFields; ++k) up[k] = upstream_run[k * kLanes];
                }
                for (uint32_t k = 0; k < kFields; ++k) x[k] = F::fma(c, F::sub(up[k], v[k]), v[k]);
            } else {
                for (uint32_t k = 0; k < kFields; ++k) x[k] = F::fnma(c, v[k], v[k]);   // inflow delta is 0
            }
            // heat: walls, radiant load, evaporative cooling of the open surface
            x[kFieldT] = F::add(F::fnma(h[kHotKT], x[kFieldT], x[kFieldT]), h[kHotBT]);
            // O2 exchange with the gully air (saturation at the absolute temperature)
            x[kFieldDO] = F::fma(h[kHotKO], F::sub(do_sat<kFtz>(F::add(refT, x[kFieldT])), F::add(refDO, x[kFieldDO])),
                                 x[kFieldDO]);
            // plant site: uptake and root respiration, booked as what was actually removed
            const int site = site_on(j, t);
            if (site >= 0) {
                float *sr = sites + (size_t)site * kSite;
                for (uint32_t k = 1; k < kFields; ++k) {
                    const float before = x[k];
                    x[k] = F::max(F::sub(x[k], sr[kSiteDrop + k * kLanes]), floor_[k]);
                    sr[kSiteRemoved + k * kLanes] = F::add(sr[kSiteRemoved + k * kLanes], F::sub(before, x[k]));
                }
            }
            for (uint32_t k = 0; k < kFields; ++k) row[k * kLanes] = x[k];
            if (j > j0)
                for (uint32_t k = 0; k < kFields; ++k) v[k] = up[k];
        }
    }
    if (owns_last)
        for (uint32_t k = 0; k < kFields; ++k) t.out_sum[(size_t)g * kRow + k * kLanes + l] = out[k];
    __syncthreads();
    // water evaporated from the film this window, summed inlet -> outlet (nft.cpp:1101-1105)
    if (q == 0) {
        float evap = 0.0f;
        for (uint32_t j = 0; j < cells; ++j)
            evap = F::fma(cold[(size_t)j * kCold + kColdEV], F::fma(t.es_slope, rows[(size_t)j * kRow + kFieldT * kLanes], t.e0), evap);
        t.evap_kg[(size_t)g * kLanes + l] = F::mul(evap, (float)t.substeps);
    }
}

// A channel in registers: kWpc = blockDim / 32 / (channels per CTA) warps hold one channel, lane i of
// warp p the slots (32 p + i) kRun .. + kRun; the channel's cells fill the LAST slots, so its outlet is
// always the last lane's last slot and the unused slots stay zero, as the inflow delta is (the
// reference's inlet update is the general one with an upstream of 0, bit for bit). Slots of one
// warp's neighbour come through shared memory (double-buffered by substep parity, one barrier).
// site_slots: sites at most in a lane's run; shared memory: [site_slots][16][threads] drop and
// removed, then [2][warps][9] boundary values and the evaporation carry.
constexpr int kMaxRun = 9;
constexpr uint32_t kMaxResidentWarps = 8;      // 255 registers a thread

template <bool kFtz, int kRun>
__global__ void __launch_bounds__(256) nft_resident_kernel(const __grid_constant__ GpuNftTransport t, uint32_t wpc,
                                                           uint32_t site_slots) {
    using F = F32<kFtz>;
    extern __shared__ float sm[];
    const uint32_t threads = blockDim.x, warps = threads / 32, warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const uint32_t part = warp % wpc, channel = blockIdx.x * (warps / wpc) + warp / wpc;
    const bool live = channel < t.groups * kLanes;   // whole warps
    const uint32_t g = live ? channel / kLanes : 0u, l = channel % kLanes;
    const uint32_t cells = t.cells, pad = wpc * 32 * kRun - cells;
    const uint32_t slot0 = (part * 32 + lane) * kRun;
    float *rows = t.rows + (size_t)g * cells * kRow + l;
    float *hot = t.hot + (size_t)g * cells * kHot + l;
    const float *cold = t.cold + (size_t)g * cells * kCold + l;
    float *sites = t.sites + (size_t)g * t.sites_count * kSite + l;
    float *site_sm = sm + threadIdx.x;
    float *edge = sm + (size_t)site_slots * 16 * threads;   // [2][warps][9]
    float *carry = edge + 2 * warps * kFields;              // [warps]

    float v[kRun][kFields], c[kRun], kT[kRun], bT[kRun], ko[kRun];
    uint32_t valid = 0, on = 0;   // slots that hold a cell; cells with a plant site
    const float tamb_rel = F::sub(t.T_amb, t.ref[kFieldT]);
#pragma unroll
    for (int j = 0; j < kRun; ++j) {
        c[j] = kT[j] = bT[j] = ko[j] = 0.0f;
#pragma unroll
        for (uint32_t k = 0; k < kFields; ++k) v[j][k] = 0.0f;
        if (!live || slot0 + j < pad) continue;
        const uint32_t cell = slot0 + j - pad;
        valid |= 1u << j;
        // this window's heat coefficients, linear in the cell temperature delta (nft.cpp:1036-1047)
        const float *cd = cold + (size_t)cell * kCold;
        float *h = hot + (size_t)cell * kHot;
        const float kw = cd[kColdKW], ge = cd[kColdGE], kr = cd[kColdKR];
        kT[j] = F::fma(ge, t.es_slope, kw);
        bT[j] = F::fnma(ge, t.e0, F::fma(kw, tamb_rel, F::mul(kr, t.radiant)));
        h[kHotKT] = kT[j];
        h[kHotBT] = bT[j];
        c[j] = h[kHotC];
        ko[j] = h[kHotKO];
#pragma unroll
        for (uint32_t k = 0; k < kFields; ++k) v[j][k] = rows[(size_t)cell * kRow + k * kLanes];
        const int site = site_on(cell, t);
        if (site >= 0) {
            const uint32_t at = __popc(on);
            on |= 1u << j;
            const float *sr = sites + (size_t)site * kSite;
#pragma unroll
            for (uint32_t k = 1; k < kFields; ++k) {
                site_sm[(at * 16 + k - 1) * threads] = sr[kSiteDrop + k * kLanes];
                site_sm[(at * 16 + 7 + k) * threads] = sr[kSiteRemoved + k * kLanes];
            }
        }
    }
    const uint32_t any = __reduce_or_sync(0xffffffffu, on);   // slots where some lane has a site
    const float refT = t.ref[kFieldT], refDO = t.ref[kFieldDO];
    float out[kFields];
#pragma unroll
    for (uint32_t k = 0; k < kFields; ++k) out[k] = 0.0f;

    for (uint32_t s = 0; s < t.substeps; ++s) {
        float in[kFields];   // the old state upstream of slot 0
#pragma unroll
        for (uint32_t k = 0; k < kFields; ++k) {
            out[k] = F::add(out[k], v[kRun - 1][k]);   // kept by the outlet's lane
            in[k] = __shfl_up_sync(0xffffffffu, v[kRun - 1][k], 1);
        }
        if (wpc > 1) {
            float *e = edge + (s & 1) * warps * kFields;
            if (lane == 31)
#pragma unroll
                for (uint32_t k = 0; k < kFields; ++k) e[warp * kFields + k] = v[kRun - 1][k];
            __syncthreads();
            if (lane == 0)
#pragma unroll
                for (uint32_t k = 0; k < kFields; ++k) in[k] = part ? e[(warp - 1) * kFields + k] : 0.0f;
        } else if (lane == 0) {
#pragma unroll
            for (uint32_t k = 0; k < kFields; ++k) in[k] = 0.0f;
        }
#pragma unroll
        for (int j = kRun - 1; j >= 0; --j) {
            float x[kFields];
#pragma unroll
            for (uint32_t k = 0; k < kFields; ++k) {
                const float up = j ? v[j ? j - 1 : 0][k] : in[k];
                x[k] = F::fma(c[j], F::sub(up, v[j][k]), v[j][k]);
            }
            // heat: walls, radiant load, evaporative cooling of the open surface
            x[kFieldT] = F::add(F::fnma(kT[j], x[kFieldT], x[kFieldT]), bT[j]);
            // O2 exchange with the gully air (saturation at the absolute temperature)
            x[kFieldDO] = F::fma(ko[j], F::sub(do_sat<kFtz>(F::add(refT, x[kFieldT])), F::add(refDO, x[kFieldDO])), x[kFieldDO]);
            // plant site: uptake and root respiration, booked as what was actually removed
            if ((any >> j) & 1u) {   // the same for the whole warp
                if ((on >> j) & 1u) {
                    float *sr = site_sm + __popc(on & ((1u << j) - 1u)) * 16 * threads;
                    float drop[kFields], removed[kFields];   // all loads ahead of the stores
#pragma unroll
                    for (uint32_t k = 1; k < kFields; ++k) {
                        drop[k] = sr[(k - 1) * threads];
                        removed[k] = sr[(7 + k) * threads];
                    }
#pragma unroll
                    for (uint32_t k = 1; k < kFields; ++k) {
                        const float before = x[k];
                        x[k] = F::max(F::sub(x[k], drop[k]), -t.ref[k]);
                        sr[(7 + k) * threads] = F::add(removed[k], F::sub(before, x[k]));
                    }
                }
            }
            const bool cell = (valid >> j) & 1u;   // a slot without a cell keeps its zeros whatever the air is
            x[kFieldT] = cell ? x[kFieldT] : 0.0f;
            x[kFieldDO] = cell ? x[kFieldDO] : 0.0f;
#pragma unroll
            for (uint32_t k = 0; k < kFields; ++k) v[j][k] = x[k];
        }
    }
    float ev[kRun], e[kRun];
#pragma unroll
    for (int j = 0; j < kRun; ++j) {
        ev[j] = e[j] = 0.0f;
        if (!((valid >> j) & 1u)) continue;
        const uint32_t cell = slot0 + j - pad;
#pragma unroll
        for (uint32_t k = 0; k < kFields; ++k) rows[(size_t)cell * kRow + k * kLanes] = v[j][k];
        ev[j] = cold[(size_t)cell * kCold + kColdEV];
        e[j] = F::fma(t.es_slope, v[j][kFieldT], t.e0);
        if ((on >> j) & 1u) {
            float *sr = sites + (size_t)site_on(cell, t) * kSite;
            const float *from = site_sm + __popc(on & ((1u << j) - 1u)) * 16 * threads;
#pragma unroll
            for (uint32_t k = 1; k < kFields; ++k) sr[kSiteRemoved + k * kLanes] = from[(7 + k) * threads];
        }
    }
    const bool outlet = live && part + 1 == wpc && lane == 31;
    if (outlet)
#pragma unroll
        for (uint32_t k = 0; k < kFields; ++k) t.out_sum[(size_t)g * kRow + k * kLanes + l] = out[k];
    // water evaporated from the film this window, summed inlet -> outlet (nft.cpp:1101-1105): lane by
    // lane, warp by warp
    float evap = 0.0f;
    for (uint32_t p = 0; p < wpc; ++p) {
        if (part == p) {
            if (p) evap = carry[warp - 1];
            for (int i = 0; i < 32; ++i) {
                if ((int)lane == i)
#pragma unroll
                    for (int j = 0; j < kRun; ++j)
                        if ((valid >> j) & 1u) evap = F::fma(ev[j], e[j], evap);
                evap = __shfl_sync(0xffffffffu, evap, i);
            }
            if (lane == 0) carry[warp] = evap;
        }
        if (wpc > 1) __syncthreads();
    }
    if (outlet) t.evap_kg[(size_t)g * kLanes + l] = F::mul(evap, (float)t.substeps);
}

// Runs per channel and cells per run of nft_transport_kernel: as many runs as a 1,024-thread CTA
// holds, then runs of equal length (the last may be shorter).
void launch_shape(uint32_t cells, uint32_t *runs, uint32_t *run_len) {
    const uint32_t len = (cells + kMaxRuns - 1) / kMaxRuns;
    *run_len = len;
    *runs = (cells + len - 1) / len;
}

// Shape of nft_resident_kernel: cells per lane, warps per channel, channels per CTA, site slots per lane.
struct Resident {
    uint32_t run, wpc, channels, slots;
    size_t smem;
};
// The run with the least estimated time per substep: instructions of a warp (30 per slot, 64 per slot
// that has a site in some lane -- one per stride where the stride divides the run, so that every
// lane has its sites at the same slots, else every slot -- and the exchange) times 2.5 + 1.75 x
// (warps per scheduler) cycles, times the waves. Fitted to 240 cells, sites every 3, 253 substeps, us at runs of
// 2 / 3 / 6 / 9: one group 103 / 101 / 181 / 228, 64 groups 242 / 184 / 237 / 241, with the registers that the
// kernels then took (kRegs; sm_103a, nvcc 13.0, takes 116 115 101 128 255 250 213 243 now, and the choice is as good with
// either). Over 280 shapes of 24 to 1,500 cells, strides 0, 1, 3, 4 and 7 and 1 to 400 groups its run takes 1.05 times the
// best run's time on average; 47 of them lie past 1.12 (a run of 2 at a stride of 4, which has its sites in one slot
// and not in both: 1.2 to 1.4), the worst at 1.73 (400 cells without sites, 100 groups).
// False: the channel or its site slots do not fit.
bool resident_shape(const GpuNftTransport &t, uint32_t sms, Resident *best) {
    constexpr uint32_t kRegs[kMaxRun + 1] = {0, 0, 64, 107, 94, 109, 128, 229, 255, 255};
    const uint32_t stride = t.sites_count > 1 ? t.site_stride : 0u;
    double least = 0.0;
    best->run = 0;
    for (uint32_t run = 2; run <= (uint32_t)kMaxRun; ++run) {
        Resident r;
        r.run = run;
        r.wpc = (t.cells + 32 * run - 1) / (32 * run);
        if (r.wpc > kMaxResidentWarps) continue;
        r.channels = r.wpc >= 4 ? 1u : 4u / r.wpc;
        const uint32_t warps = r.wpc * r.channels;
        r.slots = t.sites_count == 0 ? 0u : stride == 0 ? 1u : (run + stride - 1) / stride;
        r.smem = ((size_t)r.slots * 16 * 32 * warps + 2 * warps * kFields + warps) * sizeof(float);
        if (r.smem > 200 * 1024) continue;
        const uint32_t blocks = t.sites_count == 0 ? 0u : stride == 0 ? 1u : run % stride == 0 ? run / stride : run;
        const double instr = 30.0 * run + 64.0 * blocks + (r.wpc > 1 ? 40.0 : 10.0);
        const uint32_t by_regs = 65536u / (kRegs[run] * 32u * warps), by_smem = (uint32_t)(227 * 1024 / (r.smem + 1024));
        const uint32_t fit = by_regs < by_smem ? (by_regs ? by_regs : 1u) : (by_smem ? by_smem : 1u);
        const uint32_t ctas = (t.groups * kLanes + r.channels - 1) / r.channels, per_sm = (ctas + sms - 1) / sms;
        const uint32_t busy = per_sm < fit ? per_sm : fit, waves = (per_sm + fit - 1) / fit;
        const double time = waves * instr * (2.5 + 1.75 * ((busy * warps + 3) / 4));
        if (best->run == 0 || time < least) {
            *best = r;
            least = time;
        }
    }
    return best->run != 0;
}

// Whether a window has substeps enough for what the resident kernel does around them: it loads and stores the
// whole state by single floats a group's row apart, and one lane after the other sums the evaporation,
// before the old kernel's first substep is through (us resident / through memory, sites every 3): 100 cells in 16
// groups, 4 substeps 18 / 16, 16 21 / 37; 240 in 64, 4 49 / 28, 12 53 / 57, 24 57 / 104; 500 in 1, 1 24 / 28; 1,000 in 200,
// 4 410 / 370, 8 445 / 545; 2,304 in 200, 4 980 / 802, 8 1,040 / 1,234. One cell in 200 groups: 60 20.1 / 19.2.
bool resident_pays(const GpuNftTransport &t) {
    if (t.groups >= 32) return t.cells > 1 && t.substeps >= (t.cells < 200 ? 32u : t.cells < 1200 ? 24u : 12u);
    return t.substeps >= (t.cells < 200 ? 16u : t.cells < 400 ? 6u : t.cells < 1000 ? 3u : 1u);
}

template <bool kFtz> void (*resident_kernel(uint32_t run))(GpuNftTransport, uint32_t, uint32_t) {
    switch (run) {
        case 2: return nft_resident_kernel<kFtz, 2>;
        case 3: return nft_resident_kernel<kFtz, 3>;
        case 4: return nft_resident_kernel<kFtz, 4>;
        case 5: return nft_resident_kernel<kFtz, 5>;
        case 6: return nft_resident_kernel<kFtz, 6>;
        case 7: return nft_resident_kernel<kFtz, 7>;
        case 8: return nft_resident_kernel<kFtz, 8>;
        default: return nft_resident_kernel<kFtz, kMaxRun>;
    }
}

bool aligned16(const void *p) { return ((uintptr_t)p & 15u) == 0; }

}   // namespace

SGB_API int32_t gpu_nft_transport(const GpuNftTransport *t, float *kernel_ms) {
    if (!t || !t->rows || !t->hot || !t->cold || !t->out_sum || !t->evap_kg) return (int32_t)cudaErrorInvalidValue;
    if (t->groups == 0 || t->cells == 0 || (t->sites_count && !t->sites)) return (int32_t)cudaErrorInvalidValue;
    if (t->groups > 0x7fffffffu) return (int32_t)cudaErrorInvalidValue;
    // the reference's last site row is a u32: refuse layouts where it would wrap
    if (t->sites_count && (uint64_t)t->site_offset + (uint64_t)(t->sites_count - 1) * t->site_stride > 0xffffffffull)
        return (int32_t)cudaErrorInvalidValue;
    if (!aligned16(t->rows) || !aligned16(t->hot) || !aligned16(t->cold) || (t->sites && !aligned16(t->sites)))
        return (int32_t)cudaErrorInvalidValue;
    int dev = 0, sms = 0;
    cudaError_t q = cudaGetDevice(&dev);
    if (q == cudaSuccess) q = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (q != cudaSuccess) return (int32_t)q;
    Resident r;
    if (t->groups <= 0x0fffffffu && resident_pays(*t) && resident_shape(*t, (uint32_t)sms, &r)) {   // the channel count fits the grid
        auto kernel = t->flush_denormals ? resident_kernel<true>(r.run) : resident_kernel<false>(r.run);
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)r.smem);
        if (e == cudaSuccess) e = module_mark_start();
        if (e != cudaSuccess) return (int32_t)e;
        kernel<<<(t->groups * kLanes + r.channels - 1) / r.channels, 32 * r.wpc * r.channels, r.smem, module_stream()>>>(*t, r.wpc,
                                                                                                                        r.slots);
        e = cudaGetLastError();
        if (e != cudaSuccess) return (int32_t)e;
        return (int32_t)module_finish(kernel_ms);
    }
    uint32_t runs = 0, run_len = 0;
    launch_shape(t->cells, &runs, &run_len);
    const uint32_t threads = runs * kLanes;
    const size_t smem = (size_t)2 * runs * kRow * sizeof(float);
    auto kernel = t->flush_denormals ? nft_transport_kernel<true> : nft_transport_kernel<false>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int32_t)e;
    e = module_mark_start();
    if (e != cudaSuccess) return (int32_t)e;
    kernel<<<t->groups, threads, smem, module_stream()>>>(*t, run_len);
    e = cudaGetLastError();
    if (e != cudaSuccess) return (int32_t)e;
    return (int32_t)module_finish(kernel_ms);
}
