// Host side of the lane-group kernels: the device images of one mechanism and the launch.
#pragma once
#include <cuda_runtime.h>
#include <string.h>

#include "group_tab.h"
#include "kin_group.cuh"

namespace sgb {

typedef void (*GroupFn)(DevArgs, GroupArgs);
// The kernel of a lane precision for mechanisms of at most NM species (kern_group.cu).
template <int PREC, int NM> GroupFn group_kernel(uint32_t G, bool rodas3);
template <> GroupFn group_kernel<0, 12>(uint32_t, bool);
template <> GroupFn group_kernel<0, 17>(uint32_t, bool);
template <> GroupFn group_kernel<0, 20>(uint32_t, bool);
template <> GroupFn group_kernel<0, 32>(uint32_t, bool);
template <> GroupFn group_kernel<1, 12>(uint32_t, bool);
template <> GroupFn group_kernel<1, 17>(uint32_t, bool);
template <> GroupFn group_kernel<1, 20>(uint32_t, bool);
template <> GroupFn group_kernel<1, 32>(uint32_t, bool);
template <> GroupFn group_kernel<4, 12>(uint32_t, bool);
template <> GroupFn group_kernel<4, 17>(uint32_t, bool);
template <> GroupFn group_kernel<4, 20>(uint32_t, bool);
template <> GroupFn group_kernel<4, 32>(uint32_t, bool);
template <int PREC> GroupFn group_kernel_for(uint32_t n, uint32_t G, bool rodas3) {
    // FP64 at 8 lanes is faster without (4,096 cells x 1 s: 23.2 against 24.6 ms)
    if (n == kGroupExact && rodas3 && !(PREC == 0 && G == 8)) return group_kernel<PREC, (int)kGroupExact>(G, true);
    return n <= 12 ? group_kernel<PREC, 12>(G, rodas3) : n <= 20 ? group_kernel<PREC, 20>(G, rodas3) : group_kernel<PREC, 32>(G, rodas3);
}

// Lanes per cell of the three images.
constexpr uint32_t kGroupLanes[3] = {8, 16, 32};

// The group shape (index into kGroupLanes) for a batch of `lanes` cells on `sms` SMs, or -1: the lane
// kernels. Lines in cells per SM, from one advance of 1 s (GB300, 152 SMs; ms for 32 / 16 / 8
// lanes per cell and the lane kernel with its hand-off):
//   shipped mechanism  600 cells: FP64 12.6 / 13.8 / 18.4 / 40.1   mixed  8.8 /  8.9 / 11.7 / 18.9
//                    1,300 cells: FP64 17.0 / 14.2 / 18.5 / 42.0   mixed  9.4 /  9.0 / 11.9 / 19.7
//                    2,048 cells: FP64 20.8 / 15.9 / 20.2 / 41.5   mixed 10.9 /  9.9 / 13.0 / 20.0
//                    2,600 cells: FP64 24.3 / 19.6 / 20.6 / 41.2   mixed 12.2 / 10.8 / 13.1 / 20.1
//                    4,096 cells: FP64 34.1 / 26.5 / 21.9 / 42.1   mixed 17.1 / 14.9 / 14.4 / 20.9
//                    6,144 cells: FP64 47.9 / 34.7 / 30.1 / 45.7   mixed 23.3 / 19.5 / 18.8 / 22.3
//                    7,168 cells: FP64 54.9 / 38.8 / 32.5 / 45.1   mixed 25.7 / 21.2 / 20.6 / 21.6
//                    8,192 cells: FP64 62.3 / 43.7 / 36.4 / 44.8   mixed 29.9 / 24.7 / 23.0 / 21.7
//                   11,856 cells: FP64 8 lanes 45.4, lane kernel 46.3; 12,500: 47.0, 46.0
// 8 lanes per cell end where an SM's 64 groups (FP64; mixed 32) are all taken: cells of like numbers of attempts then
// take a second wave, which only cells that differ fill (averaged zones, one 20 ms step, 8 lanes / the lane kernel: FP64 64 cells
// per SM 5.1 / 5.1, 68 6.5 / 5.1, 78 7.1 / 5.1; mixed 34 2.2 / 2.2, 36 2.6 / 2.2, 42 2.9 / 2.1; air cells, 0.1 s: FP64 68 36.1 / 40.4,
// 78 39.8 / 39.8; mixed 36 15.0 / 18.7, 42 16.3 / 18.8).
//   table FP64, 0.05 s, 1,230 cells (9 per SM), 32 / 16 lanes: 16 species 14.2 / 11.4, 24 species
//                    19.7 / 17.3, 32 species (0.02 s) 26.7 / 22.9; 1,660 cells 15.6 / 11.9, 20.8 / 17.8, 28.8 / 24.7
// How far table mechanisms go is group_most's.
inline uint32_t group_most(uint32_t lane_prec, uint32_t n);
inline int group_rule(uint32_t lane_prec, bool generated, uint32_t n, uint32_t lanes, int sms) {
    const uint32_t c = (lanes + (uint32_t)sms - 1) / (uint32_t)sms;
    if (lane_prec != 0 && lane_prec != 1 && lane_prec != 4) return -1;   // the other mixed variants: lanes only
    if (!generated && c > group_most(lane_prec, n)) return -1;
    if (generated && lane_prec == 1) return -1;   // f32 lanes are as fast from one zone on (64 zones pulsed: 20.6 against 22.2)
    if (c <= (generated ? (lane_prec == 4 ? 10u : 8u) : lane_prec == 1 ? 11u : 8u)) return 2;
    if (c <= (lane_prec == 4 ? 26u : 16u)) return 1;
    return !generated || c <= (lane_prec == 4 ? 34u : 64u) ? 0 : -1;
}

// Cells per SM of a table mechanism of n species up to which the group kernels take it. The table-driven lane
// kernels keep a cell's arrays in local memory, so the larger the mechanism the longer they lose (24
// species: 1 ms per attempt), but a few species' arrays stay in the caches, and a group of 8 lanes has no
// work for most of them. Each line is the least over seeded mechanisms of n to 5 n reactions, from the time of
// 8-lane groups over that of the lanes without a hand-off (0.01 s, at most 120 attempts):
//   FP64   1 species 16 cells per SM 0.79, 30 1.05; 3: 52 1.02, 98 1.55; 6: 90 0.93, 120 1.14; 8: 120 0.98, 197 1.15;
//          12: 197 0.96, 300 1.11; 14: 300 0.93, 431 1.05; 16: 300 0.69, 431 0.85; 21: 300 1.01, 430 1.31; 24: 300 0.73, 431 0.88;
//          32: 140 0.65, 300 1.16
//   f32    1: 30 0.77, 60 1.37; 2: 60 0.93, 100 1.70; 3: 150 0.75, 197 1.19; 4: 250 0.98, 400 1.11; 6: 400 0.94, 700 1.20; 8: 700 0.94,
//          1,500 1.21; 10: 1,500 0.90, 3,000 1.07; 12: 2,631 0.59; 24: 1,973 0.53
//   mixed  1: 50 0.76, 100 1.44; 2: 50 0.58, 100 1.10; 3: 197 0.92, 300 1.08; 4: 500 0.94, 900 1.07; 5: 900 0.89, 2,000 1.13; 6: 2,000 0.92;
//          7: 2,000 0.80; 16: 986 0.37
inline uint32_t group_most(uint32_t lane_prec, uint32_t n) {
    static const uint16_t f32[11] = {0, 30, 60, 150, 250, 400, 400, 600, 750, 1400, 2500};
    static const uint16_t mixed[7] = {0, 50, 80, 230, 500, 900, 2000};
    constexpr uint32_t kAll = 0xffffffffu;
    if (lane_prec == 1) return n < 11 ? f32[n] : kAll;
    if (lane_prec == 4) return n < 7 ? mixed[n] : kAll;
    return n <= 9 ? 14 * n : n <= 12 ? 180u : n <= 14 ? 300u : n <= 17 ? 400u : n <= 24 ? 300u : 128u;
}

// Cells at which a CTA of `block` lanes of the queue kernel parks what it has left: where its attempt costs
// what a group kernel takes for as many cells at full throughput. Shipped mechanism, cycles: FP64 lanes
// 308k per 128-lane attempt against ~9.3k per cell and attempt of 8-lane groups (33 cells), mixed
// 149k per 256 lanes against ~6.5k (23). Table mechanisms, time over that without parking, CTAs of 128 that
// park from 16 / 127 cells on: FP64 3 species 431 cells per SM 1.00 / 2.07, 986 1.04 / 1.39; 8: 431 1.00 / 1.42; 24: 431 1.00 / 1.03,
// so they park none; mixed 2: 431 0.93 / 1.64, 986 0.88 / 1.51; 4: 986 0.95 / 1.28; 8: 431 1.00 / 1.07; 10: 431 1.00 / 0.92;
// 16: 300 1.00 / 0.83. (One species: the launch behind them costs more.)
inline uint32_t group_drain(uint32_t lane_prec, bool generated, uint32_t n, uint32_t block) {
    if (!generated) return lane_prec == 0 || n < 2 ? 0u : n < 10 ? block / 8 : block - 1;
    return lane_prec == 0 ? block / 4 : block / 11;
}

// One mechanism's schedule images on the device: per lanes-per-cell and lane precision (0 FP64, 1 f32
// Delta, 2 mixed). Empty (dev null) for a mechanism whose record could not be laid out.
struct GroupSet {
    unsigned char *dev = nullptr;   // set while there are images
    unsigned char *buffer = nullptr;
    size_t capacity = 0;
    uint32_t offset[3][3] = {};
    GroupHead head[3][3] = {};
    bool rodas3 = false;
    bool starved = false;   // the last build found no device memory: worth another

    // No kernel may be using the images of the mechanism before.
    cudaError_t build(const KinMech &mech, bool method_rodas3) {
        dev = nullptr;
        starved = false;
        std::vector<uint32_t> all, one;
        for (int g = 0; g < 3; ++g)
            for (int f = 0; f < 3; ++f) {
                if (!group_image(mech, kGroupLanes[g], f == 2 ? 4u : (uint32_t)f, &one)) return cudaSuccess;
                memcpy(&head[g][f], one.data(), sizeof(GroupHead));
                offset[g][f] = (uint32_t)all.size() * 4u;
                all.insert(all.end(), one.begin(), one.end());
            }
        rodas3 = method_rodas3;
        if (all.size() * 4 > capacity) {
            release();
            if (cudaMalloc((void **)&buffer, all.size() * 4) != cudaSuccess) {   // no memory: the lane kernels run alone
                cudaGetLastError();
                buffer = nullptr;
                starved = true;
                return cudaSuccess;
            }
            capacity = all.size() * 4;
        }
        const cudaError_t e = cudaMemcpy(buffer, all.data(), all.size() * 4, cudaMemcpyHostToDevice);
        if (e == cudaSuccess) dev = buffer;
        return e;
    }
    void release() {
        if (buffer) cudaFree(buffer);
        dev = buffer = nullptr;
        capacity = 0;
    }

    static int index(uint32_t lane_prec) { return lane_prec == 4 ? 2 : (int)lane_prec; }

    // The kernel's arguments for G = kGroupLanes[g], and the shared memory of a CTA of `warps` warps.
    GroupArgs args(uint32_t lane_prec, int g) const {
        const int f = index(lane_prec);
        GroupArgs a;
        a.image = dev + offset[g][f];
        a.image32 = dev + offset[2][f];
        a.bytes = head[g][f].words * 4;
        a.bytes32 = head[2][f].words * 4;
        a.cell_bytes = group_cell_bytes(head[g][f], lane_prec, kGroupLanes[g]);
        const uint32_t cells = 32u / kGroupLanes[g] * a.cell_bytes, one = group_cell_bytes(head[2][f], lane_prec, 32);
        a.warp_bytes = kGroupStateBytes + (cells > one ? cells : one);
        return a;
    }
    static size_t smem(const GroupArgs &a, int g, uint32_t warps) {
        return (size_t)a.bytes + (g < 2 ? a.bytes32 : 0u) + (size_t)warps * a.warp_bytes;
    }

    // Enqueues the kernel on cells of `A` (A.cursor zeroed by the caller; A.resume: the parked
    // ones): `want` cells, as many warps as they need up to what `sms` SMs hold.
    cudaError_t launch(uint32_t lane_prec, int g, const DevArgs &A, uint32_t want, int sms, cudaStream_t s) const {
        constexpr size_t kSmemMax = 227 * 1024;
        const uint32_t G = kGroupLanes[g], n = head[g][0].n;
        const GroupFn fn = lane_prec == 0 ? group_kernel_for<0>(n, G, rodas3)
                                          : lane_prec == 1 ? group_kernel_for<1>(n, G, rodas3) : group_kernel_for<4>(n, G, rodas3);
        const GroupArgs a = args(lane_prec, g);
        const uint32_t need = (want + 32 / G - 1) / (32 / G);   // warps
        const uint32_t each = (need + (uint32_t)sms - 1) / (uint32_t)sms;   // warps per SM, evenly spread
        // FP64: one CTA per SM with just its share of warps up to 8. The FP64 unit is busy with four, so an SM
        // with two CTAs of four where others have one takes twice as long (1 s of the shipped mechanism, 4,096 cells: 256
        // CTAs on 152 SMs; 0.3 s, CTAs of four / of the share: 1,501 cells 14.8 / 13.2 ms, 3,000 21.2 / 19.1,
        // 4,096 21.3 / 20.5; 24 species, 0.05 s, 2,400 cells 30.8 / 20.1). Else, as the mixed lanes
        // wait for their chains and not for the unit (2,000 cells 9.0 / 9.3): few cells one or two warps per CTA,
        // so that they spread over the SMs, and from there one warp per scheduler and CTA.
        uint32_t warps = lane_prec == 0 && each <= 8 ? each : each <= 2 ? each : 4u;
        while (warps > 1 && smem(a, g, warps) > kSmemMax) --warps;
        const size_t bytes = smem(a, g, warps);
        cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        int per_sm = 0;
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, (int)(32 * warps), bytes);
        if (e != cudaSuccess) return e;
        if (per_sm < 1) per_sm = 1;
        const uint32_t resident = (uint32_t)per_sm * (uint32_t)sms, ctas = (need + warps - 1) / warps;
        fn<<<resident < ctas ? resident : ctas, 32 * warps, bytes, s>>>(A, a);
        return cudaGetLastError();
    }
};

}   // namespace sgb
