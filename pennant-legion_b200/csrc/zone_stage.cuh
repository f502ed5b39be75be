// zone_stage.cuh -- the FP64 pass A's inputs, a warp's 32 zones at a time,
// through shared-memory stages that the warp fills for itself.
//
// The zone body (pass_a_zone_fast) needs about 250 registers to interleave
// its quotients without spilling, so 8 warps fit an SM, and warps that load
// and then compute leave it idle while they load (1024^2 Sedov, 12 warps and
// plain loads: 2.7 of 7 stalled cycles an instruction on the loads).  Here a
// warp walks tiles of 32 consecutive zones: while it computes one, cp.async
// copies bring the next one's inputs into its other stage, and the tile after
// that has its point indices loaded.  A lane copies and reads only its own
// zone's slots (structure of arrays over the lanes: conflict-free), so
// cp.async.wait_group alone orders them and there is no barrier at all.
#pragma once

#include "hydro_dev.h"
#include "zone_tiles.cuh"

#include <cuda_runtime.h>

namespace pnt {
namespace zstage {

constexpr int kT = 32;                          // zones a tile
constexpr int kOffX = 0;                        // start-of-cycle positions of the zone's points [k][lane]
constexpr int kOffU = kOffX + 4 * 16 * kT;      // velocities
constexpr int kOffMf = kOffU + 4 * 16 * kT;     // side mass fractions
constexpr int kOffZ = kOffMf + 4 * 8 * kT;      // zm, zr, ze, zwrate, zvol
constexpr int kBytes = kOffZ + 5 * 8 * kT;
constexpr int kSmem = 2 * kBytes;               // a warp's two stages

// What the copies of one zone need: its sides and points.
struct Idx {
    int32_t z, s0, n;
    int32_t p[4];
};

// Zone z of a rect-numbered mesh whose first zone and point are zo and po
// (row_tiles.cuh has the numbering): no loads.
__device__ __forceinline__ Idx rect_idx(int32_t z, int32_t nzx, int32_t zo, int32_t po) {
    const int32_t zl = z - zo, j = zl / nzx;
    const int32_t p = po + zl + j;   // j (nzx + 1) + (zl - j nzx)
    return Idx{z, 4 * z, 4, {p, p + 1, p + nzx + 2, p + nzx + 1}};
}
__device__ __forceinline__ Idx load_idx(const DevArrays& a, int32_t z, bool quads) {
    Idx r;
    r.z = z;
    if (quads) {
        const int4 p = __ldg(reinterpret_cast<const int4*>(a.mapsp1) + z);
        r.s0 = 4 * z;
        r.n = 4;
        r.p[0] = p.x, r.p[1] = p.y, r.p[2] = p.z, r.p[3] = p.w;
    } else {
        r.s0 = __ldg(a.zfirst + z);
        r.n = __ldg(a.znump + z);
#pragma unroll
        for (int k = 0; k < 4; ++k) r.p[k] = __ldg(a.mapsp1 + r.s0 + (k < r.n ? k : 0));
    }
    return r;
}

// The copies of one zone's inputs into the lane's slots of a stage.
__device__ __forceinline__ void issue(const DevArrays& a, int cur, unsigned char* st, const Idx& ix) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (k < ix.n) {
            tiles::cp16a(st + kOffX + (k * kT + lane) * 16, a.px[cur] + ix.p[k]);
            tiles::cp16a(st + kOffU + (k * kT + lane) * 16, a.pu[cur] + ix.p[k]);
            tiles::cp8(st + kOffMf + (k * kT + lane) * 8, a.smf + ix.s0 + k);
        }
    }
    const double* zf[5] = {a.zm, a.zr, a.ze, a.zwrate, a.zvol};
#pragma unroll
    for (int f = 0; f < 5; ++f) tiles::cp8(st + kOffZ + (f * kT + lane) * 8, zf[f] + ix.z);
}

// A lane's zone of a stage, read as fp64::GlobalZoneIn reads global memory.
struct ZoneIn {
    const unsigned char* st;
    int lane;
    __device__ __forceinline__ double2 x0(int k) const {
        return reinterpret_cast<const double2*>(st + kOffX)[k * kT + lane];
    }
    __device__ __forceinline__ double2 u0(int k) const {
        return reinterpret_cast<const double2*>(st + kOffU)[k * kT + lane];
    }
    __device__ __forceinline__ double mf(int k) const {
        return reinterpret_cast<const double*>(st + kOffMf)[k * kT + lane];
    }
    __device__ __forceinline__ double zs(int f) const {
        return reinterpret_cast<const double*>(st + kOffZ)[f * kT + lane];
    }
    __device__ __forceinline__ double zm() const { return zs(0); }
    __device__ __forceinline__ double zr() const { return zs(1); }
    __device__ __forceinline__ double ze() const { return zs(2); }
    __device__ __forceinline__ double zwrate() const { return zs(3); }
    __device__ __forceinline__ double zvol() const { return zs(4); }
};

}  // namespace zstage
}  // namespace pnt
