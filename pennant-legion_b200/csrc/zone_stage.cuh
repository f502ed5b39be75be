// zone_stage.cuh -- pass A's inputs (the FP64 cycle's, and the mixed and
// learned cycles'), a warp's 32 zones at a time, through shared-memory stages
// that the warp fills for itself.
//
// The FP64 zone body (pass_a_zone_fast) needs about 250 registers to interleave
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

// How a mesh's zones and sides are numbered: any way, quads at sides 4z ..
// 4z + 3, or as the rect generator does (row_tiles.cuh).
enum MeshKind { kGeneral, kQuads, kRect };

// The zones of one mesh, one warp's share: tiles w, w + nw, ...  compute(in,
// g, z, s0, n, own) is called by whole warps for each tile g: the lane's zone
// z with sides s0 .. s0 + n - 1 (own = false past the last zone).
template <MeshKind kKind, typename Compute>
__device__ __forceinline__ void for_tiles(const DevArrays& a, int cur, unsigned char* smem, int w, int nw,
                                          Compute&& compute) {
    const int lane = threadIdx.x & 31;
    const int ntiles = (a.numz + kT - 1) / kT;
    auto index = [&](int g) {
        const int z = min(g * kT + lane, a.numz - 1);
        if (kKind == kRect) return rect_idx(z, a.rect_nzx, 0, 0);
        return load_idx(a, z, kKind == kQuads);
    };
    if (w >= ntiles) return;
    Idx ix = index(w), nx = ix;
    issue(a, cur, smem, ix);
    tiles::commit();
    if (w + nw < ntiles) nx = index(w + nw);
    int s = 0;
    for (int g = w; g < ntiles; g += nw) {
        const int32_t z = ix.z, s0 = ix.s0, n = kKind == kGeneral ? ix.n : 4;
        ix = nx;
        if (g + nw < ntiles) issue(a, cur, smem + (s ^ 1) * kBytes, ix);
        tiles::commit();
        if (g + 2 * nw < ntiles) nx = index(g + 2 * nw);
        tiles::wait_groups<1>();   // this lane's copies of tile g have landed
        compute(ZoneIn{smem + s * kBytes, lane}, g, z, s0, n, g * kT + lane < a.numz);
        __syncwarp();
        s ^= 1;
    }
}

// Raises the shared-memory limit of a kernel of one-warp CTAs and returns its
// persistent grid: resident CTAs per SM x nsm, at most one per tile.  Where
// nw tiles are (nearly) whole rows of a rect mesh, a warp would keep to the
// same columns, and the warps whose columns a shock crosses would have all
// the compressing zones (1024^2 Sedov: 37 rows a round, 5.9 of 8 warps active
// on average); the grid is then cut by up to 2% so that the columns move on.
template <typename K>
inline cudaError_t prepare(K k, int32_t rect_nzx, int32_t numz, int nsm, int32_t* grid) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    if (e != cudaSuccess) return e;
    int occ = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, 32, kSmem);
    if (e != cudaSuccess) return e;
    if (occ < 1) return cudaErrorInvalidConfiguration;
    const int tiles = (numz + kT - 1) / kT;
    int nw = occ * nsm < tiles ? occ * nsm : tiles;
    if (rect_nzx > 0 && tiles > nw) {
        // how far a round moves a warp along the rows, and over the mesh
        auto drift = [&](int n) {
            const double f = (double)n * kT / rect_nzx, d = f - (double)(long long)f;
            return (d < 0.5 ? d : 1. - d) * tiles / n;
        };
        if (drift(nw) < 1.) {
            int best = nw;
            for (int n = nw; n >= nw - nw / 50 && n > 0; --n)
                if (drift(n) > drift(best)) best = n;
            nw = best;
        }
    }
    *grid = nw;
    return cudaSuccess;
}

}  // namespace zstage
}  // namespace pnt
