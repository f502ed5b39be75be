// batch_tiles.cuh -- the FP64 pass A's walk over the zone tiles of a batch:
// one-warp CTAs through the stages of zone_stage.cuh, as the single-mesh
// kernels walk one mesh, a zone tile in `subs` warp tiles of 32 zones; and
// the fold of a warp's results into its instance, for the mixed pass A too.
#pragma once

#include "batch_dev.h"
#include "hydro_fp64_body.cuh"
#include "zone_stage.cuh"

namespace pnt {
namespace btiles {

// A zone tile's entry as loaded: inst, beg, end, quads; nzx, zo, po, nzy.
struct Entry {
    int4 e0, e1;
};
__device__ __forceinline__ Entry load_entry(const BatchDev& b, int g) {
    const int4* e = reinterpret_cast<const int4*>(b.ztiles + g / b.subs);
    return Entry{__ldg(e), __ldg(e + 1)};
}

// Warp tile g: its instance, whether it has zones to advance, and the lane's
// zone (own: the lane has one; else the tile's last).  Nothing here is looked
// at before the tile's copies are issued, a tile later, so the loads of the
// instance's state and of the indices are not waited for.
struct WarpTile {
    int inst, z0, end;
    int done, cycle, stop_at;
    zstage::Idx ix;
    __device__ __forceinline__ bool any() const { return z0 < end && !done && cycle < stop_at; }
    __device__ __forceinline__ bool own() const { return any() && z0 + (int)(threadIdx.x & 31) < end; }
};

template <bool kAllQuads>
__device__ __forceinline__ WarpTile warp_tile(const BatchDev& b, int g, const Entry& e) {
    const int lane = threadIdx.x & 31;
    WarpTile r;
    r.inst = e.e0.x;
    r.z0 = e.e0.y + (g % b.subs) * zstage::kT;
    r.end = e.e0.z;
    const Ctl* ctl = b.ctls + r.inst;
    r.done = ctl->done;
    r.cycle = ctl->cycle;
    r.stop_at = ctl->stop_at;
    const int zl = min(r.z0 + lane, r.end - 1);
    r.ix = e.e1.x > 0 ? zstage::rect_idx(zl, e.e1.x, e.e1.y, e.e1.z) : zstage::load_idx(b.a, zl, kAllQuads || e.e0.w);
    return r;
}

// One warp's share: warp tiles w, w + nw, ...  compute(in, g, inst, c, dt, z,
// s0, n, own) is called by whole warps for each that has zones to advance.
template <bool kAllQuads, typename Compute>
__device__ __forceinline__ void for_tiles(const BatchDev& b, unsigned char* smem, int w, int nw, Compute&& compute) {
    const int lane = threadIdx.x & 31;
    const int ntiles = b.nztiles * b.subs;
    if (w >= ntiles) return;
    auto issue = [&](int s, const WarpTile& t) {
        if (t.any()) zstage::issue(b.a, t.cycle & 1, smem + s * zstage::kBytes, t.ix);
    };
    const int last = ntiles - 1;   // entries past the end: the last one's, not used
    WarpTile cur = warp_tile<kAllQuads>(b, w, load_entry(b, w));
    Entry e = load_entry(b, min(w + nw, last));
    issue(0, cur);
    tiles::commit();
    WarpTile next = warp_tile<kAllQuads>(b, min(w + nw, last), e);
    e = load_entry(b, min(w + 2 * nw, last));
    int s = 0;
    for (int g = w; g < ntiles; g += nw) {
        if (g + nw < ntiles) issue(s ^ 1, next);
        tiles::commit();
        const WarpTile after = warp_tile<kAllQuads>(b, min(g + 2 * nw, last), e);
        e = load_entry(b, min(g + 3 * nw, last));
        tiles::wait_groups<1>();
        if (cur.any())
            compute(zstage::ZoneIn{smem + s * zstage::kBytes, lane}, g, cur.inst, b.consts[cur.inst],
                    b.ctls[cur.inst].dt, cur.ix.z, cur.ix.s0, cur.ix.n, cur.own());
        __syncwarp();
        cur = next;
        next = after;
        s ^= 1;
    }
}

// A warp's running minimum dt and inverted sides of one instance, handed to
// the instance when the warp comes to another one.
struct InstFold {
    int inst = -1;
    double v = 1.e99;
    int bad = 0;
    __device__ __forceinline__ void flush(const BatchDev& b) {
        if (inst < 0) return;
        double m = v;
        for (int o = 16; o > 0; o >>= 1) m = fp64::dmin(m, __shfl_xor_sync(fp64::kFull, m, o));
        const int n = (int)__reduce_add_sync(fp64::kFull, (unsigned)bad);
        if ((threadIdx.x & 31) == 0) {
            long long* r = b.inst_red + 2 * inst;
            if (m < fp64::dkey_value(*(volatile long long*)r)) atomicMin(r, fp64::dkey(m));
            if (n) atomicAdd(reinterpret_cast<unsigned long long*>(r + 1), (unsigned long long)n);
        }
        v = 1.e99;
        bad = 0;
    }
    __device__ __forceinline__ void at(const BatchDev& b, int i) {
        if (i != inst) flush(b);
        inst = i;
    }
};

}  // namespace btiles
}  // namespace pnt
