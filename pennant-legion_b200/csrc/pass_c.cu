// pass_c.cu -- pass C of the single-mesh cycles: the corrector zone pass
// (calcCtrs, calcVols, calcWork, calcWorkRate, calcEnergy, calcRho,
// calcDvol; Hydro.cc:924-983) as the persistent staged kernel of
// pass_c_staged.cuh, in its FP64 form (bit-identical to a serial run of the
// reference: this file is compiled with -fmad=false) and its mixed form
// (the mixed and learned cycles).  Each CTA adds the maximum |dV/V0| and
// the count of inverted sides over its tiles to the cycle's reductions; the
// last CTA to finish ends the cycle (calcDt, checkBadSides, time/cycle, the
// next calcGlobalDt), so a cycle needs no separate finalize launch.
#include "hydro_fp64_body.cuh"
#include "pass_c_staged.cuh"
#include "row_tiles.cuh"
#include "zone_stage.cuh"

namespace pnt {
namespace {

// ---------------------------------------------------------------------
// Pass C over row tiles of a rect mesh (row_tiles.cuh): per tile of up to
// kRowT zones, the bottom and top point rows of px0, pu0, px, pu and four
// zone fields arrive by bulk copies; each thread reads its zone's sfp + sfq
// (64 contiguous bytes) from global memory, and the BC plane masks of its four
// points as one word of four bits a point, a tile ahead (the masks point by
// point were a second memory latency a tile; a flag a zone with the masks
// behind it, the same latency again in every tile of a boundary row or
// column).  64 zones and two stages a CTA, shared memory for 10 CTAs an SM.
// Bound by latency and HBM: 1920^2 Sedov 0.126 ms (its 190 bytes a zone take
// 0.107 ms); 0.135 ms with the flag, 0.134 ms with the masks of every zone,
// 0.146 ms with those and the division operator, 0.150 ms without the prefetch
// of sfp + sfq into L2 too; 480^2 Noh 17.8 us, 20.2 with the flag, 19.5 with
// the masks, 19.0 with those and neither prefetch nor straight-line quotients
// (Sedov, whose zones at rest divide zeros: 18.1, 20.2, 19.5, 20.3).  The
// 0.150 ms against 0.163 ms with sfp + sfq in the stages
// (7 CTAs an SM), 0.152 ms with the zone fields also from global memory,
// 0.174-0.185 ms with three stages or sfp + sfq held a tile ahead in registers
// (8 CTAs) and 0.173 ms for the staged gathers.
// ---------------------------------------------------------------------
#ifndef PNT_ROWS_C_T
#define PNT_ROWS_C_T 64
#endif
#ifndef PNT_ROWS_C_STAGES
#define PNT_ROWS_C_STAGES 2
#endif
constexpr int kRowT = PNT_ROWS_C_T;
constexpr int kRowStages = PNT_ROWS_C_STAGES;
constexpr int kRowRB = (kRowT + 1) * 16;               // one point row of a double2 field
constexpr int kRowOffZs = 8 * kRowRB;                  // [X0 b,t][U0 b,t][X b,t][U b,t], then zm, zetot, zvol, zp: kRowT + 2 each
constexpr int kRowZB = (kRowT + 2) * 8;
constexpr int kRowStageBytes = kRowOffZs + 4 * kRowZB;
constexpr int kRowSmemBytes = kRowStages * kRowStageBytes;
static_assert(kRowT % 2 == 0 && kRowStageBytes % 16 == 0, "16-byte aligned stages");

// From here on the sfp + sfq of a mesh do not stay in L2 until pass C and are
// prefetched a tile ahead (1920^2: 0.150 -> 0.146 ms; at 480^2, where they do
// stay, the prefetch cost 2%).
constexpr int32_t kPrefetchZones = 500000;

constexpr int kWordPlanes = 4;   // planes of a zone's word: bits a point

// kFew: at most kWordPlanes planes, the masks of the zone's points in a word.
// Decks of more planes, which no case has, read them point by point.
template <bool kFew>
struct RowIn {
    static constexpr bool kStraight = true;
    const unsigned char* st;
    const uint16_t* bcmask;
    int64_t pb, npx;
    int t, shift;
    __device__ __forceinline__ int row(int k) const { return k >= 2 ? 1 : 0; }
    __device__ __forceinline__ int col(int k) const { return t + ((k == 1 || k == 2) ? 1 : 0); }
    __device__ __forceinline__ const double2* f(int field, int k) const {
        return reinterpret_cast<const double2*>(st + (2 * field + row(k)) * kRowRB) + col(k);
    }
    __device__ __forceinline__ double x0x(int k) const { return f(0, k)->x; }
    __device__ __forceinline__ double2 u0(int k) const { return *f(1, k); }
    __device__ __forceinline__ double2 x(int k) const { return *f(2, k); }
    __device__ __forceinline__ double2 u(int k) const { return *f(3, k); }
    const double2* sfg;   // the zone's sfp + sfq (global memory)
    __device__ __forceinline__ double2 sf(int k) const { return sfg[k]; }
    unsigned word;
    __device__ __forceinline__ unsigned mask(int k) const {
        return kFew ? (word >> (kWordPlanes * k)) & ((1u << kWordPlanes) - 1u) : __ldg(bcmask + pb + row(k) * npx + col(k));
    }
    __device__ __forceinline__ double zs(int fld) const {
        return reinterpret_cast<const double*>(st + kRowOffZs + fld * kRowZB)[shift + t];
    }
    __device__ __forceinline__ double zm() const { return zs(0); }
    __device__ __forceinline__ double zetot() const { return zs(1); }
    __device__ __forceinline__ double zvol() const { return zs(2); }
    __device__ __forceinline__ double zp() const { return zs(3); }
};

template <bool kMixed, bool kFew>
__global__ void __launch_bounds__(kRowT) pass_c_rows(DevArrays a, HydroConst c) {
    extern __shared__ __align__(128) unsigned char smem_r[];
    __shared__ __align__(8) uint64_t bars[kRowStages];
    pdl_wait();
    // the learned cycle's closure pass and pass B are done with this cycle's
    // zone records
    if (a.closure_nrec && blockIdx.x == 0 && threadIdx.x == 0) *a.closure_nrec = 0;
    const Ctl* ctl = a.ctl;
    if (fp64::skip_cycle(ctl)) return;
    const int cur = ctl->cycle & 1;
    const double dt = ctl->dt, dtinv = ctl->dtinv;
    const int32_t nzx = a.rect_nzx;
    const int64_t npx = (int64_t)nzx + 1;
    const int64_t ntiles = rows::num_tiles<kRowT>(nzx, a.numz);
    const int t = threadIdx.x;
    double dvm = 1.e-99;
    int nbad = 0;
    auto bytes = [&](int64_t g) -> uint32_t {
        const rows::Tile tl = rows::tile_of<kRowT>(g, nzx);
        const rows::ZoneRun zr = rows::zone_run(tl);
        return (uint32_t)(8 * (tl.nt + 1) * 16 + 4 * zr.count * 8);
    };
    auto issue = [&](unsigned char* st, int64_t g, uint32_t bar) {
        const rows::Tile tl = rows::tile_of<kRowT>(g, nzx);
        const rows::ZoneRun zr = rows::zone_run(tl);
        const uint32_t rb = (uint32_t)(tl.nt + 1) * 16;
        const double2* fields[4] = {a.px[cur], a.pu[cur], a.px[cur ^ 1], a.pu[cur ^ 1]};
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            rows::bulk_g2s(st + (2 * f) * kRowRB, fields[f] + tl.pb, rb, bar);
            rows::bulk_g2s(st + (2 * f + 1) * kRowRB, fields[f] + tl.pb + npx, rb, bar);
        }
        const double* zf[4] = {a.zm, a.zetot, a.zvol, a.zp};
#pragma unroll
        for (int f = 0; f < 4; ++f)
            rows::bulk_g2s(st + kRowOffZs + f * kRowZB, zf[f] + zr.zs, (uint32_t)(zr.count * 8), bar);
    };
    // the plane masks of the thread's zone of tile g, a tile ahead; and that
    // tile's sfp + sfq into L2
    const bool far = a.numz > kPrefetchZones;
    auto look_ahead = [&](int64_t g) -> unsigned {
        if (g >= ntiles || !(kFew || far)) return 0;
        const rows::Tile tn = rows::tile_of<kRowT>(g, nzx);
        if (t >= tn.nt) return 0;
        if (far) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.sftot + 4 * (tn.z0 + t)));
        return kFew ? __ldg(a.zone_bc + tn.z0 + t) : 0u;
    };
    unsigned next_word = look_ahead(blockIdx.x);
    auto compute = [&](const unsigned char* st, int64_t g) {
        const rows::Tile tl = rows::tile_of<kRowT>(g, nzx);
        const unsigned word = next_word;
        next_word = look_ahead(g + gridDim.x);
        if (t >= tl.nt) return;
        const RowIn<kFew> in{st, a.bcmask, tl.pb, npx, t, (int)(tl.z0 & 1), a.sftot + 4 * (tl.z0 + t), word};
        const double d = stagedc::zone_core<true, kMixed>(a, c, 4, in, tl.z0 + t, dt, dtinv, nbad);
        dvm = (d > dvm) ? d : dvm;
    };
    if (!rows::for_tiles<kRowStages, kRowStageBytes>(ntiles, smem_r, bars, bytes, issue, compute) && t == 0)
        atomicOr(reinterpret_cast<unsigned long long*>(a.cyc_red + 4), 1ull);
    const int nb = tiles::block_isum<kRowT>(nbad);
    fp64::block_to_cycle<false, kRowT>(a.cyc_red, dvm, nb);
    fp64::end_cycle_if_last(a, c);
}

template <bool kQuads, bool kMixed>
__global__ void __launch_bounds__(stagedc::kTile) pass_c_staged(DevArrays a, HydroConst c) {
    extern __shared__ __align__(16) unsigned char smem_c[];
    pdl_wait();
    if (a.closure_nrec && blockIdx.x == 0 && threadIdx.x == 0) *a.closure_nrec = 0;
    if (fp64::skip_cycle(a.ctl)) return;
    double dvm = 1.e-99;
    int nbad = 0;
    stagedc::pass_c_tiles<kQuads, kMixed>(a, c, smem_c, dvm, nbad);
    const int nb = tiles::block_isum<stagedc::kTile>(nbad);
    fp64::block_to_cycle<false, stagedc::kTile>(a.cyc_red, dvm, nb);
    fp64::end_cycle_if_last(a, c);
}

// ---------------------------------------------------------------------
// Pass C of a small mesh: four lanes a zone, lane k its point and side k
// (lane 3 idle in a triangle), plain loads, 32 zones a CTA.  The arithmetic is
// zone_core's, its sums over the sides in side order through shuffles.
// ---------------------------------------------------------------------
constexpr int kSmallThreads = 128;

template <zstage::MeshKind kKind, bool kMixed>
__global__ void __launch_bounds__(kSmallThreads) pass_c_small(DevArrays a, HydroConst c) {
    pdl_wait();
    if (a.closure_nrec && blockIdx.x == 0 && threadIdx.x == 0) *a.closure_nrec = 0;
    const Ctl* ctl = a.ctl;
    if (fp64::skip_cycle(ctl)) return;
    const int cur = ctl->cycle & 1;
    const double dt = ctl->dt, dtinv = ctl->dtinv;
    const int zl = (int)blockIdx.x * (kSmallThreads / 4) + (int)(threadIdx.x >> 2);
    const bool live = zl < a.numz;
    const int z = live ? zl : a.numz - 1;
    const zstage::Idx ix = kKind == zstage::kRect ? zstage::rect_idx(z, a.rect_nzx, 0, 0)
                                                  : zstage::load_idx(a, z, kKind == zstage::kQuads);
    const int lane = threadIdx.x & 31, q = lane & 3, gl = lane & ~3, n = ix.n;
    const int k = q < n ? q : 0;                   // an idle lane repeats side 0
    const int ln = gl + ((k + 1 < n) ? k + 1 : 0);
    const int32_t p = k == 0 ? ix.p[0] : (k == 1 ? ix.p[1] : (k == 2 ? ix.p[2] : ix.p[3]));
    const double2 x = a.px[cur ^ 1][p], u = a.pu[cur ^ 1][p], u0 = a.pu[cur][p];
    const double x0x = a.px[cur][p].x;
    const double2 sf = a.sftot[ix.s0 + k];
    const unsigned mask = a.bcmask[p];
    double zm = 0., zetot0 = 0., zvol0 = 0., zp = 0.;
    if (live) {   // the last zone's energy and volume may be its own warp's results by now
        zm = a.zm[z];
        zetot0 = a.zetot[z];
        zvol0 = a.zvol[z];
        zp = a.zp[z];
    }
    const double dth = 0.5 * dt;
    const double xpx = x0x + u0.x * dth;
    double2 ub = u0;
    if (mask) {
        for (int b = 0; b < c.nbc; ++b)
            if (mask & (1u << b)) ub = stagedc::proj(ub, c.vfix[b][0], c.vfix[b][1]);
    }
    __syncwarp();
    const double2 x2 = fp64::shfl2(x, ln);
    const double2 us = stagedc::mk2(ub.x + u.x, ub.y + u.y);
    const double2 us2 = fp64::shfl2(us, ln);
    const double xpx2 = fp64::shfl(xpx, ln);
    // in side order; the FP64 cycle's sums start from zero
    auto sum = [&](double v) {
        const double s0 = fp64::shfl(v, gl), s1 = fp64::shfl(v, gl + 1), s2 = fp64::shfl(v, gl + 2),
                     s3 = fp64::shfl(v, gl + 3);
        double s = kMixed ? s0 : __dadd_rn(0.0, s0);
        s = s + s1;
        s = s + s2;
        return n == 4 ? s + s3 : s;
    };
    const double rn = 1. / (double)n;
    const double zxx = sum(x.x * rn), zxy = sum(x.y * rn);
    const double third = 1. / 3.;
    const double sa = 0.5 * ((x2.x - x.x) * (zxy - x.y) - (x2.y - x.y) * (zxx - x.x));
    const double sv = third * sa * (x.x + x2.x + zxx);
    const double sd1 = sf.x * us.x + sf.y * us.y;
    const double sd2 = (-sf.x) * us2.x + (-sf.y) * us2.y;
    const double dwork = -dth * (sd1 * xpx + sd2 * xpx2);
    const double zvol = sum(sv), zw = sum(dwork);
    double zetot;
    if (kMixed) {
        zetot = zetot0 + zw;
    } else {
        const double w0 = fp64::shfl(dwork, gl), w1 = fp64::shfl(dwork, gl + 1), w2 = fp64::shfl(dwork, gl + 2),
                     w3 = fp64::shfl(dwork, gl + 3);
        zetot = zetot0 + w0;
        zetot = zetot + w1;
        zetot = zetot + w2;
        if (n == 4) zetot = zetot + w3;
    }
    double dvm = 1.e-99;
    if (live && q == 0) {
        const double d = stagedc::zone_results<true>(a, z, zm, zvol0, zp, dtinv, zvol, zetot, zw);
        dvm = (d > dvm) ? d : dvm;
    }
    const int nb = tiles::block_isum<kSmallThreads>((live && q < n && sv <= 0.) ? 1 : 0);
    fp64::block_to_cycle<false, kSmallThreads>(a.cyc_red, dvm, nb);
    fp64::end_cycle_if_last(a, c);
}

// The BC plane masks of each zone's points in a word.
__global__ void find_zone_bc(DevArrays a, uint16_t* zone_bc) {
    const int64_t z = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (z >= a.numz) return;
    unsigned m = 0;
    for (int k = 0; k < a.znump[z]; ++k) m |= (unsigned)a.bcmask[a.mapsp1[a.zfirst[z] + k]] << (kWordPlanes * k);
    zone_bc[z] = (uint16_t)m;
}

using Kernel = void (*)(DevArrays, HydroConst);

// Up to here four lanes a zone are faster: cycle of 48^2 zones 11.4 against
// 13.3 us, 128^2 15.1 / 17.3, 200^2 20.7 / 21.3, 256^2 23.3 / 22.6 us (200 x
// 200 pie 24.3 / 25.6).
constexpr int32_t kSmallZones = 40000;

template <bool kMixed>
Kernel pick_small(int32_t rect_nzx, bool quads) {
    return rect_nzx > 0 ? pass_c_small<zstage::kRect, kMixed>
                        : (quads ? pass_c_small<zstage::kQuads, kMixed> : pass_c_small<zstage::kGeneral, kMixed>);
}

Kernel pick_rows(bool mixed, bool few) {
    if (mixed) return few ? pass_c_rows<true, true> : pass_c_rows<true, false>;
    return few ? pass_c_rows<false, true> : pass_c_rows<false, false>;
}

Kernel pick_kernel(bool mixed, bool quads) {
    if (mixed) return quads ? pass_c_staged<true, true> : pass_c_staged<false, true>;
    return quads ? pass_c_staged<true, false> : pass_c_staged<false, false>;
}

}  // namespace

cudaError_t prepare_pass_c(bool mixed, bool quads, int32_t rect_nzx, int32_t nbc, int32_t numz, int nsm,
                           int32_t* grid) {
    if (numz <= kSmallZones) {
        *grid = (numz + kSmallThreads / 4 - 1) / (kSmallThreads / 4);
        return cudaSuccess;
    }
    if (rect_nzx > 0) {
        const Kernel k = pick_rows(mixed, nbc <= kWordPlanes);
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kRowSmemBytes);
        if (e != cudaSuccess) return e;
        int occ = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, kRowT, kRowSmemBytes);
        if (e != cudaSuccess) return e;
        if (occ < 1) return cudaErrorInvalidConfiguration;
        int64_t g = (int64_t)occ * nsm;
        const int64_t nt = rows::num_tiles<kRowT>(rect_nzx, numz);
        if (g > nt) g = nt;
        *grid = (int32_t)(g < 1 ? 1 : g);
        return cudaSuccess;
    }
    return tiles::prepare(pick_kernel(mixed, quads), stagedc::kTile, stagedc::kSmemBytes, numz, nsm, grid);
}

bool pass_c_reads_words(int32_t rect_nzx, int32_t nbc, int32_t numz) {
    return rect_nzx > 0 && numz > kSmallZones && nbc <= kWordPlanes;
}

cudaError_t launch_find_zone_bc(const DevArrays& a, uint16_t* zone_bc, cudaStream_t stream) {
    find_zone_bc<<<(unsigned)((a.numz + 255) / 256), 256, 0, stream>>>(a, zone_bc);
    return cudaGetLastError();
}

void launch_pass_c(const DevArrays& a, const HydroConst& c, bool mixed, cudaStream_t stream) {
    if (a.numz <= kSmallZones) {
        launch_pdl(mixed ? pick_small<true>(a.rect_nzx, a.quads != 0) : pick_small<false>(a.rect_nzx, a.quads != 0),
                   a.gridC, kSmallThreads, 0, stream, a, c);
        return;
    }
    if (a.rect_nzx > 0) {
        launch_pdl(pick_rows(mixed, c.nbc <= kWordPlanes), a.gridC, kRowT, kRowSmemBytes, stream, a, c);
        return;
    }
    launch_pdl(pick_kernel(mixed, a.quads != 0), a.gridC, stagedc::kTile, stagedc::kSmemBytes, stream, a, c);
}

}  // namespace pnt
