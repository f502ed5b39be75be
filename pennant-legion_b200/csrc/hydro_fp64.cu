// hydro_fp64.cu -- the plain FP64 hydro cycle on sm_100a (one mesh).
//
// One cycle of Hydro::doCycle (Hydro.cc:342-983) runs as three kernels:
//
//   pass A  zone pass, predictor: advPosHalf, calcCtrs, calcVols,
//           calcSurfVecs, calcEdgeLen, calcCharLen, calcRho, calcCrnrMass,
//           PolyGas::calcStateHalf/calcForce, TTS::calcForce, QCS
//           setCornerDiv/setQCnForce/setForce/setVelDiff, the side part of
//           sumCrnrForce, calcDtNew (block minimum)
//   pass B  point pass: corner mass and force gathered through the
//           point->corner CSR in ascending side order (no float atomics),
//           applyFixedBC, calcAccel, advPosFull
//   pass C  zone pass, corrector: calcCtrs, calcVols, calcWork,
//           calcWorkRate, calcEnergy, calcRho, calcDvol (block maximum);
//           its last CTA then runs calcDt, checkBadSides, the time/cycle
//           update and the next cycle's calcGlobalDt (Driver.cc:213-245)
// Passes A and C add their blocks' dt minimum, dV/V maximum and inverted
// sides to the cycle's reductions with atomics (exact in any order).
//
// Pass A runs one thread per zone (four lanes a zone on small meshes): the
// zone's sides in the reference's side order, each zone-level quantity
// (centre, sums, EOS) formed once, its quotients and roots in straight-line
// code (ieee_div.cuh).  Pass C is in pass_c.cu.  The batched kernels run the
// same bodies.  1/elen is formed
// once per side and shared with the neighbouring corner; QCS terms the
// reference computes and then discards (evol and du unless cdiv < 0, zkur
// when cdiv > 0) are not computed, which leaves every stored value
// unchanged.  The arithmetic lives in hydro_fp64_body.cuh (shared with the
// batched kernels); this file is compiled with -fmad=false, so the results
// match a serial CPU run of the reference bit for bit.
#include "hydro_fp64_body.cuh"

#include <algorithm>
#include "zone_stage.cuh"

namespace pnt {
namespace {

using namespace fp64;

// Pass A: one warp a CTA, 8 an SM, each walking tiles of 32 zones through its
// two stages (zone_stage.cuh).  Zones that the straight-line body refuses are noted in
// a.redo and formed after the loop with the operators, from global memory:
// inlined into the loop, that body's registers would spill the fast one's.
// 1920^2 Sedov: 0.370 ms, against 0.515 ms for one zone a thread with plain
// loads and the division operator at 16 warps an SM; with this body 0.44 ms
// at 12 warps and 0.52 ms at 16.  Its 766 FP64 instructions a zone, comparisons
// among them, would keep the FP64 pipe busy 0.152 ms; the pipe is active 53% of
// the time at 1024^2 and the issue slots 46%.
using zstage::MeshKind;
using zstage::kGeneral;
using zstage::kQuads;
using zstage::kRect;

template <MeshKind kKind>
__global__ void __launch_bounds__(32, 8) pass_a(DevArrays a, HydroConst c) {
    extern __shared__ __align__(16) unsigned char smem_a[];
    pdl_wait();
    const Ctl* ctl = a.ctl;
    if (skip_cycle(ctl)) return;
    const int cur = ctl->cycle & 1;
    const double dt = ctl->dt;
    const int lane = threadIdx.x;
    const int w = (int)blockIdx.x, nw = (int)gridDim.x;
    double zdthyd = 1.e99;
    int bad = 0;
    bool again = false;   // a zone of this warp is out of the straight-line form's range
    zstage::for_tiles<kKind>(a, cur, smem_a, w, nw,
                             [&](const zstage::ZoneIn& in, int g, int32_t z, int32_t s0, int n, bool own) {
        bool ok = true;
        if (own) {
            double v = 1.e99;
            int b = 0;
            if (kKind != kGeneral || n == 4) ok = pass_a_zone_fast<4>(a, c, in, dt, z, s0, v, b);
            else ok = pass_a_zone_fast<3>(a, c, in, dt, z, s0, v, b);
            if (ok) {
                zdthyd = dmin(zdthyd, v);
                bad += b;
            }
        }
        __syncwarp();
        const unsigned m = __ballot_sync(kFull, !ok);
        if (lane == 0) a.redo[g] = m;
        again = again || m != 0;
    });
    if (again) {
        __syncwarp();   // lane 0's notes
        const int ntiles = (a.numz + zstage::kT - 1) / zstage::kT;
        for (int g = w; g < ntiles; g += nw) {
            if (!((a.redo[g] >> lane) & 1)) continue;
            const int32_t z = g * zstage::kT + lane;
            const int32_t s0 = kKind == kGeneral ? a.zfirst[z] : 4 * z;
            const GlobalZoneIn in{a, cur, z, s0};
            double v = 1.e99;
            if (kKind != kGeneral || a.znump[z] == 4) pass_a_zone_thread<4>(a, c, in, dt, z, s0, v, bad);
            else pass_a_zone_thread<3>(a, c, in, dt, z, s0, v, bad);
            zdthyd = dmin(zdthyd, v);
        }
    }
    warp_to_cycle<true>(a.cyc_red, zdthyd, bad);
}

// Pass A of a small mesh: four lanes a zone, 32 zones a CTA.
constexpr int kSmallThreads = 128;
template <MeshKind kKind>
__global__ void __launch_bounds__(kSmallThreads) pass_a_small(DevArrays a, HydroConst c) {
    pdl_wait();
    const Ctl* ctl = a.ctl;
    if (skip_cycle(ctl)) return;
    const int cur = ctl->cycle & 1;
    const double dt = ctl->dt;
    const int lane = threadIdx.x & 31;
    const int zl = (int)(blockIdx.x * kSmallThreads + threadIdx.x) >> 2;
    const bool live = zl < a.numz;
    const int z = live ? zl : a.numz - 1;
    const zstage::Idx ix =
        kKind == kRect ? zstage::rect_idx(z, a.rect_nzx, 0, 0) : zstage::load_idx(a, z, kKind == kQuads);
    double zdthyd = 1.e99;
    int bad = 0;
    if (!pass_a_zone_lanes(a, c, cur, dt, z, ix.s0, ix.n, ix.p, live, zdthyd, bad)) {
        zdthyd = 1.e99;
        bad = 0;
        if (live && (lane & 3) == 0) {
            const GlobalZoneIn in{a, cur, z, ix.s0};
            if (kKind != kGeneral || ix.n == 4) pass_a_zone_thread<4>(a, c, in, dt, z, ix.s0, zdthyd, bad);
            else pass_a_zone_thread<3>(a, c, in, dt, z, ix.s0, zdthyd, bad);
        }
    }
    __syncwarp();
    const int nbad = tiles::block_isum<kSmallThreads>(bad);
    block_to_cycle<true, kSmallThreads>(a.cyc_red, dmin(1.e99, zdthyd), nbad);   // a NaN is left out
}

template <PointKind kKind>
__global__ void __launch_bounds__(kPointThreads) pass_b(DevArrays a, HydroConst c) {
    pdl_wait();
    const Ctl* ctl = a.ctl;
    if (skip_cycle(ctl)) return;
    const int64_t p = (int64_t)blockIdx.x * kPointThreads + threadIdx.x;
    if (kKind == kRectPoints) {
        if (p < a.nump) pass_b_point_rect<false>(a, c, ctl->cycle & 1, ctl->dt, p, a.rect_nzx, a.numz / a.rect_nzx);
    } else {
        pass_b_point_csr<false, kKind == kPointsOfMany>(a, c, ctl->cycle & 1, ctl->dt, p, p < a.nump);
    }
}

// Multi-piece runs: the corner values the neighbours need, and the end of
// the cycle from the reduction over all pieces (min dtnew, max dvovmax,
// summed inverted sides: exact in any order).
__global__ void piece_pack(DevArrays a, const int32_t* __restrict__ send_side, int32_t nsend,
                           unsigned char* __restrict__ send, size_t foff, bool mixed) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nsend) return;
    const int32_t s = send_side[i];
    if (mixed) {
        reinterpret_cast<float*>(send)[i] = a.cmass_f[s];
        reinterpret_cast<float2*>(send + foff)[i] = a.cforce_f[s];
    } else {
        reinterpret_cast<double*>(send)[i] = a.cmass[s];
        reinterpret_cast<double2*>(send + foff)[i] = a.cforce[s];
    }
}

// The first non-finite element of a[0 .. n): its index into *first by
// atomic minimum (a thread's indices grow along its grid-stride loop, so it
// stops at its first).
__global__ void find_nonfinite(const double* __restrict__ a, int64_t n, unsigned long long* first) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        if (!isfinite(__ldg(a + i))) {
            atomicMin(first, (unsigned long long)i);
            return;
        }
    }
}

__global__ void piece_finish(DevArrays a, HydroConst c) {
    Ctl* ctl = a.ctl;
    if (skip_cycle(ctl)) return;
    const double* r = a.piece_red;
    finish_cycle(ctl, c, r[0], -r[1], (int)r[2], (int)r[3]);
}

// Up to here a zone's four lanes beat its one thread: at 128^2 zones (14
// warps an SM against 3.5) 10.6 against 11.0 us, at 48^2 8.5 against 10.5 us,
// at 160^2 12.3 against 11.7 us (with the launch, about 3 us, in each; the
// operators, a zone a thread, 13.9 us at 48^2).
constexpr int kSmallZones = 16384;

using PassA = void (*)(DevArrays, HydroConst);
PassA pass_a_kernel(int32_t rect_nzx, bool quads) {
    return rect_nzx > 0 ? pass_a<kRect> : (quads ? pass_a<kQuads> : pass_a<kGeneral>);
}

}  // namespace
cudaError_t launch_cycle_fp64(const DevArrays& a, const HydroConst& c, cudaStream_t stream, cudaEvent_t* ev,
                              int phases) {
    const int pb = (int)((a.nump + kPointThreads - 1) / kPointThreads);
    cudaError_t e = cudaSuccess;
    if (phases & kPhaseForces) {
        if (ev) cudaEventRecord(ev[0], stream);
        if (a.numz <= kSmallZones)
            e = launch_pdl(a.rect_nzx > 0 ? pass_a_small<kRect> : (a.quads ? pass_a_small<kQuads> : pass_a_small<kGeneral>),
                           (a.numz + kSmallThreads / 4 - 1) / (kSmallThreads / 4), kSmallThreads, 0, stream, a, c);
        else
            e = launch_pdl(pass_a_kernel(a.rect_nzx, a.quads != 0), a.gridA, 32, zstage::kSmem, stream, a, c);
        if (ev) cudaEventRecord(ev[1], stream);
        if (ev) cudaEventRecord(ev[2], stream);   // no closure pass
    }
    if (phases & kPhaseAdvance) {
        const cudaError_t eb =
            launch_pdl(a.rect_nzx > 0 ? pass_b<kRectPoints> : (a.many ? pass_b<kPointsOfMany> : pass_b<kPointsOfFew>), pb,
                       kPointThreads, 0, stream, a, c);
        if (e == cudaSuccess) e = eb;
        if (ev) cudaEventRecord(ev[3], stream);
        launch_pass_c(a, c, false, stream);   // its last CTA ends the cycle
        if (ev) cudaEventRecord(ev[4], stream);
        if (ev) cudaEventRecord(ev[5], stream);   // no separate finalize step
    }
    return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t prepare_pass_a_fp64(int32_t rect_nzx, bool quads, int32_t numz, int nsm, int32_t* grid, int32_t* ntiles) {
    *ntiles = (numz + zstage::kT - 1) / zstage::kT;
    return zstage::prepare(pass_a_kernel(rect_nzx, quads), rect_nzx, numz, nsm, grid);
}

void launch_piece_pack(const DevArrays& a, const int32_t* send_side, int32_t nsend, unsigned char* send,
                       size_t foff, bool mixed, cudaStream_t stream) {
    if (nsend > 0) piece_pack<<<(nsend + 255) / 256, 256, 0, stream>>>(a, send_side, nsend, send, foff, mixed);
}

void launch_find_nonfinite(const double* a, int64_t n, unsigned long long* first, cudaStream_t stream) {
    if (n <= 0) return;
    const int64_t blocks = std::min<int64_t>((n + 255) / 256, 148 * 8);
    find_nonfinite<<<(int)blocks, 256, 0, stream>>>(a, n, first);
}

void launch_piece_finish(const DevArrays& a, const HydroConst& c, cudaStream_t stream) {
    piece_finish<<<1, 1, 0, stream>>>(a, c);
}


}  // namespace pnt
