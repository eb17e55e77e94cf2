// transport.cu -- exact Siddon flights and macro-cell delta tracking (sm_103a), and the
// launchers of every transport kernel (the default Woodcock tracking: woodcock.cu).
//
// Every lane owns one photon and is in one of five states: stepping, waiting for
// a Compton interaction, waiting for a Rayleigh interaction, waiting for the
// fluorescence of a photoelectric absorption (correction level 2), or dead.  Each
// loop iteration of a warp has three phases whose branches are warp-uniform:
//
//   refill    dead lanes start new histories (source sampling, entry into the
//             grid) once at least `refillBatch` lanes are dead, from a warp-private
//             pool of history indices that the warp takes from a global work-queue
//             head in chunks of kChunk (one atomic per chunk);
//   interact  lanes waiting for an interaction run it together once at least
//             `interactBatch` lanes wait (Compton and Rayleigh: the angle from the
//             material's quantile tables, at level 2 the Doppler energy of a bound
//             electron; fluorescence: K-shell vacancy and yield);
//   step      stepping lanes take one free flight with exact Siddon path lengths, or one
//             flight against the macro cells' majorants; a real collision picks its type
//             at once: photoelectric absorption is scored on the spot below level 2, the
//             other events park the lane until the next interact phase.
//
// Parking interactions and batching refills regroups the expensive, divergent
// work so that it runs with many lanes active instead of one or two.  A history
// draws its uniforms in a fixed order from its own stream, so its result does not
// depend on when, or in which lane, each phase runs.
#include <algorithm>
#include <cfloat>
#include <algorithm>
#include <cmath>
#include <cstdint>

#include "transport_common.cuh"

namespace dxmcg {
namespace {
    // kPhoto: a photoelectric absorption waiting for its fluorescence (correction level 2)
    enum LaneState : int { kDead = 0, kStepping = 1, kCompton = 2, kRayleigh = 3, kPhoto = 4 };

    // Kahan-compensated FP32 sum; value() returns it in FP64 once, at the end.
    struct KahanSum {
        float s = 0.0f, c = 0.0f;
        __device__ __forceinline__ void add(float x)
        {
            const float y = x - c;
            const float t = s + y;
            c = (t - s) - y;
            s = t;
        }
        __device__ __forceinline__ double value() const { return static_cast<double>(s) - static_cast<double>(c); }
    };

    // One free flight with exact voxel path lengths; true on a collision.
    template <bool PACKED>
    __device__ __forceinline__ bool siddonFlight(const DevJob& J, Photon& ph, Rng& rng, const EnergyCache& ec,
        bool& escaped, uint32_t& v, int& m, unsigned& visits)
    {
        const float tau = -logf(rng.u());
        const float o[3] = { ph.px, ph.py, ph.pz };
        const float d[3] = { ph.dx, ph.dy, ph.dz };
        const int dims[3] = { J.nx, J.ny, J.nz };
        Siddon sd;
        float thit = 0.0f;
        bool hit = false;
        if (sd.begin(o, d, dims, J.sp)) {
            float acc = 0.0f;
            while (!sd.done) {
                long long vox;
                float len, t0;
                sd.next(vox, len, t0);
                if (len <= 0.0f)
                    continue;
                ++visits;
                int mm;
                const float rho = voxelAt<PACKED>(J, static_cast<uint32_t>(vox), mm);
                if (mm == DXMCG_TRANSPARENT_MATERIAL)
                    continue;
                const float mu = rho * lerp1(J.tot + mm * kTableNE, ec.ie, ec.fe);
                if (mu > 0.0f && acc + mu * len >= tau) {
                    hit = true;
                    v = static_cast<uint32_t>(vox);
                    m = mm;
                    thit = t0 + (tau - acc) / mu;
                    break;
                }
                acc += mu * len;
            }
        }
        if (!hit) {
            escaped = true;
            return false;
        }
        ph.px = fminf(fmaxf(fmaf(thit, ph.dx, ph.px), 0.0f), J.Lin[0]);
        ph.py = fminf(fmaxf(fmaf(thit, ph.dy, ph.py), 0.0f), J.Lin[1]);
        ph.pz = fminf(fmaxf(fmaf(thit, ph.dz, ph.pz), 0.0f), J.Lin[2]);
        return true;
    }

    // Delta tracking against the macro cell's majorant s_c mu_max(E): the sampled
    // optical depth is spent cell by cell (cell indices advance as integers, so every
    // crossing makes progress); a tentative collision in the cell is real with
    // probability mu(voxel) / (s_c mu_max).  True on a real collision.
    template <bool PACKED>
    __device__ __forceinline__ bool macroFlight(const DevJob& J, Photon& ph, Rng& rng, const EnergyCache& ec, int& cx,
        int& cy, int& cz, bool& escaped, uint32_t& v, int& m, unsigned& visits, unsigned& crossings, unsigned& err)
    {
        float tau = fmaxf(-__logf(rng.u()), 0.0f);
        const float ix = __frcp_rn(ph.dx), iy = __frcp_rn(ph.dy), iz = __frcp_rn(ph.dz);
        float muc = 0.0f;
        for (int guard = 0;; ++guard) {
            if (guard > (1 << 16)) { // cannot happen: each pass moves one cell along a fixed direction
                err |= kErrStepLimit;
                escaped = true;
                return false;
            }
            muc = __ldg(J.mscale + cx + J.mc[0] * (cy + J.mc[1] * cz)) * ec.mmax;
            float tx = FLT_MAX;
            int ax = 0;
            if (ph.dx != 0.0f) {
                const float b = fminf(static_cast<float>(cx + (ph.dx > 0.0f ? 1 : 0)) * J.cellL[0], J.L[0]);
                tx = (b - ph.px) * ix;
            }
            if (ph.dy != 0.0f) {
                const float b = fminf(static_cast<float>(cy + (ph.dy > 0.0f ? 1 : 0)) * J.cellL[1], J.L[1]);
                const float t = (b - ph.py) * iy;
                if (t < tx) {
                    tx = t;
                    ax = 1;
                }
            }
            if (ph.dz != 0.0f) {
                const float b = fminf(static_cast<float>(cz + (ph.dz > 0.0f ? 1 : 0)) * J.cellL[2], J.L[2]);
                const float t = (b - ph.pz) * iz;
                if (t < tx) {
                    tx = t;
                    ax = 2;
                }
            }
            tx = fmaxf(tx, 0.0f);
            if (tau < muc * tx) {
                const float t = tau / muc;
                ph.px = fmaf(t, ph.dx, ph.px);
                ph.py = fmaf(t, ph.dy, ph.py);
                ph.pz = fmaf(t, ph.dz, ph.pz);
                break;
            }
            tau -= muc * tx;
            ph.px = fmaf(tx, ph.dx, ph.px);
            ph.py = fmaf(tx, ph.dy, ph.py);
            ph.pz = fmaf(tx, ph.dz, ph.pz);
            ++crossings;
            bool out;
            if (ax == 0) {
                cx += ph.dx > 0.0f ? 1 : -1;
                out = cx < 0 || cx >= J.mc[0];
            } else if (ax == 1) {
                cy += ph.dy > 0.0f ? 1 : -1;
                out = cy < 0 || cy >= J.mc[1];
            } else {
                cz += ph.dz > 0.0f ? 1 : -1;
                out = cz < 0 || cz >= J.mc[2];
            }
            if (out) {
                escaped = true;
                return false;
            }
        }
        // the voxel of the tentative collision, kept inside the current cell
        const int vx = min(max(static_cast<int>(ph.px * J.isp[0]), cx * J.mb), min(cx * J.mb + J.mb, J.nx) - 1);
        const int vy = min(max(static_cast<int>(ph.py * J.isp[1]), cy * J.mb), min(cy * J.mb + J.mb, J.ny) - 1);
        const int vz = min(max(static_cast<int>(ph.pz * J.isp[2]), cz * J.mb), min(cz * J.mb + J.mb, J.nz) - 1);
        ph.px = fminf(fmaxf(ph.px, 0.0f), J.Lin[0]);
        ph.py = fminf(fmaxf(ph.py, 0.0f), J.Lin[1]);
        ph.pz = fminf(fmaxf(ph.pz, 0.0f), J.Lin[2]);
        ++visits;
        v = static_cast<uint32_t>(vx + J.nx * (vy + J.ny * vz));
        const float rho = voxelAt<PACKED>(J, v, m);
        if (m == DXMCG_TRANSPARENT_MATERIAL)
            return false;
        const float mu = rho * lerp1(J.tot + m * kTableNE, ec.ie, ec.fe);
        return rng.u() * muc < mu;
    }

    // MULTI: one queue over the concatenated history ranges of nJobs jobs (offsets[j] is the
    // first global history of job j, offsets[nJobs] the total); each lane reads its job's
    // descriptor from `jobs`.  Otherwise J0 is the only job.
    template <int TRACKING, bool PACKED, bool MULTI>
    __device__ __forceinline__ void transportRun(const DevJob& J0, const DevJob* __restrict__ jobs,
        const unsigned long long* __restrict__ offsets, int nJobs, unsigned long long h_end,
        DevCounters* __restrict__ ctr, int refillBatch, int interactBatch)
    {
        int jid = 0;
        // event counters per warp (no block-wide barrier: warps finish independently)
        __shared__ unsigned long long sCountAll[256 / 32][cNum];
        const unsigned lane = threadIdx.x & 31u;
        unsigned long long* sCount = sCountAll[threadIdx.x >> 5];
        if (lane < cNum)
            sCount[lane] = 0ull;
        __syncwarp();

        const unsigned ltMask = (1u << lane) - 1u;
        KahanSum sum[3];                      // kSumSource, kSumEscaped, kSumDeposited
        unsigned long long poolNext = 0, poolEnd = 0; // the warp's pool of history indices
        bool exhausted = false;
        int st = kDead;
        Photon ph;
        Rng rng;
        EnergyCache ec { 0, 0.0f, 1.0f, 1.0f };
        uint32_t pv = 0; // voxel of the parked interaction
        int pm = 0;      // its material
        unsigned steps = 0, visits = 0, crossings = 0, err = 0;
        int cx = 0, cy = 0, cz = 0; // macro cell of the photon (MACRO tracking)
        bool fresh = false;

        for (;;) {
            const unsigned stepping = __ballot_sync(kFull, st == kStepping);
            const unsigned parked = __ballot_sync(kFull, st >= kCompton);
            const unsigned dead = ~(stepping | parked);
            const int nStep = __popc(stepping);

            // ---- refill
            if (dead && !exhausted && (__popc(dead) >= refillBatch || nStep == 0)) {
                if (poolNext >= poolEnd) {
                    unsigned long long base = 0;
                    if (lane == 0)
                        base = atomicAdd(&ctr->next, static_cast<unsigned long long>(kChunk));
                    base = __shfl_sync(kFull, base, 0);
                    if (base >= h_end) {
                        exhausted = true;
                        poolNext = poolEnd = 0;
                    } else {
                        poolNext = base;
                        poolEnd = min(base + kChunk, h_end);
                    }
                }
                const unsigned long long avail = poolEnd - poolNext;
                const unsigned rank = __popc(dead & ltMask);
                const bool start = st == kDead && rank < avail;
                bool entered = false;
                if (start) {
                    unsigned long long h = poolNext + rank;
                    if (MULTI) { // the queue spans all jobs: find this history's
                        int lo = 0, hi = nJobs;
                        while (hi - lo > 1) {
                            const int mid = (lo + hi) >> 1;
                            if (__ldg(offsets + mid) <= h)
                                lo = mid;
                            else
                                hi = mid;
                        }
                        jid = lo;
                        h -= __ldg(offsets + lo);
                    }
                    const DevJob& J = MULTI ? jobs[jid] : J0;
                    rng.init(J.key, h);
                    sampleSource(J, h, ph, rng);
                    sum[kSumSource].add(ph.w * ph.E);
                    entered = enterGrid(J, ph);
                    if (entered) {
                        st = kStepping;
                        steps = 0;
                        fresh = true;
                        if (TRACKING == DXMCG_TRACK_SIDDON)
                            gridPos(ph.E, ec.ie, ec.fe);
                        else
                            ec.set(J, ph.E);
                        if (TRACKING == DXMCG_TRACK_MACRO) {
                            cx = min(static_cast<int>(ph.px / J.cellL[0]), J.mc[0] - 1);
                            cy = min(static_cast<int>(ph.py / J.cellL[1]), J.mc[1] - 1);
                            cz = min(static_cast<int>(ph.pz / J.cellL[2]), J.mc[2] - 1);
                        }
                    } else {
                        sum[kSumEscaped].add(ph.w * ph.E);
                    }
                }
                poolNext += min(static_cast<unsigned long long>(__popc(dead)), avail);
                const unsigned mStart = __ballot_sync(kFull, start);
                const unsigned mIn = __ballot_sync(kFull, entered);
                if (lane == 0 && mStart) {
                    atomicAdd(&sCount[cHist], static_cast<unsigned long long>(__popc(mStart)));
                    atomicAdd(&sCount[cMissed], static_cast<unsigned long long>(__popc(mStart & ~mIn)));
                }
            }

            // the lane's job, after the refill may have changed it
            const DevJob& J = MULTI ? jobs[jid] : J0;

            // ---- interact
            const int nPark = __popc(parked);
            if (parked && (nPark >= interactBatch || nPark >= nStep)) {
                const bool compton = st == kCompton;
                const bool rayleigh = st == kRayleigh;
                bool cut = false, fluor = false;
                // the samplers diverge; the direction update they share runs once
                float cost = 1.0f, Ep = ph.E;
                if (compton)
                    Ep = sampleCompton<false>(ph.E, J.mats + pm, J.ctab + pm * (kTableNE * kCTabK), ec.ie, ec.fe,
                        J.correction, rng, cost, err);
                else if (rayleigh)
                    cost = sampleRayleigh(J.rtab + pm * (kTableNE * kCTabK), ec.ie, ec.fe, rng);
                if (compton || rayleigh)
                    scatterDirection(ph.dx, ph.dy, ph.dz, cost, rng.u());
                if (compton) {
                    const float e = ph.w * (ph.E - Ep);
                    deposit(J.tally, pv, e);
                    sum[kSumDeposited].add(e);
                    ph.E = Ep;
                    if (Ep < 1.0f) {
                        const float r = ph.w * Ep;
                        deposit(J.tally, pv, r);
                        sum[kSumDeposited].add(r);
                        st = kDead;
                        cut = true;
                    } else {
                        st = kStepping;
                        if (TRACKING == DXMCG_TRACK_SIDDON)
                            gridPos(ph.E, ec.ie, ec.fe);
                        else
                            ec.set(J, ph.E);
                    }
                } else if (rayleigh) {
                    st = kStepping;
                } else if (st == kPhoto) {
                    // correction level 2: the atom may emit a K-alpha photon, which the lane
                    // follows from the absorption point in an isotropic direction
                    const float Ef = samplePhotoFluorescence(ph.E, J.mats + pm, rng);
                    const float e = ph.w * (ph.E - Ef);
                    deposit(J.tally, pv, e);
                    sum[kSumDeposited].add(e);
                    if (Ef > 0.0f) {
                        const float u1 = rng.u();
                        isotropicDirection(ph.dx, ph.dy, ph.dz, u1, rng.u());
                        ph.E = Ef;
                        st = kStepping;
                        fluor = true;
                        if (TRACKING == DXMCG_TRACK_SIDDON)
                            gridPos(ph.E, ec.ie, ec.fe);
                        else
                            ec.set(J, ph.E);
                    } else {
                        st = kDead;
                    }
                }
                const unsigned mC = __ballot_sync(kFull, compton);
                const unsigned mR = __ballot_sync(kFull, rayleigh);
                const unsigned mCut = __ballot_sync(kFull, cut);
                const unsigned mF = __ballot_sync(kFull, fluor);
                if (lane == 0) {
                    if (mC)
                        atomicAdd(&sCount[cCompton], static_cast<unsigned long long>(__popc(mC)));
                    if (mR)
                        atomicAdd(&sCount[cRayleigh], static_cast<unsigned long long>(__popc(mR)));
                    if (mCut)
                        atomicAdd(&sCount[cCutoff], static_cast<unsigned long long>(__popc(mCut)));
                    if (mF)
                        atomicAdd(&sCount[cFluorescence], static_cast<unsigned long long>(__popc(mF)));
                }
            }

            if (__ballot_sync(kFull, st != kDead) == 0u) {
                if (exhausted)
                    break;
                continue;
            }

            // ---- step
            bool photo = false, first = false, error = false;
            if (st == kStepping) {
                bool escaped = false;
                uint32_t v = 0;
                int m = 0;
                bool real = false;
                if (TRACKING == DXMCG_TRACK_SIDDON)
                    real = siddonFlight<PACKED>(J, ph, rng, ec, escaped, v, m, visits);
                else
                    real = macroFlight<PACKED>(J, ph, rng, ec, cx, cy, cz, escaped, v, m, visits, crossings, err);
                if (escaped) {
                    sum[kSumEscaped].add(ph.w * ph.E);
                    st = kDead;
                } else if (real) {
                    first = fresh;
                    fresh = false;
                    const float4 a = __ldg(J.xs + m * kTableNE + ec.ie);
                    const float4 b = __ldg(J.xs + m * kTableNE + ec.ie + 1);
                    const float pe = fmaf(ec.fe, b.x - a.x, a.x);
                    const float ic = fmaf(ec.fe, b.y - a.y, a.y);
                    const float co = fmaf(ec.fe, b.z - a.z, a.z);
                    const float rt = rng.u() * (pe + ic + co);
                    if (rt < pe) {
                        photo = true;
                        if (J.correction >= 2) {
                            pv = v;
                            pm = m;
                            st = kPhoto;
                        } else {
                            const float e = ph.w * ph.E;
                            deposit(J.tally, v, e);
                            sum[kSumDeposited].add(e);
                            st = kDead;
                        }
                    } else {
                        pv = v;
                        pm = m;
                        st = rt < pe + ic ? kCompton : kRayleigh;
                    }
                }
                if (st != kDead && ++steps > J.maxSteps) {
                    err |= kErrStepLimit;
                    st = kDead;
                    error = true;
                }
            }
            const unsigned mPhoto = __ballot_sync(kFull, photo);
            const unsigned mFirst = __ballot_sync(kFull, first);
            const unsigned mErr = __ballot_sync(kFull, error);
            if (lane == 0) {
                if (mPhoto)
                    atomicAdd(&sCount[cPhoto], static_cast<unsigned long long>(__popc(mPhoto)));
                if (mFirst)
                    atomicAdd(&sCount[cInteracted], static_cast<unsigned long long>(__popc(mFirst)));
                if (mErr)
                    atomicAdd(&sCount[cErrors], static_cast<unsigned long long>(__popc(mErr)));
            }
        }

        // ---- flush: per-lane sums by warp, block counters by one thread
        const unsigned long long vi = warpSum(static_cast<unsigned long long>(visits));
        const unsigned long long cr = warpSum(static_cast<unsigned long long>(crossings));
        const double es = warpSum(sum[kSumSource].value());
        const double ee = warpSum(sum[kSumEscaped].value());
        const double ed = warpSum(sum[kSumDeposited].value());
        unsigned errAll = err;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            errAll |= __shfl_xor_sync(kFull, errAll, o);
        __syncwarp();
        if (lane == 0) {
            atomicAdd(&ctr->visits, vi);
            if (cr)
                atomicAdd(&ctr->crossings, cr);
            atomicAdd(&ctr->e_source, es);
            atomicAdd(&ctr->e_escaped, ee);
            atomicAdd(&ctr->e_deposited, ed);
            if (errAll)
                atomicOr(&ctr->error_flags, errAll);
            flushCounts(ctr, sCount);
        }
    }

    template <int TRACKING, bool PACKED>
    __global__ void __launch_bounds__(256) transportKernel(const DevJob J, unsigned long long h_end,
        DevCounters* __restrict__ ctr, int refillBatch, int interactBatch, int)
    {
        transportRun<TRACKING, PACKED, false>(J, nullptr, nullptr, 1, h_end, ctr, refillBatch, interactBatch);
    }
    template <int TRACKING>
    __global__ void __launch_bounds__(256) transportPackKernel(const __grid_constant__ JobPack pack)
    {
        const JobPack::Entry& e = pack.e[packJob(pack)];
        transportRun<TRACKING, true, false>(e.job, nullptr, nullptr, 1, e.h_end, e.ctr, e.refill, e.interact);
    }
    template <int TRACKING>
    __global__ void __launch_bounds__(256) transportQueueKernel(const DevJob* __restrict__ jobs,
        const unsigned long long* __restrict__ offsets, int nJobs, unsigned long long h_end,
        DevCounters* __restrict__ ctr, int refillBatch, int interactBatch)
    {
        transportRun<TRACKING, true, true>(jobs[0], jobs, offsets, nJobs, h_end, ctr, refillBatch, interactBatch);
    }

} // namespace

namespace {
    // kernel instance for a tracking mode on the packed (world) or unpacked
    // (caller-owned arrays) voxel layout with n_mats materials, with or without the gather
    // skip's cell bounds, at correction level 2 (bound) or below; nullptr where no instance
    // exists
    TransportFn kernelFor(int tracking, bool packed, int n_mats, bool skip, bool bound)
    {
        switch (tracking) {
        case DXMCG_TRACK_WOODCOCK: return woodcockKernelFor(packed, false, n_mats, skip, bound);
        case kTrackWoodcockBox: return woodcockKernelFor(packed, true, n_mats, skip, bound);
        case DXMCG_TRACK_SIDDON:
            return packed ? transportKernel<DXMCG_TRACK_SIDDON, true> : transportKernel<DXMCG_TRACK_SIDDON, false>;
        case DXMCG_TRACK_MACRO: return packed ? transportKernel<DXMCG_TRACK_MACRO, true> : nullptr;
        default: return nullptr;
        }
    }

    // the same for a launch of several jobs, all of one instance
    PackFn packFor(int tracking, int n_mats, bool skip, bool bound)
    {
        switch (tracking) {
        case DXMCG_TRACK_WOODCOCK: return woodcockPackFor(false, n_mats, skip, bound);
        case kTrackWoodcockBox: return woodcockPackFor(true, n_mats, skip, bound);
        case DXMCG_TRACK_SIDDON: return transportPackKernel<DXMCG_TRACK_SIDDON>;
        case DXMCG_TRACK_MACRO: return transportPackKernel<DXMCG_TRACK_MACRO>;
        default: return nullptr;
        }
    }

    bool isWoodcock(int tracking) { return tracking == DXMCG_TRACK_WOODCOCK || tracking == kTrackWoodcockBox; }

    // The batch sizes and steps of a shape, defaults filled in.  Batches are counted in lanes:
    // of the Woodcock kernel's two photon slots a lane, twice as many (32 at most, a phase's
    // lanes).
    void phaseSizes(const LaunchShape& shape, bool woodcock, int& refill, int& interact, int& steps)
    {
        const auto size = [&](int batch, int woodcockDefault) {
            if (batch <= 0)
                return woodcock ? woodcockDefault : 8;
            return woodcock ? std::min(32, 2 * batch) : batch;
        };
        refill = size(shape.refill_batch, kWoodcockRefillBatch);
        interact = size(shape.interact_batch, kWoodcockInteractBatch);
        steps = shape.woodcock_steps > 0 ? shape.woodcock_steps : 8;
    }

    cudaError_t launch(bool packed, const DevJob& job, unsigned long long h_end, DevCounters* ctr, LaunchShape shape,
        cudaStream_t s)
    {
        const int tracking = kernelTracking(job);
        const bool woodcock = isWoodcock(tracking);
        const TransportFn fn = kernelFor(tracking, packed, job.n_mats, job.cbound != nullptr,
            job.correction >= 2);
        if (!fn)
            return cudaErrorInvalidValue;
        int refill = 0, interact = 0, wsteps = 0;
        phaseSizes(shape, woodcock, refill, interact, wsteps);
        const size_t smem = woodcock ? woodcockSharedBytes(shape.block, job.n_mats) : 0;
        fn<<<shape.grid, shape.block, smem, s>>>(job, h_end, ctr, refill, interact, wsteps);
        return cudaGetLastError();
    }

    // resident blocks per SM of the instance that needs most shared memory
    int residentBlocks(int tracking, bool packed, int block)
    {
        int n = 0;
        const bool woodcock = isWoodcock(tracking);
        const TransportFn fn = kernelFor(tracking, packed, kSharedTableMaterials, false, true);
        const size_t smem = woodcock ? woodcockSharedBytes(block, kSharedTableMaterials) : 0;
        if (!fn || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, block, smem) != cudaSuccess)
            return 1;
        return n > 0 ? n : 1;
    }
} // namespace

cudaError_t launchTransport(const DevJob& job, unsigned long long h_end, DevCounters* ctr, LaunchShape shape,
    cudaStream_t s)
{
    return launch(true, job, h_end, ctr, shape, s);
}

int transportInstance(const DevJob& job)
{
    const int tracking = kernelTracking(job);
    if (!isWoodcock(tracking))
        return tracking;
    return tracking | (job.n_mats <= kSharedTableMaterials ? 8 : 0) | (job.cbound ? 16 : 0)
        | (job.correction >= 2 ? 32 : 0);
}

cudaError_t launchTransportPack(const PackedJob* jobs, int n, cudaStream_t s)
{
    if (n < 1 || n > kPackJobs)
        return cudaErrorInvalidValue;
    const DevJob& J = *jobs[0].job;
    const int tracking = kernelTracking(J);
    const bool woodcock = isWoodcock(tracking);
    const PackFn fn = packFor(tracking, J.n_mats, J.cbound != nullptr, J.correction >= 2);
    if (!fn)
        return cudaErrorInvalidValue;
    JobPack pack;
    pack.n = n;
    int mats = 0;
    unsigned blocks = 0;
    for (int k = 0; k < n; ++k) {
        const PackedJob& p = jobs[k];
        if (transportInstance(*p.job) != transportInstance(J) || p.shape.block != jobs[0].shape.block
            || p.shape.grid < 1)
            return cudaErrorInvalidValue;
        JobPack::Entry& e = pack.e[k];
        e.job = *p.job;
        e.h_end = p.h_end;
        e.ctr = p.ctr;
        phaseSizes(p.shape, woodcock, e.refill, e.interact, e.steps);
        pack.first[k] = blocks;
        blocks += static_cast<unsigned>(p.shape.grid);
        mats = std::max(mats, p.job->n_mats);
    }
    pack.first[n] = blocks;
    const size_t smem = woodcock ? woodcockSharedBytes(jobs[0].shape.block, mats) : 0;
    fn<<<blocks, jobs[0].shape.block, smem, s>>>(pack);
    return cudaGetLastError();
}

cudaError_t launchTransportQueue(int tracking, const DevJob* jobs, const unsigned long long* offsets, int nJobs,
    unsigned long long h_end, DevCounters* ctr, LaunchShape shape, cudaStream_t s)
{
    if (!jobs || !offsets || nJobs < 1 || (tracking != DXMCG_TRACK_SIDDON && tracking != DXMCG_TRACK_MACRO))
        return cudaErrorInvalidValue;
    int refill = 0, interact = 0, wsteps = 0;
    phaseSizes(shape, false, refill, interact, wsteps);
    const auto fn = tracking == DXMCG_TRACK_SIDDON ? transportQueueKernel<DXMCG_TRACK_SIDDON>
                                                   : transportQueueKernel<DXMCG_TRACK_MACRO>;
    fn<<<shape.grid, shape.block, 0, s>>>(jobs, offsets, nJobs, h_end, ctr, refill, interact);
    return cudaGetLastError();
}

cudaError_t loadTransport(const DevJob& J, LaunchKind kind)
{
    const int tracking = kernelTracking(J);
    const bool skip = J.cbound != nullptr, bound = J.correction >= 2;
    cudaFuncAttributes a {};
    if (kind == LaunchKind::kPack)
        return cudaFuncGetAttributes(&a, packFor(tracking, J.n_mats, skip, bound));
    if (kind == LaunchKind::kQueue)
        return tracking == DXMCG_TRACK_SIDDON ? cudaFuncGetAttributes(&a, transportQueueKernel<DXMCG_TRACK_SIDDON>)
                                              : cudaFuncGetAttributes(&a, transportQueueKernel<DXMCG_TRACK_MACRO>);
    return cudaFuncGetAttributes(&a, kernelFor(tracking, true, J.n_mats, skip, bound));
}

cudaError_t launchTransportUnpacked(const DevJob& job, unsigned long long h_end, DevCounters* ctr,
    LaunchShape shape, cudaStream_t s)
{
    return launch(false, job, h_end, ctr, shape, s);
}

int transportMaxBlocksPerSMUnpacked(int block, int tracking) { return residentBlocks(tracking, false, block); }

int transportMaxBlocksPerSM(int block, int tracking) { return residentBlocks(tracking, true, block); }

int transportRegistersPerThread(int tracking)
{
    cudaFuncAttributes a {};
    const TransportFn fn = kernelFor(tracking, true, kSharedTableMaterials, false, true);
    return fn && cudaFuncGetAttributes(&a, fn) == cudaSuccess ? a.numRegs : -1;
}

} // namespace dxmcg
