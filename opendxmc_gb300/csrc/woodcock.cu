// woodcock.cu -- the Woodcock transport kernel (sm_103a), the default tracking mode and
// the dominant kernel of the path: one region, or two with a box (see outerFlight).
#include <cfloat>
#include <cmath>
#include <cstdint>

#include "transport_common.cuh"

namespace dxmcg {
namespace {
    // a slot's packed word: energy-grid index below, flags, steps taken from bit 12
    constexpr unsigned kPackOuter = 1u << 9, kPackFresh = 1u << 10;
    constexpr int kPackSteps = 12;
    static_assert(kTableNE <= 512 && kMaxStepsPerHistory + 64 < (1u << 20), "packed word layout");

    // Voxel (ix, iy, iz) lies outside the two-region box.
    __device__ __forceinline__ bool outsideBox(const DevJob& J, int ix, int iy, int iz)
    {
        return (static_cast<unsigned>(ix - J.b0[0]) >= J.bn[0]) | (static_cast<unsigned>(iy - J.b0[1]) >= J.bn[1])
            | (static_cast<unsigned>(iz - J.b0[2]) >= J.bn[2]);
    }

    // Distance along the flight to the widened box (FLT_MAX if the line misses it, 0
    // from inside it).  Approximate reciprocals: the margin of the box absorbs their
    // error, so the entry is never found late.
    __device__ __forceinline__ float boxEntry(const DevJob& J, const Photon& ph)
    {
        const float p[3] = { ph.px, ph.py, ph.pz };
        const float d[3] = { ph.dx, ph.dy, ph.dz };
        float tn = 0.0f, tf = FLT_MAX;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float inv = __fdividef(1.0f, d[a]);
            const float t1 = (J.blo[a] - p[a]) * inv, t2 = (J.bhi[a] - p[a]) * inv;
            tn = fmaxf(tn, fminf(t1, t2));
            tf = fminf(tf, fmaxf(t1, t2));
        }
        return tn <= tf ? tn : FLT_MAX;
    }

    // Voxel indices of the photon's position, by rounding down; outside the grid one of
    // them is negative (huge as unsigned) or >= its dimension (conversions saturate far
    // away) and the result is false.
    __device__ __forceinline__ bool voxelOf(const DevJob& J, const Photon& ph, int& ix, int& iy, int& iz)
    {
        ix = __float2int_rd(ph.px * J.isp[0]);
        iy = __float2int_rd(ph.py * J.isp[1]);
        iz = __float2int_rd(ph.pz * J.isp[2]);
        return (static_cast<unsigned>(ix) < static_cast<unsigned>(J.nx))
            & (static_cast<unsigned>(iy) < static_cast<unsigned>(J.ny))
            & (static_cast<unsigned>(iz) < static_cast<unsigned>(J.nz));
    }

    // Free path to the next tentative collision (an error of negLog near u = 1 is one of less
    // than 1e-6 mean free paths).
    __device__ __forceinline__ float freePath(Rng& rng, float invMmax)
    {
        return fmaxf(negLog(rng.u()), 0.0f) * invMmax;
    }

    __device__ __forceinline__ void fly(Photon& ph, float s)
    {
        ph.px = fmaf(s, ph.dx, ph.px);
        ph.py = fmaf(s, ph.dy, ph.py);
        ph.pz = fmaf(s, ph.dz, ph.pz);
    }

    // What a photon is after a step: in flight, parked at a real collision, gone, or in
    // flight outside the two-region box.
    enum SlotKind : int { kFly = 0, kPark = 1, kFree = 2, kOuter = 3 };

    // Total attenuation of material m at the photon's energy: from the block's shared
    // tables (TAB), or the world's.  A gather of 23 lanes takes about 18 L1 wavefronts from
    // global memory and 5 from shared (1e7 histories of the DX cylinder: 1.41 -> 1.33 ms).
    template <bool TAB>
    __device__ __forceinline__ float attenuation(const DevJob& J, const float* sTot, int m, const EnergyCache& ec)
    {
        if (TAB) {
            const float* t = sTot + m * kTableNE + ec.ie;
            const float a = t[0], b = t[1];
            return fmaf(ec.fe, b - a, a);
        }
        return lerp1(J.tot + m * kTableNE, ec.ie, ec.fe);
    }

    // Woodcock step against maj; returns what the photon is after it: kPark at a real
    // collision in voxel v / material m, kFree outside the grid, kOuter when a virtual
    // collision lies outside the two-region box (BOX), else kFly.
    //
    // Gather skip (SKIP, J.cbound set): the tentative collision is real when u mu_max(E) <
    // rho mu_m(E).  The cell's bound b_c satisfies rho mu_m(E) <= b_c mu_max(E) for each
    // of its voxels, with a margin larger than the FP32 roundings of both sides, so
    // u mu_max >= b_c mu_max settles the step as virtual without reading the voxel.
    // Otherwise the voxel is read and the usual test decides, on the same uniform: the
    // decisions, and so the histories, are those of the plain step.  Cells holding a
    // transparent voxel (b_c = +inf) take the plain step, which draws the uniform only
    // for a voxel that is not transparent.
    //
    // BOX: a flight that ends outside the box decides its tentative collision as usual
    // (maj bounds every voxel); the flights after it are outerFlight's, and `packed` is
    // marked.
    template <bool PACKED, bool BOX, bool TAB, bool SKIP>
    __device__ __forceinline__ int woodcockStep(const DevJob& J, const float* sTot, Photon& ph, Rng& rng,
        const EnergyCache& ec, unsigned& packed, uint32_t& v, int& m, unsigned& visits, unsigned& skipped)
    {
        fly(ph, freePath(rng, ec.invMmax));
        int ix, iy, iz;
        if (!voxelOf(J, ph, ix, iy, iz))
            return kFree;
        ++visits;
        v = static_cast<uint32_t>(ix + J.nx * (iy + J.ny * iz));
        const bool left = BOX && outsideBox(J, ix, iy, iz);
        if (left)
            packed |= kPackOuter;
        const int on = left ? kOuter : kFly;
        float t = -1.0f;
        if (SKIP) {
            const float b = __ldg(J.cbound
                + ((ix >> kCellShift) + J.cb[0] * ((iy >> kCellShift) + J.cb[1] * (iz >> kCellShift))));
            if (b <= FLT_MAX) {
                t = rng.u() * ec.mmax;
                if (t >= b * ec.mmax) {
                    ++skipped;
                    return on;
                }
            }
        }
        const float rho = voxelAt<PACKED>(J, v, m);
        if (m == DXMCG_TRANSPARENT_MATERIAL)
            return on;
        const float mu = rho * attenuation<TAB>(J, sTot, m, ec);
        if (!SKIP || !(t >= 0.0f))
            t = rng.u() * ec.mmax;
        return t < mu ? kPark : on;
    }

    // Two-region Woodcock: a flight that starts outside the box, against majOut.  If the
    // box comes first, the photon moves to it and steps on against maj (the flight is
    // memoryless; kFly), drawing no acceptance uniform.  Every decision keeps the
    // tentative-collision rate at or above rho mu(E) on the path, so the transport is
    // that of plain Woodcock with fewer tentative collisions.  The cell bounds (relative
    // to maj) are not used here.
    template <bool PACKED, bool TAB>
    __device__ __forceinline__ int outerFlight(const DevJob& J, const float* sTot, Photon& ph, Rng& rng,
        EnergyCache& ec, uint32_t& v, int& m, unsigned& visits)
    {
        ec.setMajorant(J.majOut);
        const float s = freePath(rng, ec.invMmax);
        const float te = boxEntry(J, ph);
        const bool entered = te < s;
        fly(ph, entered ? te : s);
        if (entered) {
            ec.setMajorant(J.maj);
            return kFly;
        }
        int ix, iy, iz;
        if (!voxelOf(J, ph, ix, iy, iz))
            return kFree;
        ++visits;
        v = static_cast<uint32_t>(ix + J.nx * (iy + J.ny * iz));
        const float rho = voxelAt<PACKED>(J, v, m);
        if (m == DXMCG_TRANSPARENT_MATERIAL)
            return kOuter;
        return rng.u() * ec.mmax < rho * attenuation<TAB>(J, sTot, m, ec) ? kPark : kOuter;
    }

    // A warp owns a pool of kSlots photons in shared memory: a stack of photons in flight
    // growing up from the pool's first slot and one of photons parked at a real collision
    // growing down from its last; the slots between are free.  Each iteration takes up to
    // 32 photons off one stack, or starts up to 32 histories, does that kind's work in
    // all lanes and pushes every photon onto the stack of its new kind:
    //
    //   refill    new histories (source sampling, entry into the grid);
    //   interact  parked photons choose their interaction type and take it;
    //   step      photons in flight take Woodcock steps until no more than half of the
    //             lanes still fly (or woodcockSteps is reached).
    //
    // With two photons per lane some kind always holds most of a warp, so the kinds of
    // work, which diverge from each other, each run with nearly full warps, and no
    // photon's state lives in registers from one phase to the next.  Photons move between
    // phases as whole 64-byte states: the lanes read and write consecutive slots of four
    // float4 arrays, free of bank conflicts.  A history draws its uniforms in a fixed
    // order from its own stream, so its result does not depend on when, or in which lane,
    // its phases run.
    //
    // Issue bounds the kernel (about 85 % of the issue slots in steady state, 117 warp
    // instructions a history of the torso), with the L1/shared pipe next (28 to 30
    // wavefronts a history).  Against one photon per lane, parked in registers until enough lanes of a
    // warp waited: 13 -> 23 active lanes an instruction; 2e8 histories of the 256x256x200
    // torso 34.9 -> 26.0 ms, 3e8 of the 512x512x400 torso 67.7 -> 54.7 ms, 1e7 of the DX
    // cylinder 1.48 -> 1.26 ms (with the instances below and shorter arithmetic since: 22.5,
    // 50.1 and 1.15).  Measured beside it at that time: stacks of slot numbers in place of
    // moved photons (random slots conflict 2.5-fold: 25.9 / 53.5 / 1.33 ms), slots bound to
    // lanes by residue (no conflicts, fuller warps lost: 27.4 / 56.8 / 1.37 ms), 48
    // registers for 40 warps (spills: 33.5 ms), three blocks an SM (27.8 / 60.9 / 1.33 ms).
    // Batches of 28 parked photons or free slots: 24 and 32 measured within 1 %, 20 3 %
    // slower.  The step phase's end at half the lanes: 3/8 and 1/4 measured 2 % and 4 %
    // slower on the cylinder.  The last chunks of the queue shrink to 16 histories, which
    // spreads a short run over all warps: 1e5 histories 0.203 -> 0.115 ms.
    constexpr int kSlots = 64;

    constexpr size_t kPoolBytes = kSlots * 64 + 6 * 32 * sizeof(float) + 10 * sizeof(unsigned long long);

    // TAB: the block keeps the job's attenuation tables in shared memory, behind the pools.
    // SKIP: with cell bounds (J.cbound).  BOUND: correction level 2 (Doppler-broadened
    // Compton, fluorescence).  An instance each: asked at run time, the cell bounds and the
    // level-2 samplers held registers (the steps spilled) and issue slots where they are off.
    // 1e7 histories of the DX cylinder 1.26 -> 1.18 ms, 2e8 of the torso 24.9 -> 23.2, 3e8 of
    // the 512 x 512 x 400 torso 53.3 -> 51.2, 1e7 of a level-2 CBCT 3.65 -> 3.32.
    // blocks: the blocks that work on this job.
    template <bool PACKED, bool BOX, bool TAB, bool SKIP, bool BOUND>
    __device__ __forceinline__ void woodcockRun(const DevJob& J, unsigned long long h_end,
        DevCounters* __restrict__ ctr, int refillBatch, int interactBatch, int woodcockSteps, unsigned blocks)
    {
        extern __shared__ __align__(16) unsigned char sRaw[];
        const int lane = static_cast<int>(threadIdx.x & 31u);
        const unsigned ltMask = (1u << lane) - 1u;
        const int warps = static_cast<int>(blockDim.x >> 5);
        unsigned char* const base = sRaw + (threadIdx.x >> 5) * kPoolBytes;
        // slot state: A position, energy; B direction, weight; C generator; D in flight:
        // {packed, fe, majorant, its inverse}, parked: {packed, fe, voxel, material}
        float4* const A = reinterpret_cast<float4*>(base);
        float* const sums = reinterpret_cast<float*>(A + 4 * kSlots) + lane; // [2K] sum, [2K + 1] compensation, x 32
        unsigned long long* const counts = reinterpret_cast<unsigned long long*>(sums - lane + 6 * 32);
        float* const sTot = reinterpret_cast<float*>(sRaw + warps * kPoolBytes);

#pragma unroll
        for (int k = 0; k < 6; ++k)
            sums[32 * k] = 0.0f;
        if (lane < 10)
            counts[lane] = 0ull;
        if (TAB) {
            for (int i = static_cast<int>(threadIdx.x); i < J.n_mats * kTableNE; i += static_cast<int>(blockDim.x))
                sTot[i] = __ldg(&J.tot[i].x);
            __syncthreads();
        }

        int nFly = 0, nPark = 0;
        unsigned long long next = 0, end = 0; // the warp's history indices
        bool exhausted = false;
        unsigned visits = 0, skipped = 0, outerVisits = 0, err = 0;
        // half the warps' share of the histories left
        const float halfShare = 0.5f / static_cast<float>(blocks * static_cast<unsigned>(warps));

        const auto addSum = [&](int K, float x) { // Kahan step of the lane's sum K
            const float c = sums[32 * (2 * K + 1)], s0 = sums[32 * (2 * K)];
            const float y = x - c;
            const float t = s0 + y;
            sums[32 * (2 * K + 1)] = (t - s0) - y;
            sums[32 * (2 * K)] = t;
        };
        const auto count = [&](BlockCount c, unsigned mask) { // lane 0 only
            counts[c] += static_cast<unsigned long long>(__popc(mask));
        };
        const auto store = [&](int slot, const Photon& ph, const Rng& rng, unsigned packed, float fe, float z, float w) {
            float4* const p = A + slot;
            p[0] = make_float4(ph.px, ph.py, ph.pz, ph.E);
            p[kSlots] = make_float4(ph.dx, ph.dy, ph.dz, ph.w);
            p[2 * kSlots] = make_float4(__uint_as_float(rng.s0), __uint_as_float(rng.s1), __uint_as_float(rng.s2),
                __uint_as_float(rng.s3));
            p[3 * kSlots] = make_float4(__uint_as_float(packed), fe, z, w);
        };

        for (;;) {
            __syncwarp(); // the last phase's photons, for the other lanes
            // a full batch of parked photons or free slots first, else the larger stack
            const int nFree = next < end || !exhausted ? min(kSlots - nFly - nPark, 32) : 0;
            const bool refill = nFree > 0 && (nFree >= refillBatch || nFly + nPark == 0);
            if (refill && nPark < interactBatch) {
                // ---- refill
                unsigned long long avail = end - next, base2 = 0, avail2 = 0;
                if (avail < static_cast<unsigned long long>(nFree) && !exhausted) {
                    // a chunk of half the warp's share of what is left, 16 to kChunk histories:
                    // large ones cost few atomics, small ones near the end keep the warps level
                    if (lane == 0) {
                        const unsigned long long seen = *reinterpret_cast<volatile unsigned long long*>(&ctr->next);
                        const float left = seen < h_end ? static_cast<float>(h_end - seen) : 0.0f;
                        const unsigned long long size = static_cast<unsigned long long>(
                            fminf(fmaxf(left * halfShare, 16.0f), static_cast<float>(kChunk)));
                        base2 = atomicAdd(&ctr->next, size);
                        avail2 = base2 < h_end ? min(size, h_end - base2) : 0ull;
                    }
                    base2 = __shfl_sync(kFull, base2, 0);
                    avail2 = __shfl_sync(kFull, avail2, 0);
                    exhausted = avail2 == 0;
                }
                // the lane's history: of what was left, then of the new chunk
                const unsigned long long rank = static_cast<unsigned long long>(lane);
                const unsigned long long n = min(static_cast<unsigned long long>(nFree), avail + avail2);
                const bool start = rank < n;
                const unsigned long long h = rank < avail ? next + rank : base2 + (rank - avail);
                Photon ph;
                Rng rng;
                EnergyCache ec { 0, 0.0f, 0.0f, 0.0f };
                unsigned packed = kPackFresh;
                bool entered = false;
                if (start) {
                    rng.init(J.key, h);
                    sampleSource(J, h, ph, rng);
                    addSum(kSumSource, ph.w * ph.E);
                    entered = enterGrid(J, ph);
                    if (entered) {
                        gridPos(ph.E, ec.ie, ec.fe);
                        packed |= static_cast<unsigned>(ec.ie);
                        if (BOX
                            && outsideBox(J, __float2int_rd(ph.px * J.isp[0]), __float2int_rd(ph.py * J.isp[1]),
                                __float2int_rd(ph.pz * J.isp[2])))
                            packed |= kPackOuter;
                        else
                            ec.setMajorant(J.maj);
                    } else {
                        addSum(kSumEscaped, ph.w * ph.E);
                    }
                }
                if (n < avail) {
                    next += n;
                } else if (avail2 > 0) {
                    next = base2 + (n - avail);
                    end = base2 + avail2;
                } else {
                    next = end = 0;
                }
                const unsigned mIn = __ballot_sync(kFull, entered);
                if (entered)
                    store(nFly + __popc(mIn & ltMask), ph, rng, packed, ec.fe, ec.mmax, ec.invMmax);
                nFly += __popc(mIn);
                if (lane == 0) {
                    counts[cHist] += n;
                    counts[cMissed] += n - static_cast<unsigned long long>(__popc(mIn));
                }
            } else if (nPark > 0 && (nPark >= interactBatch || nPark > nFly)) {
                // ---- interact
                const int n = min(nPark, 32);
                const bool has = lane < n;
                const float4* const src = A + (kSlots - nPark + (has ? lane : 0));
                const float4 a = src[0], b = src[kSlots], c = src[2 * kSlots], d = src[3 * kSlots];
                nPark -= n;
                __syncwarp(); // before the pushes overwrite what other lanes read
                Photon ph { a.x, a.y, a.z, b.x, b.y, b.z, a.w, b.w };
                Rng rng { __float_as_uint(c.x), __float_as_uint(c.y), __float_as_uint(c.z), __float_as_uint(c.w) };
                const unsigned packed = __float_as_uint(d.x);
                EnergyCache ec { static_cast<int>(packed & 0x1ffu), d.y, 0.0f, 0.0f };
                const uint32_t pv = __float_as_uint(d.z);
                const int pm = __float_as_int(d.w);
                bool photo = false, compton = false, rayleigh = false, cut = false, fluor = false, error = false;
                bool alive = false, outer = false;
                if (has) {
                    const float4 x0 = __ldg(J.xs + pm * kTableNE + ec.ie);
                    const float4 x1 = __ldg(J.xs + pm * kTableNE + ec.ie + 1);
                    const float pe = fmaf(ec.fe, x1.x - x0.x, x0.x);
                    const float ic = fmaf(ec.fe, x1.y - x0.y, x0.y);
                    const float co = fmaf(ec.fe, x1.z - x0.z, x0.z);
                    const float rt = rng.u() * (pe + ic + co);
                    photo = rt < pe;
                    compton = !photo && rt < pe + ic;
                    rayleigh = !photo && !compton;
                    const bool atomic = BOUND && photo; // may emit fluorescence
                    error = (!photo || atomic) && (packed >> kPackSteps) > J.maxSteps;
                    if (error) {
                        err |= kErrStepLimit;
                    } else {
                        float Ep = ph.E;
                        if (!photo) {
                            float cost;
                            if (BOUND && compton) {
                                Ep = sampleCompton<true>(ph.E, J.mats + pm, J.ctab + pm * (kTableNE * kCTabK), ec.ie, ec.fe,
                                    2, rng, cost, err);
                            } else {
                                // one path for both: the angle from the kind's quantile table
                                const float omu = oneMinusCos((compton ? J.ctab : J.rtab) + pm * (kTableNE * kCTabK),
                                    ec.ie, ec.fe, rng.u());
                                cost = 1.0f - omu;
                                if (compton)
                                    Ep = ph.E * reciprocal(comptonRatio(ph.E, omu));
                            }
                            scatterDirection(ph.dx, ph.dy, ph.dz, cost, rng.u());
                            alive = true;
                        } else if (atomic) {
                            // correction level 2: the atom may emit a K-alpha photon, which is
                            // followed from the absorption point in an isotropic direction
                            Ep = samplePhotoFluorescence(ph.E, J.mats + pm, rng);
                            if (Ep > 0.0f) {
                                const float u1 = rng.u();
                                isotropicDirection(ph.dx, ph.dy, ph.dz, u1, rng.u());
                                alive = fluor = true;
                            }
                        } else {
                            Ep = 0.0f;
                        }
                        if (!rayleigh) {
                            const float e = ph.w * (ph.E - Ep);
                            deposit(J.tally, pv, e);
                            addSum(kSumDeposited, e);
                            ph.E = Ep;
                            if (compton && Ep < 1.0f) {
                                const float r = ph.w * Ep;
                                deposit(J.tally, pv, r);
                                addSum(kSumDeposited, r);
                                cut = true;
                                alive = false;
                            }
                        }
                        // Rayleigh keeps the flight's region, the others fly against maj again
                        outer = BOX && rayleigh && (packed & kPackOuter) != 0u;
                        if (!rayleigh)
                            gridPos(ph.E, ec.ie, ec.fe);
                        if (!outer)
                            ec.setMajorant(J.maj);
                    }
                }
                const unsigned mAlive = __ballot_sync(kFull, alive);
                if (alive)
                    store(nFly + __popc(mAlive & ltMask), ph, rng,
                        static_cast<unsigned>(ec.ie) | (outer ? kPackOuter : 0u) | (packed >> kPackSteps << kPackSteps),
                        ec.fe, ec.mmax, ec.invMmax);
                nFly += __popc(mAlive);
                const unsigned mFirst = __ballot_sync(kFull, has && (packed & kPackFresh) != 0u);
                const unsigned mP = __ballot_sync(kFull, photo);
                const unsigned mC = __ballot_sync(kFull, compton && !error);
                const unsigned mR = __ballot_sync(kFull, rayleigh && !error);
                const unsigned mRare = __ballot_sync(kFull, cut || fluor || error);
                if (lane == 0) {
                    count(cInteracted, mFirst);
                    count(cPhoto, mP);
                    count(cCompton, mC);
                    count(cRayleigh, mR);
                }
                if (mRare) {
                    const unsigned mCut = __ballot_sync(kFull, cut);
                    const unsigned mF = __ballot_sync(kFull, fluor);
                    const unsigned mErr = __ballot_sync(kFull, error);
                    if (lane == 0) {
                        count(cCutoff, mCut);
                        count(cFluorescence, mF);
                        count(cErrors, mErr);
                    }
                }
            } else if (nFly > 0) {
                // ---- step
                const int n = min(nFly, 32);
                const bool has = lane < n;
                nFly -= n;
                const float4* const src = A + (nFly + (has ? lane : 0));
                const float4 a = src[0], b = src[kSlots], c = src[2 * kSlots], d = src[3 * kSlots];
                __syncwarp(); // before the pushes overwrite what other lanes read
                Photon ph { a.x, a.y, a.z, b.x, b.y, b.z, a.w, b.w };
                Rng rng { __float_as_uint(c.x), __float_as_uint(c.y), __float_as_uint(c.z), __float_as_uint(c.w) };
                unsigned packed = __float_as_uint(d.x);
                EnergyCache ec { static_cast<int>(packed & 0x1ffu), d.y, d.z, d.w };
                uint32_t v = 0;
                int m = 0, to = has ? kFly : kFree;
                if (BOX) {
                    // photons outside the box first fly to it, out of the grid or to a collision
                    if (to == kFly && (packed & kPackOuter) != 0u) {
                        do {
                            const unsigned v0 = visits;
                            to = outerFlight<PACKED, TAB>(J, sTot, ph, rng, ec, v, m, visits);
                            outerVisits += visits - v0;
                            packed += 1u << kPackSteps;
                        } while (to == kOuter && (packed >> kPackSteps) <= J.maxSteps);
                        if (to == kFly)
                            packed &= ~kPackOuter;
                    }
                }
                for (int k = 0;;) {
                    if (to == kFly) {
                        to = woodcockStep<PACKED, BOX, TAB, SKIP>(J, sTot, ph, rng, ec, packed, v, m, visits, skipped);
                        packed += 1u << kPackSteps;
                    }
                    if (++k >= woodcockSteps || __popc(__ballot_sync(kFull, to == kFly)) <= (n >> 1))
                        break;
                }
                if (has && to == kFree)
                    addSum(kSumEscaped, ph.w * ph.E);
                bool on = to == kFly || (BOX && to == kOuter); // still in flight
                const bool error = on && (packed >> kPackSteps) > J.maxSteps;
                if (__any_sync(kFull, error)) {
                    const unsigned mErr = __ballot_sync(kFull, error);
                    if (lane == 0)
                        count(cErrors, mErr);
                    err |= error ? kErrStepLimit : 0u;
                    on = on && !error;
                }
                const bool real = to == kPark;
                const unsigned mOn = __ballot_sync(kFull, on), mReal = __ballot_sync(kFull, real);
                if (on || real)
                    store(real ? kSlots - 1 - nPark - __popc(mReal & ltMask) : nFly + __popc(mOn & ltMask), ph, rng,
                        packed, ec.fe, real ? __uint_as_float(v) : ec.mmax, real ? __int_as_float(m) : ec.invMmax);
                nFly += __popc(mOn);
                nPark += __popc(mReal);
            } else {
                break; // no photon and no history left
            }
        }

        // ---- flush: per-lane sums by warp, then one lane
        const unsigned long long vi = warpSum(static_cast<unsigned long long>(visits));
        const unsigned long long sk = warpSum(static_cast<unsigned long long>(skipped));
        const unsigned long long ov = BOX ? warpSum(static_cast<unsigned long long>(outerVisits)) : 0ull;
        double es[3];
#pragma unroll
        for (int k = 0; k < 3; ++k)
            es[k] = warpSum(static_cast<double>(sums[64 * k]) - static_cast<double>(sums[64 * k + 32]));
        const unsigned errAll = __reduce_or_sync(kFull, err);
        if (lane == 0) {
            atomicAdd(&ctr->visits, vi);
            if (sk)
                atomicAdd(&ctr->skipped, sk);
            if (ov)
                atomicAdd(&ctr->outer, ov);
            atomicAdd(&ctr->e_source, es[kSumSource]);
            atomicAdd(&ctr->e_escaped, es[kSumEscaped]);
            atomicAdd(&ctr->e_deposited, es[kSumDeposited]);
            if (errAll)
                atomicOr(&ctr->error_flags, errAll);
            flushCounts(ctr, counts);
        }
    }

    template <bool PACKED, bool BOX, bool TAB, bool SKIP, bool BOUND>
    __global__ void __launch_bounds__(256, 4) woodcockKernel(const DevJob J, unsigned long long h_end,
        DevCounters* __restrict__ ctr, int refillBatch, int interactBatch, int woodcockSteps)
    {
        woodcockRun<PACKED, BOX, TAB, SKIP, BOUND>(J, h_end, ctr, refillBatch, interactBatch, woodcockSteps,
            gridDim.x);
    }
    template <bool BOX, bool TAB, bool SKIP, bool BOUND>
    __global__ void __launch_bounds__(256, 4) woodcockPackKernel(const __grid_constant__ JobPack pack)
    {
        const int k = packJob(pack);
        const JobPack::Entry& e = pack.e[k];
        woodcockRun<true, BOX, TAB, SKIP, BOUND>(e.job, e.h_end, e.ctr, e.refill, e.interact, e.steps,
            pack.first[k + 1] - pack.first[k]);
    }

    template <bool BOX, bool TAB, bool SKIP>
    PackFn packByLevel(bool bound)
    {
        return bound ? woodcockPackKernel<BOX, TAB, SKIP, true> : woodcockPackKernel<BOX, TAB, SKIP, false>;
    }
    template <bool BOX>
    PackFn packInstance(bool tab, bool skip, bool bound)
    {
        if (skip)
            return tab ? packByLevel<BOX, true, true>(bound) : packByLevel<BOX, false, true>(bound);
        return tab ? packByLevel<BOX, true, false>(bound) : packByLevel<BOX, false, false>(bound);
    }

    template <bool PACKED, bool BOX, bool TAB, bool SKIP>
    TransportFn byLevel(bool bound)
    {
        return bound ? woodcockKernel<PACKED, BOX, TAB, SKIP, true> : woodcockKernel<PACKED, BOX, TAB, SKIP, false>;
    }
    template <bool PACKED, bool BOX>
    TransportFn instance(bool tab, bool skip, bool bound)
    {
        if constexpr (PACKED) // the unpacked layout has no cell bounds
            if (skip)
                return tab ? byLevel<true, BOX, true, true>(bound) : byLevel<true, BOX, false, true>(bound);
        return tab ? byLevel<PACKED, BOX, true, false>(bound) : byLevel<PACKED, BOX, false, false>(bound);
    }
} // namespace

// lanes a warp wants of a kind before it runs that kind's phase
extern const int kWoodcockRefillBatch = 28, kWoodcockInteractBatch = 28;

TransportFn woodcockKernelFor(bool packed, bool box, int n_mats, bool skip, bool bound)
{
    const bool tab = n_mats <= kSharedTableMaterials;
    if (packed)
        return box ? instance<true, true>(tab, skip, bound) : instance<true, false>(tab, skip, bound);
    return box ? instance<false, true>(tab, false, bound) : instance<false, false>(tab, false, bound);
}

PackFn woodcockPackFor(bool box, int n_mats, bool skip, bool bound)
{
    const bool tab = n_mats <= kSharedTableMaterials;
    return box ? packInstance<true>(tab, skip, bound) : packInstance<false>(tab, skip, bound);
}

size_t woodcockSharedBytes(int block, int n_mats)
{
    const size_t pools = static_cast<size_t>(block / 32) * kPoolBytes;
    const bool tab = n_mats <= kSharedTableMaterials;
    return pools + (tab ? static_cast<size_t>(n_mats) * kTableNE * sizeof(float) : 0);
}

// the tables and pools of 8 warps fit the 48 KB a launch may use without opting in
static_assert(8 * kPoolBytes + kSharedTableMaterials * kTableNE * sizeof(float) <= 48 * 1024, "shared memory");

} // namespace dxmcg
