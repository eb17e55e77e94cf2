// transport_common.cuh -- what the transport kernels share (woodcock.cu: Woodcock
// tracking; transport.cu: exact Siddon flights and macro cells): event counters, the
// photon's cached majorant, voxel reads.
#pragma once

#include "device.cuh"

namespace dxmcg {
namespace {
    using namespace dev;

    constexpr int kChunk = 256; // histories a warp takes from the queue at once

    enum BlockCount : int {
        cHist,
        cMissed,
        cPhoto,
        cCompton,
        cRayleigh,
        cCutoff,
        cErrors,
        cInteracted,
        cFluorescence,
        cNum
    };

    __device__ __forceinline__ unsigned long long warpSum(unsigned long long v)
    {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            v += __shfl_xor_sync(kFull, v, o);
        return v;
    }
    __device__ __forceinline__ double warpSum(double v)
    {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            v += __shfl_xor_sync(kFull, v, o);
        return v;
    }

    constexpr int kSumSource = 0, kSumEscaped = 1, kSumDeposited = 2; // per-lane energy sums

    // The photon's energy-grid position and the majorant its next flight steps against.
    // reciprocal is the correctly rounded 1 / mmax, as a division gives (tables hold 1e-30 or
    // more).
    struct EnergyCache {
        int ie;
        float fe, mmax, invMmax;
        __device__ __forceinline__ void set(const DevJob& J, float E)
        {
            gridPos(E, ie, fe);
            setMajorant(J.maj);
        }
        __device__ __forceinline__ void setMajorant(const float2* maj)
        {
            mmax = lerp1(maj, ie, fe);
            invMmax = reciprocal(mmax);
        }
    };

    // Density and material of voxel v: one 4-byte word in the packed layout, or two
    // loads from caller-owned arrays in the unpacked layout.
    template <bool PACKED>
    __device__ __forceinline__ float voxelAt(const DevJob& J, uint32_t v, int& m)
    {
        if (PACKED) {
            const uint32_t word = __ldg(J.vox + v);
            m = static_cast<int>(word & 0xffu);
            return __uint_as_float(word & 0xffffff00u);
        }
        m = static_cast<int>(__ldg(J.mat + v));
        return __ldg(J.dens + v);
    }

    __device__ __forceinline__ void flushCounts(DevCounters* __restrict__ ctr, const unsigned long long* c)
    {
        atomicAdd(&ctr->histories, c[cHist]);
        atomicAdd(&ctr->missed, c[cMissed]);
        atomicAdd(&ctr->photo, c[cPhoto]);
        atomicAdd(&ctr->compton, c[cCompton]);
        atomicAdd(&ctr->rayleigh, c[cRayleigh]);
        atomicAdd(&ctr->cutoff, c[cCutoff]);
        atomicAdd(&ctr->errors, c[cErrors]);
        atomicAdd(&ctr->interacted, c[cInteracted]);
        if (c[cFluorescence])
            atomicAdd(&ctr->fluorescence, c[cFluorescence]);
    }

} // namespace

// Jobs that share a launch: block b works on job k with first[k] <= b < first[k + 1].  They
// are kernel parameters, so that a block reads its job from the constant bank, as it does
// where the launch has only one; kPackJobs of them stay below the 32,764 bytes a launch
// can pass.
constexpr int kPackJobs = kMaxPackedJobs;
struct JobPack {
    struct Entry {
        DevJob job;
        unsigned long long h_end;
        DevCounters* ctr;
        int refill, interact, steps;
    };
    int n;
    unsigned first[kPackJobs + 1];
    Entry e[kPackJobs];
};
static_assert(sizeof(JobPack) <= 32764, "kernel parameters");

namespace {
    // the job of this block (first[0] = 0, every job has a block)
    __device__ __forceinline__ int packJob(const JobPack& p)
    {
        int lo = 0, hi = p.n;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (p.first[mid] <= blockIdx.x)
                lo = mid;
            else
                hi = mid;
        }
        return lo;
    }
} // namespace

using TransportFn = void (*)(const DevJob, unsigned long long, DevCounters*, int, int, int);
using PackFn = void (*)(const JobPack);

// woodcock.cu: the Woodcock kernel's instance for a voxel layout, one region or two and
// n_mats materials (for several jobs: in the packed layout); its dynamic shared memory at a
// block size; its default batch sizes
TransportFn woodcockKernelFor(bool packed, bool box, int n_mats, bool skip, bool bound);
PackFn woodcockPackFor(bool box, int n_mats, bool skip, bool bound);
size_t woodcockSharedBytes(int block, int n_mats);
extern const int kWoodcockRefillBatch, kWoodcockInteractBatch;
// materials whose attenuation tables a block holds in shared memory: with the photon
// pools of 8 warps, as many as fit the 48 KB a launch may use without opting in
constexpr int kSharedTableMaterials = 6;

} // namespace dxmcg
