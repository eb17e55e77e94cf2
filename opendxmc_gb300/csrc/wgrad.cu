// wgrad.cu -- weight and bias gradients of the dose denoiser's 3x3x3 convolutions.
// This part has no counterpart in the reference.
//
// dW[co][tap][ci] += sum over output voxels v of dz[v][co] * x[v + off(tap)][ci], and
// db[co] += sum of dz[v][co] (by the CTAs of input slice 0, from the same fragments).
// grid: x = CTAs looping over bricks of 8 x 8 x 8 voxels, y = 16-output-channel tile,
// z = 16-channel input slice.
//
// bf16 mma.sync with the voxels as the K dimension (for tcgen05 the channel counts, 16 at
// level 0, would be M and N: a quarter of its narrowest tile).  Its rate, one m16n8k16 per
// two cycles and SM, is the bound to reach.  So
//   * warp (p, g) owns the nine taps of z-plane p and the brick's z-slices 2 g, 2 g + 1: a
//     16-voxel step (two rows of 8) multiplies one fragment of dz with 9 x 2 fragments of x,
//     and of the four halo rows those need, two stay in registers from the step before: 4
//     ldmatrix.x4 for 18 MMAs (one tap a warp and step, re-reading dz for each, took 2 for 2);
//   * one thread fetches a brick with two TMA loads, two bricks ahead (the warps take turns:
//     always the same one held the others back, 74 us in place of 71), and the warps pass from
//     brick to brick on mbarriers.  When the threads copied the bricks themselves
//     (cp.async, nine copies each), their addresses and bounds took more issue slots than
//     the MMAs, and all warps took them at once, between two barriers;
//   * a half-resolution input is staged as it is, 6 x 6 x 6 voxels instead of 10 x 10 x 10,
//     and expanded by the addresses that ldmatrix gets.
// Halo rows are 12 (8) voxels of 32 bytes apart and the copies are swizzled, so that the
// eight rows of every matrix fall in distinct banks.  The four z-groups' sums meet in shared
// memory and leave by one atomic per four weights and CTA.
// 8 x 64^3 voxels: 16 to 16 channels 98 -> 71 us (48 at the MMA rate), 48 to 16 channels, 32
// of them from half resolution, 289 -> 204 us; 8 x 32^3, 96 to 32, 159 -> 110 us.
#include <algorithm>
#include <cstdint>

#include <cuda_bf16.h>

#include "chain.cuh"
#include "denoiser.hpp"
#include "tensor_map.hpp"
#include "umma.cuh"

namespace dxmcg {
namespace nn {
namespace {

    constexpr int kWarps = 12;
    constexpr int kThreads = 32 * kWarps;
    constexpr int kStages = 4; // two bricks on their way, one read, one that warps may still read
    constexpr int kAhead = 2;
    constexpr uint32_t kPolls = 1u << 24;

    // bytes of a brick's halo, of the half-resolution halo and of its dz
    constexpr int kRow = 12 * 32, kPlane = 10 * kRow, kHalo = 10 * kPlane;
    constexpr int kRowHalf = 8 * 32, kPlaneHalf = 6 * kRowHalf, kHaloHalf = 6 * kPlaneHalf;
    constexpr int kDz = 512 * 32;
    constexpr int kStage = kHalo + kDz;
    constexpr int kSumPitch = 27 * 16 + 8; // floats an output channel: no bank conflicts
    constexpr int kSmem = kStages * kStage + 256; // rounded up to the swizzle's 256 bytes
    static_assert(4 * 16 * kSumPitch * 4 <= kStages * kStage, "");
    static_assert(kHalo % 256 == 0 && kStage % 256 == 0 && kSmem <= 227 * 1024, "");
    // the swizzle goes by address bit 7; a plane and a pair of rows leave it as it is
    static_assert(kPlane % 256 == 0 && (2 * kRow) % 256 == 0 && kRow % 256 == 128, "");
    static_assert(kPlaneHalf % 256 == 0 && kRowHalf % 256 == 0, "");

    __device__ __forceinline__ void ldsm4t(uint32_t addr, unsigned& r0, unsigned& r1, unsigned& r2, unsigned& r3)
    {
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                     : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                     : "r"(addr)
                     : "memory");
    }
    // D = A (16x16, row) * B (16x8, col) + D, bf16 inputs, f32 accumulators
    __device__ __forceinline__ void mma16816(float (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3,
        unsigned b0, unsigned b1)
    {
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                     "{%0,%1,%2,%3};\n"
                     : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                     : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    }
    __device__ __forceinline__ float pairSum(unsigned p) // of two bf16
    {
        return __uint_as_float(p << 16) + __uint_as_float(p & 0xffff0000u);
    }

    // The warp's share of one staged brick: acc += its taps' products, sb += dz (of output
    // channels lane / 4 and lane / 4 + 8)
    template <bool HALF>
    __device__ __forceinline__ void brickProducts(uint32_t base, int plane, int group, int lane, bool bias,
        float (&acc)[9][2][4], float (&sb)[2])
    {
        const int q = lane >> 3, r = lane & 7;
        // this lane's rows: halo row q >> 1 of a pair, voxel r + dx, half q & 1; dz row q >> 1
        // of the step, voxel r, half q & 1
        uint32_t xOff[3];
#pragma unroll
        for (int dx = 0; dx < 3; ++dx) {
            const int hx = HALF ? (r + dx + 1) >> 1 : r + dx;
            const uint32_t at = static_cast<uint32_t>((q >> 1) * (HALF ? kRowHalf : kRow) + hx * 32);
            xOff[dx] = base + at + (((q & 1) ^ (at >> 7 & 1u)) << 4);
        }
        const uint32_t zAt = static_cast<uint32_t>(((q >> 1) * 8 + r) * 32);
        const uint32_t zOff = base + kHalo + zAt + (((q & 1) ^ (zAt >> 7 & 1u)) << 4);
#pragma unroll 1
        for (int s = 0; s < 2; ++s) {
            const int z = 2 * group + s;
            const int hz = z + plane;
            const uint32_t xz = static_cast<uint32_t>(HALF ? ((hz + 1) >> 1) * kPlaneHalf : hz * kPlane);
            const uint32_t zz = zOff + static_cast<uint32_t>(z) * (64 * 32);
            unsigned b[4][3][2]; // halo rows (rotating), dx, channel half
            const auto rows = [&](int hy) { // halo rows hy and hy + 1, hy even
#pragma unroll
                for (int dx = 0; dx < 3; ++dx)
                    ldsm4t(xOff[dx] + xz + (HALF ? (hy >> 1) * kRowHalf : hy * kRow), b[hy & 3][dx][0],
                        b[hy & 3][dx][1], b[(hy + 1) & 3][dx][0], b[(hy + 1) & 3][dx][1]);
            };
            // a step starts on what the step before fetched: its first six MMAs (dy = -1)
            // need dz and the two rows at hand, and cover the fetch of the next two
            unsigned a[2][4];
            ldsm4t(zz, a[0][0], a[0][1], a[0][2], a[0][3]);
            rows(0);
#pragma unroll
            for (int yb = 0; yb < 8; yb += 2) {
                const int u = yb >> 1 & 1;
                rows(yb + 2);
                if (yb < 6)
                    ldsm4t(zz + (yb + 2) * 256, a[u ^ 1][0], a[u ^ 1][1], a[u ^ 1][2], a[u ^ 1][3]);
                const unsigned a0 = a[u][0], a1 = a[u][1], a2 = a[u][2], a3 = a[u][3];
                if (bias) {
                    sb[0] += pairSum(a0) + pairSum(a2);
                    sb[1] += pairSum(a1) + pairSum(a3);
                }
#pragma unroll
                for (int t = 0; t < 9; ++t) {
                    const int dy = t / 3, dx = t % 3;
                    const int r0 = (yb + dy) & 3, r1 = (yb + dy + 1) & 3;
                    mma16816(acc[t][0], a0, a1, a2, a3, b[r0][dx][0], b[r1][dx][0]);
                    mma16816(acc[t][1], a0, a1, a2, a3, b[r0][dx][1], b[r1][dx][1]);
                }
            }
        }
    }

    // mapA, mapB: the inputs (a at half resolution with in.halfA), mapZ: dz.  *errors is set
    // when a wait ran out; the sums are then wrong.
    __global__ void __launch_bounds__(kThreads, 1) wgradKernel(const __grid_constant__ CUtensorMap mapA,
        const __grid_constant__ CUtensorMap mapB, const __grid_constant__ CUtensorMap mapZ, int ca, int halfA, int D,
        int H, int W, int Cin, int nBricks, float* __restrict__ dW, float* __restrict__ db, unsigned* errors)
    {
        extern __shared__ __align__(256) unsigned char smemRaw[];
        __shared__ __align__(8) uint64_t full[kStages];  // stage landed
        __shared__ __align__(8) uint64_t empty[kStages]; // every warp is done with it
        __shared__ int abortFlag;
        __shared__ int fetched; // bricks asked for (read after a wait ran out)
        const uint32_t base = (umma::smemAddr(smemRaw) + 255u) & ~255u;
        const int n0 = blockIdx.y * 16;
        const int c0 = blockIdx.z * 16;
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const int plane = warp % 3, group = warp / 3;
        const bool inA = c0 < ca;
        const bool half = inA && halfA;
        volatile int* abortp = &abortFlag;
        if (threadIdx.x == 0) {
            for (int i = 0; i < kStages; ++i) {
                umma::mbarInit(&full[i], 1);
                umma::mbarInit(&empty[i], kWarps);
            }
            abortFlag = 0;
            fetched = 0;
        }
        umma::fenceProxyAsync();
        __syncthreads();
        chain::afterPrevious();
        chain::letNextStart();

        const int first = static_cast<int>(blockIdx.x), hop = static_cast<int>(gridDim.x);
        const int mine = first < nBricks ? (nBricks - 1 - first) / hop + 1 : 0;
        // brick i of this CTA into stage i % kStages, once all warps are done with the brick
        // that was there
        const auto fetch = [&](int i) {
            const int st = i % kStages, use = i / kStages;
            if (use > 0 && !umma::mbarWaitOrAbort(&empty[st], static_cast<uint32_t>(use - 1) & 1u, kPolls, abortp))
                return false;
            int v = first + i * hop;
            const int nbx = (W + 7) >> 3, nby = (H + 7) >> 3, nbz = (D + 7) >> 3;
            const int x0 = (v % nbx) * 8;
            v /= nbx;
            const int y0 = (v % nby) * 8;
            v /= nby;
            const int z0 = (v % nbz) * 8, b = v / nbz;
            const uint32_t dst = base + st * kStage;
            umma::mbarArriveExpectTx(&full[st], (half ? kHaloHalf : kHalo) + kDz);
            if (half)
                umma::tmaLoad5d(dst, &mapA, c0, (x0 >> 1) - 1, (y0 >> 1) - 1, (z0 >> 1) - 1, b, &full[st]);
            else
                umma::tmaLoad5d(dst, inA ? &mapA : &mapB, inA ? c0 : c0 - ca, x0 - 1, y0 - 1, z0 - 1, b, &full[st]);
            umma::tmaLoad5d(dst + kHalo, &mapZ, n0, x0, y0, z0, b, &full[st]);
            atomicMax(&fetched, i + 1);
            return true;
        };

        float acc[9][2][4];
#pragma unroll
        for (int t = 0; t < 9; ++t)
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    acc[t][n][k] = 0.0f;
        const bool bias = blockIdx.z == 0 && plane == 0;
        float sb[2] = { 0.0f, 0.0f };

        if (threadIdx.x == 0)
            for (int i = 0; i < kAhead && i < mine; ++i)
                fetch(i);
        __syncwarp();
        for (int i = 0; i < mine; ++i) {
            // the warps fetch in turn
            if (i + kAhead < mine && warp == i % kWarps) {
                if (lane == 0 && !fetch(i + kAhead))
                    *abortp = 1;
                __syncwarp();
            }
            const int st = i % kStages;
            const bool there
                = umma::mbarWaitOrAbort(&full[st], static_cast<uint32_t>(i / kStages) & 1u, kPolls, abortp);
            if (!__all_sync(0xffffffffu, there)) {
                *abortp = 1;
                break;
            }
            if (half)
                brickProducts<true>(base + st * kStage, plane, group, lane, bias, acc, sb);
            else
                brickProducts<false>(base + st * kStage, plane, group, lane, bias, acc, sb);
            __syncwarp();
            if (lane == 0)
                umma::mbarArrive(&empty[st]);
        }

        // the z-groups' sums meet, then one atomic per four weights
        float* sum = reinterpret_cast<float*>(smemRaw); // [group][16 co][27 taps][16 ci]
        const int g = lane >> 2, tq = lane & 3;
        __syncthreads(); // every warp is done with the stages
        if (abortFlag) { // loads may still be on their way
            if (threadIdx.x == 0)
                for (int i = max(0, fetched - kStages); i < fetched; ++i)
                    umma::mbarWait(&full[i % kStages], static_cast<uint32_t>(i / kStages) & 1u, kPolls);
            __syncthreads();
        }
#pragma unroll
        for (int t = 0; t < 9; ++t)
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int k = 0; k < 2; ++k)
                    *reinterpret_cast<float2*>(sum + (group * 16 + g + 8 * k) * kSumPitch + (9 * plane + t) * 16 + n * 8
                        + 2 * tq)
                        = make_float2(acc[t][n][2 * k], acc[t][n][2 * k + 1]);
        __syncthreads();
        for (int j = threadIdx.x; j < 16 * 27 * 4; j += kThreads) {
            const int co = j / (27 * 4), w = j % (27 * 4); // w: tap and ci / 4
            const float4* v = reinterpret_cast<const float4*>(sum + co * kSumPitch) + w;
            float4 f = v[0];
#pragma unroll
            for (int k = 1; k < 4; ++k) {
                const float4 o = v[k * 16 * (kSumPitch / 4)];
                f.x += o.x;
                f.y += o.y;
                f.z += o.z;
                f.w += o.w;
            }
            atomicAdd(reinterpret_cast<float4*>(dW + static_cast<size_t>((n0 + co) * 27 + (w >> 2)) * Cin + c0)
                    + (w & 3),
                f);
        }
        if (bias) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                sb[j] += __shfl_xor_sync(0xffffffffu, sb[j], 1);
                sb[j] += __shfl_xor_sync(0xffffffffu, sb[j], 2);
                if (tq == 0)
                    atomicAdd(db + n0 + g + 8 * j, sb[j]);
            }
        }
        if (threadIdx.x == 0) {
            if (abortFlag)
                atomicOr(errors, 1u);
            for (int k = 0; k < kStages; ++k) {
                umma::mbarInval(&full[k]);
                umma::mbarInval(&empty[k]);
            }
        }
    }

} // namespace

cudaError_t wgradConfigure()
{
    return cudaFuncSetAttribute(wgradKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
}

cudaError_t launchWgrad(const ConvIn& in, const __nv_bfloat16* dz, int B, int D, int H, int W, int Cin, int Cout,
    float* dW, float* db, cudaStream_t s)
{
    if (Cin % 16 || Cout % 16 || in.ca % 16 || (in.b && in.cb % 16) || in.ca + (in.b ? in.cb : 0) != Cin
        || (in.halfA && ((D | H | W) & 1)))
        return cudaErrorInvalidValue;
    CUtensorMap mapA {}, mapB {}, mapZ {};
    const int sh = in.halfA ? 1 : 0;
    if (!brickTensorMap(&mapA, in.a, B, D >> sh, H >> sh, W >> sh, in.ca, sh ? 8 : 12, sh ? 6 : 10, sh ? 6 : 10)
        || (in.b && !brickTensorMap(&mapB, in.b, B, D, H, W, in.cb, 12, 10, 10))
        || !brickTensorMap(&mapZ, dz, B, D, H, W, Cout, 8, 8, 8))
        return cudaErrorInvalidValue;
    unsigned* errors = nullptr;
    const cudaError_t e = convErrorFlags(&errors);
    if (e != cudaSuccess)
        return e;
    const int bricks = B * ((D + 7) / 8) * ((H + 7) / 8) * ((W + 7) / 8);
    const int tiles = (Cout / 16) * (Cin / 16);
    // one CTA an SM: as many per tile as fill the SMs once
    const int gx = std::max(1, std::min(bricks, smCount() / tiles));
    return chain::launchChained(wgradKernel, dim3(gx, Cout / 16, Cin / 16), kThreads, kSmem, s, mapA, mapB, mapZ, in.ca,
        in.halfA ? 1 : 0, D, H, W, Cin, bricks, dW, db, errors);
}

} // namespace nn
} // namespace dxmcg
