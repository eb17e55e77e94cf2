// denoiser_kernels.cu -- kernels of the dose denoiser (a 3D convolutional
// encoder-decoder trained on the transport's own low/high-history dose pairs).
// This part has no counterpart in the reference.
//
// Tensors are [B][D][H][W][C] bfloat16 with C a multiple of 16 ("channels last"),
// so that 16 channels of one voxel are one 32-byte row.  A 3x3x3 convolution is an
// implicit GEMM: rows = output voxels, columns = output channels, reduction =
// 27 taps x input channels.  A CTA owns an 8x8x8 brick of output voxels and
// NT output channels; per 16-channel slice of the input it stages the 10x10x10
// halo brick and the slice's weights in shared memory (cp.async, double
// buffered), and every tap then reads the same halo brick shifted by one voxel:
// each input element is fetched from global memory once per CTA instead of 27
// times.  The products run on the tensor cores as bf16 mma.sync m16n8k16 with
// FP32 accumulation; rows are loaded with ldmatrix from shared memory whose
// 16-byte halves are XOR-swizzled so that the eight rows of a matrix fall in
// distinct banks.
#include <algorithm>
#include <cstdint>

#include <cuda_bf16.h>

#include "chain.cuh"
#include "denoiser.hpp"
#include "device.cuh"

namespace dxmcg {
namespace nn {
namespace {

    constexpr int kHaloVox = 1000;            // 10 x 10 x 10
    constexpr int kHaloBytes = kHaloVox * 32; // 16 channels of bf16 per voxel

    __device__ __forceinline__ unsigned smemAddr(const void* p)
    {
        return static_cast<unsigned>(__cvta_generic_to_shared(p));
    }

    // 16-byte asynchronous copy global -> shared; zero fill when !valid (no read)
    __device__ __forceinline__ void cpAsync16(unsigned dst, const void* src, bool valid)
    {
        const int n = valid ? 16 : 0;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(n));
    }
    __device__ __forceinline__ void cpAsyncCommit() { asm volatile("cp.async.commit_group;\n" ::); }
    template <int N>
    __device__ __forceinline__ void cpAsyncWait()
    {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
    }

    __device__ __forceinline__ void ldsm4(unsigned addr, unsigned& r0, unsigned& r1, unsigned& r2, unsigned& r3)
    {
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                     : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                     : "r"(addr));
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

    __device__ __forceinline__ int tapDz(int t) { return t / 9 - 1; }
    __device__ __forceinline__ int tapDy(int t) { return (t / 3) % 3 - 1; }
    __device__ __forceinline__ int tapDx(int t) { return t % 3 - 1; }

    struct BrickPos {
        int b, z0, y0, x0;
    };
    __device__ __forceinline__ BrickPos brickOf(int brick, int D, int H, int W)
    {
        const int nbx = (W + 7) >> 3, nby = (H + 7) >> 3, nbz = (D + 7) >> 3;
        BrickPos p;
        p.x0 = (brick % nbx) * 8;
        brick /= nbx;
        p.y0 = (brick % nby) * 8;
        brick /= nby;
        p.z0 = (brick % nbz) * 8;
        p.b = brick / nbz;
        return p;
    }

    // Stage the halo brick of one 16-channel input slice: halo voxel v = (hz*10 + hy)*10
    // + hx holds its two 16-byte halves at v*32 + ((h ^ ((hx >> 2) & 1)) << 4).
    __device__ __forceinline__ void loadHalo(const ConvIn& in, int c0, const BrickPos& p, int D, int H, int W,
        unsigned sbase)
    {
        const bool inA = c0 < in.ca;
        const __nv_bfloat16* src = inA ? in.a : in.b;
        const int cs = inA ? in.ca : in.cb;
        const int cc = inA ? c0 : c0 - in.ca;
        const bool half = inA && in.halfA;
        const int Ds = half ? D >> 1 : D, Hs = half ? H >> 1 : H, Ws = half ? W >> 1 : W;
        for (int i = threadIdx.x; i < 2 * kHaloVox; i += blockDim.x) {
            const int v = i >> 1, h = i & 1;
            const int hz = v / 100, hy = (v / 10) % 10, hx = v % 10;
            const int gz = p.z0 + hz - 1, gy = p.y0 + hy - 1, gx = p.x0 + hx - 1;
            const bool ok = gz >= 0 && gz < D && gy >= 0 && gy < H && gx >= 0 && gx < W;
            const __nv_bfloat16* q = src;
            if (ok) {
                const int sz = half ? gz >> 1 : gz, sy = half ? gy >> 1 : gy, sx = half ? gx >> 1 : gx;
                q = src + ((((static_cast<size_t>(p.b) * Ds + sz) * Hs + sy) * Ws + sx) * cs + cc + h * 8);
            }
            cpAsync16(sbase + v * 32 + ((h ^ ((hx >> 2) & 1)) << 4), q, ok);
        }
    }

    // two channels at index `at` of a convolution's output, 0 where mask is not positive
    __device__ __forceinline__ void storePair(__nv_bfloat16* out, const __nv_bfloat16* mask, size_t at, float v0,
        float v1)
    {
        if (mask) {
            const float2 m = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(mask + at));
            v0 = m.x > 0.0f ? v0 : 0.0f;
            v1 = m.y > 0.0f ? v1 : 0.0f;
        }
        *reinterpret_cast<__nv_bfloat162*>(out + at) = __floats2bfloat162_rn(v0, v1);
    }

    // ------------------------------------------------------------------ forward conv
    template <int NT>
    __global__ void __launch_bounds__(256, 1) conv3Kernel(const ConvIn in, int D, int H, int W, int Cin,
        const __nv_bfloat16* __restrict__ wgt, const float* __restrict__ bias, int Cout, int relu,
        __nv_bfloat16* __restrict__ out, const __nv_bfloat16* __restrict__ mask)
    {
        extern __shared__ __align__(128) unsigned char smem[];
        constexpr int kWBytes = 27 * NT * 32;
        constexpr int kStage = kHaloBytes + kWBytes;
        const BrickPos p = brickOf(blockIdx.x, D, H, W);
        const int n0 = blockIdx.y * NT;
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const int nChunks = Cin >> 4;

        auto load = [&](int chunk, int stage) {
            const unsigned sbase = smemAddr(smem + stage * kStage);
            const int c0 = chunk * 16;
            loadHalo(in, c0, p, D, H, W, sbase);
            const unsigned wbase = sbase + kHaloBytes;
            for (int i = threadIdx.x; i < 27 * NT * 2; i += blockDim.x) {
                const int h = i & 1, row = i >> 1; // row = tap * NT + co
                const int tap = row / NT, co = row % NT;
                const bool ok = n0 + co < Cout;
                const __nv_bfloat16* q
                    = ok ? wgt + ((static_cast<size_t>(n0 + co) * 27 + tap) * Cin + c0 + h * 8) : wgt;
                cpAsync16(wbase + row * 32 + ((h ^ ((co >> 2) & 1)) << 4), q, ok);
            }
            cpAsyncCommit();
        };

        float acc[4][NT / 8][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < NT / 8; ++j)
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    acc[i][j][k] = 0.0f;

        const int q = lane >> 3, r = lane & 7;
        load(0, 0);
        for (int chunk = 0; chunk < nChunks; ++chunk) {
            if (chunk + 1 < nChunks) {
                load(chunk + 1, (chunk + 1) & 1);
                cpAsyncWait<1>();
            } else {
                cpAsyncWait<0>();
            }
            __syncthreads();
            const unsigned sbase = smemAddr(smem + (chunk & 1) * kStage);
            const unsigned wbase = sbase + kHaloBytes;
#pragma unroll 1
            for (int tap = 0; tap < 27; ++tap) {
                const int dz = tapDz(tap), dy = tapDy(tap), dx = tapDx(tap);
                unsigned bf[NT / 8][2];
#pragma unroll
                for (int j = 0; j < NT / 16; ++j) {
                    const int co = j * 16 + ((q >> 1) << 3) + r;
                    const int h = q & 1;
                    ldsm4(wbase + (tap * NT + co) * 32 + ((h ^ ((co >> 2) & 1)) << 4), bf[2 * j][0], bf[2 * j][1],
                        bf[2 * j + 1][0], bf[2 * j + 1][1]);
                }
                const int hz = warp + dz + 1, hx = r + dx + 1;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int hy = 2 * i + (q & 1) + dy + 1;
                    const int v = (hz * 10 + hy) * 10 + hx;
                    const int h = q >> 1;
                    unsigned a0, a1, a2, a3;
                    ldsm4(sbase + v * 32 + ((h ^ ((hx >> 2) & 1)) << 4), a0, a1, a2, a3);
#pragma unroll
                    for (int j = 0; j < NT / 8; ++j)
                        mma16816(acc[i][j], a0, a1, a2, a3, bf[j][0], bf[j][1]);
                }
            }
            __syncthreads(); // the next iteration's load reuses this stage
        }

        const int g = lane >> 2, t = lane & 3;
        const int z = p.z0 + warp;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                const int y = p.y0 + 2 * i + hf, x = p.x0 + g;
                if (z >= D || y >= H || x >= W)
                    continue;
                const size_t at = (((static_cast<size_t>(p.b) * D + z) * H + y) * W + x) * Cout;
#pragma unroll
                for (int j = 0; j < NT / 8; ++j) {
                    const int co = n0 + 8 * j + 2 * t;
                    if (co >= Cout)
                        continue;
                    float v0 = acc[i][j][2 * hf], v1 = acc[i][j][2 * hf + 1];
                    if (bias) {
                        v0 += bias[co];
                        v1 += bias[co + 1];
                    }
                    if (relu) {
                        v0 = fmaxf(v0, 0.0f);
                        v1 = fmaxf(v1, 0.0f);
                    }
                    storePair(out, mask, at + co, v0, v1);
                }
            }
    }

    // ------------------------------------------------------------------ forward conv, small grids
    // The same sums in the same order (input slices, then taps) on bricks of 8 x 4 x 2
    // voxels and 16 output channels: an eighth of conv3Kernel's brick and half its
    // channels, so that a volume of a few thousand voxels still gives every SM a CTA.  A
    // warp owns 16 voxels (8 x 2) and all 16 channels: a chain of 27 Cin / 16 dependent
    // MMAs (23 cycles each), with the fragments of tap t + 3 read while tap t multiplies
    // and the slices arriving through a ring of kSmallStages cp.async stages.  A slice
    // takes about 1 us, bound by the shared-memory pipe: two fragment loads and a share of
    // the copies for every two MMAs.
    constexpr int kSmallStages = 3;
    constexpr int kSmallHaloVox = 4 * 6 * 10;
    constexpr int kSmallHalo = kSmallHaloVox * 32;
    constexpr int kSmallStage = kSmallHalo + 27 * 16 * 32;

    __global__ void __launch_bounds__(128) conv3SmallKernel(const ConvIn in, int D, int H, int W, int Cin,
        const __nv_bfloat16* __restrict__ wgt, const float* __restrict__ bias, int Cout, int relu,
        __nv_bfloat16* __restrict__ out, const __nv_bfloat16* __restrict__ mask)
    {
        chain::afterPrevious();
        chain::letNextStart();
        extern __shared__ __align__(128) unsigned char smem[];
        const int nbx = (W + 7) >> 3, nby = (H + 3) >> 2, nbz = (D + 1) >> 1;
        int brick = static_cast<int>(blockIdx.x);
        const int x0 = (brick % nbx) * 8;
        brick /= nbx;
        const int y0 = (brick % nby) * 4;
        brick /= nby;
        const int z0 = (brick % nbz) * 2;
        const int bi = brick / nbz;
        const int n0 = blockIdx.y * 16;
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const int nChunks = Cin >> 4;
        // this thread's share of a slice, 16 bytes a copy: the halo voxels (tid >> 1) + 64 k
        // (their index in a full- and a half-resolution input, or -1) and the weight rows
        // tap = (tid >> 5) + 4 k of output channel (tid >> 1) & 15; half tid & 1
        constexpr int kHaloCopies = (2 * kSmallHaloVox + 127) / 128;
        constexpr int kWeightCopies = (27 * 16 * 2 + 127) / 128;
        const int tid = static_cast<int>(threadIdx.x), h = tid & 1;
        int full[kHaloCopies], low[kHaloCopies];
        unsigned haloDst[kHaloCopies];
#pragma unroll
        for (int k = 0; k < kHaloCopies; ++k) {
            const int v = (tid >> 1) + 64 * k;
            const int hz = v / 60, hy = (v / 10) % 6, hx = v % 10;
            const int gz = z0 + hz - 1, gy = y0 + hy - 1, gx = x0 + hx - 1;
            const bool ok = gz >= 0 && gz < D && gy >= 0 && gy < H && gx >= 0 && gx < W;
            full[k] = ok ? ((bi * D + gz) * H + gy) * W + gx : -1;
            low[k] = ok ? ((bi * (D >> 1) + (gz >> 1)) * (H >> 1) + (gy >> 1)) * (W >> 1) + (gx >> 1) : -1;
            haloDst[k] = static_cast<unsigned>(v * 32 + ((h ^ ((hx >> 2) & 1)) << 4));
        }
        const int wco = (tid >> 1) & 15;
        const unsigned wDst
            = static_cast<unsigned>(kSmallHalo + (tid >> 1) * 32 + ((h ^ ((wco >> 2) & 1)) << 4));
        const __nv_bfloat16* const wSrc
            = wgt + (static_cast<size_t>(n0 + wco) * 27 + (tid >> 5)) * Cin + h * 8;
        const auto load = [&](int chunk) {
            const unsigned sbase = smemAddr(smem + (chunk % kSmallStages) * kSmallStage);
            const int c0 = chunk * 16;
            const bool inA = c0 < in.ca;
            const int cs = inA ? in.ca : in.cb;
            const __nv_bfloat16* src = (inA ? in.a + c0 : in.b + (c0 - in.ca)) + h * 8;
            const bool half = inA && in.halfA;
#pragma unroll
            for (int k = 0; k < kHaloCopies; ++k) {
                const int v = half ? low[k] : full[k];
                if (k < kHaloCopies - 1 || tid + 128 * k < 2 * kSmallHaloVox)
                    cpAsync16(sbase + haloDst[k], src + (v >= 0 ? static_cast<size_t>(v) * cs : 0), v >= 0);
            }
#pragma unroll
            for (int k = 0; k < kWeightCopies; ++k)
                if (k < kWeightCopies - 1 || (tid >> 5) + 4 * k < 27)
                    cpAsync16(sbase + wDst + k * 64 * 32, wSrc + c0 + 4 * k * Cin, true);
        };

        const int q = lane >> 3, r = lane & 7;
        // lane's A rows: voxel x = r, y = 2 (warp & 1) + (q & 1), z = warp >> 1; half q >> 1
        unsigned aOff[3];
#pragma unroll
        for (int dx = 0; dx < 3; ++dx) {
            const int hx = r + dx;
            aOff[dx] = static_cast<unsigned>((((warp >> 1) * 6 + 2 * (warp & 1) + (q & 1)) * 10 + hx) * 32
                + (((q >> 1) ^ ((hx >> 2) & 1)) << 4));
        }
        // its B rows: output channel co, half q & 1
        const int bco = ((q >> 1) << 3) + r;
        const unsigned bOff = static_cast<unsigned>(kSmallHalo + bco * 32 + (((q & 1) ^ ((bco >> 2) & 1)) << 4));

        float acc[2][4] = {};
        for (int c = 0; c < kSmallStages - 1; ++c) {
            if (c < nChunks)
                load(c);
            cpAsyncCommit();
        }
        for (int chunk = 0; chunk < nChunks; ++chunk) {
            cpAsyncWait<kSmallStages - 2>();
            __syncthreads(); // slice `chunk` landed, and slice chunk - 1 was read by all
            if (chunk + kSmallStages - 1 < nChunks)
                load(chunk + kSmallStages - 1);
            cpAsyncCommit();
            const unsigned sbase = smemAddr(smem + (chunk % kSmallStages) * kSmallStage);
            unsigned a[4][4], b[4][4];
            const auto fragments = [&](int tap, unsigned (&fa)[4], unsigned (&fb)[4]) {
                const int dz = tap / 9, dy = (tap / 3) % 3, dx = tap % 3;
                ldsm4(sbase + aOff[dx] + (dz * 60 + dy * 10) * 32, fa[0], fa[1], fa[2], fa[3]);
                ldsm4(sbase + bOff + tap * 512, fb[0], fb[1], fb[2], fb[3]);
            };
#pragma unroll
            for (int tap = 0; tap < 3; ++tap)
                fragments(tap, a[tap], b[tap]);
#pragma unroll
            for (int tap = 0; tap < 27; ++tap) {
                const int k = tap & 3;
                if (tap + 3 < 27)
                    fragments(tap + 3, a[(tap + 3) & 3], b[(tap + 3) & 3]);
                mma16816(acc[0], a[k][0], a[k][1], a[k][2], a[k][3], b[k][0], b[k][1]);
                mma16816(acc[1], a[k][0], a[k][1], a[k][2], a[k][3], b[k][2], b[k][3]);
            }
        }

        const int g = lane >> 2, t = lane & 3;
        const int z = z0 + (warp >> 1), x = x0 + g;
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const int y = y0 + 2 * (warp & 1) + hf;
            if (z >= D || y >= H || x >= W)
                continue;
            const size_t at = (((static_cast<size_t>(bi) * D + z) * H + y) * W + x) * Cout + n0 + 2 * t;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                float v0 = acc[j][2 * hf], v1 = acc[j][2 * hf + 1];
                if (bias) {
                    v0 += bias[n0 + 8 * j + 2 * t];
                    v1 += bias[n0 + 8 * j + 2 * t + 1];
                }
                if (relu) {
                    v0 = fmaxf(v0, 0.0f);
                    v1 = fmaxf(v1, 0.0f);
                }
                storePair(out, mask, at + 8 * j, v0, v1);
            }
        }
    }

    // ------------------------------------------------------------------ elementwise passes
    __device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8])
    {
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float2 v = __bfloat1622float2(h[k]);
            f[2 * k] = v.x;
            f[2 * k + 1] = v.y;
        }
    }
    __device__ __forceinline__ uint4 pack8(const float (&f)[8])
    {
        uint4 u;
        __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
        for (int k = 0; k < 4; ++k)
            h[k] = __floats2bfloat162_rn(f[2 * k], f[2 * k + 1]);
        return u;
    }

    // f where y > 0, 0 elsewhere
    __device__ __forceinline__ void reluMask(float (&f)[8], const uint4& y)
    {
        float m[8];
        unpack8(y, m);
#pragma unroll
        for (int k = 0; k < 8; ++k)
            f[k] = m[k] > 0.0f ? f[k] : 0.0f;
    }

    // x_{l+1} = mean over the 2x2x2 children (half resolution output)
    __global__ void avgPoolKernel(const uint4* __restrict__ x, uint4* __restrict__ out, int B, int D, int H, int W,
        int groups)
    {
        chain::afterPrevious();
        chain::letNextStart();
        const int Dh = D >> 1, Hh = H >> 1, Wh = W >> 1;
        const size_t items = static_cast<size_t>(B) * Dh * Hh * Wh * groups;
        for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < items;
             i += static_cast<size_t>(gridDim.x) * blockDim.x) {
            const int g = static_cast<int>(i % groups);
            size_t v = i / groups;
            const int x0 = static_cast<int>(v % Wh) * 2;
            v /= Wh;
            const int y0 = static_cast<int>(v % Hh) * 2;
            v /= Hh;
            const int z0 = static_cast<int>(v % Dh) * 2;
            const size_t b = v / Dh;
            float s[8] = { 0, 0, 0, 0, 0, 0, 0, 0 };
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const size_t src = (((b * D + z0 + (c >> 2)) * H + y0 + ((c >> 1) & 1)) * W + x0 + (c & 1)) * groups + g;
                float f[8];
                unpack8(x[src], f);
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    s[k] += f[k];
            }
#pragma unroll
            for (int k = 0; k < 8; ++k)
                s[k] *= 0.125f;
            out[i] = pack8(s);
        }
    }

    // Gradient of the decoder's concat input, split: du (half resolution, channels
    // [0, cu)) = sum of the 2x2x2 children; de (full resolution, channels [cu, cu+cs))
    // = dcat + dxNext(parent) / 8, the skip path plus the pooled path of the encoder; both
    // through the ReLU they go back to (yu, ye: its outputs).
    __global__ void splitConcatGradKernel(const uint4* __restrict__ dcat, int gu, int gs,
        const uint4* __restrict__ dxNext, const uint4* __restrict__ yu, uint4* __restrict__ du,
        const uint4* __restrict__ ye, uint4* __restrict__ de, int B, int D, int H, int W)
    {
        chain::afterPrevious();
        chain::letNextStart();
        const int gc = gu + gs;
        const int Dh = D >> 1, Hh = H >> 1, Wh = W >> 1;
        const size_t nU = du ? static_cast<size_t>(B) * Dh * Hh * Wh * gu : 0;
        const size_t nE = de ? static_cast<size_t>(B) * D * H * W * gs : 0;
        const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
        for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < nU + nE; i += stride) {
            if (i < nU) {
                const int g = static_cast<int>(i % gu);
                size_t v = i / gu;
                const int x0 = static_cast<int>(v % Wh) * 2;
                v /= Wh;
                const int y0 = static_cast<int>(v % Hh) * 2;
                v /= Hh;
                const int z0 = static_cast<int>(v % Dh) * 2;
                const size_t b = v / Dh;
                float s[8] = { 0, 0, 0, 0, 0, 0, 0, 0 };
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const size_t src
                        = (((b * D + z0 + (c >> 2)) * H + y0 + ((c >> 1) & 1)) * W + x0 + (c & 1)) * gc + g;
                    float f[8];
                    unpack8(dcat[src], f);
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        s[k] += f[k];
                }
                reluMask(s, yu[i]);
                du[i] = pack8(s);
            } else {
                const size_t j = i - nU;
                const int g = static_cast<int>(j % gs);
                size_t v = j / gs;
                const int x = static_cast<int>(v % W);
                v /= W;
                const int y = static_cast<int>(v % H);
                v /= H;
                const int z = static_cast<int>(v % D);
                const size_t b = v / D;
                float a[8], n[8];
                unpack8(dcat[(((b * D + z) * H + y) * W + x) * gc + gu + g], a);
                unpack8(dxNext[(((b * Dh + (z >> 1)) * Hh + (y >> 1)) * Wh + (x >> 1)) * gs + g], n);
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    a[k] += n[k] * 0.125f;
                reluMask(a, ye[j]);
                de[j] = pack8(a);
            }
        }
    }

    // Head: pred = d . w + b per voxel; in training also the L1 loss and its
    // gradients (dd = g w through the ReLU that d comes from, dw += g d, db += g with g =
    // sign(pred - target) / N).
    template <int C0>
    __global__ void headKernel(const __nv_bfloat16* __restrict__ d, const float* __restrict__ hw, size_t nvox,
        const float* __restrict__ target, float invN, float* __restrict__ pred, double predScale,
        double* __restrict__ predOut, __nv_bfloat16* __restrict__ dd, float* __restrict__ dhw,
        double* __restrict__ lossSum)
    {
        chain::afterPrevious();
        chain::letNextStart();
        float w[C0];
#pragma unroll
        for (int c = 0; c < C0; ++c)
            w[c] = hw[c];
        const float b = hw[C0];
        float gw[C0];
#pragma unroll
        for (int c = 0; c < C0; ++c)
            gw[c] = 0.0f;
        float gb = 0.0f, loss = 0.0f;
        for (size_t v = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; v < nvox;
             v += static_cast<size_t>(gridDim.x) * blockDim.x) {
            float x[C0];
            const uint4* src = reinterpret_cast<const uint4*>(d + v * C0);
#pragma unroll
            for (int k = 0; k < C0 / 8; ++k) {
                float f[8];
                unpack8(src[k], f);
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    x[8 * k + j] = f[j];
            }
            float p = b;
#pragma unroll
            for (int c = 0; c < C0; ++c)
                p = fmaf(x[c], w[c], p);
            if (pred)
                pred[v] = p;
            if (predOut)
                predOut[v] = static_cast<double>(p) * predScale;
            if (target) {
                const float diff = p - target[v];
                loss += fabsf(diff);
                const float g = diff > 0.0f ? invN : (diff < 0.0f ? -invN : 0.0f);
                gb += g;
                float o[C0];
#pragma unroll
                for (int c = 0; c < C0; ++c) {
                    gw[c] = fmaf(g, x[c], gw[c]);
                    o[c] = x[c] > 0.0f ? g * w[c] : 0.0f;
                }
                uint4* dst = reinterpret_cast<uint4*>(dd + v * C0);
#pragma unroll
                for (int k = 0; k < C0 / 8; ++k) {
                    float f[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        f[j] = o[8 * k + j];
                    dst[k] = pack8(f);
                }
            }
        }
        if (!target)
            return;
        // warp sums, block sums, then one atomic per block and sum: the addresses are the same
        // for all, and one atomic per warp held the pass (8 x 64^3 voxels: 196 -> 38 us).  The
        // bias' own sum stays at an atomic per warp: its terms are all +-invN, round alike,
        // and in coarser steps it comes out up to 3e-5 of itself elsewhere.
        __shared__ float part[8][C0 + 1];
        const int warp = threadIdx.x >> 5;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            gb += __shfl_xor_sync(0xffffffffu, gb, o);
            loss += __shfl_xor_sync(0xffffffffu, loss, o);
#pragma unroll
            for (int c = 0; c < C0; ++c)
                gw[c] += __shfl_xor_sync(0xffffffffu, gw[c], o);
        }
        if ((threadIdx.x & 31) == 0) {
#pragma unroll
            for (int c = 0; c < C0; ++c)
                part[warp][c] = gw[c];
            part[warp][C0] = loss;
            atomicAdd(dhw + C0, gb);
        }
        __syncthreads();
        if (threadIdx.x < C0) {
            float v = 0.0f;
            for (int w = 0; w < 8; ++w)
                v += part[w][threadIdx.x];
            atomicAdd(dhw + threadIdx.x, v);
        } else if (threadIdx.x == C0) { // the loss: in FP64 from the warps' sums on
            double v = 0.0;
            for (int w = 0; w < 8; ++w)
                v += static_cast<double>(part[w][C0]);
            atomicAdd(lossSum, v);
        }
    }

    // Adam (Kingma & Ba 2015) on the FP32 master copy; writes the bf16 copy the
    // convolutions read.  c1 = 1 / (1 - beta1^t), c2 = 1 / (1 - beta2^t).
    __global__ void adamKernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
        float* __restrict__ v, __nv_bfloat16* __restrict__ pb, size_t n, float lr, float b1, float b2, float eps,
        float c1, float c2)
    {
        chain::afterPrevious();
        chain::letNextStart();
        for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
             i += static_cast<size_t>(gridDim.x) * blockDim.x) {
            const float gi = g[i];
            const float mi = b1 * m[i] + (1.0f - b1) * gi;
            const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
            m[i] = mi;
            v[i] = vi;
            const float pi = p[i] - lr * (mi * c1) / (sqrtf(vi * c2) + eps);
            p[i] = pi;
            pb[i] = __float2bfloat16_rn(pi);
        }
    }

    __global__ void toBf16Kernel(const float* __restrict__ p, __nv_bfloat16* __restrict__ pb, size_t n)
    {
        for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
             i += static_cast<size_t>(gridDim.x) * blockDim.x)
            pb[i] = __float2bfloat16_rn(p[i]);
    }

    // Copies of every layer's weights W[co][tap][ci]: for the input gradients
    // Wt[ci][tap][co] = W[co][26 - tap][ci], and the prepared forms of both (conv3Tc's:
    // [slice][in-plane tap][half][z-tap][output channel][8 input channels], z-taps from the
    // last to the first).  A thread moves 8 input channels of a (co, tap) for W and 8 output
    // channels of a (ci, tap) for Wt, lanes on neighbouring channels of the other kind.
    __global__ void arrangeWeightsKernel(const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ wt,
        __nv_bfloat16* __restrict__ wPrep, __nv_bfloat16* __restrict__ wtPrep, const LayerTable layers)
    {
        chain::afterPrevious();
        chain::letNextStart();
        const auto prepared = [](int tap, int c8, int n, int N) { // in units of 8 channels
            return (((c8 >> 1) * 9 + tap % 9) * 2 + (c8 & 1)) * 3 * N + (2 - tap / 9) * N + n;
        };
        for (int k = static_cast<int>(blockIdx.y); k < layers.n; k += static_cast<int>(gridDim.y)) {
            const int Cout = layers.cout[k], Cin = layers.cin[k];
            const __nv_bfloat16* const src = w + layers.w[k];
            const int n = Cout * 27 * Cin / 8;
            for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < 2 * n; j += gridDim.x * blockDim.x) {
                if (j < n) {
                    const int co = j % Cout, tap = (j / Cout) % 27, c8 = j / (Cout * 27);
                    reinterpret_cast<uint4*>(wPrep + layers.w[k])[prepared(tap, c8, co, Cout)]
                        = *reinterpret_cast<const uint4*>(src + (co * 27 + tap) * Cin + c8 * 8);
                } else {
                    const int i = j - n;
                    const int ci = i % Cin, tap = (i / Cin) % 27, c8 = i / (Cin * 27);
                    __align__(16) __nv_bfloat16 v[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        v[e] = src[((c8 * 8 + e) * 27 + (26 - tap)) * Cin + ci];
                    const uint4 u = *reinterpret_cast<const uint4*>(v);
                    *reinterpret_cast<uint4*>(wt + layers.wt[k] + (ci * 27 + tap) * Cout + c8 * 8) = u;
                    reinterpret_cast<uint4*>(wtPrep + layers.wt[k])[prepared(tap, c8, ci, Cin)] = u;
                }
            }
        }
    }

    // Network input channels for one volume: [log(1 + d / s), density, one-hot of
    // material 0..5, zeros]; d, density and material come either from arrays or
    // straight from a world (tally energy -> dose, packed voxel words), in which case
    // the bricks holding a non-air voxel are marked too when marks.active is set.
    __global__ void prepareInputKernel(const float* __restrict__ dose, const float* __restrict__ dens,
        const uint8_t* __restrict__ mat, const Tally* __restrict__ tally, const uint32_t* __restrict__ vox,
        DoseScale toDose, size_t n, float invScale, uint4* __restrict__ out, const BrickMarks marks)
    {
        for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
             i += static_cast<size_t>(gridDim.x) * blockDim.x) {
            float d, rho;
            int m;
            if (tally) {
                const uint32_t w = vox[i];
                rho = __uint_as_float(w & 0xffffff00u);
                m = static_cast<int>(w & 0xffu);
                // air (material 0) enters with zero dose, as the worker's readout deletes it
                d = rho > 0.0f && m != 0 ? static_cast<float>(tally[i].e * dev::doseFactor(toDose, w)) : 0.0f;
                if (marks.active && m != 0) {
                    const uint32_t v = static_cast<uint32_t>(i);
                    const uint32_t row = v / static_cast<uint32_t>(marks.nx);
                    const int x = static_cast<int>(v - row * static_cast<uint32_t>(marks.nx));
                    const int y = static_cast<int>(row % static_cast<uint32_t>(marks.ny));
                    const int z = static_cast<int>(row / static_cast<uint32_t>(marks.ny));
                    marks.active[x / marks.bx + marks.cx * (y / marks.by + marks.cy * (z / marks.bz))] = 1;
                }
            } else {
                d = dose[i];
                rho = dens[i];
                m = mat[i];
            }
            float f[8];
            f[0] = log1pf(fmaxf(d, 0.0f) * invScale);
            f[1] = rho;
#pragma unroll
            for (int k = 0; k < 6; ++k)
                f[2 + k] = m == k ? 1.0f : 0.0f;
            out[2 * i] = pack8(f);
            out[2 * i + 1] = make_uint4(0u, 0u, 0u, 0u);
        }
    }

    // Copy nPatch cubes of edge P from volumes (input 16 channels, target f32) at the
    // given origins into batch tensors.  origins[p] = {volume, z, y, x}.
    __global__ void gatherPatchesKernel(const uint4* const* __restrict__ inputs, const float* const* __restrict__ targets,
        const int* __restrict__ dims, int nVolumes, const int4* __restrict__ origins, int nPatch, int P,
        uint4* __restrict__ xin, float* __restrict__ tgt)
    {
        const size_t per = static_cast<size_t>(P) * P * P;
        const size_t items = per * nPatch * 3; // two 16-byte halves of input + one target per voxel
        for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < items;
             i += static_cast<size_t>(gridDim.x) * blockDim.x) {
            const int part = static_cast<int>(i % 3);
            const size_t v = i / 3;
            const int pt = static_cast<int>(v / per);
            const size_t w = v % per;
            const int x = static_cast<int>(w % P), y = static_cast<int>((w / P) % P), z = static_cast<int>(w / (P * P));
            const int4 o = origins[pt];
            bool ok = o.x >= 0 && o.x < nVolumes;
            int D = 0, H = 0, W = 0;
            if (ok) {
                D = dims[3 * o.x];
                H = dims[3 * o.x + 1];
                W = dims[3 * o.x + 2];
                ok = o.y >= 0 && o.z >= 0 && o.w >= 0 && o.y + z < D && o.z + y < H && o.w + x < W;
            }
            const size_t src = ok ? (static_cast<size_t>(o.y + z) * H + (o.z + y)) * W + (o.w + x) : 0;
            if (part < 2)
                xin[2 * v + part] = ok ? inputs[o.x][2 * src + part] : make_uint4(0u, 0u, 0u, 0u);
            else
                tgt[v] = ok ? targets[o.x][src] : 0.0f;
        }
    }

    // sum and count of the dose over voxels denser than rhoMin (the normalisation scale).
    // The factor toDose / rho is formed in FP32 (relative error ~1e-7, well inside what
    // a normalisation needs): an FP64 division per voxel made this pass FP64-bound.
    __global__ void doseMeanKernel(const Tally* __restrict__ tally, const uint32_t* __restrict__ vox, float toDose,
        size_t n, float rhoMin, double* __restrict__ sum, unsigned long long* __restrict__ count)
    {
        double s = 0.0;
        unsigned long long c = 0;
        for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
             i += static_cast<size_t>(gridDim.x) * blockDim.x) {
            const float rho = __uint_as_float(vox[i] & 0xffffff00u);
            if (rho > rhoMin) {
                s += tally[i].e * static_cast<double>(toDose / rho);
                ++c;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            s += __shfl_xor_sync(0xffffffffu, s, o);
            c += __shfl_xor_sync(0xffffffffu, c, o);
        }
        if ((threadIdx.x & 31) == 0 && c) {
            atomicAdd(sum, s);
            atomicAdd(count, c);
        }
    }

    int grid1d(size_t items)
    {
        const size_t blocks = (items + 255) / 256;
        const size_t cap = static_cast<size_t>(smCount()) * 8;
        return static_cast<int>(blocks < 1 ? 1 : (blocks < cap ? blocks : cap));
    }
} // namespace

int smCount()
{
    static const int sms = [] {
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        return n > 0 ? n : 1;
    }();
    return sms;
}

size_t conv3SmemBytes(int nt) { return 2 * static_cast<size_t>(kHaloBytes + 27 * nt * 32); }

cudaError_t conv3Configure()
{
    cudaError_t e = cudaFuncSetAttribute(conv3Kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
        static_cast<int>(conv3SmemBytes(16)));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(conv3Kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
            static_cast<int>(conv3SmemBytes(32)));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(conv3SmallKernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
            kSmallStages * kSmallStage);
    if (e == cudaSuccess)
        e = wgradConfigure();
    return e;
}

int conv3SmallCtas(int B, int D, int H, int W, int Cout)
{
    return B * ((D + 1) / 2) * ((H + 3) / 4) * ((W + 7) / 8) * (Cout / 16);
}

cudaError_t launchConv3(const ConvIn& in, int B, int D, int H, int W, int Cin, const __nv_bfloat16* w,
    const float* bias, int Cout, bool relu, __nv_bfloat16* out, cudaStream_t s, const __nv_bfloat16* mask)
{
    if (Cin % 16 || Cout % 16 || (in.ca % 16) || (in.b && in.cb % 16) || in.ca + (in.b ? in.cb : 0) != Cin)
        return cudaErrorInvalidValue;
    const int bricks = B * ((D + 7) / 8) * ((H + 7) / 8) * ((W + 7) / 8);
    // the small bricks where conv3Kernel would leave three quarters of the SMs without a
    // CTA (voxel indices are ints there).  8^3 voxels, 128 to 128 channels: 56 -> 12 us;
    // 8 x 8^3: 55 -> 36 us; 16^3, 192 to 64: 83 -> 22 us.  From a quarter of the SMs on,
    // conv3Kernel's reuse wins: 32^3, 96 to 32 channels (64 CTAs) 43 against 45 us, 8 x 16^3
    // 64 to 64 (128 CTAs) 30 against 51 us.
    if (4 * bricks * (Cout / (Cout % 32 == 0 ? 32 : 16)) <= smCount()
        && static_cast<size_t>(B) * D * H * W < (1ull << 31)) {
        const int small = conv3SmallCtas(B, D, H, W, Cout) / (Cout / 16);
        return chain::launchChained(conv3SmallKernel, dim3(small, Cout / 16), 128, kSmallStages * kSmallStage, s, in, D,
            H, W, Cin, w, bias, Cout, relu ? 1 : 0, out, mask);
    } else if (Cout % 32 == 0) {
        conv3Kernel<32><<<dim3(bricks, Cout / 32), 256, conv3SmemBytes(32), s>>>(in, D, H, W, Cin, w, bias, Cout,
            relu ? 1 : 0, out, mask);
    } else {
        conv3Kernel<16><<<dim3(bricks, Cout / 16), 256, conv3SmemBytes(16), s>>>(in, D, H, W, Cin, w, bias, Cout,
            relu ? 1 : 0, out, mask);
    }
    return cudaGetLastError();
}

cudaError_t launchAvgPool(const __nv_bfloat16* x, __nv_bfloat16* out, int B, int D, int H, int W, int C,
    cudaStream_t s)
{
    const size_t items = static_cast<size_t>(B) * (D / 2) * (H / 2) * (W / 2) * (C / 8);
    return chain::launchChained(avgPoolKernel, grid1d(items), 256, 0, s, reinterpret_cast<const uint4*>(x),
        reinterpret_cast<uint4*>(out), B, D, H, W, C / 8);
}

cudaError_t launchSplitConcatGrad(const __nv_bfloat16* dcat, int cu, int cs, const __nv_bfloat16* dxNext,
    const __nv_bfloat16* yu, __nv_bfloat16* du, const __nv_bfloat16* ye, __nv_bfloat16* de, int B, int D, int H, int W,
    cudaStream_t s)
{
    const size_t items = (du ? static_cast<size_t>(B) * (D / 2) * (H / 2) * (W / 2) * (cu / 8) : 0)
        + (de ? static_cast<size_t>(B) * D * H * W * (cs / 8) : 0);
    return chain::launchChained(splitConcatGradKernel, grid1d(items), 256, 0, s, reinterpret_cast<const uint4*>(dcat),
        cu / 8, cs / 8, reinterpret_cast<const uint4*>(dxNext), reinterpret_cast<const uint4*>(yu),
        reinterpret_cast<uint4*>(du), reinterpret_cast<const uint4*>(ye), reinterpret_cast<uint4*>(de), B, D, H, W);
}

cudaError_t launchHead(const __nv_bfloat16* d, int C0, const float* hw, size_t nvox, const float* target,
    float* pred, double predScale, double* predOut, __nv_bfloat16* dd, float* dhw, double* lossSum, cudaStream_t s)
{
    const float invN = nvox ? 1.0f / static_cast<float>(nvox) : 0.0f;
    const int g = grid1d(nvox);
    if (C0 != 16 && C0 != 32)
        return cudaErrorInvalidValue;
    return chain::launchChained(C0 == 16 ? headKernel<16> : headKernel<32>, g, 256, 0, s, d, hw, nvox, target, invN, pred,
        predScale, predOut, dd, dhw, lossSum);
}

cudaError_t launchAdam(float* p, const float* g, float* m, float* v, __nv_bfloat16* pb, size_t n, float lr, float b1,
    float b2, float eps, float c1, float c2, cudaStream_t s)
{
    return chain::launchChained(adamKernel, grid1d(n), 256, 0, s, p, g, m, v, pb, n, lr, b1, b2, eps, c1, c2);
}

cudaError_t launchToBf16(const float* p, __nv_bfloat16* pb, size_t n, cudaStream_t s)
{
    toBf16Kernel<<<grid1d(n), 256, 0, s>>>(p, pb, n);
    return cudaGetLastError();
}

cudaError_t launchArrangeWeights(const __nv_bfloat16* w, __nv_bfloat16* wt, __nv_bfloat16* wPrep,
    __nv_bfloat16* wtPrep, const LayerTable& layers, cudaStream_t s)
{
    return chain::launchChained(arrangeWeightsKernel, dim3(smCount(), std::max(1, layers.n)), 256, 0, s, w, wt, wPrep,
        wtPrep, layers);
}

cudaError_t launchPrepareInput(const float* dose, const float* dens, const uint8_t* mat, const Tally* tally,
    const uint32_t* vox, DoseScale toDose, size_t n, float invScale, __nv_bfloat16* out, cudaStream_t s,
    const BrickMarks* marks)
{
    const BrickMarks none {};
    const BrickMarks& bm = marks ? *marks : none;
    if (bm.active
        && (!tally || n >= (1ull << 32) || bm.nx < 1 || bm.ny < 1 || bm.bx < 1 || bm.by < 1 || bm.bz < 1
            || static_cast<size_t>(bm.nx) * bm.ny == 0 || n % (static_cast<size_t>(bm.nx) * bm.ny) != 0
            || bm.cx < (bm.nx + bm.bx - 1) / bm.bx || bm.cy < (bm.ny + bm.by - 1) / bm.by))
        return cudaErrorInvalidValue;
    prepareInputKernel<<<grid1d(n), 256, 0, s>>>(dose, dens, mat, tally, vox, toDose, n, invScale,
        reinterpret_cast<uint4*>(out), bm);
    return cudaGetLastError();
}

cudaError_t launchGatherPatches(const __nv_bfloat16* const* inputs, const float* const* targets, const int* dims,
    int nVolumes, const int* origins, int nPatch, int P, __nv_bfloat16* xin, float* tgt, cudaStream_t s)
{
    const size_t items = static_cast<size_t>(P) * P * P * nPatch * 3;
    gatherPatchesKernel<<<grid1d(items), 256, 0, s>>>(reinterpret_cast<const uint4* const*>(inputs), targets, dims,
        nVolumes, reinterpret_cast<const int4*>(origins), nPatch, P, reinterpret_cast<uint4*>(xin), tgt);
    return cudaGetLastError();
}

cudaError_t launchDoseMean(const Tally* tally, const uint32_t* vox, double toDose, size_t n, float rhoMin,
    double* sum, unsigned long long* count, cudaStream_t s)
{
    doseMeanKernel<<<grid1d(n), 256, 0, s>>>(tally, vox, static_cast<float>(toDose), n, rhoMin, sum, count);
    return cudaGetLastError();
}

} // namespace nn
} // namespace dxmcg
