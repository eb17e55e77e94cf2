// denoiser.hpp -- launchers of the denoiser kernels (denoiser_kernels.cu) and the
// network that drives them (denoiser.cpp).  Tensors are [B][D][H][W][C] bf16,
// C a multiple of 16; weights [Cout][27][Cin] bf16 with tap (dz+1)*9+(dy+1)*3+(dx+1).
#pragma once

#include <cstddef>
#include <cstdint>

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "engine.hpp"

namespace dxmcg {
namespace nn {

// Input of a convolution: channels [0, ca) from tensor a (at half resolution,
// nearest-upsampled on the fly, when halfA), channels [ca, ca + cb) from b.
struct ConvIn {
    const __nv_bfloat16* a = nullptr;
    int ca = 0;
    int halfA = 0;
    const __nv_bfloat16* b = nullptr;
    int cb = 0;
};

size_t conv3SmemBytes(int nt);
cudaError_t conv3Configure(); // opt the kernels into their shared-memory size (once per device)
cudaError_t wgradConfigure(); // the same for launchWgrad's (conv3Configure calls it)
int smCount();                // streaming multiprocessors of the device

// Options of the tcgen05 convolution beyond launchConv3's:
//   list:   device array of output-brick indices (conv3TcBrickDims, x fastest, then y,
//           z, batch) and *listLen, its length, on the device: only those bricks are
//           computed, the others' output is left as it was;
//   pooled: also the 2x2x2 average of the (bf16) output, as launchAvgPool gives it up
//           to the order of the eight additions (D, H, W even);
//   head:   for a 16-channel output, the 1x1x1 head (16 weights, then the bias) in
//           place of the output, exactly as launchHead without a target: headPred[v]
//           = the prediction, headOut[v] = it times headScale (either may be null);
//   mask:   the output where `mask` (its layout) is positive, 0 elsewhere: an input
//           gradient times the derivative of the ReLU whose output `mask` is;
//   handoverPolls: polls of each wait by which one role of the kernel hands work to
//           another before it gives up (0: 2^24); the waits for copies and MMAs already
//           in flight keep the default limit, so a kernel that gives up still returns
//           only after its own asynchronous work has landed.
struct ConvOptions {
    const int* list = nullptr;
    const int* listLen = nullptr;
    __nv_bfloat16* pooled = nullptr;
    const float* head = nullptr;
    float* headPred = nullptr;
    double* headOut = nullptr;
    double headScale = 1.0;
    const __nv_bfloat16* mask = nullptr;
    uint32_t handoverPolls = 0;
};

// tcgen05 (5th-generation tensor core) form of launchConv3 (conv_tc.cu): the same result,
// plus the optional epilogue work; w are the prepared weights (launchArrangeWeights)
cudaError_t conv3TcConfigure();
cudaError_t launchConv3Tc(const ConvIn& in, int B, int D, int H, int W, int Cin, const __nv_bfloat16* w,
    const float* bias, int Cout, bool relu, __nv_bfloat16* out, cudaStream_t s, const ConvOptions* ep = nullptr);
cudaError_t conv3TcErrors(unsigned* flags);
cudaError_t convErrorFlags(unsigned** flags); // where kernels set what conv3TcErrors reads
// whether the tcgen05 launch's own brick shape (conv3TcBrickDims, which a list goes by) has
// a CTA for every SM
bool conv3TcFills(int B, int D, int H, int W, int Cout);
// whether launchConv3Tc, which takes thinner bricks for smaller grids, is the faster one: not
// where launchConv3's smallest bricks leave SMs idle.  The network on 64^3, 32^3, 2 x 48^3 and
// 8 x 32^3 voxels: 153, 99, 155 and 156 us with the line at one such brick an SM; at two 168,
// 99, 171 and 162; tcgen05 everywhere 160, 122, 158 and 158.
bool conv3TcPays(int B, int D, int H, int W, int Cout);
int conv3SmallCtas(int B, int D, int H, int W, int Cout); // CTAs of launchConv3's smallest bricks
// the output bricks of the tcgen05 launch for this shape: (x, y, z) voxels per brick
// and the brick counts along x, y, z (per batch item)
void conv3TcBrickDims(int D, int H, int W, int Cout, int brick[3], int count[3]);
// Brick sets of the world path (one byte per brick, bricks x fastest, all on the device;
// the tissue set comes from launchPrepareInput's brick marks):
//   sets:     bricks of other brick grids (count per axis) that a marked brick needs: the
//             union over marked bricks (cx, cy, cz) of the boxes X(cx) x Y(cy) x Z(cz), where
//             `ranges` (device) holds for each output brick index b along x, then y, then z,
//             the range [lo, hi] of input brick indices whose interval holds b (lo > hi:
//             none); up to kMaxBrickLists sets at once (bits: brickBitWords(inCount) words
//             of scratch);
//   list:     the marked indices in increasing order, and how many (*listLen);
//             launchBrickLists compacts up to kMaxBrickLists masks in one launch.
constexpr int kMaxBrickLists = 12;
struct BrickSetJobs {
    uint8_t* mask[kMaxBrickLists] = {};
    const int* ranges[kMaxBrickLists] = {};
    int count[kMaxBrickLists][3] = {};
    int n = 0;
};
size_t brickBitWords(const int count[3]);
cudaError_t launchBrickSets(const uint8_t* in, const int inCount[3], uint32_t* bits, const BrickSetJobs& jobs,
    cudaStream_t s);
cudaError_t launchBrickList(const uint8_t* mask, int nb, int* list, int* listLen, cudaStream_t s);
struct BrickListJobs {
    const uint8_t* mask[kMaxBrickLists] = {};
    int* list[kMaxBrickLists] = {};
    int* len[kMaxBrickLists] = {};
    int nb[kMaxBrickLists] = {};
    int n = 0;
    void add(const uint8_t* m, int count, int* l, int* lenOut)
    {
        if (n < kMaxBrickLists) {
            mask[n] = m;
            nb[n] = count;
            list[n] = l;
            len[n] = lenOut;
        }
        ++n; // beyond kMaxBrickLists the launch refuses
    }
};
cudaError_t launchBrickLists(const BrickListJobs& jobs, cudaStream_t s);
// out = act(conv3(in) + bias), act = relu or identity; bias and mask (as ConvOptions') may
// be null
cudaError_t launchConv3(const ConvIn& in, int B, int D, int H, int W, int Cin, const __nv_bfloat16* w,
    const float* bias, int Cout, bool relu, __nv_bfloat16* out, cudaStream_t s,
    const __nv_bfloat16* mask = nullptr);
// dW[co][t][ci] += sum_v dz[v][co] x[v + off(t)][ci], db[co] += sum_v dz[v][co]  (FP32 atomics)
cudaError_t launchWgrad(const ConvIn& in, const __nv_bfloat16* dz, int B, int D, int H, int W, int Cin, int Cout,
    float* dW, float* db, cudaStream_t s);
cudaError_t launchAvgPool(const __nv_bfloat16* x, __nv_bfloat16* out, int B, int D, int H, int W, int C,
    cudaStream_t s);
// du (half res) = sum of children of dcat[:, :cu] where yu > 0; de = dcat[:, cu:] +
// dxNext(parent) / 8 where ye > 0 (either may be null); 0 elsewhere
cudaError_t launchSplitConcatGrad(const __nv_bfloat16* dcat, int cu, int cs, const __nv_bfloat16* dxNext,
    const __nv_bfloat16* yu, __nv_bfloat16* du, const __nv_bfloat16* ye, __nv_bfloat16* de, int B, int D, int H, int W,
    cudaStream_t s);
// head: pred = d . w + b; with a target also the L1 loss sum and the gradients (dd: of the
// last convolution before its ReLU, 0 where d is)
cudaError_t launchHead(const __nv_bfloat16* d, int C0, const float* hw, size_t nvox, const float* target,
    float* pred, double predScale, double* predOut, __nv_bfloat16* dd, float* dhw, double* lossSum, cudaStream_t s);
cudaError_t launchAdam(float* p, const float* g, float* m, float* v, __nv_bfloat16* pb, size_t n, float lr, float b1,
    float b2, float eps, float c1, float c2, cudaStream_t s);
cudaError_t launchToBf16(const float* p, __nv_bfloat16* pb, size_t n, cudaStream_t s);
// where the layers' weights lie in the parameter vector (w) and transposed (wt)
constexpr int kMaxLayers = 18;
struct LayerTable {
    int n = 0;
    int cout[kMaxLayers] = {}, cin[kMaxLayers] = {};
    size_t w[kMaxLayers] = {}, wt[kMaxLayers] = {};
};
// of every layer's weights: the input gradient's (wt: taps flipped, channels exchanged) and
// both as launchConv3Tc reads them (wPrep at the offsets of w, wtPrep at those of wt)
cudaError_t launchArrangeWeights(const __nv_bfloat16* w, __nv_bfloat16* wt, __nv_bfloat16* wPrep,
    __nv_bfloat16* wtPrep, const LayerTable& layers, cudaStream_t s);
// Bricks to mark while the input is prepared from a world: active[b] = 1 for each
// brick b holding a voxel whose material is not 0 (bricks of bx, by, bz voxels, cx and
// cy of them along x and y, x fastest; the grid nx voxels along x, ny along y).  The
// caller zeroes `active`.
struct BrickMarks {
    uint8_t* active = nullptr;
    int nx = 1, ny = 1, bx = 1, by = 1, bz = 1, cx = 1, cy = 1;
};
// input channels [log1p(d / s), density, one-hot(material 0..5), 0 x 8] from arrays
// (dose, dens, mat) or from a world (tally, vox, toDose); with a world, optionally
// the brick marks above (fewer than 2^32 voxels)
cudaError_t launchPrepareInput(const float* dose, const float* dens, const uint8_t* mat, const Tally* tally,
    const uint32_t* vox, DoseScale toDose, size_t n, float invScale, __nv_bfloat16* out, cudaStream_t s,
    const BrickMarks* marks = nullptr);
// patches outside their volume (or of a volume index out of range) are written as zeros
cudaError_t launchGatherPatches(const __nv_bfloat16* const* inputs, const float* const* targets, const int* dims,
    int nVolumes, const int* origins, int nPatch, int P, __nv_bfloat16* xin, float* tgt, cudaStream_t s);
cudaError_t launchDoseMean(const Tally* tally, const uint32_t* vox, double toDose, size_t n, float rhoMin,
    double* sum, unsigned long long* count, cudaStream_t s);

// a world's dose through the network (denoiser.cpp); dims nx, ny, nz (x fastest)
int denoiseWorld(dxmcg_denoiser* d, int device, const Tally* tally, const uint32_t* vox, int nx, int ny, int nz,
    DoseScale toDose, double scale, double* hostOut, double* scaleUsed, cudaStream_t s);

} // namespace nn
} // namespace dxmcg
