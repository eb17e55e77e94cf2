// Device functions of the transport against what they stand in for: the arithmetic forms
// against CUDA's functions for every float of their ranges, and the bound-electron samplers
// against their plain loops.  Prints a line a check, "name mismatches of total"; exits 0.
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include <cuda_runtime.h>

#include "../../opendxmc_gb300/csrc/device.cuh"

using namespace dxmcg;
using namespace dxmcg::dev;

namespace {

enum Form { kReciprocal, kSquareRoot, kUnitRsqrt, kNegLog };

template <int FORM>
__global__ void compareForms(uint32_t first, unsigned long long n, unsigned long long* bad)
{
    unsigned long long wrong = 0;
    for (unsigned long long i = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<unsigned long long>(gridDim.x) * blockDim.x) {
        float got, want;
        if (FORM == kNegLog) {
            const float u = toUniform(static_cast<uint32_t>(i) << 9); // i: the uniform's 23 bits
            got = negLog(u);
            want = -__logf(u);
        } else {
            const float x = __uint_as_float(first + static_cast<uint32_t>(i));
            got = FORM == kReciprocal ? reciprocal(x) : (FORM == kSquareRoot ? squareRoot(x) : unitRsqrt(x));
            want = FORM == kReciprocal ? __frcp_rn(x) : (FORM == kSquareRoot ? __fsqrt_rn(x) : rsqrtf(x));
        }
        wrong += __float_as_uint(got) != __float_as_uint(want);
    }
    if (wrong)
        atomicAdd(bad, wrong);
}

// dopplerEnergy as a plain loop: the shell by two passes over the shells, every draw tried
template <bool FUSED, class U>
__device__ bool plainDoppler(float E, float A, float omu, const DevMaterial* M, U& r, float& Ep)
{
    float tot = 0.0f;
    for (int k = 0; k < M->nShell; ++k)
        if (M->shellBinding[k] < E)
            tot += M->shellElectrons[k];
    const float target = r.u() * tot;
    int sh = -1;
    float acc = 0.0f;
    for (int k = 0; k < M->nShell; ++k)
        if (M->shellBinding[k] < E) {
            sh = k;
            acc += M->shellElectrons[k];
            if (target <= acc)
                break;
        }
    if (sh < 0)
        return false;
    const float c = 1.0f - omu, am = A - c, sin2 = omu * (2.0f - omu);
    for (int t = 0; t < kPzTries; ++t) {
        const float a = 2.0f * r.u() - 1.0f;
        const float b = 2.0f * r.u() - 1.0f;
        const float w = __fmaf_rn(a, a, __fmul_rn(b, b));
        if (w >= 1.0f)
            continue;
        const float rho = M->shellMomentum[sh] * a * sqrtf((powf(w, -0.4f) - 1.0f) / w);
        const float rho2 = __fmul_rn(rho, rho);
        const float den = FUSED ? __fmaf_rn(A, A, -rho2) : __fsub_rn(__fmul_rn(A, A), rho2);
        const float rest = __fsub_rn(1.0f, rho2);
        const float disc
            = FUSED ? __fmaf_rn(am, am, __fmul_rn(sin2, rest)) : __fmaf_rn(sin2, rest, __fmul_rn(am, am));
        if (!(den > 0.0f) || !(disc >= 0.0f))
            continue;
        const float e1 = E * (__fmaf_rn(rho, sqrtf(disc), __fmaf_rn(-rho2, c, A)) / den);
        if (e1 > 0.0f && E - e1 > M->shellBinding[sh]) {
            Ep = e1;
            return true;
        }
    }
    return false;
}

// per draw: energy 1 to 150 keV and an angle; the same uniforms to both forms
template <bool FUSED>
__global__ void compareSamplers(const DevMaterial* mats, int nMats, int n, unsigned long long* badDoppler,
    unsigned long long* badFluorescence, unsigned long long* taken)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const DevMaterial* M = mats + i % nMats;
        Rng seed;
        seed.init(77ull, static_cast<unsigned long long>(i));
        const float E = expf(seed.u() * 5.0106f), omu = 2.0f * seed.u() * seed.u();
        Rng a = seed, b = seed;
        float ea = 0.0f, eb = 0.0f;
        const float A = comptonRatio(E, omu);
        const bool ta = dopplerEnergy<FUSED>(E, A, omu, M, a, ea), tb = plainDoppler<FUSED>(E, A, omu, M, b, eb);
        // taken or not, the energy, and the uniforms used (the generators' states)
        if (ta != tb || __float_as_uint(ea) != __float_as_uint(eb) || a.s0 != b.s0 || a.s3 != b.s3)
            atomicAdd(badDoppler, 1ull);
        if (ta)
            atomicAdd(taken, 1ull);
        // material nMats + k is material k with an edge above every energy: the plain loop
        a = b = seed;
        ea = samplePhotoFluorescence(E, M, a);
        eb = samplePhotoFluorescence(E, M + nMats, b);
        if (__float_as_uint(ea) != __float_as_uint(eb) || a.s0 != b.s0 || a.s3 != b.s3)
            atomicAdd(badFluorescence, 1ull);
    }
}

struct Lcg {
    unsigned long long s;
    double u() { return static_cast<double>((s = s * 6364136223846793005ull + 1442695040888963407ull) >> 11) * 0x1p-53; }
};

// a material of random shells, K and L edges and shares, with the running sums of its definition
DevMaterial randomMaterial(Lcg& r, int elements)
{
    DevMaterial d {};
    d.n = elements;
    d.nShell = 3 * elements;
    d.invJumpK = 0.15f;
    d.invJumpL = 0.4f;
    float acc = 0.0f;
    for (int i = 0; i < d.n; ++i) {
        d.nZ4[i] = static_cast<float>(std::exp(6.0 * r.u()));
        d.eK[i] = static_cast<float>(std::exp(4.5 * r.u()));
        d.eL[i] = d.eK[i] * 0.15f;
        d.kAlpha[i] = 0.9f * d.eK[i];
        d.omegaK[i] = static_cast<float>(r.u());
        d.z4Cum[i] = acc += d.nZ4[i];
        d.edgeTop = std::fmax(d.edgeTop, std::fmax(d.eK[i], d.eL[i]));
    }
    acc = 0.0f;
    for (int k = 0; k < d.nShell; ++k) {
        d.shellElectrons[k] = static_cast<float>(0.01 + 8.0 * r.u() * r.u());
        d.shellBinding[k] = static_cast<float>(0.005 * std::exp(9.5 * r.u()));
        d.shellMomentum[k] = static_cast<float>(0.005 * std::exp(5.0 * r.u()));
        d.shellCum[k] = acc += d.shellElectrons[k];
        d.shellTop = std::fmax(d.shellTop, d.shellBinding[k]);
    }
    for (int c = 0; c < 64; ++c) {
        int k = 0;
        while (k + 1 < d.nShell && static_cast<float>(c) * 0.015625f * acc > d.shellCum[k])
            ++k;
        d.shellStart[c] = static_cast<uint8_t>(k);
    }
    return d;
}

unsigned long long take(unsigned long long* p)
{
    unsigned long long v = 0;
    if (cudaMemcpy(&v, p, sizeof v, cudaMemcpyDeviceToHost) != cudaSuccess)
        std::exit(2);
    cudaMemset(p, 0, sizeof v);
    return v;
}

uint32_t bits(float x)
{
    uint32_t b;
    std::memcpy(&b, &x, sizeof b);
    return b;
}

template <int FORM>
void forms(const char* name, float lo, float hi, unsigned long long* bad) // lo <= x < hi
{
    const unsigned long long n = FORM == kNegLog ? 1ull << 23 : bits(hi) - bits(lo);
    compareForms<FORM><<<2048, 256>>>(bits(lo), n, bad);
    std::printf("%s %llu of %llu\n", name, take(bad), n);
}

} // namespace

int main()
{
    unsigned long long* c = nullptr;
    if (cudaMalloc(&c, 3 * sizeof *c) != cudaSuccess || cudaMemset(c, 0, 3 * sizeof *c) != cudaSuccess)
        return 2;
    forms<kReciprocal>("reciprocal", 0x1p-112f, 0x1p107f, c);
    forms<kSquareRoot>("squareRoot", 0x1p-102f, 0x1p107f, c);
    forms<kSquareRoot>("squareRootOfZero", 0.0f, FLT_TRUE_MIN, c);
    forms<kUnitRsqrt>("unitRsqrt", 0.25f, 4.0f, c);
    forms<kNegLog>("negLog", 0.0f, 0.0f, c);

    Lcg r { 5ull };
    constexpr int kMats = 64, kDraws = 1 << 23;
    std::vector<DevMaterial> mats;
    for (int k = 0; k < kMats; ++k)
        mats.push_back(randomMaterial(r, 1 + k % DXMCG_MAX_ELEMENTS));
    for (int k = 0; k < kMats; ++k) {
        mats.push_back(mats[k]);
        mats.back().edgeTop = FLT_MAX;
    }
    DevMaterial* m = nullptr;
    if (cudaMalloc(&m, mats.size() * sizeof *m) != cudaSuccess
        || cudaMemcpy(m, mats.data(), mats.size() * sizeof *m, cudaMemcpyHostToDevice) != cudaSuccess)
        return 2;
    const auto samplers = [&](auto kernel, const char* which) {
        kernel<<<2048, 128>>>(m, kMats, kDraws, c, c + 1, c + 2);
        std::printf("dopplerEnergy%s %llu of %d\n", which, take(c), kDraws);
        std::printf("samplePhotoFluorescence%s %llu of %d\n", which, take(c + 1), kDraws);
        std::printf("taken%s %llu of %d\n", which, take(c + 2), kDraws);
    };
    samplers(compareSamplers<true>, "Fused");
    samplers(compareSamplers<false>, "Plain");
    return cudaDeviceSynchronize() == cudaSuccess ? 0 : 2;
}
