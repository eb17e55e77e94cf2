// device.cuh -- device functions of the photon-transport hot path shared by the
// transport kernel and the test kernels: per-history random streams, table
// interpolation, interaction samplers, direction update, exact voxel traversal,
// source sampling.
#pragma once

#include <cfloat>
#include <cmath>
#include <cstdint>

#include "engine.hpp"

namespace dxmcg {
namespace dev {

    constexpr unsigned kFull = 0xffffffffu;
    constexpr float kMeKeV = 510.99895f;
    constexpr float kInvHc = 1.0f / 12.398419843f;

    // (2k + 1) / 2^24 from the top 23 bits k: exact in FP32 and FP64, never 0 or 1.
    // Formed as the float 1 + k / 2^23 (k in the mantissa) minus 1 - 2^-24; both are
    // in [1/2, 2] of each other, so the difference is exact (Sterbenz) and no
    // integer-to-float conversion is needed.
    __device__ __forceinline__ float toUniform(uint32_t x)
    {
        return __fsub_rn(__uint_as_float(0x3f800000u | (x >> 9)), 0.99999994039535522461f);
    }

    // Stream of one history: a xoshiro128+ generator (Blackman & Vigna 2018) whose
    // 128-bit state is two SplitMix64 outputs, at the counters key + (2h + 1) gamma and
    // key + (2h + 2) gamma of the run's key (the seeding the generator's authors give),
    // so every history's draws depend only on (seed, stream word, h).  Then seven 32-bit
    // ALU operations per draw with no data-dependent branch, so lanes stay converged
    // while drawing.  Every draw is used through its top 23 bits (uniforms, alias
    // columns), where the '+' output (s0 + s3) is as good as the scrambled '**' one;
    // only its lowest bits are weak, and they are never used.
    struct Rng {
        uint32_t s0, s1, s2, s3;

        __device__ __forceinline__ void init(unsigned long long key, unsigned long long h)
        {
            const unsigned long long x = key + (2ull * h + 1ull) * kGolden64;
            const unsigned long long a = splitMix64(x), b = splitMix64(x + kGolden64);
            s0 = static_cast<uint32_t>(a);
            s1 = static_cast<uint32_t>(a >> 32);
            s2 = static_cast<uint32_t>(b);
            s3 = static_cast<uint32_t>(b >> 32);
            if ((s0 | s1 | s2 | s3) == 0u)
                s0 = 0x9E3779B9u;
        }
        __device__ __forceinline__ uint32_t raw()
        {
            const uint32_t out = s0 + s3;
            const uint32_t t = s1 << 9;
            s2 ^= s0;
            s3 ^= s1;
            s1 ^= s2;
            s0 ^= s3;
            s2 ^= t;
            s3 = __funnelshift_l(s3, s3, 11);
            return out;
        }
        __device__ __forceinline__ float u() { return toUniform(raw()); }
    };

    // Injected uniforms (sampler tests).
    struct InjectedUniforms {
        const float* p;
        int n, used;
        __device__ float u()
        {
            if (used >= n)
                return 0.5f;
            return p[used++];
        }
    };

    // ---------------------------------------------------------------- tables
    __device__ __forceinline__ void gridPos(float E, int& i, float& f)
    {
        const float x = (E - 1.0f) * 2.0f;
        int k = static_cast<int>(x);
        k = k < 0 ? 0 : (k > kTableNE - 2 ? kTableNE - 2 : k);
        i = k;
        f = x - static_cast<float>(k);
    }

    // t[i] holds the table's values at i and i + 1: one 8-byte load
    __device__ __forceinline__ float lerp1(const float2* t, int i, float f)
    {
        const float2 ab = __ldg(t + i);
        return fmaf(f, ab.y - ab.x, ab.x);
    }

    // Correctly rounded 1 / x for 2^-112 <= x < 2^107 and sqrt(x) for 0 and 2^-102 <= x <
    // 2^107: the hardware's approximation and one Newton step in fused arithmetic (Markstein,
    // IBM J. Res. Dev. 34, 111, 1990).  Below 2^-102 the root's residual is no multiple of the
    // least subnormal, and for 1 / x the theorem leaves out the significand of all ones; every
    // float of these ranges is checked against __frcp_rn and __fsqrt_rn
    // (tests/cpp/arithmetic.cu).  Majorants are 1e-30 and more, the roots' arguments 0 or
    // 2^-72 and more (of 1 - s^2 - t^2 with floats s, t).  In place of those functions: 1e7
    // histories of the DX cylinder 1.18 -> 1.15 ms, 2e8 of the torso 23.2 -> 22.5 ms.
    __device__ __forceinline__ float reciprocal(float x)
    {
        float r;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
        return __fmaf_rn(__fmaf_rn(-x, r, 1.0f), r, r);
    }
    __device__ __forceinline__ float squareRoot(float x)
    {
        float y;
        asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
        const float g = __fmul_rn(x, y);
        const float s = __fmaf_rn(__fmaf_rn(-g, g, x), __fmul_rn(0.5f, y), g);
        return x > 0.0f ? s : 0.0f;
    }
    // 1 / sqrt(x) of a squared length near 1, by the hardware's approximation; rsqrtf's bits
    // there (checked between 1/4 and 4, as above).
    __device__ __forceinline__ float unitRsqrt(float x)
    {
        float y;
        asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
        return y;
    }
    // -ln u = -ln 2 log2 u of a uniform (toUniform), by the hardware's log2: |error| <=
    // 2^-21.4 near u = 1.  __logf's bits for each of the 2^23 uniforms (checked, as above).
    // 1e7 histories of the DX cylinder 1518 -> 1502 us in its place, 2e8 of the torso 27.10
    // -> 26.88 ms.
    __device__ __forceinline__ float negLog(float u)
    {
        float l;
        asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(u));
        return __fmul_rn(l, -0.693147180559945309f);
    }

    // ---------------------------------------------------------------- samplers
    constexpr float kCutoffKeV = 1.0f; // photons below this energy are absorbed on the spot
    constexpr int kPzTries = 32;       // electron-momentum draws per accepted scattering angle

    // Correction level 2 (impulse approximation): the scattered energy for a bound
    // electron.  A = E / E_C (E_C: the Compton line) and omu = 1 - cos(theta) come
    // from the angle already sampled.  A shell is picked by its electrons among the
    // shells bound by less than E; its projected momentum p_z = p_s t / sqrt(5) with t
    // Student-t of 5 degrees of freedom, which is the profile (1 + (p_z/p_s)^2)^-3,
    // drawn by Bailey's polar method (Math. Comp. 62, 779, 1994).  rho = p_z / m_e c
    // gives E' from the impulse-approximation energy relation (Ribberfors 1975)
    //   rho = (E E' (1 - cos) / m_e c^2 - (E - E')) / |E - E'| (photon momenta in keV),
    // solved as E'/E = (A - rho^2 cos + rho sqrt((A - cos)^2 + omu (2 - omu) (1 - rho^2)))
    //                  / (A^2 - rho^2).
    // Accepted when E' > 0 and E - E' exceeds the shell's binding; false after
    // kPzTries draws (the caller then samples a new angle).
    //
    // What a trip costs decides the rate here, since a warp waits for its unluckiest lane:
    //   * above every binding energy the shell comes from the material's running sums (one
    //     guide entry, a short scan) instead of two loops over up to 48 shells;
    //   * the polar draw loops by itself, so that lanes meet at the power function;
    //   * a shell bound more strongly than the Compton line's energy loss accepts only
    //     p_z well below zero: rho < rho_b, the rho of E' = E - binding.  A draw short of
    //     it, by a bound wider than the roundings of both, is dropped on a hardware power
    //     function, or on its sign alone.
    // The accepted draws, and so the histories, are those of the plain loop.  Which products
    // are fused is written out: left to the compiler, a job's energies differed with the launch
    // it was part of, by one unit in the last place.  FUSED: in the Woodcock kernel; Siddon and
    // macro tracking keep the roundings that they had.  1e7
    // histories of a CBCT run at level 2: 4.36 -> 3.60 ms.
    template <bool FUSED, class U>
    __device__ bool dopplerEnergy(float E, float A, float omu, const DevMaterial* __restrict__ M, U& r, float& Ep)
    {
        const int ns = M->nShell;
        int sh = -1;
        if (ns > 0 && E > __ldg(&M->shellTop)) {
            const float u = r.u();
            const float target = u * __ldg(&M->shellCum[ns - 1]);
            sh = M->shellStart[static_cast<int>(u * 64.0f)];
            while (sh < ns - 1 && target > __ldg(&M->shellCum[sh]))
                ++sh;
        } else {
            float tot = 0.0f;
            for (int k = 0; k < ns; ++k)
                if (__ldg(&M->shellBinding[k]) < E)
                    tot += __ldg(&M->shellElectrons[k]);
            const float target = r.u() * tot;
            float acc = 0.0f;
            for (int k = 0; k < ns; ++k) {
                if (__ldg(&M->shellBinding[k]) < E) {
                    sh = k;
                    acc += __ldg(&M->shellElectrons[k]);
                    if (target <= acc)
                        break;
                }
            }
            if (sh < 0)
                return false;
        }
        const float bind = __ldg(&M->shellBinding[sh]);
        const float ps = __ldg(&M->shellMomentum[sh]);
        const float c = 1.0f - omu;
        const float am = A - c;
        const float sin2 = omu * (2.0f - omu);
        // |rho_b|^2 where rho_b < 0, else 0: of E' = E - bind + 2e-5 E, so that a draw on
        // the near side of it fails the test below whatever its rounding
        float need2 = 0.0f;
        {
            const float be = __fdividef(bind, E) - 2e-5f, x = 1.0f - be, loss = A - 1.0f;
            const float lack = be - loss * x - 4e-7f * (1.0f + loss);
            if (lack > 0.0f) {
                const float n2 = __fdividef(lack * lack, be * be + 2.0f * x * omu);
                need2 = fminf(n2, 0.25f) * 0.999f;
            }
        }
        const float ps2 = ps * ps;
        for (int t = 0;;) {
            float a, w;
            do {
                if (t == kPzTries)
                    return false;
                ++t;
                a = 2.0f * r.u() - 1.0f;
                const float b = 2.0f * r.u() - 1.0f;
                w = __fmaf_rn(a, a, __fmul_rn(b, b));
            } while (w >= 1.0f
                || (need2 > 0.0f
                    && (a >= 0.0f || ps2 * a * a * (__powf(w, -0.4f) - 1.0f + 1e-5f) * 1.001f < need2 * w)));
            const float rho = ps * a * sqrtf((powf(w, -0.4f) - 1.0f) / w);
            const float rho2 = __fmul_rn(rho, rho);
            const float den = FUSED ? __fmaf_rn(A, A, -rho2) : __fsub_rn(__fmul_rn(A, A), rho2);
            const float rest = __fsub_rn(1.0f, rho2);
            const float disc = FUSED ? __fmaf_rn(am, am, __fmul_rn(sin2, rest))
                                     : __fmaf_rn(sin2, rest, __fmul_rn(am, am));
            if (!(den > 0.0f) || !(disc >= 0.0f))
                continue;
            const float e1 = E * (__fmaf_rn(rho, sqrtf(disc), __fmaf_rn(-rho2, c, A)) / den);
            if (e1 > 0.0f && E - e1 > bind) {
                Ep = e1;
                return true;
            }
        }
    }

    // 1 - cos theta from a material's angle quantile table (row ie of tab, interpolated
    // towards row ie + 1 by fe, at the same probability): one uniform, no rejection.
    // The table's probability grid u_j = (1 - cos(pi j/(K-1)))/2 is inverted by
    // j = (K - 1) acos(1 - 2u) / pi.
    __device__ __forceinline__ float oneMinusCos(const float* __restrict__ tab, int ie, float fe, float u)
    {
        const float jf = static_cast<float>(kCTabK - 1) * 0.31830988618379067f * acosf(fmaf(-2.0f, u, 1.0f));
        const int j = min(static_cast<int>(jf), kCTabK - 2);
        const float g = jf - static_cast<float>(j);
        const float* a = tab + ie * kCTabK + j;
        const float a0 = __ldg(a), a1 = __ldg(a + 1);
        const float b0 = __ldg(a + kCTabK), b1 = __ldg(a + kCTabK + 1);
        const float lo = fmaf(g, a1 - a0, a0);
        const float hi = fmaf(g, b1 - b0, b0);
        return fmaf(fe, hi - lo, lo);
    }

    // E / E_C of the Compton line at 1 - cos theta = omu, product and sum rounded
    // separately: histories must not depend on where the compiler fuses them
    __device__ __forceinline__ float comptonRatio(float E, float omu)
    {
        return __fadd_rn(1.0f, __fmul_rn(E * (1.0f / kMeKeV), omu));
    }

    // Compton scattering: the angle from the Klein-Nishina x S table, E' from the
    // Compton relation (correction 0 and 1), or Doppler-broadened by a bound electron's
    // momentum (correction 2, which may send the draw back for a new angle).
    template <bool FUSED, class U>
    __device__ float sampleCompton(float E, const DevMaterial* __restrict__ M, const float* __restrict__ ctab,
        int ie, float fe, int correction, U& r, float& cost, unsigned& err)
    {
        for (int guard = 0; guard < kMaxRejections; ++guard) {
            const float omu = oneMinusCos(ctab, ie, fe, r.u());
            const float ratio = comptonRatio(E, omu);
            cost = 1.0f - omu;
            if (correction >= 2) {
                float Ep;
                if (!dopplerEnergy<FUSED>(E, ratio, omu, M, r, Ep))
                    continue;
                return Ep;
            }
            return E * reciprocal(ratio);
        }
        err |= kErrRejectLimit;
        cost = 1.0f;
        return E;
    }

    // Rayleigh scattering: cos theta from the material's quantile table of
    // (1 + cos^2)/2 F^2(x), as for the Compton angle: one uniform, no rejection.
    template <class U>
    __device__ __forceinline__ float sampleRayleigh(const float* __restrict__ rtab, int ie, float fe, U& r)
    {
        return 1.0f - oneMinusCos(rtab, ie, fe, r.u());
    }

    // Correction level 2, photoelectric absorption: the absorbing element by its share
    // n_i Z_i^4 (/ J_K below its K edge, / J_L below its L edge) of the cross-section,
    // a K vacancy with probability 1 - 1/J_K above the element's K edge, then a K-alpha
    // photon with the element's K fluorescence yield.  Returns the fluorescence
    // energy, or 0 when no photon above the cutoff leaves the atom (all of E is then
    // deposited).  Draws: element; above the K edge the shell; for a K vacancy the
    // yield.
    __device__ __forceinline__ float photoShare(float E, const DevMaterial* __restrict__ M, int i)
    {
        float w = __ldg(&M->nZ4[i]);
        if (E < __ldg(&M->eK[i]))
            w *= __ldg(&M->invJumpK);
        if (E < __ldg(&M->eL[i]))
            w *= __ldg(&M->invJumpL);
        return w;
    }

    template <class U>
    __device__ float samplePhotoFluorescence(float E, const DevMaterial* __restrict__ M, U& r)
    {
        const int n = M->n;
        int e = n - 1;
        if (E >= __ldg(&M->edgeTop)) { // no share is below an edge
            const float target = r.u() * __ldg(&M->z4Cum[n - 1]);
            for (int i = 0; i < n; ++i)
                if (target <= __ldg(&M->z4Cum[i])) {
                    e = i;
                    break;
                }
        } else {
            float tot = 0.0f;
            for (int i = 0; i < n; ++i)
                tot += photoShare(E, M, i);
            const float target = r.u() * tot;
            float acc = 0.0f;
            for (int i = 0; i < n; ++i) {
                acc += photoShare(E, M, i);
                if (target <= acc) {
                    e = i;
                    break;
                }
            }
        }
        if (E < __ldg(&M->eK[e]))
            return 0.0f;
        if (r.u() >= 1.0f - __ldg(&M->invJumpK))
            return 0.0f; // L or outer shell: its fluorescence stays below the cutoff here
        if (r.u() >= __ldg(&M->omegaK[e]))
            return 0.0f; // Auger electrons: local
        const float ka = __ldg(&M->kAlpha[e]);
        return ka >= kCutoffKeV ? ka : 0.0f;
    }

    // isotropic direction from two uniforms: cos(theta) = 2 u1 - 1, phi = 2 pi u2
    __device__ __forceinline__ void isotropicDirection(float& dx, float& dy, float& dz, float u1, float u2)
    {
        const float ct = 2.0f * u1 - 1.0f;
        const float st = squareRoot(fmaxf(0.0f, 1.0f - ct * ct));
        float sp, cp;
        sincospif(2.0f * u2, &sp, &cp);
        dx = st * cp;
        dy = st * sp;
        dz = ct;
    }

    __device__ __forceinline__ void scatterDirection(float& dx, float& dy, float& dz, float cost, float phiU)
    {
        const float sint = squareRoot(fmaxf(0.0f, 1.0f - cost * cost));
        float sp, cp;
        sincospif(2.0f * phiU, &sp, &cp);
        float nx, ny, nz;
        if (fabsf(dz) > 0.99999f) {
            nx = sint * cp;
            ny = sint * sp;
            nz = (dz > 0.0f ? 1.0f : -1.0f) * cost;
        } else {
            const float tmp = squareRoot(1.0f - dz * dz);
            const float it = reciprocal(tmp);
            nx = sint * (dx * dz * cp - dy * sp) * it + dx * cost;
            ny = sint * (dy * dz * cp + dx * sp) * it + dy * cost;
            nz = -sint * cp * tmp + dz * cost;
        }
        const float inv = unitRsqrt(nx * nx + ny * ny + nz * nz);
        dx = nx * inv;
        dy = ny * inv;
        dz = nz * inv;
    }

    // ---------------------------------------------------------------- Siddon
    // Exact voxel stepping in grid-local coordinates; the FP32 operation order is
    // fixed with _rn intrinsics (no FMA contraction) so that a host restatement
    // compiled without contraction produces the same voxel sequence bit for bit.
    // Ray parameter of the crossing with the plane k * sp; the plane position is a
    // double-float (hi + fma remainder) so grazing rays do not amplify its rounding.
    __device__ __forceinline__ float crossF32(int k, float sp, float o, float d)
    {
        const float kf = __int2float_rn(k);
        const float hi = __fmul_rn(kf, sp);
        const float lo = __fmaf_rn(kf, sp, -hi);
        return __fdiv_rn(__fadd_rn(__fsub_rn(hi, o), lo), d);
    }

    struct Siddon {
        int i[3], st[3];
        float o[3], d[3], sp[3];
        float t, tmax;
        int n[3];

        // returns false if the ray misses the grid
        __device__ bool begin(const float* org, const float* dir, const int* dims, const float* spacing)
        {
            float tmin = 0.0f;
            tmax = FLT_MAX;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                n[a] = dims[a];
                sp[a] = spacing[a];
                o[a] = org[a];
                d[a] = dir[a];
                if (dir[a] != 0.0f) {
                    float t1 = crossF32(0, spacing[a], org[a], dir[a]);
                    float t2 = crossF32(dims[a], spacing[a], org[a], dir[a]);
                    if (t1 > t2) {
                        const float tt = t1;
                        t1 = t2;
                        t2 = tt;
                    }
                    if (t1 > tmin)
                        tmin = t1;
                    if (t2 < tmax)
                        tmax = t2;
                } else if (org[a] < 0.0f || org[a] >= __fmul_rn(__int2float_rn(dims[a]), spacing[a])) {
                    return false;
                }
            }
            if (!(tmin < tmax))
                return false;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const float p = __fadd_rn(org[a], __fmul_rn(tmin, dir[a]));
                int k = static_cast<int>(floorf(__fdiv_rn(p, sp[a])));
                k = k < 0 ? 0 : (k > n[a] - 1 ? n[a] - 1 : k);
                i[a] = k;
                st[a] = dir[a] > 0.0f ? 1 : (dir[a] < 0.0f ? -1 : 0);
            }
            t = tmin;
            return true;
        }

        // next segment: returns false when the ray has left the grid.
        // *len may be 0 for degenerate steps (callers skip them).
        __device__ bool next(long long& voxel, float& len, float& t0)
        {
            float tn[3];
#pragma unroll
            for (int a = 0; a < 3; ++a)
                tn[a] = st[a] != 0 ? crossF32(i[a] + (st[a] > 0 ? 1 : 0), sp[a], o[a], d[a]) : FLT_MAX;
            int ax = 0;
            if (tn[1] < tn[ax])
                ax = 1;
            if (tn[2] < tn[ax])
                ax = 2;
            const float tnext = tn[ax] < tmax ? tn[ax] : tmax;
            const float l = __fsub_rn(tnext, t);
            voxel = static_cast<long long>(i[0]) + static_cast<long long>(n[0])
                    * (static_cast<long long>(i[1]) + static_cast<long long>(n[1]) * i[2]);
            t0 = t;
            if (l > 0.0f) {
                len = l;
                t = tnext;
            } else {
                len = 0.0f;
            }
            if (tnext >= tmax) {
                done = true;
                return true;
            }
            i[ax] += st[ax];
            if (i[ax] < 0 || i[ax] >= n[ax])
                done = true;
            return true;
        }
        bool done = false;
    };

    // ---------------------------------------------------------------- photon
    struct Photon {
        float px, py, pz;
        float dx, dy, dz;
        float E, w;
    };

    // FP64 reductions into the voxel's 32-byte record (one L2 sector).
    // The deposit is formed in FP32 and widened only for the reductions.
    __device__ __forceinline__ void deposit(Tally* __restrict__ tally, uint32_t v, float e)
    {
        atomicAdd(&tally[v].e, static_cast<double>(e));
        atomicAdd(&tally[v].e2, static_cast<double>(e * e));
        atomicAdd(&tally[v].n, 1ull);
    }

    // toDose / rho of a packed voxel word, 0 without density; the same double as the
    // division gives (see DoseScale).  FP64 runs at 2 lanes a clock and SM here, and a
    // division is some ten FP64 operations: one 8-byte load of a table that stays in L1
    // (a material's +-2 % of density are a few hundred entries) takes its place.
    __device__ __forceinline__ double doseFactor(const DoseScale& c, uint32_t word)
    {
        const uint32_t bits = word & 0xffffff00u;
        if (bits == 0u)
            return 0.0;
        const int e = static_cast<int>(bits >> 23); // densities are positive
        if (!c.factors || e == 0)
            return c.toDose / static_cast<double>(__uint_as_float(bits));
        const long long f = __double_as_longlong(__ldg(c.factors + (bits >> 8 & 0x7fffu)));
        return __longlong_as_double(f - (static_cast<long long>(e - 127) << 52));
    }

    // relative bowtie weight of tube `tube` at |fan angle| a (1 when that tube has none)
    __device__ __forceinline__ float bowtieAt(const DevBowtie* __restrict__ b, int tube, float a)
    {
        const int n = b->n[tube];
        const float* __restrict__ ang = b->ang[tube];
        const float* __restrict__ w = b->w[tube];
        if (n <= 0)
            return 1.0f;
        if (a <= ang[0])
            return w[0];
        if (a >= ang[n - 1])
            return w[n - 1];
        // the segment with ang[lo] <= a < ang[lo + 1], from the cell's entry (the two
        // scans correct a cell misplaced by the rounding of a * cellScale)
        const int c = min(static_cast<int>(a * b->cellScale[tube]), kBowtieCells - 1);
        int lo = b->seg[tube][c];
        while (lo > 0 && ang[lo] > a)
            --lo;
        while (ang[lo + 1] <= a)
            ++lo;
        const int hi = lo + 1;
        const float t = (a - ang[lo]) / (ang[hi] - ang[lo]);
        return w[lo] + t * (w[hi] - w[lo]);
    }

    // exposure of history h (histories are numbered exposure-major)
    __device__ __forceinline__ unsigned exposureOf(const DevJob& J, unsigned long long h)
    {
        if ((h >> 32) == 0ull && (J.ppe >> 32) == 0ull)
            return static_cast<uint32_t>(h) / static_cast<uint32_t>(J.ppe);
        return static_cast<unsigned>(h / J.ppe);
    }

    // Source sampling (draw order: 2 raw for the energy, fan, cone).  Leaves the
    // photon at its source position (grid-local).
    __device__ __forceinline__ void sampleSource(const DevJob& J, unsigned long long h, Photon& ph, Rng& r)
    {
        // the 64-byte exposure record as four 16-byte loads: (pos, c0.x), (c0.y, c0.z,
        // c1.x, c1.y), (c1.z, n), (half, weight, tube)
        const float4* __restrict__ ex4 = reinterpret_cast<const float4*>(J.exps + exposureOf(J, h));
        const float4 q3 = __ldg(ex4 + 3);
        const int tube = __float_as_int(q3.w);
        if (J.beam_type == DXMCG_BEAM_PENCIL) {
            (void)r.raw();
            (void)r.raw();
            ph.E = J.pencil_energy;
        } else {
            const DevSpectrum* __restrict__ S = J.spec + tube;
            const uint32_t x0 = r.raw() >> 9;
            const uint32_t x1 = r.raw() >> 9;
            const int n = S->n;
            int k = static_cast<int>((static_cast<unsigned long long>(x0) * static_cast<unsigned long long>(n)) >> 23);
            k = x1 < __ldg(&S->thr[k]) ? k : __ldg(&S->alias[k]);
            ph.E = __ldg(&S->E[k]);
        }
        const float ax = (2.0f * r.u() - 1.0f) * q3.x;
        const float ay = (2.0f * r.u() - 1.0f) * q3.y;
        // |angle| < pi/2: the hardware sine is within 2^-21.4
        const float sx = __sinf(ax), sy = __sinf(ay);
        const float sz = squareRoot(fmaxf(0.0f, 1.0f - sx * sx - sy * sy));
        const float4 q0 = __ldg(ex4), q1 = __ldg(ex4 + 1), q2 = __ldg(ex4 + 2);
        ph.dx = q0.w * sx + q1.z * sy + q2.y * sz;
        ph.dy = q1.x * sx + q1.w * sy + q2.z * sz;
        ph.dz = q1.y * sx + q2.x * sy + q2.w * sz;
        ph.px = q0.x;
        ph.py = q0.y;
        ph.pz = q0.z;
        float w = q3.z;
        if (J.bowtie)
            w *= bowtieAt(J.bowtie, tube, fabsf(ax)) * J.bowtie->inv_norm[tube];
        ph.w = w;
    }

    // Move a source photon to its entry point on the grid box; false if it misses.
    __device__ __forceinline__ bool enterGrid(const DevJob& J, Photon& ph)
    {
        float p[3] = { ph.px, ph.py, ph.pz };
        const float d[3] = { ph.dx, ph.dy, ph.dz };
        float tmin = 0.0f, tmax = FLT_MAX;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if (d[a] != 0.0f) {
                const float inv = __frcp_rn(d[a]); // the correctly rounded 1 / d, as a division gives
                float t1 = (0.0f - p[a]) * inv, t2 = (J.L[a] - p[a]) * inv;
                if (t1 > t2) {
                    const float tt = t1;
                    t1 = t2;
                    t2 = tt;
                }
                tmin = fmaxf(tmin, t1);
                tmax = fminf(tmax, t2);
            } else if (p[a] < 0.0f || p[a] >= J.L[a]) {
                tmax = -1.0f;
            }
        }
        if (!(tmin < tmax))
            return false;
#pragma unroll
        for (int a = 0; a < 3; ++a)
            p[a] = fminf(fmaxf(p[a] + tmin * d[a], 0.0f), J.Lin[a]);
        ph.px = p[0];
        ph.py = p[1];
        ph.pz = p[2];
        return true;
    }

} // namespace dev
} // namespace dxmcg
