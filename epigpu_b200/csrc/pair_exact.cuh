// pair_exact.cuh -- the FP64 statistics of one pair from its exact integer cell counts and
// digit sums, shared by the tensor form's epilogue and by the kernel that evaluates the
// screen's candidates.
#pragma once
#include "epi_internal.cuh"

namespace epi {

// 1/x for x > 0: single-precision seed (__frcp_rn) refined by one Newton step in FP64,
// e = 1 - x r, r' = r + r e, which squares the seed's relative error (2^-24 -> ~2^-48).
__device__ __forceinline__ double rcp_d(double x)
{
    double r = (double)__frcp_rn((float)x);
    const double e = fma(-x, r, 1.0);
    return fma(r, e, r);
}

// num / den in FP64: by rcp_d when den is a normal single-precision magnitude (relative error
// ~2^-46), else by IEEE division (zero, tiny or huge denominators keep division's inf / NaN).
__device__ __forceinline__ double div_fast(double num, double den)
{
    const double ad = fabs(den);
    return (ad > 1e-30 && ad < 1e30) ? num * rcp_d(den) : num / den;
}

// The reference's 8 df / 4 df statistics (src/EpiOpenCL.c:231-247, :452-486) in FP64 from
// the exact integer cell counts n and digit sums si (S = si * sc), and Q = sum of y^2 over
// the pair's valid individuals. Same quantities as pair_stat, arranged to avoid division
// chains: reciprocals by rcp_d. A pair whose individuals all have one value of y has nothing to explain:
// F and F2 are 0/0 (NaN, never a hit or a maximum), although SSB may hold a rounding of the cell means.
__device__ __forceinline__ PairStat pair_stat_exact(const int n[9], const double si[9], double sc, double Q,
                                                    bool want_int)
{
    // si are integers below 2^53 in magnitude (digit sums), so every sum of them is exact
    PairStat r;
    int N = 0, nfac = 0;
    double St_i = 0.0;
#pragma unroll
    for (int c = 0; c < 9; ++c) {
        N += n[c];
        St_i += si[c];
        nfac += n[c] > 0;
    }
    const double St = St_i * sc;
    const double m = St * rcp_d((double)N);
    double mc[9], SSB = 0.0;
#pragma unroll
    for (int c = 0; c < 9; ++c) {
        mc[c] = 0.0;
        if (n[c] > 0) {
            mc[c] = si[c] * sc * rcp_d((double)n[c]);
            const double d = mc[c] - m;
            SSB = fma((double)n[c] * d, d, SSB);
        }
    }
    const double SSY = Q - St * m;
    const double SSW = ssw_floored(SSY, SSB, SSW_FLOOR_EXACT);
    r.nfac = nfac;
    r.d1 = nfac - 1;
    r.d2 = N - nfac;
    r.F = div_fast(SSB * (double)r.d2, SSW * (double)r.d1);
    r.F2 = 0.0;
    if (!(SSY > 0.0)) {
        r.F = r.F2 = __longlong_as_double(0x7ff8000000000000ll);
        return r;
    }
    if (want_int) {
        double row[3], col[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const double rs = si[3 * i] + si[3 * i + 1] + si[3 * i + 2];
            const double cs = si[i] + si[i + 3] + si[i + 6];
            const int rn = n[3 * i] + n[3 * i + 1] + n[3 * i + 2];
            const int cn = n[i] + n[i + 3] + n[i + 6];
            row[i] = rn > 0 ? rs * sc * rcp_d((double)rn) : 0.0;
            col[i] = cn > 0 ? cs * sc * rcp_d((double)cn) : 0.0;
        }
        double SSI = 0.0;
#pragma unroll
        for (int c = 0; c < 9; ++c) {
            if (n[c] > 0) {
                const double t = mc[c] - row[c / 3] - col[c % 3] + m;
                SSI = fma((double)n[c] * t, t, SSI);
            }
        }
        r.F2 = div_fast(SSI * (double)r.d2, 4.0 * SSW);
    }
    return r;
}

// Sum of ytilde^2 over the phenotype-valid individuals missing at both SNPs, by the whole warp
// (every lane gets it): the intersection of the two SNPs' missing bits.
__device__ __forceinline__ double missing_both_q(const ScanArgs &a, int t, int snp1, int snp2)
{
    const int lane = threadIdx.x & 31;
    const uint32_t *mbi = a.missbits + (size_t)snp1 * a.Wp, *mbj = a.missbits + (size_t)snp2 * a.Wp;
    const uint32_t *wm = a.wmask + (size_t)t * a.Wp;
    const double *qdt = a.qd + (size_t)t * a.Np;
    double part = 0.0;
    for (int w = lane; w < a.Wp; w += 32) {
        uint32_t bits = mbi[w] & mbj[w] & wm[w];
        while (bits) {
            part += qdt[32 * w + __ffs(bits) - 1];
            bits &= bits - 1;
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) part += __shfl_xor_sync(0xffffffffu, part, off);
    return part;
}

template <class T>
__device__ __forceinline__ T pick3(T x0, T x1, T x2, int idx)
{
    return idx == 0 ? x0 : (idx == 1 ? x1 : x2);
}

// approximate reciprocal of the screen (one MUFU operation, relative error ~2^-23; 1/0 = +inf)
__device__ __forceinline__ float rcp_fast(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// approximate square root (relative error ~2^-23)
__device__ __forceinline__ float sqrt_fast(float x)
{
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// x lowered by the screen's margin (relative 1e-3); -inf and NaN stay as they are
__device__ __forceinline__ float screen_lo(float x) { return x - 1e-3f * fabsf(x); }

}  // namespace epi
