// prep.cu -- device-side genotype preparation.
//
// Turns the reference's packed rows (src/readplink.c:1066-1102: 16 codes per int32, first
// individual in bits 31:30, tail word right-aligned with `remain` codes) into
//   planes  uint4 [nsnp][Wp]: bits of [g==0], [g==1], [g==2], [g!=3] per 32 individuals
//   codes   uint32 [nsnp][Wc]: 2-bit codes, LSB first, padding individuals coded 3
// The decoding is the kernel's own (EpiOpenCL.c:116-228), done once per load instead of
// once per pair.
#include <cstdint>
#include <cuda_runtime.h>

#include "epi_internal.cuh"

namespace epi {

__device__ __forceinline__ uint32_t ref_code(const int32_t *row, int k, int nid, int npack, int remain)
{
    if (k >= nid) return 3u;
    if (k < 16 * npack) return ((uint32_t)row[k >> 4] >> (30 - 2 * (k & 15))) & 3u;
    const int t = k - 16 * npack;
    return ((uint32_t)row[npack] >> (2 * (remain - 1 - t))) & 3u;
}

// One thread per (SNP, 32-individual word). Also writes the tensor form's one-hot code
// bytes (1 << g, 0 when missing or padding), its genotype-indicator rows h3 (row 3s + a holds
// the byte [g == a] per individual) and the missing-genotype bits.
__global__ void k_unpack(const int32_t *__restrict__ raw, int nsnp, int nid, int npack, int remain,
                         int npack1, uint4 *__restrict__ planes, int Wp, uint32_t *__restrict__ codes, int Wc,
                         uint8_t *__restrict__ hcodes, uint8_t *__restrict__ h3, uint32_t *__restrict__ missbits)
{
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long total = (long long)nsnp * Wp;
    if (gid >= total) return;
    const int s = (int)(gid / Wp), w = (int)(gid % Wp);
    const int32_t *row = raw + (size_t)s * npack1;
    uint32_t p0 = 0, p1 = 0, p2 = 0, c0 = 0, c1 = 0, miss = 0;
    uint32_t h[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int t = 0; t < 32; ++t) {
        const int k = 32 * w + t;
        const uint32_t c = ref_code(row, k, nid, npack, remain);
        p0 |= (uint32_t)(c == 0u) << t;
        p1 |= (uint32_t)(c == 1u) << t;
        p2 |= (uint32_t)(c == 2u) << t;
        miss |= (uint32_t)(c == 3u && k < nid) << t;
        h[t >> 2] |= (c < 3u ? (1u << c) : 0u) << (8 * (t & 3));
        if (t < 16) c0 |= c << (2 * t);
        else c1 |= c << (2 * (t - 16));
    }
    planes[(size_t)s * Wp + w] = make_uint4(p0, p1, p2, p0 | p1 | p2);
    if (hcodes != nullptr) {
        uint4 *dst = reinterpret_cast<uint4 *>(hcodes + ((size_t)s * Wp + w) * 32);
        dst[0] = make_uint4(h[0], h[1], h[2], h[3]);
        dst[1] = make_uint4(h[4], h[5], h[6], h[7]);
    }
    if (h3 != nullptr) {
        const size_t Np = (size_t)Wp * 32;
#pragma unroll
        for (int g = 0; g < 3; ++g) {
            uint32_t e[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) e[q] = (h[q] >> g) & 0x01010101u;
            uint4 *dst = reinterpret_cast<uint4 *>(h3 + (3 * (size_t)s + g) * Np + (size_t)w * 32);
            dst[0] = make_uint4(e[0], e[1], e[2], e[3]);
            dst[1] = make_uint4(e[4], e[5], e[6], e[7]);
        }
    }
    if (missbits != nullptr) missbits[(size_t)s * Wp + w] = miss;
    if (codes != nullptr) {
        if (2 * w < Wc) codes[(size_t)s * Wc + 2 * w] = c0;
        if (2 * w + 1 < Wc) codes[(size_t)s * Wc + 2 * w + 1] = c1;
    }
}

// Sum over the block of a few values at once; every thread gets the sums. `sv` holds
// 32 x N doubles.
template <int N>
__device__ __forceinline__ void block_sum(double (&v)[N], double *sv)
{
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < N; ++i)
        for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
    __syncthreads();
    if (l == 0)
        for (int i = 0; i < N; ++i) sv[N * w + i] = v[i];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < N; ++i) {
        double x = l < (int)(blockDim.x >> 5) ? sv[N * l + i] : 0.0;
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        v[i] = x;
    }
}

// The largest of each of two values over the block (NaN is never the larger one).
__device__ __forceinline__ void block_max2(double &a, double &b, double *sv)
{
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    auto warp_max = [](double x) {
        for (int o = 16; o > 0; o >>= 1) {
            const double y = __shfl_xor_sync(0xffffffffu, x, o);
            x = y > x ? y : x;
        }
        return x;
    };
    a = warp_max(a);
    b = warp_max(b);
    __syncthreads();
    if (l == 0) {
        sv[2 * w] = a;
        sv[2 * w + 1] = b;
    }
    __syncthreads();
    const int nw = blockDim.x >> 5;
    a = warp_max(sv[2 * (l < nw ? l : 0)]);
    b = warp_max(sv[2 * (l < nw ? l : 0) + 1]);
}

// Everything that the scans need of a phenotype column, one block per trait, in FP64:
//   * centred by its valid mean and scaled by the power of two that brings its largest magnitude
//     into [0.5, 1). F and F2 do not depend on the trait's scale, and a power-of-two factor is
//     exact in binary floating point, so in the normal range every result is bit-identical to
//     the unscaled computation; a trait in units of 1e20 or 1e-20 no longer overflows or
//     underflows the single-precision sums of squares;
//   * tensor form: Y = round(y 2^sy) (|Y| <= 8355711), three balanced base-256 digits of it
//     and the valid flag; ytilde^2 = (Y 2^-sy)^2 (exact in FP64: |Y| < 2^23) and Y; their sums;
//   * the screen's 8-bit phenotype D = round(s (ytilde - c)), c the middle of the values and s
//     the scale that spreads them over -127..127, d0 = -s c (the D of the mean), and the norm
//     E of what the rounding leaves, that of ytilde against y included; the same for the two upper
//     digits of Y (scan_mma.cu).
// Four passes over the column; at 10,000 individuals about 15 us, where the same loops on one
// host core and the upload of their eight arrays took 200 to 300 us.
__global__ void __launch_bounds__(1024) k_traits(const float *__restrict__ yraw, const uint8_t *__restrict__ valid,
                                                 int mode, int nid, int Np, int ntraits, TraitArrays o,
                                                 TraitInfo *__restrict__ info)
{
    __shared__ double sv[32 * 5];
    const int t = blockIdx.x, tid = threadIdx.x, nt = blockDim.x;
    const float *y = yraw + (size_t)t * nid;
    const uint8_t *vb = mode == VALID_BYTES ? valid + (size_t)t * nid : nullptr;
    auto ok = [&](int k) { return k < nid && (mode == VALID_ALL || (vb ? vb[k] != 0 : y[k] != -9.0f)); };
    // trait 0's
    auto ok0 = [&](int k) { return k < nid && (mode == VALID_ALL || (vb ? valid[k] != 0 : yraw[k] != -9.0f)); };
    bool differs = false;

    double s0[2] = {0.0, 0.0};
    for (int k = tid; k < Np; k += nt) {  // (Np and the block are multiples of a warp)
        const bool v = ok(k);
        const unsigned int bits = __ballot_sync(0xffffffffu, v);
        if ((tid & 31) == 0) o.wmask[((size_t)t * Np + k) >> 5] = bits;
        if (v) {
            s0[0] += (double)y[k];
            s0[1] += 1.0;
        }
        differs = differs || v != ok0(k);
    }
    differs = __syncthreads_or(differs);
    block_sum(s0, sv);
    const double nv = s0[1], mu = nv > 0.0 ? s0[0] / nv : 0.0;

    double maxabs = 0.0, unused = 0.0;
    for (int k = tid; k < nid; k += nt)
        if (ok(k)) {
            const double d = fabs((double)y[k] - mu);
            maxabs = d > maxabs ? d : maxabs;
        }
    block_max2(maxabs, unused, sv);
    const bool scaled = maxabs > 0.0 && isfinite(maxabs);
    const double p2 = scaled ? ldexp(1.0, -(ilogb(maxabs) + 1)) : 1.0;
    // the largest power of two with maxabs p2 2^sy <= 8355000, maxabs p2 in [0.5, 1)
    const double scale = scaled ? (maxabs * p2 * 8388608.0 <= 8355000.0 ? 8388608.0 : 4194304.0) : 1.0;
    const double unit = 1.0 / scale;  // 2^-sy

    int8_t *dg = o.ydig + (size_t)t * 5 * Np;  // rows D, w, d2, d1, d0
    double s1[5] = {0.0, 0.0, 0.0, 0.0, 0.0};  // sums of y^2 (as floats), ytilde^2, Y, d0^2, (y - ytilde)^2
    double ymax = -INFINITY, nymin = -INFINITY;
    for (int k = tid; k < Np; k += nt) {
        float yc = 0.0f;
        long long Y = 0;
        const bool v = ok(k);
        if (v) {
            const double x = ((double)y[k] - mu) * p2, z = x * scale;
            yc = (float)x;
            Y = isfinite(z) ? llround(z) : -8355711LL;
            Y = min(8355711LL, max(-8355711LL, Y));
        }
        const long long a0 = ((Y + 128) & 255) - 128, Y1 = (Y - a0) / 256;
        const long long a1 = ((Y1 + 128) & 255) - 128, a2 = (Y1 - a1) / 256;
        const double yq = (double)Y * unit;
        if (o.y) o.y[(size_t)t * Np + k] = yc;
        dg[(size_t)Np + k] = (int8_t)v;
        dg[2 * (size_t)Np + k] = (int8_t)a2;
        dg[3 * (size_t)Np + k] = (int8_t)a1;
        dg[4 * (size_t)Np + k] = (int8_t)a0;
        if (o.qd) {
            o.qd[(size_t)t * Np + k] = yq * yq;
            o.qd[((size_t)ntraits + t) * Np + k] = (double)Y;
        }
        if (v) {
            s1[0] += (double)yc * (double)yc;
            s1[1] += yq * yq;
            s1[2] += (double)Y;
            s1[3] += (double)(a0 * a0);
            s1[4] += ((double)yc - yq) * ((double)yc - yq);
            ymax = yq > ymax ? yq : ymax;
            nymin = -yq > nymin ? -yq : nymin;
        }
    }
    block_sum(s1, sv);
    block_max2(ymax, nymin, sv);

    const double mid = nv > 0.0 ? 0.5 * (ymax - nymin) : 0.0, half = nv > 0.0 ? 0.5 * (ymax + nymin) : 0.0;
    const double s = half > 0.0 ? 127.0 / half : 1.0;
    const float dm = (float)(-s * mid);
    double e[1] = {0.0};
    for (int k = tid; k < Np; k += nt) {  // (each thread reads what it wrote)
        double D = 0.0;
        if (dg[(size_t)Np + k]) {
            const int Y = dg[4 * (size_t)Np + k] + 256 * dg[3 * (size_t)Np + k] + 65536 * dg[2 * (size_t)Np + k];
            const double x = s * ((double)Y * unit);
            D = fmin(127.0, fmax(-127.0, rint(x + (double)dm)));
            const double r = x - (D - (double)dm);
            e[0] += r * r;
        }
        dg[k] = (int8_t)D;
    }
    block_sum(e, sv);
    if (tid != 0) return;
    const double s16 = scale / 256.0, e16 = s1[3] / 65536.0;  // two digits: D = d1 + 256 d2 = (Y - d0) / 256
    const double q8 = s * s * s1[1], q16 = s16 * s16 * s1[1];
    o.ysq[t] = s1[0];
    o.qtot[t] = s1[1];
    o.yscale[t] = unit;
    o.yscale[ntraits + t] = s1[2];
    o.yscale[2 * (size_t)ntraits + t] = nv;
    const double ey = sqrt(s1[4]);
    o.tscr[2 * t] = make_float4(dm, (float)((sqrt(e[0]) + s * ey) * (1.0 + 1e-6)), (float)q8, (float)(s * s));
    o.tscr[2 * t + 1] = make_float4(0.0f, (float)((sqrt(e16) + s16 * ey) * (1.0 + 1e-6)), (float)q16, (float)(s16 * s16));
    info[t].nv = nv;
    info[t].same_mask = differs ? 0.0 : 1.0;
    info[t].r1 = q8 > 0.0 ? sqrt(e[0] * nv / q8) : INFINITY;
    info[t].r2 = q16 > 0.0 ? sqrt(e16 * nv / q16) : INFINITY;
}

// Per trait t and SNP s, over the individuals missing at s (and phenotype-valid for t):
// qm[t][s] = sum of qd[t][k], rm[t][s] = sum of qr[t][k] and nm[t][s] = their number; qmf[t][s]
// = qm as a float. One warp per (t, s), lanes over the words (one thread per SNP walked its words
// one after the other: 200 us for 20,000 SNPs at 10,000 individuals, and as long for few SNPs).
__global__ void k_qmiss(const uint32_t *__restrict__ missbits, int nsnp, int Wp, const uint32_t *__restrict__ wmask,
                        const double *__restrict__ qd, const double *__restrict__ qr, int Np, int ntraits,
                        double *__restrict__ qm, double *__restrict__ rm, double *__restrict__ nm,
                        float *__restrict__ qmf)
{
    const long long gid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (gid >= (long long)nsnp * ntraits) return;
    const int t = (int)(gid / nsnp), s = (int)(gid % nsnp);
    double x = 0.0, r = 0.0;
    int cnt = 0;
    const uint32_t *mb = missbits + (size_t)s * Wp;
    for (int w = lane; w < Wp; w += 32) {
        uint32_t bits = mb[w] & wmask[(size_t)t * Wp + w];
        cnt += __popc(bits);
        while (bits) {
            const size_t k = (size_t)t * Np + 32 * w + __ffs(bits) - 1;
            x += qd[k];
            r += qr[k];
            bits &= bits - 1;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        x += __shfl_xor_sync(0xffffffffu, x, o);
        r += __shfl_xor_sync(0xffffffffu, r, o);
    }
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (lane == 0) {
        qm[gid] = x;
        rm[gid] = r;
        nm[gid] = (double)cnt;
        qmf[gid] = (float)x;
    }
}

// The streamed-B variant's expanded B rows: row (u nsnp + s) R + r of the u-th set of R = 3 G rows
// per SNP holds [g_s(k) == b] * digit(k) for every individual k, r = G b + i and digit the i-th of
// the set's G digit rows -- the rows the tensor form's producers otherwise build in shared
// memory. GROUP: one set per group of five traits with the same mask, w and their D's (zero past
// the last trait). Full digits: two sets of G = 2 rows per trait, (w, d2) for CTA 0's half and (d1, d0) for
// CTA 1's; the screen: one set per trait, (w, D) or (w, d2, d1). ydig's rows per trait are D, w,
// d2, d1, d0. One thread per 16 individuals of (set, s).
template <int G, bool FULL, bool GROUP = false>
__global__ void k_expand(const uint8_t *__restrict__ hcodes, const int8_t *__restrict__ ydig, int nsnp, int Np,
                         int sets, int ntraits, int8_t *__restrict__ x)
{
    const int nc = Np / 16;
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= (long long)sets * nsnp * nc) return;
    const int c = (int)(gid % nc);
    const long long rest = gid / nc;
    const int s = (int)(rest % nsnp), u = (int)(rest / nsnp);
    const int trait = FULL ? u / 2 : u;
    const uint4 hc = reinterpret_cast<const uint4 *>(hcodes + (size_t)s * Np)[c];
    uint4 d[G];
#pragma unroll
    for (int i = 0; i < G; ++i) {
        const int row = FULL ? 1 + 2 * (u & 1) + i : GROUP ? (i == 0 ? 1 : 0) : G == 2 ? 1 - i : 1 + i;
        const int tr = GROUP ? (G - 1) * u + (i == 0 ? 0 : i - 1) : trait;
        d[i] = tr < ntraits ? reinterpret_cast<const uint4 *>(ydig + ((size_t)tr * 5 + row) * Np)[c]
                            : make_uint4(0u, 0u, 0u, 0u);
    }
    uint4 *out = reinterpret_cast<uint4 *>(x + ((size_t)u * nsnp + s) * 3 * G * (size_t)Np) + c;
#pragma unroll
    for (int b = 0; b < 3; ++b) {
        uint4 m;
        m.x = ((hc.x >> b) & 0x01010101u) * 0xFFu;
        m.y = ((hc.y >> b) & 0x01010101u) * 0xFFu;
        m.z = ((hc.z >> b) & 0x01010101u) * 0xFFu;
        m.w = ((hc.w >> b) & 0x01010101u) * 0xFFu;
#pragma unroll
        for (int i = 0; i < G; ++i)
            out[(size_t)(G * b + i) * nc] = make_uint4(m.x & d[i].x, m.y & d[i].y, m.z & d[i].z, m.w & d[i].w);
    }
}

// Per SNP the most frequent genotype (ties to the lower code), one warp per SNP: the plain
// form derives that genotype's row of the 3x3 table from the SNP's marginals.
__global__ void k_major(const uint4 *__restrict__ planes, int nsnp, int Wp, uint8_t *__restrict__ maj)
{
    const long long s = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (s >= nsnp) return;
    int c0 = 0, c1 = 0, c2 = 0;
    for (int w = lane; w < Wp; w += 32) {
        const uint4 P = planes[(size_t)s * Wp + w];
        c0 += __popc(P.x);
        c1 += __popc(P.y);
        c2 += __popc(P.z);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        c0 += __shfl_xor_sync(0xffffffffu, c0, o);
        c1 += __shfl_xor_sync(0xffffffffu, c1, o);
        c2 += __shfl_xor_sync(0xffffffffu, c2, o);
    }
    if (lane == 0) maj[s] = (uint8_t)((c0 >= c1 && c0 >= c2) ? 0 : (c1 >= c2 ? 1 : 2));
}

// Plain-form marginals, one warp per (trait t, SNP s), lane = individual within each 32-word:
// pmC[t][s][b] = sum of y over g_s = b, pmN[t][s][b] = number of phenotype-valid individuals
// with g_s = b, pmQ[t][s] = sum of y^2 over the valid individuals missing at s. FP64 per lane,
// then a warp-shuffle reduction.
__global__ void k_marg(const uint4 *__restrict__ planes, int nsnp, int Wp, const float *__restrict__ y,
                       const uint32_t *__restrict__ wmask, int Np, int ntraits, double *__restrict__ pmC,
                       int32_t *__restrict__ pmN, double *__restrict__ pmQ)
{
    const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (gw >= (long long)nsnp * ntraits) return;
    const int t = (int)(gw / nsnp), s = (int)(gw % nsnp);
    double c0 = 0.0, c1 = 0.0, c2 = 0.0, q = 0.0;
    int n0 = 0, n1 = 0, n2 = 0;
    const float *yt = y + (size_t)t * Np;
    const uint32_t *wt = wmask + (size_t)t * Wp;
    for (int w = 0; w < Wp; ++w) {
        const uint4 P = planes[(size_t)s * Wp + w];
        const uint32_t W = wt[w];
        const double yv = (double)yt[32 * w + lane];
        const int ok = (W >> lane) & 1u;
        if ((P.x >> lane) & 1u) {
            c0 += yv;
            n0 += ok;
        } else if ((P.y >> lane) & 1u) {
            c1 += yv;
            n1 += ok;
        } else if ((P.z >> lane) & 1u) {
            c2 += yv;
            n2 += ok;
        } else if (ok) {
            q += yv * yv;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        c0 += __shfl_xor_sync(0xffffffffu, c0, o);
        c1 += __shfl_xor_sync(0xffffffffu, c1, o);
        c2 += __shfl_xor_sync(0xffffffffu, c2, o);
        q += __shfl_xor_sync(0xffffffffu, q, o);
        n0 += __shfl_xor_sync(0xffffffffu, n0, o);
        n1 += __shfl_xor_sync(0xffffffffu, n1, o);
        n2 += __shfl_xor_sync(0xffffffffu, n2, o);
    }
    if (lane == 0) {
        const size_t o = (size_t)gw;
        pmC[3 * o] = c0;
        pmC[3 * o + 1] = c1;
        pmC[3 * o + 2] = c2;
        pmN[3 * o] = n0;
        pmN[3 * o + 1] = n1;
        pmN[3 * o + 2] = n2;
        pmQ[o] = q;
    }
}

cudaError_t launch_traits(const float *yraw, const uint8_t *valid, int mode, int nid, int Np, int ntraits,
                          const TraitArrays &o, TraitInfo *info, cudaStream_t stream)
{
    k_traits<<<ntraits, Np < 1024 ? Np : 1024, 0, stream>>>(yraw, valid, mode, nid, Np, ntraits, o, info);
    return cudaGetLastError();
}

cudaError_t launch_major(const uint4 *planes, int nsnp, int Wp, uint8_t *maj, cudaStream_t stream)
{
    const long long threads = 32LL * nsnp;
    k_major<<<(unsigned)((threads + 255) / 256), 256, 0, stream>>>(planes, nsnp, Wp, maj);
    return cudaGetLastError();
}

cudaError_t launch_marg(const uint4 *planes, int nsnp, int Wp, const float *y, const uint32_t *wmask, int Np,
                        int ntraits, double *pmC, int32_t *pmN, double *pmQ, cudaStream_t stream)
{
    const long long threads = 32LL * nsnp * ntraits;
    k_marg<<<(unsigned)((threads + 255) / 256), 256, 0, stream>>>(planes, nsnp, Wp, y, wmask, Np, ntraits, pmC, pmN,
                                                                 pmQ);
    return cudaGetLastError();
}

cudaError_t launch_unpack(const int32_t *raw, int nsnp, int nid, int npack, int remain, uint4 *planes, int Wp,
                          uint32_t *codes, int Wc, uint8_t *hcodes, uint8_t *h3, uint32_t *missbits,
                          cudaStream_t stream)
{
    const int npack1 = remain ? npack + 1 : npack;
    const long long total = (long long)nsnp * Wp;
    const int nt = 256;
    const long long nb = (total + nt - 1) / nt;
    k_unpack<<<(unsigned)nb, nt, 0, stream>>>(raw, nsnp, nid, npack, remain, npack1, planes, Wp, codes, Wc, hcodes,
                                              h3, missbits);
    return cudaGetLastError();
}

cudaError_t launch_qmiss(const uint32_t *missbits, int nsnp, int Wp, const uint32_t *wmask, const double *qd,
                        const double *qr, int Np, int ntraits, double *qm, double *rm, double *nm,
                        float *qmf, cudaStream_t stream)
{
    const long long total = 32LL * nsnp * ntraits;
    const int nt = 256;
    k_qmiss<<<(unsigned)((total + nt - 1) / nt), nt, 0, stream>>>(missbits, nsnp, Wp, wmask, qd, qr, Np, ntraits, qm,
                                                              rm, nm, qmf);
    return cudaGetLastError();
}

cudaError_t launch_expand(const uint8_t *hcodes, const int8_t *ydig, int nsnp, int Np, int ntraits, int screen,
                          int8_t *x, cudaStream_t stream)
{
    const int sets = screen == 0 ? 2 * ntraits : screen == 3 ? (ntraits + GROUP_TRAITS - 1) / GROUP_TRAITS : ntraits;
    const long long total = (long long)sets * nsnp * (Np / 16);
    const int nt = 256;
    const unsigned nb = (unsigned)((total + nt - 1) / nt);
    if (screen == 0) k_expand<2, true><<<nb, nt, 0, stream>>>(hcodes, ydig, nsnp, Np, sets, ntraits, x);
    else if (screen == 1) k_expand<2, false><<<nb, nt, 0, stream>>>(hcodes, ydig, nsnp, Np, sets, ntraits, x);
    else if (screen == 2) k_expand<3, false><<<nb, nt, 0, stream>>>(hcodes, ydig, nsnp, Np, sets, ntraits, x);
    else k_expand<GROUP_TRAITS + 1, false, true><<<nb, nt, 0, stream>>>(hcodes, ydig, nsnp, Np, sets, ntraits, x);
    return cudaGetLastError();
}

}  // namespace epi
