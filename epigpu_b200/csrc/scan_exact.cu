// scan_exact.cu -- the exact statistics of the pairs that the tensor form's screen could not
// settle (the candidate list of k_scan_mma's screened variants, scan_mma.cu).
//
// One warp per candidate: the 3x3 counts and the three digit sums of every cell over the
// one-hot genotype bytes and the trait's digit rows, 16 individuals per lane and step, as byte
// masks and dp4a (36 accumulators; int32, so the sums are the same integers that the full
// MMA gives), then the same FP64 statistics (pair_stat_exact). The reference's per-pair loop is
// src/EpiOpenCL.c:110-247 and :452-489.
// FROM_Y: from y itself in FP64 instead of the digits, which hold it to 2^-24 of the trait's largest value:
// for the few individuals whose automatic form was the plain one before there was a screen, so that the
// results keep its precision (200 individuals with an outlier of 1,000 standard deviations: F of a pair
// that misses it is good to 1e-7 from y and to 2e-5 from the digits).
// About 57 instructions per 128 individuals and warp: 5,000 per candidate at 10,000
// individuals. At 1e-4 of the pairs that is under 1% of the screen's time, which is why the
// list is worked off pair by pair and not as tiles.
#include "epi_internal.cuh"
#include "pair_exact.cuh"

namespace epi {

constexpr int EXACT_NT = 256;

// RAW (epi_scan_block_noalloc): the genotypes come from the reference's packed words, ytilde from
// the digits, the missing sums by the SNP's place in the block (qm, sm, nm of the i side, then of
// the j side), and the hits go out as 24-byte rows.

// the sum of ytilde^2 over the individuals missing at both SNPs, as missing_both_q, from the packed words
__device__ __forceinline__ double missing_both_packed(const ScanArgs &a, const uint32_t *ri, const uint32_t *rj)
{
    const int8_t *dg = a.ydig;
    double part = 0.0;
    for (int w = threadIdx.x & 31; 16 * w < a.nid; w += 32) {
        const uint32_t x = packed_word(ri, w, a.npack, a.remain) & packed_word(rj, w, a.npack, a.remain);
        uint32_t m = x & (x >> 1) & 0x55555555u;  // both bits of both codes
        while (m) {
            const int k = 16 * w + 15 - ((31 - __clz(m)) >> 1);
            m &= ~(0x80000000u >> __clz(m));
            if (k < a.nid && dg[a.Np + k]) {
                const int Y = dg[4 * a.Np + k] + 256 * dg[3 * a.Np + k] + 65536 * dg[2 * a.Np + k];
                const double yq = (double)Y * a.yscale[0];
                part += yq * yq;
            }
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) part += __shfl_xor_sync(0xffffffffu, part, off);
    return part;
}

// FROM_Y: the pair's counts and sums of y by cell, and its sum of y^2, four individuals per lane and
// step (every lane gets them).
__device__ __forceinline__ void cells_from_y(const ScanArgs &a, int t, int snp1, int snp2, int n[9], double S[9], double &Q)
{
    const uint8_t *hi = a.hcodes + (size_t)snp1 * a.Np, *hj = a.hcodes + (size_t)snp2 * a.Np;
    const int8_t *w = a.ydig + ((size_t)t * 5 + 1) * a.Np;
    const float *y = a.y + (size_t)t * a.Np;
    Q = 0.0;
#pragma unroll
    for (int c = 0; c < 9; ++c) {
        n[c] = 0;
        S[c] = 0.0;
    }
    for (int k = threadIdx.x & 31; k < a.Np; k += 128) {  // (Np is a multiple of 128; a step's loads together)
        int gi[4], gj[4], wk[4];  // 1 << genotype, 0: missing
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            gi[e] = hi[k + 32 * e];
            gj[e] = hj[k + 32 * e];
            wk[e] = w[k + 32 * e];
            v[e] = y[k + 32 * e];
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int cell = gi[e] && gj[e] && wk[e] ? 3 * (gi[e] >> 1) + (gj[e] >> 1) : 9;
            const double x = (double)v[e];
#pragma unroll
            for (int c = 0; c < 9; ++c)
                if (cell == c) {
                    ++n[c];
                    S[c] += x;
                }
            if (cell < 9) Q = fma(x, x, Q);
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        Q += __shfl_xor_sync(0xffffffffu, Q, off);
#pragma unroll
        for (int c = 0; c < 9; ++c) S[c] += __shfl_xor_sync(0xffffffffu, S[c], off);
    }
#pragma unroll
    for (int c = 0; c < 9; ++c) n[c] = __reduce_add_sync(0xffffffffu, n[c]);
}

template <bool RAW, bool FROM_Y>
__global__ void __launch_bounds__(EXACT_NT, 2) k_exact(ScanArgs a)
{
    const int lane = threadIdx.x & 31;
    const long long warp = ((long long)blockIdx.x * EXACT_NT + threadIdx.x) >> 5, nwarps = (long long)gridDim.x * (EXACT_NT / 32);
    const long long found = (long long)a.counters[CNT_CAND + a.segment];
    if (found > a.cand_cap || a.counters[CNT_OVERFLOW]) {
        // the list does not hold them all: the host scans again without the screen
        if (blockIdx.x == 0 && threadIdx.x == 0) a.counters[CNT_OVERFLOW] = 1ull;
        return;
    }
    const float t1c = screen_lo(a.t1), t2c = screen_lo(a.t2);
    const int nc = a.Np / 16;
    for (long long q = warp; q < found; q += nwarps) {
        const Cand c = a.cand[q];
        const int t = c.trait;
        const bool report = a.report_trait < 0 || a.report_trait == t;
        // against the lower bounds of the maxima as they stand now (the same for every lane)
        unsigned int lF = 0u, lI = 0u;
        if (lane == 0) {
            lF = reinterpret_cast<volatile unsigned int *>(a.lowf)[t];
            lI = reinterpret_cast<volatile unsigned int *>(a.lowf2)[t];
        }
        const float mF = screen_lo(ord2f(__shfl_sync(0xffffffffu, lF, 0)));
        const float mI = screen_lo(ord2f(__shfl_sync(0xffffffffu, lI, 0)));
        if (c.fu < (report ? fminf(t1c, mF) : mF) && (!a.test_int || c.f2u < (report ? fminf(t2c, mI) : mI))) continue;

        int n[9];
        double si[9], sc = 1.0, Q;
        if constexpr (FROM_Y) {
            cells_from_y(a, t, c.snp1, c.snp2, n, si, Q);
        } else {
            const uint4 *hi = nullptr, *hj = nullptr;
            const uint32_t *ri = nullptr, *rj = nullptr;
            if (RAW) {
                const size_t npack1 = a.npack + (a.remain > 0);
                ri = reinterpret_cast<const uint32_t *>(a.gpack) + c.snp1 * npack1;
                rj = reinterpret_cast<const uint32_t *>(a.gpack) + c.snp2 * npack1;
            } else {
                hi = reinterpret_cast<const uint4 *>(a.hcodes + (size_t)c.snp1 * a.Np);
                hj = reinterpret_cast<const uint4 *>(a.hcodes + (size_t)c.snp2 * a.Np);
            }
            const uint4 *dg = reinterpret_cast<const uint4 *>(a.ydig + ((size_t)t * 5 + 1) * a.Np);
            int acc[9][4];
#pragma unroll
            for (int k = 0; k < 9; ++k)
#pragma unroll
                for (int r = 0; r < 4; ++r) acc[k][r] = 0;
            // the chunks of the next step are fetched while this one's are worked on: a step waits about as
            // long for its loads as it computes, and few candidates leave few warps to hide that
            uint4 vi, vj, d[4];
            uint32_t pi = 0u, pj = 0u;
            auto fetch = [&](int k) {
                if (k >= nc) return;
                if (RAW) {
                    pi = packed_raw(ri, k, a.npack + (a.remain > 0));
                    pj = packed_raw(rj, k, a.npack + (a.remain > 0));
                } else {
                    vi = hi[k];
                    vj = hj[k];
                }
#pragma unroll
                for (int r = 0; r < 4; ++r) d[r] = dg[r * nc + k];
            };
            fetch(lane);
            for (int k = lane; k < nc; k += 32) {
                uint4 ci = vi, cj = vj;
                const uint4 e[4] = {d[0], d[1], d[2], d[3]};
                if (RAW) {
                    const auto one_hot = [&](uint32_t w) {
                        uint32_t sel[4];
                        packed_selectors(packed_aligned(w, k, a.npack, a.remain), sel);
                        return packed_lookup(PACKED_TABLE(1u, 2u, 4u, 0u), sel);
                    };
                    ci = one_hot(pi);
                    cj = one_hot(pj);
                }
                fetch(k + 32);
                const uint32_t wi[4] = {ci.x, ci.y, ci.z, ci.w}, wj[4] = {cj.x, cj.y, cj.z, cj.w};
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    int dx[4];
#pragma unroll
                    for (int r = 0; r < 4; ++r) dx[r] = (int)(x == 0 ? e[r].x : x == 1 ? e[r].y : x == 2 ? e[r].z : e[r].w);
#pragma unroll
                    for (int g = 0; g < 3; ++g) {
                        const uint32_t mi = (wi[x] >> g) & 0x01010101u;
#pragma unroll
                        for (int b = 0; b < 3; ++b) {
                            const int m = (int)(mi & (wj[x] >> b));
#pragma unroll
                            for (int r = 0; r < 4; ++r) acc[3 * g + b][r] = __dp4a(m, dx[r], acc[3 * g + b][r]);
                        }
                    }
                }
            }
            int N = 0;
            double st = 0.0;
#pragma unroll
            for (int k = 0; k < 9; ++k) {
                n[k] = __reduce_add_sync(0xffffffffu, acc[k][0]);
                const int x3 = __reduce_add_sync(0xffffffffu, acc[k][1]);
                const int x2 = __reduce_add_sync(0xffffffffu, acc[k][2]);
                const int x1 = __reduce_add_sync(0xffffffffu, acc[k][3]);
                si[k] = fma(65536.0, (double)x3, fma(256.0, (double)x2, (double)x1));
                st += si[k];
                N += n[k];
            }
            // the sum of squares: see scan_mma.cu
            size_t mi = (size_t)t * a.nsnp + c.snp1, mj = (size_t)t * a.nsnp + c.snp2;
            if (RAW) {
                mi = c.snp1 - a.blocks[0].start1;
                mj = RAW_SNPS + c.snp2 - a.blocks[0].start2;
            }
            sc = a.yscale[t];
            const int nmm = N + (int)(a.nm[mi] - a.nvalid[t] + a.nm[mj]);
            double qmm = 0.0;
            if (nmm == 1) {
                const double ymm = (st - a.ytot[t] + a.sm[mi] + a.sm[mj]) * sc;
                qmm = ymm * ymm;
            } else if (nmm >= 2) {
                qmm = RAW ? missing_both_packed(a, ri, rj) : missing_both_q(a, t, c.snp1, c.snp2);
            }
            Q = a.qtot[t] - a.qm[mi] - a.qm[mj] + qmm;
        }
        const PairStat s = pair_stat_exact(n, si, sc, Q, a.test_int != 0);
        const bool hit = lane == 0 && report && is_hit(a, s);
        if (RAW) emit_row(a, hit, c.snp1, c.snp2, s);
        else emit_hit(a, hit, c.snp1, c.snp2, s, t, c.block);
        if (lane == 0) {
            auto raise = [](unsigned int *max, unsigned int *low, double F) {
                if (!(F == F)) return;
                const unsigned int v = f2ord((float)F);
                if (v > *reinterpret_cast<volatile unsigned int *>(max)) atomicMax(max, v);
                if (v > *reinterpret_cast<volatile unsigned int *>(low)) atomicMax(low, v);
            };
            raise(&a.maxf[t], &a.lowf[t], s.F);
            if (a.test_int) raise(&a.maxf2[t], &a.lowf2[t], s.F2);
        }
    }
}

cudaError_t exact_enqueue(const ScanArgs &a, int sm_count, cudaStream_t stream)
{
    if (a.gpack) k_exact<true, false><<<2 * sm_count, EXACT_NT, 0, stream>>>(a);
    else if (a.from_y) k_exact<false, true><<<2 * sm_count, EXACT_NT, 0, stream>>>(a);
    else k_exact<false, false><<<2 * sm_count, EXACT_NT, 0, stream>>>(a);
    return cudaGetLastError();
}

}  // namespace epi
