// scan_popc.cu -- the plain form of the pair scan: the reference's per-individual method
// (src/EpiOpenCL.c:110-228: unpack two SNPs, count the 3x3 genotype cells, add the
// phenotype into its cell) redone for the B200's CUDA cores.
//
// Persistent kernel, one 512-thread CTA per SM, pulling (SNP-pair tile, trait) units from a
// queue over the tile schedule of the chromosome blocks (tile shapes: the table at the end of
// this file, chosen by the autotuner). The genotype bit-plane words of the tile's i-SNPs and
// j-SNPs (planes of g==0, g==1, g==2, g!=3 per 32 individuals)
// arrive by TMA, 64 individuals per stage, in a three-stage ring. Each SNP's two genotypes
// other than its most frequent one are its dense genotypes A and B. Per stage:
//   * expansion (all threads, double-buffered): the phenotype-masked plane words of A, B and of the
//     missing calls of each i-SNP, and 13 tables of 32 partial sums: entry e of table g is the sum of
//     y over the individuals 5g + b whose bit b is set in e (the last table has four);
//   * cell counts of the dense 2x2 cells and of the individuals missing at j: AND + __popc of
//     32-bit plane words, 16-bit packed counters;
//   * cell sums S_{Ai,Aj}, S_{Ai,Bj}, S_{Bi,Aj}, S_{Bi,Bj}: the same ANDed words, five individuals at
//     a time, select an entry of each table. A lane holds entry `lane` of the 13 tables in
//     registers, so a look-up is one shift and one warp shuffle (which reads the low five bits of its
//     index) and one add; three chains of adds per cell;
//   * individuals missing at the j-SNP (per lane, sparse): their sums by the i genotype;
//   * individuals missing at the i-SNP (warp-uniform, sparse): their sums and counts by the
//     j genotype, and the sum of y^2 of individuals missing at both SNPs.
// Four FP32 adds per pair and individual, predicated by the bits, took 93 cycles of an SM per 32
// individuals and 32 pairs (32 of them the packed adds, 16 the shared-memory broadcasts of the
// i-SNP's values, much of the rest read-modify-writes of the sparse sums in shared memory). The
// look-ups take 60 (26 shuffles, LSU at 63%, issue at 65%: bound by their latency chains), and the
// sparse sums stand in registers, which four pairs per thread leave room for: 69 cycles at 1%
// missing calls, 10.0 -> 7.4 ms at N = 4,000 x 4,001 SNPs. More warps with two pairs each (768 or
// 1,024 threads), look-ups in shared memory instead of shuffles and for the individuals missing at j
// measured 7.8 to 9.4 ms. Their partial sums of five add fewer roundings than one add per
// individual.
// The most frequent genotypes' row and column and the sum of squares come from per-(trait,
// SNP) FP64 marginals in the epilogue: S_{a,Mj} = R_a(i) - S_{a,Aj} - S_{a,Bj} - S_{a,3}
// (R_a(i) = sum of y over g_i = a), then S_{Mi,b} = C_b(j) - S_{Ai,b} - S_{Bi,b} - S_{3,b},
// likewise the counts, and Q = Qtot - QM_i - QM_j + QMM. Deriving the most frequent
// genotypes keeps the FP32 sums to the smaller cells. Each thread owns 4 whole pairs (the
// warp's 4 i-SNPs x the lane's j-SNP), so the reduction over individuals stays in registers.
// Epilogue: an FP32 screen (upper bounds of F and F2) settles all pairs but those that may be a hit
// or raise a maximum; for these FP64 SSB/SSI/F/F2 (src/EpiOpenCL.c:231-247, :452-486),
// warp-aggregated atomic hit append, per-trait maxima (warp-shuffle reductions).
#include <cuda.h>
#include <cudaTypedefs.h>

#include "epi_internal.cuh"
#include "pair_exact.cuh"
#include "tc_ptx.cuh"

namespace epi {
namespace popc {

// A tile shape: WI x WJ warps, each warp PI i-SNPs x 32 j-SNPs (PI pairs per thread); the
// tile is TI = WI * PI i-SNPs by TJ = 32 * WJ j-SNPs. The autotuner picks one per device and
// workload from the table at the end of this file.
template <int WI_, int WJ_, int PI_>
struct Shape {
    static constexpr int WI = WI_, WJ = WJ_, PI = PI_;
    static constexpr int TI = WI * PI;        // i-SNPs per tile
    static constexpr int TJ = WJ * 32;        // j-SNPs per tile
    static constexpr int NT = WI * WJ * 32;   // threads
    static constexpr int KW = 2;              // 32-individual words per stage
    static constexpr int KI = 32 * KW;        // individuals per stage
    static constexpr int RS = 3;              // TMA ring depth
    static constexpr int G = (KI + 4) / 5;    // tables of partial sums, five individuals each
    static constexpr uint32_t STAGE_BYTES = (TI + TJ) * KW * 16;  // transaction bytes per stage
    static_assert(KW == 2 && 32 * G <= NT && TI * KW <= NT - KI / 4 && TI <= 256 && TJ <= 256 && TI + TJ <= NT,
                  "expansion roles");
    static_assert(PI % 2 == 0, "i-SNPs in pairs");

    struct Smem {
        uint4 raw_i[RS][TI][KW];  // TMA: plane words of the i-tile (row = SNP)
        uint4 raw_j[RS][TJ][KW];  // TMA: plane words of the j-tile
        float tab[2][G][32];      // sums of y over the subsets of five individuals
        uint4 pm[2][KW][TI];      // (P_A & W, P_B & W, missing & W, W) of each i-SNP
        float y[2][KI];           // the stage's trait values (0 where invalid)
        uint64_t full[RS];
        uint8_t maj[TI];          // most frequent genotype of each i-SNP
        uint8_t majj[TJ];         // and of each j-SNP
        long long unit;
        int never;                // always 0: the abort flag of the bounded waits
    };
};

// One pair's accumulators and the per-SNP values its statistics need, passed out of line.
struct PairIn {
    float S[4];    // S_{Ai,Aj}, S_{Ai,Bj}, S_{Bi,Aj}, S_{Bi,Bj}
    float SJ[2];   // S_{Ai,3}, S_{Bi,3}: individuals missing at j
    uint32_t C[3]; // n_{Ai,Aj} | n_{Ai,Bj} << 16, n_{Bi,Aj} | n_{Bi,Bj} << 16, n_{Ai,3} | n_{Bi,3} << 16
    float4 sp;     // individuals missing at i, by g_j: S_{3,0..2}, and QMM
    uint2 spn;     // n_{3,0} | n_{3,1} << 16, n_{3,2}
    int maj, majj, trait, si, sj, gi, gj, size2;
};

// FP64 statistics of one pair: the most frequent genotype's row from the marginals, then the
// reference's formulas (pair_stat); also writes the optional per-pair dump. Out of line, so the
// kernel's accumulators stay in registers.
__device__ __noinline__ PairStat eval_pair(const ScanArgs &a, const PairIn p)
{
    const int Ai = p.maj == 0 ? 1 : 0, Bi = p.maj == 2 ? 1 : 2, Mi = p.maj;
    const int Aj = p.majj == 0 ? 1 : 0, Bj = p.majj == 2 ? 1 : 2, Mj = p.majj;
    const size_t mi = (size_t)p.trait * a.nsnp + p.si, mj = (size_t)p.trait * a.nsnp + p.sj;
    int n[9];
    double S[9];
    // the dense 2 x 2 cells
    n[3 * Ai + Aj] = (int)(p.C[0] & 0xffffu);
    n[3 * Ai + Bj] = (int)(p.C[0] >> 16);
    n[3 * Bi + Aj] = (int)(p.C[1] & 0xffffu);
    n[3 * Bi + Bj] = (int)(p.C[1] >> 16);
    S[3 * Ai + Aj] = (double)p.S[0];
    S[3 * Ai + Bj] = (double)p.S[1];
    S[3 * Bi + Aj] = (double)p.S[2];
    S[3 * Bi + Bj] = (double)p.S[3];
    // the j-SNP's most frequent genotype, rows Ai and Bi: the i-SNP's marginal less the row's
    // other cells and its individuals missing at j
    n[3 * Ai + Mj] = a.pmN[3 * mi + Ai] - n[3 * Ai + Aj] - n[3 * Ai + Bj] - (int)(p.C[2] & 0xffffu);
    n[3 * Bi + Mj] = a.pmN[3 * mi + Bi] - n[3 * Bi + Aj] - n[3 * Bi + Bj] - (int)(p.C[2] >> 16);
    S[3 * Ai + Mj] = a.pmC[3 * mi + Ai] - S[3 * Ai + Aj] - S[3 * Ai + Bj] - (double)p.SJ[0];
    S[3 * Bi + Mj] = a.pmC[3 * mi + Bi] - S[3 * Bi + Aj] - S[3 * Bi + Bj] - (double)p.SJ[1];
    // the i-SNP's most frequent genotype, every column: the j-SNP's marginal less the column's
    // other cells and its individuals missing at i
    const int n3[3] = {(int)(p.spn.x & 0xffffu), (int)(p.spn.x >> 16), (int)p.spn.y};
    const double S3[3] = {(double)p.sp.x, (double)p.sp.y, (double)p.sp.z};
#pragma unroll
    for (int b = 0; b < 3; ++b) {
        n[3 * Mi + b] = a.pmN[3 * mj + b] - n[3 * Ai + b] - n[3 * Bi + b] - n3[b];
        S[3 * Mi + b] = a.pmC[3 * mj + b] - S[3 * Ai + b] - S[3 * Bi + b] - S3[b];
    }
    // an empty cell's sum is 0: a derived sum of an empty cell holds only the rounding of the
    // FP32 sums it was formed from (so a pair without valid individuals keeps F = 0/0 = NaN)
#pragma unroll
    for (int c = 0; c < 9; ++c)
        if (n[c] == 0) S[c] = 0.0;
    const double Qv = a.ysq[p.trait] - a.pmQ[mi] - a.pmQ[mj] + (double)p.sp.w;
    const PairStat s = pair_stat(n, S, Qv, a.test_int != 0);
    if (p.trait == a.report_trait) {
        const size_t o = (size_t)p.gi * p.size2 + p.gj;
        if (a.dump_counts)
#pragma unroll
            for (int c = 0; c < 9; ++c) a.dump_counts[9 * o + c] = n[c];
        if (a.dump_F) a.dump_F[o] = (float)s.F;
        if (a.dump_F2) a.dump_F2[o] = (float)s.F2;
        if (a.dump_df1) a.dump_df1[o] = s.d1;
        if (a.dump_df2) a.dump_df2[o] = s.d2;
    }
    return s;
}

// What the screen keeps of this lane's j-SNP for a tile: the marginals of its genotypes A, B and
// most frequent one (count, sum of y) and the sum of y^2 over its missing calls.
struct JSide {
    float N[3], C[3], q;
};

// Upper bounds of one pair's F and F2 in FP32, from the same sums that eval_pair works with; rows
// and columns in the order A, B, most frequent (F and F2 do not depend on it). n3, s3: individuals
// missing at i by the j genotype in that order. What FP32 costs against eval_pair's FP64, with u = 2^-24:
//   * the sum of squares Q is a difference of numbers up to the trait's whole one, ysq, however little
//     of it the pair keeps (outliers that it misses): four values rounded to FP32 and three operations,
//     below 6 u ysq = 3.6e-7 ysq;
//   * the five derived cell sums are differences of marginals: each is good to 4 u (the most frequent
//     cell 8 u) of the magnitudes it was formed from, together below E = 16 u B, B the sum of all of
//     them. sqrt(P), sqrt(SSB) and sqrt(SSI), P the sum of S^2 / n, are norms of the cell sums or of
//     maps of them of norm <= 1 (scan_mma.cu: the screen), so each is within E of its own;
//   * forming P, M and SSI: below 1e-5 of Q.
// NaN where SSW is then below 1e-3 of Q, too little to be told from the subtraction's rounding.
constexpr float SLK_Q = 4e-7f, SLK_S = 1e-6f, SLK_P = 1e-5f;
__device__ __forceinline__ void upper_f32(const PairIn &p, const JSide &j, const float iN[2], const float iC[2], float iq,
                                          float ysq, const float n3[3], const float s3[3], bool want_int, float &F,
                                          float &F2)
{
    float n[9], S[9];
    n[0] = (float)(p.C[0] & 0xffffu);
    n[1] = (float)(p.C[0] >> 16);
    n[3] = (float)(p.C[1] & 0xffffu);
    n[4] = (float)(p.C[1] >> 16);
    S[0] = p.S[0];
    S[1] = p.S[1];
    S[3] = p.S[2];
    S[4] = p.S[3];
    n[2] = iN[0] - n[0] - n[1] - (float)(p.C[2] & 0xffffu);
    n[5] = iN[1] - n[3] - n[4] - (float)(p.C[2] >> 16);
    S[2] = iC[0] - S[0] - S[1] - p.SJ[0];
    S[5] = iC[1] - S[3] - S[4] - p.SJ[1];
    float N = 0.0f, St = 0.0f, nfac = 0.0f, P = 0.0f;
#pragma unroll
    for (int b = 0; b < 3; ++b) {
        n[6 + b] = j.N[b] - n[b] - n[3 + b] - n3[b];
        S[6 + b] = j.C[b] - S[b] - S[3 + b] - s3[b];
    }
    float mc[9];
#pragma unroll
    for (int c = 0; c < 9; ++c) {
        S[c] = n[c] > 0.0f ? S[c] : 0.0f;  // (a derived sum of an empty cell holds rounding only)
        N += n[c];
        St += S[c];
        nfac += n[c] > 0.0f ? 1.0f : 0.0f;
        mc[c] = S[c] * rcp_fast(n[c] + 1e-30f);
        P = fmaf(S[c], mc[c], P);
    }
    const float m = St * rcp_fast(N + 1e-30f), M = St * m;
    const float Q = fmaf(-SLK_Q, ysq, ysq - iq - j.q + p.sp.w), slack = SLK_P * Q;
    const float B = fabsf(iC[0]) + fabsf(iC[1]) + fabsf(j.C[0]) + fabsf(j.C[1]) + fabsf(j.C[2]) + fabsf(S[0]) +
                    fabsf(S[1]) + fabsf(S[3]) + fabsf(S[4]) + fabsf(p.SJ[0]) + fabsf(p.SJ[1]) + fabsf(s3[0]) +
                    fabsf(s3[1]) + fabsf(s3[2]);
    const float E = SLK_S * B;
    const float sP = sqrt_fast(P + slack) + E, sB = sqrt_fast(fmaxf(P - M + slack, 0.0f)) + E;
    const float W = Q - sP * sP;  // (Q <= 0: NaN or negative)
    const float d1 = nfac - 1.0f, d2 = N - nfac;
    const bool ok = W > 1e-3f * Q;
    const float nan = __int_as_float(0x7fc00000);
    F = ok ? sB * sB * d2 * rcp_fast(d1 * W) : nan;
    F2 = 0.0f;
    if (want_int) {
        float row[3], col[3], SSI = slack;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            row[i] = (S[3 * i] + S[3 * i + 1] + S[3 * i + 2]) * rcp_fast(n[3 * i] + n[3 * i + 1] + n[3 * i + 2] + 1e-30f);
            col[i] = (S[i] + S[3 + i] + S[6 + i]) * rcp_fast(n[i] + n[3 + i] + n[6 + i] + 1e-30f);
        }
#pragma unroll
        for (int c = 0; c < 9; ++c) {
            const float t = mc[c] - row[c / 3] - col[c % 3] + m;
            SSI = fmaf(n[c] * t, t, SSI);
        }
        const float sI = sqrt_fast(SSI) + E;
        F2 = ok ? sI * sI * d2 * rcp_fast(4.0f * W) : nan;
    }
}

__device__ __forceinline__ bool bit(uint32_t w, int t) { return (w >> t) & 1u; }

template <class Sh>
__global__ void __launch_bounds__(Sh::NT, 1) k_scan_popc(ScanArgs a, const __grid_constant__ PopcMaps maps)
{
    constexpr int WI = Sh::WI, PI = Sh::PI, TI = Sh::TI, TJ = Sh::TJ, NT = Sh::NT, KW = Sh::KW, KI = Sh::KI;
    constexpr int RS = Sh::RS;
    using Smem = typename Sh::Smem;
    extern __shared__ uint8_t smem_raw[];
    // TMA destinations: 1024-byte aligned
    const uint32_t raw_s = tc::smem_u32(smem_raw);
    Smem &sm = *reinterpret_cast<Smem *>(smem_raw + (((raw_s + 1023u) & ~1023u) - raw_s));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int wi = warp % WI, wj = warp / WI;
    const int ib = wi * PI, jl = wj * 32 + lane;  // this thread's first i row, its j row
    const int nst = a.Wp / KW;
    const long long units = a.ntiles * (long long)a.ntraits;

    // maxima of F and F2 per trait: per CTA in shared memory (flushed once, at the end) up to
    // SMAX_TRAITS traits, else the global maxima directly
    const bool smax_local = a.ntraits <= SMAX_TRAITS;
    unsigned int *smax = reinterpret_cast<unsigned int *>(reinterpret_cast<uint8_t *>(&sm) + sizeof(Smem));
    if (smax_local)
        for (int w = tid; w < 2 * a.ntraits; w += NT) smax[w] = 0u;
    unsigned int *const mxf = smax_local ? smax : a.maxf;
    unsigned int *const mxf2 = smax_local ? smax + a.ntraits : a.maxf2;
    if (tid == 0) {
        for (int r = 0; r < RS; ++r) tc::mbar_init(&sm.full[r], 1);
        sm.never = 0;
        tc::fence_barrier_init();
    }
    __syncthreads();
    uint32_t par = 0u;  // parity of each ring slot's next phase (bit r), the same in every thread

    // every thread: wait for stage `st`'s words (bounded; a timeout is recorded, and the
    // control flow stays the same in every thread)
    auto wait_stage = [&](int st) {
        const int r = st % RS;
        if (!tc::mbar_wait(&sm.full[r], (par >> r) & 1u, &sm.never, a.wait_ns) && lane == 0 &&
            atomicCAS(&a.counters[2], 0ull, 1ull) == 0ull)
            a.counters[3] = 20ull;
        par ^= 1u << r;
    };

    for (;;) {
        if (tid == 0) sm.unit = (long long)atomicAdd(&a.counters[1], 1ull);
        __syncthreads();
        const long long u = sm.unit;
        __syncthreads();
        if (u >= units) break;
        const long long tile = u / a.ntraits;
        const int t = (int)(u % a.ntraits);
        const int blk = find_block(a.blocks, a.nblocks, tile);
        const BlockDesc bd = a.blocks[blk];
        const long long lt = tile - bd.tile_base;
        const int i0 = (int)(lt / bd.tiles_j) * TI, j0 = (int)(lt % bd.tiles_j) * TJ;
        // no pair with snp1 > snp2 in this tile (upper part of a diagonal block)
        if (bd.start1 + min(i0 + TI, bd.size1) - 1 <= bd.start2 + j0) continue;

        const float *yt = a.y + (size_t)t * a.Np;
        const uint32_t *wt = a.wmask + (size_t)t * a.Wp;
        if (tid < TI) sm.maj[tid] = i0 + tid < bd.size1 ? a.maj[bd.start1 + i0 + tid] : (uint8_t)0;
        else if (tid < TI + TJ)
            sm.majj[tid - TI] = j0 + tid - TI < bd.size2 ? a.maj[bd.start2 + j0 + tid - TI] : (uint8_t)0;
        auto issue = [&](int st) {  // thread 0: the TMA loads of stage st
            const int r = st % RS;
            tc::mbar_arrive_expect_tx(&sm.full[r], Sh::STAGE_BYTES);
            tc::tma_load_2d(&sm.raw_i[r][0][0], &maps.planes_i, 4 * KW * st, bd.start1 + i0, &sm.full[r]);
            tc::tma_load_2d(&sm.raw_j[r][0][0], &maps.planes_j, 4 * KW * st, bd.start2 + j0, &sm.full[r]);
        };
        if (tid == 0)
            for (int st = 0; st < min(RS, nst); ++st) issue(st);
        __syncthreads();  // maj

        // expansion of stage st into buffer b
        auto expand = [&](int st, int b) {
            const int r = st % RS;
            if (tid < 32 * Sh::G) {
                const int g = tid >> 5;
                float v = 0.f;
#pragma unroll
                for (int e = 0; e < 5; ++e)
                    if (5 * g + e < KI && bit(lane, e)) v += __ldg(yt + KI * st + 5 * g + e);
                sm.tab[b][g][lane] = v;
            }
            if (tid < TI * KW) {
                const int i = tid % TI, w = tid / TI;
                const uint4 P = sm.raw_i[r][i][w];
                const int mj = sm.maj[i];
                const uint32_t W = __ldg(wt + KW * st + w);
                const uint32_t PA = mj == 0 ? P.y : P.x, PB = mj == 2 ? P.y : P.z;
                sm.pm[b][w][i] = make_uint4(PA & W, PB & W, ~P.w & W, W);
            } else if (tid >= NT - KI / 4) {
                const int q = tid - (NT - KI / 4);
                reinterpret_cast<float4 *>(sm.y[b])[q] = __ldg(reinterpret_cast<const float4 *>(yt + KI * st) + q);
            }
        };

        wait_stage(0);
        expand(0, 0);
        __syncthreads();

        float2 S[PI / 2][4];  // the cell sums of i-SNPs ib + 2p (x) and ib + 2p + 1 (y)
        uint32_t C[PI][3];
        float4 sps[PI];       // per pair: sums over individuals missing at i by g_j: S_30..S_32, QMM
        uint2 spn[PI];        // and counts: n_30 | n_31 << 16, n_32
        float2 spj[PI];       // per pair: sums over individuals missing at j by g_i: S_{Ai,3}, S_{Bi,3}
#pragma unroll
        for (int ii = 0; ii < PI; ++ii) {
            if (ii % 2 == 0)
#pragma unroll
                for (int c = 0; c < 4; ++c) S[ii / 2][c] = make_float2(0.f, 0.f);
            C[ii][0] = C[ii][1] = C[ii][2] = 0u;
            sps[ii] = make_float4(0.f, 0.f, 0.f, 0.f);
            spn[ii] = make_uint2(0u, 0u);
            spj[ii] = make_float2(0.f, 0.f);
        }
        const int mjj = sm.majj[jl];  // this lane's j-SNP: its dense genotypes' planes

        for (int st = 0; st < nst; ++st) {
            const int b = st & 1, r = st % RS;
            if (st + 1 < nst) {
                wait_stage(st + 1);
                expand(st + 1, b ^ 1);
            }
            float T[Sh::G];  // this lane's entries of the tables
#pragma unroll
            for (int g = 0; g < Sh::G; ++g) T[g] = sm.tab[b][g][lane];
            const uint4 pj[2] = {sm.raw_j[r][jl][0], sm.raw_j[r][jl][1]};
            const uint32_t Xj[2][2] = {{mjj == 0 ? pj[0].y : pj[0].x, mjj == 0 ? pj[1].y : pj[1].x},   // A
                                       {mjj == 2 ? pj[0].y : pj[0].z, mjj == 2 ? pj[1].y : pj[1].z}};  // B
            const uint32_t Mj[2] = {~pj[0].w, ~pj[1].w};
#pragma unroll
            for (int q = 0; q < PI / 2; ++q) {
                const uint4 pm[2][2] = {{sm.pm[b][0][ib + 2 * q], sm.pm[b][1][ib + 2 * q]},
                                        {sm.pm[b][0][ib + 2 * q + 1], sm.pm[b][1][ib + 2 * q + 1]}};
                // the dense cells: counts, and sums by look-up (all lanes of the warp are here)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    uint32_t x[2][2];
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
#pragma unroll
                        for (int w = 0; w < 2; ++w) x[e][w] = (c < 2 ? pm[e][w].x : pm[e][w].y) & Xj[c & 1][w];
                        C[2 * q + e][c >> 1] += (uint32_t)(__popc(x[e][0]) + __popc(x[e][1])) << (16 * (c & 1));
                    }
                    float2 s[3];
#pragma unroll
                    for (int g = 0; g < Sh::G; ++g) {
                        const int k = 5 * g;
                        float2 v;
                        v.x = __shfl_sync(0xffffffffu, T[g], (int)(k < 32 ? __funnelshift_r(x[0][0], x[0][1], k) : x[0][1] >> (k - 32)));
                        v.y = __shfl_sync(0xffffffffu, T[g], (int)(k < 32 ? __funnelshift_r(x[1][0], x[1][1], k) : x[1][1] >> (k - 32)));
                        if (g < 3) s[g] = v;
                        else { s[g % 3].x += v.x; s[g % 3].y += v.y; }
                    }
                    s[0].x += s[1].x; s[0].y += s[1].y; s[0].x += s[2].x; s[0].y += s[2].y;
                    S[q][c].x += s[0].x; S[q][c].y += s[0].y;
                }
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int ii = 2 * q + e;
                    // the sparse individuals missing at i
#pragma unroll
                    for (int w = 0; w < 2; ++w) {
                        uint32_t m = pm[e][w].z;  // the same in every lane of the warp
                        if (!m) continue;
                        spn[ii].x += (uint32_t)__popc(m & pj[w].x) + ((uint32_t)__popc(m & pj[w].y) << 16);
                        spn[ii].y += (uint32_t)__popc(m & pj[w].z);
#pragma unroll 1
                        while (m) {
                            const int k = __ffs(m) - 1;
                            m &= m - 1u;
                            const float yv = sm.y[b][32 * w + k];
                            if (bit(pj[w].x, k)) sps[ii].x += yv;
                            if (bit(pj[w].y, k)) sps[ii].y += yv;
                            if (bit(pj[w].z, k)) sps[ii].z += yv;
                            if (bit(Mj[w], k)) sps[ii].w = fmaf(yv, yv, sps[ii].w);
                        }
                    }
                }
            }
            // individuals missing at this lane's j-SNP (and phenotype-valid): their sums by
            // the i genotype (per lane; rare)
            uint32_t mj = Mj[0] & sm.pm[b][0][ib].w, mj1 = Mj[1] & sm.pm[b][1][ib].w;
            int w = 0;
            if (!mj) {
                mj = mj1;
                mj1 = 0u;
                w = 1;
            }
#pragma unroll 1
            while (mj) {
                const int k = __ffs(mj) - 1;
                mj &= mj - 1u;
                const float yv = sm.y[b][32 * w + k];
                const uint4 *const row = &sm.pm[b][w][ib];
                if (!mj) {
                    mj = mj1;
                    mj1 = 0u;
                    w = 1;
                }
#pragma unroll
                for (int ii = 0; ii < PI; ++ii) {
                    const uint2 pab = *reinterpret_cast<const uint2 *>(row + ii);
                    if (bit(pab.x, k)) {
                        spj[ii].x += yv;
                        C[ii][2] += 1u;
                    }
                    if (bit(pab.y, k)) {
                        spj[ii].y += yv;
                        C[ii][2] += 0x10000u;
                    }
                }
            }
            __syncwarp();
            __syncthreads();  // stage st consumed (its ring slot and expansion buffer), st + 1 expanded
            if (tid == 0 && st + RS < nst) issue(st + RS);
        }

        // epilogue
        const bool report = a.report_trait < 0 || a.report_trait == t;
        const bool dumping = t == a.report_trait && (a.dump_counts || a.dump_F || a.dump_F2 || a.dump_df1 || a.dump_df2);
        const float t1c = screen_lo(a.t1), t2c = screen_lo(a.t2);
        const float ysq = (float)a.ysq[t];
        JSide js;
        {
            const int gj = min(j0 + jl, bd.size2 - 1);
            const size_t mj = (size_t)t * a.nsnp + bd.start2 + gj;
            const int A = mjj == 0 ? 1 : 0, B = mjj == 2 ? 1 : 2;
            js.N[0] = (float)a.pmN[3 * mj + A];
            js.N[1] = (float)a.pmN[3 * mj + B];
            js.N[2] = (float)a.pmN[3 * mj + mjj];
            js.C[0] = (float)a.pmC[3 * mj + A];
            js.C[1] = (float)a.pmC[3 * mj + B];
            js.C[2] = (float)a.pmC[3 * mj + mjj];
            js.q = (float)a.pmQ[mj];
        }
        // unrolled: S and C are indexed by constants only, so they stay in registers
#pragma unroll
        for (int ii = 0; ii < PI; ++ii) {
            const int gi = i0 + ib + ii, gj = j0 + jl;
            const bool valid = gi < bd.size1 && gj < bd.size2 && (bd.start1 + gi > bd.start2 + gj);
            PairIn p;
#pragma unroll
            for (int c = 0; c < 4; ++c) p.S[c] = ii % 2 ? S[ii / 2][c].y : S[ii / 2][c].x;
            p.SJ[0] = spj[ii].x;
            p.SJ[1] = spj[ii].y;
#pragma unroll
            for (int c = 0; c < 3; ++c) p.C[c] = C[ii][c];
            p.sp = sps[ii];
            p.spn = spn[ii];
            p.maj = sm.maj[ib + ii];
            p.majj = mjj;
            p.trait = t;
            p.si = bd.start1 + gi;
            p.sj = bd.start2 + gj;
            p.gi = gi;
            p.gj = gj;
            p.size2 = bd.size2;
            bool exact = valid;
            if (!dumping) {
                const size_t mi = (size_t)t * a.nsnp + bd.start1 + min(gi, bd.size1 - 1);
                const int A = p.maj == 0 ? 1 : 0, B = p.maj == 2 ? 1 : 2;
                const float iN[2] = {(float)a.pmN[3 * mi + A], (float)a.pmN[3 * mi + B]};
                const float iC[2] = {(float)a.pmC[3 * mi + A], (float)a.pmC[3 * mi + B]};
                const float g0 = (float)(p.spn.x & 0xffffu), g1 = (float)(p.spn.x >> 16), g2 = (float)p.spn.y;
                const float n3[3] = {mjj == 0 ? g1 : g0, mjj == 2 ? g1 : g2, pick3(g0, g1, g2, mjj)};
                const float s3[3] = {mjj == 0 ? p.sp.y : p.sp.x, mjj == 2 ? p.sp.y : p.sp.z,
                                     pick3(p.sp.x, p.sp.y, p.sp.z, mjj)};
                float uF, uF2;
                upper_f32(p, js, iN, iC, (float)a.pmQ[mi], ysq, n3, s3, a.test_int != 0, uF, uF2);
                // the CTA's maxima so far are exact values and bound the final ones from below
                const unsigned int m1 = reinterpret_cast<volatile unsigned int *>(mxf)[t];
                const unsigned int m2 = a.test_int ? reinterpret_cast<volatile unsigned int *>(mxf2)[t] : 0u;
                const float l1 = m1 ? screen_lo(ord2f(m1)) : -INFINITY, l2 = m2 ? screen_lo(ord2f(m2)) : -INFINITY;
                exact = valid && (!(uF <= (report ? fminf(t1c, l1) : l1)) ||
                                  (a.test_int && !(uF2 <= (report ? fminf(t2c, l2) : l2))));
            }
            if (!__any_sync(0xffffffffu, exact)) continue;
            PairStat s;
            s.nfac = s.d1 = s.d2 = 0;
            s.F = s.F2 = 0.0;
            if (exact) s = eval_pair(a, p);
            const bool hit = exact && report && is_hit(a, s);
            emit_hit(a, hit, bd.start1 + gi, bd.start2 + gj, s, t, blk);
            fold_max(&mxf[t], exact, s.F);
            if (a.test_int) fold_max(&mxf2[t], exact, s.F2);
        }
    }
    __syncthreads();
    if (smax_local)
        for (int w = tid; w < 2 * a.ntraits; w += NT)
            if (smax[w]) atomicMax(w < a.ntraits ? &a.maxf[w] : &a.maxf2[w - a.ntraits], smax[w]);
}

}  // namespace popc

// The tile shapes the autotuner chooses among:
//   0  32 x 64 tile (8 x 2 warps)
//   1  64 x 32 tile (16 x 1 warps): the j side's words shared by more warps
//   2  16 x 128 tile (4 x 4 warps): the i side's
using Shape0 = popc::Shape<8, 2, 4>;
using Shape1 = popc::Shape<16, 1, 4>;
using Shape2 = popc::Shape<4, 4, 4>;
constexpr int POPC_SHAPES = 3;

int popc_shapes() { return POPC_SHAPES; }

// Tile size (i x j SNPs) and a description of shape v.
void popc_shape(int v, int *ti, int *tj, const char **desc)
{
    static const char *names[POPC_SHAPES] = {"32x64 tile, 4 pairs/thread, 8x2 warps",
                                             "64x32 tile, 4 pairs/thread, 16x1 warps",
                                             "16x128 tile, 4 pairs/thread, 4x4 warps"};
    const int tis[POPC_SHAPES] = {Shape0::TI, Shape1::TI, Shape2::TI};
    const int tjs[POPC_SHAPES] = {Shape0::TJ, Shape1::TJ, Shape2::TJ};
    *ti = tis[v];
    *tj = tjs[v];
    if (desc) *desc = names[v];
}

// The plane words [nsnp][Wp] (uint4) as a 2-D uint32 tensor [nsnp][4 Wp]; one box = the words
// of one stage (KW x 4 uint32 = 32 bytes) of `rows` SNPs; rows past the last SNP read as 0.
static cudaError_t encode_planes(CUtensorMap *m, const uint4 *planes, int nsnp, int Wp, int rows)
{
    static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    if (!encode) {
        cudaDriverEntryPointQueryResult q;
        void *fn = nullptr;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
        if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !fn) return cudaErrorNotSupported;
        encode = (PFN_cuTensorMapEncodeTiled_v12000)fn;
    }
    const cuuint64_t dims[2] = {4 * (cuuint64_t)Wp, (cuuint64_t)nsnp};
    const cuuint64_t strides[1] = {16 * (cuuint64_t)Wp};
    const cuuint32_t box[2] = {4 * Shape0::KW, (cuuint32_t)rows};
    const cuuint32_t es[2] = {1, 1};
    CUresult r = encode(m, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<uint4 *>(planes), dims, strides, box, es,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

cudaError_t popc_encode_planes(int v, PopcMaps *maps, const uint4 *planes, int nsnp, int Wp)
{
    int ti = 0, tj = 0;
    popc_shape(v, &ti, &tj, nullptr);
    cudaError_t e = encode_planes(&maps->planes_i, planes, nsnp, Wp, ti);
    if (e == cudaSuccess) e = encode_planes(&maps->planes_j, planes, nsnp, Wp, tj);
    return e;
}

template <class C>
static size_t shape_smem(int ntraits)
{
    return sizeof(typename C::Smem) + 1024 + smax_bytes(ntraits);
}

template <class C>
static cudaError_t prepare(void)
{
    return cudaFuncSetAttribute(popc::k_scan_popc<C>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)shape_smem<C>(SMAX_TRAITS));
}

template <class C>
static cudaError_t enqueue(const ScanArgs &a, const PopcMaps &maps, int grid, cudaStream_t stream)
{
    popc::k_scan_popc<C><<<grid, C::NT, shape_smem<C>(a.ntraits), stream>>>(a, maps);
    return cudaGetLastError();
}

// Before any stream capture: the shape's kernel attribute (the largest shared-memory size any
// trait count asks for).
cudaError_t popc_prepare(int v)
{
    switch (v) {
    case 0: return prepare<Shape0>();
    case 1: return prepare<Shape1>();
    case 2: return prepare<Shape2>();
    }
    return cudaErrorInvalidValue;
}

// The launch itself (a stream operation only, so it can be captured into a CUDA graph).
cudaError_t popc_enqueue(int v, const ScanArgs &a, const PopcMaps &maps, int grid, cudaStream_t stream)
{
    switch (v) {
    case 0: return enqueue<Shape0>(a, maps, grid, stream);
    case 1: return enqueue<Shape1>(a, maps, grid, stream);
    case 2: return enqueue<Shape2>(a, maps, grid, stream);
    }
    return cudaErrorInvalidValue;
}

}  // namespace epi
