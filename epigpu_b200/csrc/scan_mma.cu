// scan_mma.cu -- tensor-core form of the pair scan (tcgen05, kind::i8, sm_100a).
//
// Per pair (i, j) the reference accumulates, over individuals k, the 3x3 genotype-cell
// counts and phenotype sums (src/EpiOpenCL.c:110-228). Both are contractions over k:
//     n_ab = sum_k [g_i(k)=a] [g_j(k)=b] w_k        S_ab = sum_k [g_i(k)=a] [g_j(k)=b] y_k
// so for a tile of 40 i-SNPs x 21 j-SNPs they are one integer GEMM
//     D[128 x 252] = A[128 x K] * B[K x 252]
//   A rows (row 32w + l, l < 30): i-SNP 10w + l/3, genotype a = l%3: [g_i(k) == a]
//   B cols: type t = 4b + s (b = 0..2 the j genotype, s = 0..3), [g_j(k) == b] * D_s(k), with
//     D_0 = w_k (phenotype valid) and D_1..3 the balanced base-256 digits, the highest first, of
//     the fixed-point phenotype Y_k = round(y_k * 2^sy) (y centred, 0 when invalid); CTA 0 of the pair holds
//     the types of D_0 and D_1, CTA 1 those of D_2 and D_3, so each builds its half from two
//     digit rows: column of (t, j') in the pair MMA 128 (s / 2) + 6 j' + (2b + s % 2), the six
//     columns of a j-SNP side by side in each half.
// int8 operands, int32 accumulation: counts and digit sums are exact, so
//     S_ab = (65536 D1 + 256 D2 + D3) * 2^-sy exactly for the quantised phenotype.
// The sum of ytilde^2 (ytilde = Y 2^-sy) over the pair's valid individuals (both genotypes
// known, phenotype valid) follows from per-SNP sums over each SNP's missing individuals:
//     Q_ij = Qtot - QM_i - QM_j + QMM_ij,   QMM_ij = sum of ytilde^2 over the individuals
// missing at both SNPs, 0 <= QMM_ij. Their number and Y sum are exact from the cells:
//     n_mm = N_ij - Nvalid + NM_i + NM_j,   Y_mm = St_ij - Ytot + SM_i + SM_j,
// so QMM_ij = 0 when n_mm = 0 and (Y_mm 2^-sy)^2 when n_mm = 1 (exact); only a pair with two
// or more such individuals that needs exact statistics intersects the two SNPs' missing bits.
// The epilogue screens F and F2 in FP32 with Q_ij >= Qtot - QM_i - QM_j (F and F2 fall as Q
// grows, so the screen bounds them from above) and forms SSB / SSI / F / F2 in FP64 for every
// pair that could be a hit or a new maximum.
//
// That is the kernel with all digits. The screen (SCR) carries only the count and one or two
// 8-bit phenotype digits, bounds F and F2 (screen_epilogue) and lists the pairs it cannot
// settle for k_exact (scan_exact.cu): 42 or 28 j-SNPs per tile instead of 21, or 14 j-SNPs by
// five traits that share their counts (group_epilogue). RAW is the screen on the packed words.
//
// The GEMM runs on a CTA pair (a cluster of two CTAs on two SMs, tcgen05 cta_group::2): one
// MMA of M = 256 rows (each CTA's 40 i-SNPs, 3 genotype rows each, in its own shared memory)
// by N = 256 columns (the 252 columns of 21 j-SNPs plus 4 zero columns; each CTA holds and
// builds half of them), so each SM expands half of B per stage. Each CTA's TMEM receives the
// accumulator rows of its own i-SNPs, which its epilogue reads.
//
// A comes straight from HBM: the genotype-indicator rows h3 (row 3s + a = [g_s == a] bytes)
// are TMA-loaded into a 128-byte-swizzled shared-memory stage and read by the MMA from there.
//
// Per CTA, 15 warps (20 in the variants with three epilogue warps per lane quarter or two
// producer groups; Rings below):
//   warp 13       A loader (one thread): per 128-individual stage, the CTA's A stage (four
//                 2-D tiled loads of 30 h3 rows into rows 32w..32w+29); no multicast
//   warp 14       raw loader (one thread): per stage, the j-tile's 21 one-hot rows and the
//                 trait's 4 digit rows, up to RSTAGES stages ahead of the B producers
//   warps 4-7     B producers: raw rows -> this CTA's half of the B stage (K-major, 128-byte
//                 swizzle): CTA 0 the column types of digit rows 0-1, CTA 1 of rows 2-3;
//                 a second producer group (warps 16-19) takes alternate stages in one variant
//   warp 12       CTA 0: MMA issuer (one thread): 4 pair MMAs per stage; CTA 1: forwards the
//                 completion of its own A stages to CTA 0. Both: TMEM allocation (pair form)
//   warps 0-3, 8-11  epilogue, two warps per TMEM lane quarter, seven j rounds between them
// Handshakes: one operand ring (an A stage and a B stage per slot). CTA 0's `full` barrier of a
// slot counts its own A load, CTA 1's forward of its A load and the 8 producer warps of both
// CTAs, so the MMA issuer waits once per stage; its commit arrives on both CTAs' `empty`
// barrier of the slot (multicast), which the A loaders and producers wait on. CTA 0's acc_empty
// also counts CTA 1's epilogue warps; commits arrive on both CTAs' acc_full. TMEM (512
// columns per CTA): accumulators at [0, 256) and [256, 512). All waits are bounded
// (tc_ptx.cuh); a timeout sets counters[2] and every role leaves its loop; the CTAs meet in
// a cluster barrier before the TMEM is released.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "epi_internal.cuh"
#include "pair_exact.cuh"
#include "tc_ptx.cuh"

namespace epi {
namespace mma {

constexpr int TI = 40;         // i-SNPs per CTA (4 lane quarters x 10 triplets)
constexpr int TIP = 2 * TI;    // i-SNPs per pair tile
constexpr int TJ = 21;         // j-SNPs per tile of the full digits (the screen: 2 x 21)
constexpr int NTYPE = 12;      // B column types per j-SNP: b (3) x {w, d0, d1, d2}
constexpr int NCOL = TJ * NTYPE;  // 252 columns in use
constexpr int N = 256;         // MMA width (pair MMAs take multiples of 32)
constexpr int NH = N / 2;      // B columns held by each CTA
constexpr int TYH = NTYPE / 2; // column types held by each CTA (6 x 21 = 126 of its 128 rows)
constexpr int M = 256;         // MMA height over the pair
constexpr int KS = 128;        // individuals per pipeline stage
constexpr int ND = 4;          // digit rows per trait: w, Y digits (3)
constexpr int DROWS = 1 + ND;  // rows per trait in ydig: D, w, then the Y digits, the highest first
constexpr int ROUNDS = (TJ + 2) / 3;  // j rounds of the epilogue (3 j-SNPs per round)
constexpr uint32_t ACC_COL1 = N;
__host__ __device__ constexpr uint32_t acc_col(uint32_t buf) { return buf ? ACC_COL1 : 0u; }
// accumulator column of column type ty = 4b + s, j-SNP jj of the tile: digit rows s = 0, 1 in
// CTA 0's half, 2, 3 in CTA 1's; in each half the six local types q = 2b + s % 2 of a j-SNP
// are adjacent (column 6 jj + q)
__host__ __device__ constexpr int bq(int ty) { return 2 * (ty >> 2) + (ty & 1); }
__host__ __device__ constexpr int bcol(int ty, int jj) { return ((ty & 3) >> 1) * NH + 6 * jj + bq(ty); }
// the epilogue loads a round's three j-SNPs as 20 adjacent columns per half (five x4 loads)
constexpr int RCOLS = 20;
constexpr uint32_t TMEM_COLS = 512;
constexpr int A_STAGE = (M / 2) * KS;  // 16 KB
constexpr int B_STAGE = NH * KS;       // 16 KB
constexpr int A_BOX = 30;              // h3 rows per TMA box (10 i-SNPs x 3 genotypes)
constexpr uint32_t A_BYTES = 4 * A_BOX * KS;  // transaction bytes per A stage (one CTA)
constexpr uint32_t XB_BYTES = 6 * TJ * KS;     // the streamed-B variant: one CTA's B half (126 rows)
// raw stage: the j-tile's one-hot rows and the trait's digit rows, 1024-aligned sections
constexpr int RAW_J = 0, RAW_D = (TJ * KS + 1023) / 1024 * 1024;
constexpr int RAW_STAGE = 4 * 1024;
// raw stage of RAW: the packed words of 40 + 21 SNPs (32 bytes each), then the digit rows D and w
constexpr int PACKED_ROWS = TI + TJ, PACKED_D = PACKED_ROWS * 32, PACKED_STAGE = PACKED_D + 2 * KS;
static_assert(PACKED_D % 16 == 0, "digit rows are read in words of 16 bytes");
// producer work items per stage: (j-SNP, 16-individual chunk); 128 producer threads take the
// first 128 and the threads below XTRA one more (the j-SNPs 16..20, same chunk)
constexpr int XTRA = TJ * 8 - 128;

constexpr uint32_t IDESC = tc::idesc_i8(M, N);
static_assert(RAW_D % 1024 == 0 && RAW_D + ND * KS <= RAW_STAGE, "raw layout");
static_assert(B_STAGE % 1024 == 0 && A_STAGE % 1024 == 0 && N % 32 == 0 && N <= 256 && NCOL <= N, "operand tiles");
static_assert(NTYPE % 2 == 0 && TYH * TJ <= NH && TYH == 6, "B split: six types per CTA");
static_assert(XTRA >= 0 && XTRA <= 128 && (XTRA % 8) == 0 && 16 + XTRA / 8 == TJ, "producer items");
static_assert(2 * N <= (int)TMEM_COLS, "TMEM layout: two accumulators");
// the accumulator loads of a round's three j-SNPs (18 columns per half) read two columns past
// them: within each half even for the last round
static_assert(6 * 3 * (ROUNDS - 1) + RCOLS <= NH && bcol(11, TJ - 1) < N && bcol(9, TJ - 1) < NH, "epilogue loads");

// Ring depths (a kernel variant, chosen by the autotuner): STAGES operand slots, each an A stage
// (TMA from L2 / DRAM) and a B stage (built from raw rows already in shared memory), and the raw
// ring (j one-hot and digit rows, by TMA), which lets the raw loader run ahead of the B
// producers. One barrier pair per operand slot keeps the MMA issuer's work per stage to one
// wait and one commit: the issuer is the pipeline's critical path (a barrier wait costs about a
// hundred cycles even when the barrier is ready).
//
// EPW epilogue warps per TMEM lane quarter: 2 (epilogue warps 0-3 and 8-11) or 3 (also 16-19);
// 4 in the screen's streamed-B variant, which has no producers (0-3, 4-7, 8-11 and 16-19).
// PW producer groups of 4 warps: 1 (warps 4-7) or 2 (also 16-19, the groups taking alternate
// stages, so each has two stage times for its loads, stores, proxy fence and arrivals: the
// producers' per-stage latency, not their throughput, bounds the pipeline). One group and two
// epilogue warps: 15 warps. Otherwise 20 warps (warp 15 idle), launched with 96 registers each
// and rebalanced by warpgroup (setmaxnreg): epilogue warpgroups to 128, producer warpgroups to
// 56 (EPW 3) or 88 (PW 2), the loaders and MMA issuer to 40 -- 3 x 128 x 128 + 128 x 56 +
// 128 x 40 = 61,440 and 2 x 128 x 128 + 2 x 128 x 88 + 128 x 40 = 60,416, within the launch's
// pool of 640 x 96 = 61,440.
//
// XF (the streamed-B variant, single traits and sizes whose expanded B rows fit in HBM): B is
// not built in shared memory but precomputed once per genotype and trait load into HBM (12
// bytes per SNP and individual: `hx`, rows ((t 2 + half) M + snp) 6 + q) and TMA-loaded with
// the A rows, one 126-row box per CTA half per stage; no producers or raw loader run (warps 4-7
// and 14 idle); both CTAs' loads complete on CTA 0's full barrier, which counts one arrival (its
// loader) and the bytes of both.
//
// SCR (the screened scan, 1 or 2 phenotype digits; 0: all digits): B holds the column types of w
// and of the screen's digits only, 3 (1 + SCR) per j-SNP and TJH j-SNPs in each CTA's half: a
// tile is 42 j-SNPs wide with one digit, 28 with two (screen_epilogue below).
//
// RAW (epi_scan_block_noalloc: no memory for expanded rows): warps 13 and 14 copy the reference's
// packed words of the CTA's 40 i-SNPs and 21 j-SNPs into the raw ring (cp.async, 4 bytes: the
// caller's rows have no larger alignment) and three producer groups of 4 warps on alternate stages
// (4-7, 16-19, 20-23) build A and B from them; CTA 0's full barrier counts the 8 producer warps of
// a stage. 24 warps, launched with 80 registers each: epilogue 104, producers 72, the others 40
// (59,392 of 61,440).
//
// GT > 1 (streamed B, one digit): traits with the same valid individuals in groups of GT. Their counts
// are the same, so a j-SNP has 3 (1 + GT) column types for GT traits, w and their D's: 18 for five,
// and a tile of 14 j-SNPs makes 70 tests per i-SNP instead of 42 (group_epilogue below).
template <int S, int RSx, int EPW_ = 2, int PW_ = 1, bool XF_ = false, int SCR_ = 0, bool RAW_ = false, int GT_ = 1>
struct Rings {
    static constexpr int STAGES = S, RSTAGES = RSx, EPW = EPW_, PW = PW_, SCR = SCR_, GT = GT_;
    static constexpr bool XF = XF_, RAW = RAW_;
    static_assert(GT == 1 || (XF && SCR == 1 && EPW == 2 && PW == 1), "grouped traits: streamed B, one digit");
    static constexpr int TY = SCR ? 3 * (1 + SCR * GT) : TYH;  // column types of a j-SNP in a CTA's half
    static constexpr int TJH = (TYH * TJ) / TY;  // j-SNPs in a half: 21 (all digits, one), 14 (two), 7 (groups)
    static constexpr int TJT = SCR ? 2 * TJH : TJ;        // j-SNPs per tile
    using OneTrait = Rings<S, RSx, EPW_, PW_, XF_, SCR_, RAW_, 1>;
    static constexpr int RAW_ROWS = SCR == 0 ? ND : 1 + SCR;  // digit rows of a raw stage
    static constexpr uint32_t RAW_BYTES = (TJH + RAW_ROWS) * KS;
    static_assert(TY * TJH == TYH * TJ, "every variant fills 126 of a half's 128 rows");
    static_assert(!XF || (EPW == 2 && PW == 1) || (EPW == 4 && PW == 1 && SCR), "streamed-B layouts");
    static constexpr int NWARPS = RAW ? 24 : (EPW == 2 && PW == 1) ? 15 : 20;
    static constexpr int NTHREADS = NWARPS * 32;
    static constexpr int PROD_REGS = RAW ? 72 : PW == 2 ? 88 : 56, EPI_REGS = RAW ? 104 : 128;
    static constexpr int LAUNCH_REGS = RAW ? 80 : 96;
    // register budgets by warpgroup (setmaxnreg); with four epilogue warpgroups all keep the launch's 96
    static constexpr bool REBALANCE = NWARPS >= 20 && EPW < 4;
    static_assert(RAW ? EPW == 2 && PW == 3 && SCR == 1 && !XF
                      : (EPW == 2 || EPW == 3 || XF) && (PW == 1 || PW == 2) && !(EPW == 3 && PW == 2),
                  "warp roles");
    static_assert(!REBALANCE || EPW * 128 * EPI_REGS + PW * 128 * PROD_REGS + 128 * 40 <= NTHREADS * LAUNCH_REGS,
                  "register split");
    struct Smem {
        uint8_t a[STAGES][A_STAGE];
        uint8_t b[STAGES][B_STAGE];
        uint8_t raw[RSTAGES][XF ? 16 : RAW ? PACKED_STAGE : RAW_STAGE];  // (unused with streamed B)
        // full: CTA 0 -- its A stage landed (its TMA), CTA 1's forward of its own, and both B
        // halves built (4 local + 4 remote producer warps): 10 arrivals; CTA 1 -- its A stage
        // landed (1). empty: the MMAs reading the slot are done (both CTAs, one commit)
        uint64_t full[STAGES], empty[STAGES], raw_full[RSTAGES], raw_empty[RSTAGES], acc_full[2], acc_empty[2],
            drain;
        uint64_t stall;  // never arrived at: the wait of the debug_stall test hook
        uint32_t tmem_base;
        int abort;
    };
};

// 16-byte chunk c of row r of a 128-byte-swizzled tile (1024-byte aligned base)
__device__ __forceinline__ uint4 ld_sw128(const uint8_t *base, int r, int c)
{
    return *reinterpret_cast<const uint4 *>(base + r * 128 + ((c ^ (r & 7)) << 4));
}

// The units (trait, pair tile) of one cluster, in order: every npairs-th one of the tiles that
// hold a pair snp1 > snp2, of one trait after the other (with traits innermost the expanded B
// rows of the streamed-B variant, which differ per trait, came from DRAM for every i-tile). Each
// role walks its own copy. Tiles outside the
// triangle are not in the sequence at all, so the clusters' shares differ by one unit at most
// (a fixed stride over all tiles gave some clusters twice the work of others on a diagonal
// block, and a 64-bit division per unit and role). A block's tiles run in groups of xsi i-tile
// rows and within a group in chunks of xsj j-tiles, row by row inside a chunk: with xsi = 1 and
// one chunk row by row over all j-tiles; the streamed-B variant keeps super-tiles, whose A rows
// and expanded B rows then stay in L2 together.
template <class C>
struct Walker {
    BlockDesc bd;
    int block, trait, i0, j0;  // the unit: its block, trait, first i-SNP (of the pair) and first j-SNP
    bool done;

    __device__ __forceinline__ Walker(const ScanArgs &args, int first, int step_)
        : block(args.seg0.block), trait(args.seg0.trait), done(false), a(args), step(step_), grp(args.seg0.group - 1),
          jc(0), q(0), rows(0), chunks(0), off(0), len(0)
    {
        bd = a.blocks[block];
        move(first);
    }
    __device__ __forceinline__ void next() { move(step); }

private:
    const ScanArgs &a;
    int step;
    int grp, jc, q, rows, chunks;  // the row group, the chunk of j-tiles, the row in the group
    int off, len;                  // the tile in the row's part of the chunk, and that part's length

    // how many tiles of row ti hold a pair: those that begin below the row's last i-SNP
    __device__ __forceinline__ int valid_tiles(int ti) const
    {
        const int x = bd.start1 + min((ti + 1) * TIP, bd.size1) - 1 - bd.start2;
        return x <= 0 ? 0 : min(bd.tiles_j, (x + C::TJT - 1) / C::TJT);
    }
    __device__ __forceinline__ bool at_end() const
    {
        if (trait != a.seg1.trait) return trait > a.seg1.trait;
        return block > a.seg1.block || (block == a.seg1.block && grp >= a.seg1.group);
    }
    __device__ __forceinline__ bool next_row()
    {
        ++q;
        while (q >= rows) {  // next chunk
            q = 0;
            if (++jc < chunks) break;
            jc = 0;
            ++grp;
            while (!at_end() && grp * a.xsi >= bd.tiles_i) {  // next block, or trait
                grp = 0;
                if (++block == a.nblocks) {
                    block = 0;
                    ++trait;
                }
                if (!at_end()) bd = a.blocks[block];
            }
            if (at_end()) return false;
            rows = min(a.xsi, bd.tiles_i - grp * a.xsi);
            chunks = (valid_tiles(grp * a.xsi + rows - 1) + a.xsj - 1) / a.xsj;
            if (chunks == 0) q = rows;  // a group above the diagonal
        }
        len = max(0, min(a.xsj, valid_tiles(grp * a.xsi + q) - jc * a.xsj));
        return true;
    }
    __device__ __forceinline__ void move(int tiles)
    {
        off += tiles;
        while (off >= len) {
            off -= len;
            if (!next_row()) {
                done = true;
                return;
            }
        }
        i0 = (grp * a.xsi + q) * TIP;
        j0 = (jc * a.xsj + off) * C::TJT;
    }
};

template <class Smem>
__device__ __forceinline__ void fail(const ScanArgs &a, Smem &sm, int where)
{
    sm.abort = 1;
    if (atomicCAS(&a.counters[2], 0ull, 1ull) == 0ull) a.counters[3] = (unsigned long long)where;
}

__device__ __forceinline__ uint32_t sel3(const uint32_t v[3], int idx)
{
    return idx == 0 ? v[0] : (idx == 1 ? v[1] : v[2]);
}

// The same statistics in FP32, as a screen: relative error ~1e-6 for the centred trait and
// the exact integer cells this gets (no cancellation beyond SSW = Q - ... at large N).
// A pair whose screened F and F2 are clearly below every threshold and below the running
// maxima cannot be a hit or a new maximum, and keeps these values; every other pair is
// recomputed by pair_stat_exact.
__device__ __forceinline__ void pair_stat_f32(const int n[9], const float sd[9], float sc, float Q, bool want_int,
                                              float &F, float &F2)
{
    float N = 0.0f, St = 0.0f, nfac = 0.0f, sf[9];
#pragma unroll
    for (int c = 0; c < 9; ++c) {
        sf[c] = sd[c] * sc;
        N += (float)n[c];
        St += sf[c];
        nfac += n[c] > 0 ? 1.0f : 0.0f;
    }
    const float m = St * rcp_fast(N);
    float mc[9], SSB = 0.0f;
#pragma unroll
    for (int c = 0; c < 9; ++c) {
        mc[c] = n[c] > 0 ? sf[c] * rcp_fast((float)n[c]) : 0.0f;
        const float d = mc[c] - m;
        SSB = fmaf((float)n[c] * d, d, SSB);
    }
    const float SSY = Q - St * m;  // sum of squares about the pair's mean
    const float SSW = SSY - SSB;
    // SSW carries an absolute error of a few ulps of SSY; while SSW > 1e-3 SSY its relative
    // error stays below ~3e-4, inside the margin. A closer fit (or a negative SSW from
    // rounding) goes to the exact path: NaN fails every screen comparison.
    if (!(SSW > 1e-3f * SSY)) {
        F = F2 = __int_as_float(0x7fc00000);
        return;
    }
    const float d1 = nfac - 1.0f, d2 = N - nfac;
    F = (SSB * d2) * rcp_fast(SSW * d1);
    F2 = 0.0f;
    if (want_int) {
        float row[3], col[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const float rn = (float)(n[3 * i] + n[3 * i + 1] + n[3 * i + 2]);
            const float cn = (float)(n[i] + n[i + 3] + n[i + 6]);
            row[i] = rn > 0.0f ? (sf[3 * i] + sf[3 * i + 1] + sf[3 * i + 2]) * rcp_fast(rn) : 0.0f;
            col[i] = cn > 0.0f ? (sf[i] + sf[i + 3] + sf[i + 6]) * rcp_fast(cn) : 0.0f;
        }
        float SSI = 0.0f;
#pragma unroll
        for (int c = 0; c < 9; ++c) {
            const float t = mc[c] - row[c / 3] - col[c % 3] + m;
            SSI = n[c] > 0 ? fmaf((float)n[c] * t, t, SSI) : SSI;
        }
        F2 = (SSI * d2) * rcp_fast(4.0f * SSW);
    }
}

template <int RING>
__device__ __forceinline__ void advance(uint32_t &slot, uint32_t &phase)
{
    if (++slot == RING) {
        slot = 0;
        phase ^= 1u;
    }
}

// ---- the screen (SCR) ----
//
// For deciding which pairs can matter an 8-bit phenotype is enough (16 bits, the two upper
// digits of Y, where N is so large that 8 let too many pairs through). With D (|D| <= 127, one
// int8 digit) approximating s (ytilde - c) and E = ||s ytilde - (D - d0)||_2 over the valid
// individuals, SSB is the squared norm of an orthogonal projection of ytilde (onto the cells'
// indicators less the constant) and SSI that of a symmetric map of norm <= 1 (the cells' mean
// less the row and column means plus the grand mean), so in units of D
//     sqrt(SSB) <= sqrt(SSB_D) + E,     sqrt(SSI) <= sqrt(SSI_D) + E,
// and likewise from below with - E (and the same of P, the squared norm of the projection onto the
// cells' indicators with the constant: SSB = P - M). The sum of squares is exact up to the
// individuals missing at both SNPs: Qtot - QM_i - QM_j <= Q <= Qtot - max(QM_i, QM_j). A pair whose upper bounds of
// F and F2 stay below the thresholds and below the largest lower bounds met so far is neither
// a hit nor a maximum; every other pair (about 1e-4 of them at the usual thresholds) goes to
// the candidate list, which k_exact evaluates from the 24-bit digits. The bounds of FP32
// rounding: P, R, C, M and X below are sums of squares of the centred trait's cell sums, each
// at most P in magnitude and good to ~1e-6 of it, hence the slack SLK_B and SLK_I. Q is a difference
// of floats up to Qtot, however little of it the pair keeps: six roundings, below 6 x 2^-24 Qtot, hence
// SLK_Q (E is no cover for it: it is 0 for a trait of two values). The thresholds are lowered by a
// relative 1e-3, which covers the rest. A pair is settled only below a bound, never at it: where every
// F is 0 the pair that raised the lower bound to 0 has to reach k_exact, or no pair would make the maximum.
//
// Six column types (nine) instead of twelve per j-SNP: a pair MMA serves 80 x 42 (28) pairs
// instead of 80 x 21.
constexpr float SLK_B = 4e-6f, SLK_I = 1.2e-5f, SLK_Q = 4e-7f;

__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 rcp2(float2 a) { return make_float2(rcp_fast(a.x), rcp_fast(a.y)); }

__device__ __forceinline__ float int_float(uint32_t x) { return __int_as_float((int)(x + 0x4B400000u)) - 12582912.0f; }

// Integers below 2^22 in magnitude as floats (exact): an integer addition into the mantissa of
// 1.5 x 2^23 and a float subtraction. The conversion instruction runs on the pipe of the
// reciprocals, at a sixteenth of the rate: 36 of them a round made it the epilogue's bound
// (85% busy at 500 individuals).
__device__ __forceinline__ float2 int_float2(uint32_t x, uint32_t y)
{
    const float2 m = make_float2(-12582912.0f, -12582912.0f);
    return add2(make_float2(__int_as_float((int)(x + 0x4B400000u)), __int_as_float((int)(y + 0x4B400000u))), m);
}

// A lane's accumulator row of a round, the j-SNPs 3 r .. 3 r + 2 of each half (the last three
// where fewer are left): v[h][TY c + (1 + SCR) b + s], the count (s = 0) and the digit sums of
// genotype b of j-SNP c
template <class C>
__device__ __forceinline__ int round_j(int r) { return min(3 * r, C::TJH - 3); }

template <class C>
__device__ __forceinline__ void load_round(uint32_t acc, int r, uint32_t v[2][3 * C::TY])
{
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint32_t col = acc + h * NH + C::TY * round_j<C>(r);
        tc::tmem_ld16(col, v[h]);
        if constexpr (C::SCR == 2) tc::tmem_ld8(col + 16, v[h] + 16);
        tc::tmem_ld2(col + 3 * C::TY - 2 - C::SCR / 2, v[h] + 3 * C::TY - 2 - C::SCR / 2);
        if constexpr (C::SCR == 2) tc::tmem_ld1(col + 26, v[h][26]);
    }
    tc::tmem_wait_ld();
}

// The count and the sum (about the trait's mean) of a cell, of the pairs of both halves
template <class C>
__device__ __forceinline__ void cell2(const uint32_t v[2][3 * C::TY], int k, float2 md0, float2 &n, float2 &S)
{
    n = int_float2(v[0][k], v[1][k]);
    S = int_float2(v[0][k + 1], v[1][k + 1]);
    if constexpr (C::SCR == 2) S = fma2(S, make_float2(256.0f, 256.0f), int_float2(v[0][k + 2], v[1][k + 2]));
    else S = fma2(md0, n, S);  // exactly 0 in an empty cell
}

// What other warps change meanwhile, a lower bound of a trait's maximum or the number of candidates:
// lane 0's reading for the whole warp. Whether a unit's rounds run, and whether they run twice (seed),
// hangs on it, and the rounds hold full-warp operations, so lanes with different readings of it could
// end up in different passes. (Loads first, then the shuffles: each load is a trip to L2.)
template <class T>
__device__ __forceinline__ T peek(const T *p) { return *reinterpret_cast<const volatile T *>(p); }
template <class T>
__device__ __forceinline__ T lane0(T x) { return __shfl_sync(0xffffffffu, x, 0); }

// All that the screen can tell of the lane's pair in half h, from its nine cells, gathered from the
// triplet's rows (the rows' order does not matter): P, M, the count, the occupied cells, and
// I0 = 2 X - R - C - M, so that SSI_D = P + I0
struct Table {
    float P, M, N, nf, I0;
};
template <class C>
__device__ __forceinline__ Table gather_table(const uint32_t v[3 * C::TY], float d0, int ga, int s1, int s2)
{
    const int o1 = (ga + 2) % 3, o2 = (ga + 1) % 3;  // the columns this lane offers the others
    float n[9], S[9];
#pragma unroll
    for (int q = 0; q < C::TY; ++q) {
        const uint32_t x0 = v[q], x1 = v[C::TY + q], x2 = v[2 * C::TY + q];
        const uint32_t w[3] = {pick3(x0, x1, x2, ga), __shfl_sync(0xffffffffu, pick3(x0, x1, x2, o1), s1),
                               __shfl_sync(0xffffffffu, pick3(x0, x1, x2, o2), s2)};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int cell = 3 * k + q / (1 + C::SCR), s = q % (1 + C::SCR);
            const float f = (float)(int)w[k];
            if (s == 0) n[cell] = f;
            else if (C::SCR == 1) S[cell] = fmaf(-d0, n[cell], f);
            else S[cell] = s == 1 ? 256.0f * f : S[cell] + f;
        }
    }
    Table t = {0.f, 0.f, 0.f, 0.f, 0.f};
    float cb[3], St = 0.f, RC = 0.f, X = 0.f;
#pragma unroll
    for (int c = 0; c < 9; ++c) {
        t.P = fmaf(S[c], S[c] * rcp_fast(n[c] + 1e-30f), t.P);
        t.nf += n[c] > 0.0f ? 1.0f : 0.0f;
    }
#pragma unroll
    for (int b = 0; b < 3; ++b) {
        const float nb = n[b] + n[3 + b] + n[6 + b], Sb = S[b] + S[3 + b] + S[6 + b];
        cb[b] = Sb * rcp_fast(nb + 1e-30f);
        RC = fmaf(Sb, cb[b], RC);
        t.N += nb;
        St += Sb;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float na = n[3 * k] + n[3 * k + 1] + n[3 * k + 2], Sa = S[3 * k] + S[3 * k + 1] + S[3 * k + 2];
        const float ra = Sa * rcp_fast(na + 1e-30f);
        RC = fmaf(Sa, ra, RC);
        X = fmaf(ra, fmaf(n[3 * k + 2], cb[2], fmaf(n[3 * k + 1], cb[1], n[3 * k] * cb[0])), X);
    }
    t.M = St * St * rcp_fast(t.N + 1e-30f);
    t.I0 = fmaf(2.0f, X, -RC) - t.M;
    return t;
}

// One warp of the epilogue: its j rounds of every unit. A round is three j-SNPs of each B half
// (columns 18 r of either half), so a lane forms the pairs (i, j0 + 3 r + ga) and
// (i, j0 + 21 + 3 r + ga), the two halves side by side in packed FP32 (f32x2) operations. What all
// pairs need is little. With P the sum of S^2 / n over the cells, SSW = Q - P and SSB = P - M <= P, SSI
// is at most SSB (the map above has norm <= 1 on the cells' means) and d2 at most the trait's valid
// individuals, so P and the number of occupied cells settle both tests for all but a few pairs
// in a thousand: each lane forms them for its own genotype row and the three j-SNPs, and the triplet
// adds them up, three values for the two pairs instead of 36. All nine cells meet in one lane only
// where a pair passes (the columns are read again).
template <class C>
__device__ __forceinline__ void screen_epilogue(const ScanArgs &a, typename C::Smem &sm, uint32_t tmem, uint32_t rank,
                                                int pair, int npairs)
{
    constexpr int EPW = C::EPW;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    volatile int *abort = &sm.abort;
    constexpr int RND = (C::TJH + 2) / 3;
    const int e = warp & 3;  // TMEM lane quarter, and the warp's number among those of its quarter
    const int part = EPW == 4 ? (warp < 12 ? warp >> 2 : 3) : warp < 4 ? 0 : (warp < 12 ? 1 : 2);
    const int r_begin = (part * RND + EPW - 1) / EPW, r_end = ((part + 1) * RND + EPW - 1) / EPW;
    const int ii = 10 * e + lane / 3, ga = lane % 3, tbase = (lane / 3) * 3;
    const int s1 = tbase + (ga + 1) % 3, s2 = tbase + (ga + 2) % 3;  // the triplet's other rows
    const bool is1 = ga == 1, is2 = ga == 2;
    const uint32_t tl = tmem + ((uint32_t)(32 * e) << 16);
    const bool ti = a.test_int != 0;
    const float t1c = screen_lo(a.t1), t2c = screen_lo(a.t2);
    uint32_t accph = 0u;  // bit b: the parity of accumulator b's next phase
    int buf = 0;
    for (Walker<C> un(a, pair, npairs); !un.done; un.next()) {
        const int t = un.trait;
        const int di = un.i0 + TI * (int)rank + ii;
        const int gi = un.bd.start1 + di;
        const bool ivalid = lane < 30 && di < un.bd.size1;
        const float4 ts = a.tscr[2 * t + C::SCR - 1];
        const float d0 = ts.x, E = ts.y, qtot = ts.z, s2y = ts.w;
        const float *qmf_j = a.qmf_j + (size_t)t * a.nsnp;
        const float qmi = ivalid ? s2y * a.qmf[(size_t)t * a.nsnp + gi] : 0.0f;
        const bool report = a.report_trait < 0 || a.report_trait == t;
        unsigned int lF = peek(a.lowf + t), lI = ti ? peek(a.lowf2 + t) : 0u;
        // a list that has run over: what is left is listed nowhere and need not be screened
        const unsigned long long listed = lane0(peek(a.counters + CNT_CAND + a.segment));
        const int r_first = (long long)listed > a.cand_cap ? r_end : r_begin;
        lF = lane0(lF);
        lI = lane0(lI);
        auto threshold = [&](unsigned int low, float tc) {
            const float l = screen_lo(ord2f(low));
            return report ? fminf(tc, l) : l;
        };
        float tF = threshold(lF, t1c), tI = ti ? 4.0f * threshold(lI, t2c) : INFINITY;
        const float qi = fmaf(-SLK_Q, qtot, qtot - qmi), nv = (float)a.nvalid[t];
        if (!tc::mbar_wait(&sm.acc_full[buf], (accph >> buf) & 1u, abort, a.wait_ns)) {
            fail(a, sm, 3);
            break;
        }
        tc::tc_fence_after();
        const uint32_t acc = tl + acc_col(buf);
        // Nothing is known of the trait's maxima yet (its first units, which every cluster begins
        // at once): the rounds run twice, first only to raise the lower bounds. Listing pairs in
        // that pass would list a tenth of them.
        bool seed = lF == ENC_NEG_INF || (ti && lI == ENC_NEG_INF);
#pragma unroll 1
        for (int r = r_first; r < r_end; ++r) {
            const int dj = un.j0 + round_j<C>(r) + ga, gj = un.bd.start2 + dj;
            bool valid[2];
            float qmj[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                valid[h] = ivalid && dj + C::TJH * h < un.bd.size2 && gi > gj + C::TJH * h;
                // (the last round takes in the j-SNPs of the one before where three do not divide)
                if (C::TJH % 3 != 0) valid[h] = valid[h] && round_j<C>(r) + ga >= 3 * r;
                qmj[h] = valid[h] ? s2y * qmf_j[gj + C::TJH * h] : 0.0f;
            }
            uint32_t v[2][3 * C::TY];
            load_round<C>(acc, r, v);
            const float2 tiny = make_float2(1e-30f, 1e-30f), md0 = make_float2(-d0, -d0);
            float2 P2[3], nf2[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                P2[c] = nf2[c] = make_float2(0.f, 0.f);
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    float2 nb, Sb;
                    cell2<C>(v, C::TY * c + (1 + C::SCR) * b, md0, nb, Sb);
                    P2[c] = fma2(Sb, mul2(Sb, rcp2(add2(nb, tiny))), P2[c]);
                    nf2[c] = add2(nf2[c], make_float2(__saturatef(nb.x), __saturatef(nb.y)));
                }
            }
            // the pair (i, j-SNP c = ga) is this lane's: each lane adds what the triplet's other
            // two offer it, the lane of row ga + 1 its column (ga + 1) + 2 = ga (mod 3)
            auto gather = [&](float x0, float x1, float x2) {
                const float own = is1 ? x1 : is2 ? x2 : x0;
                const float for1 = is1 ? x0 : is2 ? x1 : x2, for2 = is1 ? x2 : is2 ? x0 : x1;
                return own + __shfl_sync(0xffffffffu, for1, s1) + __shfl_sync(0xffffffffu, for2, s2);
            };
            const float P[2] = {gather(P2[0].x, P2[1].x, P2[2].x), gather(P2[0].y, P2[1].y, P2[2].y)};
            // occupied cells of both halves in one value, 16 nf1 + nf0 (nf <= 9)
            const float nf01 = gather(fmaf(16.0f, nf2[0].y, nf2[0].x), fmaf(16.0f, nf2[1].y, nf2[1].x),
                                      fmaf(16.0f, nf2[2].y, nf2[2].x));
            // nf1 = (nf01 - 4.5) / 16 to the nearest integer, since 0 <= nf0 <= 9
            const float nf1 = fmaf(nf01 - 4.5f, 0.0625f, 12582912.0f) - 12582912.0f;
            const float nf[2] = {fmaf(-16.0f, nf1, nf01), nf1};
            bool cand[2];
            bool any = false;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float sB = sqrt_fast(P[h] * (1.0f + SLK_B)) + E, u = sB * sB;  // >= P >= SSB >= SSI
                const float Q = qi - qmj[h], W = Q - u, lhs = u * nv, d1 = nf[h] - 1.0f;
                // one occupied cell: F is 0/0, never a hit or a maximum (F2 is 0); none: neither is
                // defined. W too small a part of Q to be told from rounding: unknown
                cand[h] = valid[h] && d1 >= (ti ? 0.0f : 1.0f) &&
                          (!(W > 1e-3f * Q) || (d1 > 0.0f && !(lhs < tF * d1 * W)) || !(lhs < tI * W));
                any = any || cand[h];
            }
            if (__any_sync(0xffffffffu, any)) {
                // tighter bounds from all nine cells; they raise the lower bounds of the maxima first,
                // then the pairs that still matter are listed
                load_round<C>(acc, r, v);
                float fu[2], f2u[2];
                unsigned int bF = 0u, bI = 0u;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const Table x = gather_table<C>(v[h], d0, ga, s1, s2);
                    const float d1 = x.nf - 1.0f, d2 = x.N - x.nf, Q = qi - qmj[h];
                    const float sP = sqrt_fast(x.P * (1.0f + SLK_B)) + E;
                    const float sB = sqrt_fast(fmaxf(fmaf(x.P, 1.0f + SLK_B, -x.M), 0.0f)) + E;
                    const float sI = sqrt_fast(fmaxf(fmaf(x.P, 1.0f + SLK_I, x.I0), 0.0f)) + E;
                    const float W0 = Q - sP * sP, W = W0 > 1e-3f * Q ? W0 : __int_as_float(0x7fc00000);
                    fu[h] = d1 > 0.0f ? sB * sB * d2 / (d1 * W) : -INFINITY;
                    f2u[h] = ti ? sI * sI * d2 / (4.0f * W) : -INFINITY;
                    // from below: SSB, SSI and, for SSW <= Q - P from above, P
                    const float lP = fmaxf(sqrt_fast(x.P * (1.0f - SLK_B)) - E, 0.0f);
                    const float lB = fmaxf(sqrt_fast(fmaxf(fmaf(x.P, 1.0f - SLK_B, -x.M), 0.0f)) - E, 0.0f);
                    const float lo = fmaxf(sqrt_fast(fmaxf(fmaf(x.P, 1.0f - SLK_I, x.I0), 0.0f)) - E, 0.0f);
                    const float Wu = fmaf(SLK_Q, qtot, qtot - fmaxf(qmi, qmj[h])) - lP * lP;
                    if (cand[h] && W == W && Wu > 0.0f) {
                        if (d1 > 0.0f) bF = max(bF, f2ord(screen_lo(lB * lB * d2 / (d1 * Wu))));
                        if (ti) bI = max(bI, f2ord(screen_lo(lo * lo * d2 / (4.0f * Wu))));
                    }
                }
                bF = __reduce_max_sync(0xffffffffu, bF);
                bI = __reduce_max_sync(0xffffffffu, bI);
                if (bF > lF) {
                    lF = bF;
                    tF = threshold(lF, t1c);
                    if (lane == 0) atomicMax(&a.lowf[t], lF);
                }
                if (ti && bI > lI) {
                    lI = bI;
                    tI = 4.0f * threshold(lI, t2c);
                    if (lane == 0) atomicMax(&a.lowf2[t], lI);
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const bool c = cand[h] && !seed && (!(fu[h] < tF) || !(4.0f * f2u[h] < tI));
                    const unsigned int mask = __ballot_sync(0xffffffffu, c);
                    if (!mask) continue;
                    const int leader = __ffs(mask) - 1;
                    unsigned long long base = 0ull;
                    if (lane == leader)
                        base = atomicAdd(&a.counters[CNT_CAND + a.segment], (unsigned long long)__popc(mask));
                    base = __shfl_sync(0xffffffffu, base, leader) + __popc(mask & ((1u << lane) - 1u));
                    if (c && (long long)base < a.cand_cap)
                        a.cand[base] = Cand{gi, gj + C::TJH * h, t, un.block, fu[h], f2u[h]};
                }
            }
            if (seed && r + 1 == r_end) {
                seed = false;
                r = r_begin - 1;
                lF = max(lF, lane0(peek(a.lowf + t)));
                tF = threshold(lF, t1c);
                if (ti) {
                    lI = max(lI, lane0(peek(a.lowf2 + t)));
                    tI = 4.0f * threshold(lI, t2c);
                }
            }
        }
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) {
            if (rank == 0) tc::mbar_arrive(&sm.acc_empty[buf]);
            else tc::mbar_arrive_remote(&sm.acc_empty[buf], 0);
        }
        accph ^= 1u << buf;
        buf ^= 1;
    }
}

// The epilogue of grouped traits: as screen_epilogue, for GT traits at once. A round is three j-SNPs
// of one half (all its columns: 3 TY); the counts, their reciprocals and the occupied cells are
// formed once, then per trait P of the lane's own genotype row and the triplet's sum: about 90
// operations per test against 150. A trait whose bounds pass goes through the nine cells one by one
// (gather_table on its columns).
template <class C>
__device__ __forceinline__ void group_epilogue(const ScanArgs &a, typename C::Smem &sm, uint32_t tmem, uint32_t rank,
                                               int pair, int npairs)
{
    constexpr int EPW = C::EPW, GT = C::GT, TY = C::TY, NC = 3 * TY;
    constexpr int RND = (C::TJH + 2) / 3;  // rounds of a half
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    volatile int *abort = &sm.abort;
    const int e = warp & 3, part = warp < 4 ? 0 : 1;
    const int ii = 10 * e + lane / 3, ga = lane % 3, tbase = (lane / 3) * 3;
    const int s1 = tbase + (ga + 1) % 3, s2 = tbase + (ga + 2) % 3;
    const bool is1 = ga == 1, is2 = ga == 2;
    const uint32_t tl = tmem + ((uint32_t)(32 * e) << 16);
    const bool ti = a.test_int != 0;
    const float t1c = screen_lo(a.t1), t2c = screen_lo(a.t2);
    uint32_t accph = 0u;
    int buf = 0;
    auto gather = [&](float x0, float x1, float x2) {
        const float own = is1 ? x1 : is2 ? x2 : x0;
        const float for1 = is1 ? x0 : is2 ? x1 : x2, for2 = is1 ? x2 : is2 ? x0 : x1;
        return own + __shfl_sync(0xffffffffu, for1, s1) + __shfl_sync(0xffffffffu, for2, s2);
    };
    for (Walker<C> un(a, pair, npairs); !un.done; un.next()) {
        const int t0 = un.trait * GT, nt = min(GT, a.ntraits - t0);  // the group's traits
        const int di = un.i0 + TI * (int)rank + ii;
        const int gi = un.bd.start1 + di;
        const bool ivalid = lane < 30 && di < un.bd.size1;
        const float nv = (float)a.nvalid[t0];  // the same for the group
        // thresholds per trait: the report threshold or the lower bound of the maximum
        float tF[GT], tI[GT], qi[GT];
        bool unknown = false;
        unsigned int low[GT][2];
#pragma unroll
        for (int g = 0; g < GT; ++g) {
            const int t = t0 + min(g, nt - 1);
            low[g][0] = peek(a.lowf + t);
            low[g][1] = ti ? peek(a.lowf2 + t) : 0u;
        }
        const bool full = (long long)lane0(peek(a.counters + CNT_CAND + a.segment)) > a.cand_cap;
#pragma unroll
        for (int g = 0; g < GT; ++g) {
            const int t = t0 + min(g, nt - 1);
            const float4 ts = a.tscr[2 * t];
            const bool report = a.report_trait < 0 || a.report_trait == t;
            const unsigned int lF = lane0(low[g][0]), lI = lane0(low[g][1]);
            const float bF = screen_lo(ord2f(lF)), bI = screen_lo(ord2f(lI));
            tF[g] = report ? fminf(t1c, bF) : bF;
            tI[g] = !ti ? INFINITY : 4.0f * (report ? fminf(t2c, bI) : bI);
            qi[g] = ivalid ? fmaf(-SLK_Q, ts.z, ts.z - ts.w * a.qmf[(size_t)t * a.nsnp + gi]) : 0.0f;
            unknown = unknown || lF == ENC_NEG_INF || (ti && lI == ENC_NEG_INF);
        }
        if (!tc::mbar_wait(&sm.acc_full[buf], (accph >> buf) & 1u, abort, a.wait_ns)) {
            fail(a, sm, 3);
            break;
        }
        tc::tc_fence_after();
        const uint32_t acc = tl + acc_col(buf);
        // (unknown maxima: the rounds run twice, as in screen_epilogue)
        for (int pass = full ? 2 : unknown ? 0 : 1; pass < 2; ++pass) {
#pragma unroll 1
            for (int q = part; q < 2 * RND; q += EPW) {
                const int h = q / RND, r = q % RND;
                const int jr = round_j<C>(r) + ga;  // the lane's j-SNP of the half
                const int dj = un.j0 + C::TJH * h + jr, gj = un.bd.start2 + dj;
                const bool valid = ivalid && jr >= 3 * r && dj < un.bd.size2 && gi > gj;
                const uint32_t col = acc + h * NH + TY * round_j<C>(r);
                uint32_t v[NC];
                static_assert(NC == 54, "columns of a round: 32 + 16 + 4 + 2");
                tc::tmem_ld32(col, v);
                tc::tmem_ld16(col + 32, v + 32);
                tc::tmem_ld4(col + 48, v[48], v[49], v[50], v[51]);
                tc::tmem_ld2(col + 52, v + 52);
                tc::tmem_wait_ld();
                float n[3][3], rn[3][3], nf[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    nf[c] = 0.0f;
#pragma unroll
                    for (int b = 0; b < 3; ++b) {
                        n[c][b] = int_float(v[TY * c + (1 + GT) * b]);
                        rn[c][b] = rcp_fast(n[c][b] + 1e-30f);
                        nf[c] += __saturatef(n[c][b]);
                    }
                }
                const float d1 = gather(nf[0], nf[1], nf[2]) - 1.0f;
                uint32_t cand = 0u;
#pragma unroll
                for (int g = 0; g < GT; ++g) {
                    const int t = t0 + min(g, nt - 1);
                    const float4 ts = a.tscr[2 * t];
                    float P[3];
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        P[c] = 0.0f;
#pragma unroll
                        for (int b = 0; b < 3; ++b) {
                            const float S = fmaf(-ts.x, n[c][b], int_float(v[TY * c + (1 + GT) * b + 1 + g]));
                            P[c] = fmaf(S, S * rn[c][b], P[c]);
                        }
                    }
                    const float qmj = valid ? ts.w * a.qmf_j[(size_t)t * a.nsnp + gj] : 0.0f;
                    const float sB = sqrt_fast(gather(P[0], P[1], P[2]) * (1.0f + SLK_B)) + ts.y, u = sB * sB;
                    const float Q = qi[g] - qmj, W = Q - u, lhs = u * nv;
                    const bool c = valid && g < nt && d1 >= (ti ? 0.0f : 1.0f) &&
                                   (!(W > 1e-3f * Q) || (d1 > 0.0f && !(lhs < tF[g] * d1 * W)) || !(lhs < tI[g] * W));
                    if (c) cand |= 1u << g;
                }
                uint32_t some = __reduce_or_sync(0xffffffffu, cand);
                while (some) {  // traits with a pair that passes, one after the other (rare)
                    const int g = __ffs(some) - 1, t = t0 + g;
                    some &= some - 1u;
                    const float4 ts = a.tscr[2 * t];
                    const float E = ts.y;
                    // the trait's columns as a one-digit round: counts and D sums (read again, since the
                    // trait is not known at compile time)
                    uint32_t w[18];
#pragma unroll
                    for (int k = 0; k < 9; ++k) {
                        const uint32_t cc = col + TY * (k / 3) + (1 + GT) * (k % 3);
                        tc::tmem_ld1(cc, w[2 * k]);
                        tc::tmem_ld1(cc + 1 + g, w[2 * k + 1]);
                    }
                    tc::tmem_wait_ld();
                    const Table x = gather_table<typename C::OneTrait>(w, ts.x, ga, s1, s2);
                    const bool mine = cand >> g & 1u;
                    const bool report = a.report_trait < 0 || a.report_trait == t;
                    const float qm = ivalid ? ts.w * a.qmf[(size_t)t * a.nsnp + gi] : 0.0f;
                    const float qmj = valid ? ts.w * a.qmf_j[(size_t)t * a.nsnp + gj] : 0.0f;
                    const float e1 = x.nf - 1.0f, d2 = x.N - x.nf, Q = fmaf(-SLK_Q, ts.z, ts.z - qm) - qmj;
                    const float sP = sqrt_fast(x.P * (1.0f + SLK_B)) + E;
                    const float sB = sqrt_fast(fmaxf(fmaf(x.P, 1.0f + SLK_B, -x.M), 0.0f)) + E;
                    const float sI = sqrt_fast(fmaxf(fmaf(x.P, 1.0f + SLK_I, x.I0), 0.0f)) + E;
                    const float W0 = Q - sP * sP, W = W0 > 1e-3f * Q ? W0 : __int_as_float(0x7fc00000);
                    const float fu = e1 > 0.0f ? sB * sB * d2 / (e1 * W) : -INFINITY;
                    const float f2u = ti ? sI * sI * d2 / (4.0f * W) : -INFINITY;
                    const float lP = fmaxf(sqrt_fast(x.P * (1.0f - SLK_B)) - E, 0.0f);
                    const float lB = fmaxf(sqrt_fast(fmaxf(fmaf(x.P, 1.0f - SLK_B, -x.M), 0.0f)) - E, 0.0f);
                    const float lo = fmaxf(sqrt_fast(fmaxf(fmaf(x.P, 1.0f - SLK_I, x.I0), 0.0f)) - E, 0.0f);
                    const float Wu = fmaf(SLK_Q, ts.z, ts.z - fmaxf(qm, qmj)) - lP * lP;
                    unsigned int bF = 0u, bI = 0u;
                    if (mine && W == W && Wu > 0.0f) {
                        if (e1 > 0.0f) bF = f2ord(screen_lo(lB * lB * d2 / (e1 * Wu)));
                        if (ti) bI = f2ord(screen_lo(lo * lo * d2 / (4.0f * Wu)));
                    }
                    bF = __reduce_max_sync(0xffffffffu, bF);
                    bI = __reduce_max_sync(0xffffffffu, bI);
                    // what is known now of this trait's maxima, this round's pairs included
                    unsigned int oF = 0u, oI = 0u;
                    if (lane == 0) {
                        oF = atomicMax(&a.lowf[t], bF);
                        if (ti) oI = atomicMax(&a.lowf2[t], bI);
                    }
                    bF = max(bF, __shfl_sync(0xffffffffu, oF, 0));
                    bI = max(bI, __shfl_sync(0xffffffffu, oI, 0));
                    const float kF = screen_lo(ord2f(bF)), kI = screen_lo(ord2f(bI));
                    const float hF = report ? fminf(t1c, kF) : kF, hI = report ? fminf(t2c, kI) : kI;
#pragma unroll
                    for (int k = 0; k < GT; ++k)
                        if (k == g) {
                            tF[k] = hF;
                            if (ti) tI[k] = 4.0f * hI;
                        }
                    const bool c = mine && pass == 1 && (!(fu < hF) || (ti && !(f2u < hI)));
                    const unsigned int mask = __ballot_sync(0xffffffffu, c);
                    if (!mask) continue;
                    const int leader = __ffs(mask) - 1;
                    unsigned long long base = 0ull;
                    if (lane == leader)
                        base = atomicAdd(&a.counters[CNT_CAND + a.segment], (unsigned long long)__popc(mask));
                    base = __shfl_sync(0xffffffffu, base, leader) + __popc(mask & ((1u << lane) - 1u));
                    if (c && (long long)base < a.cand_cap) a.cand[base] = Cand{gi, gj, t, un.block, fu, f2u};
                }
            }
        }
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) {
            if (rank == 0) tc::mbar_arrive(&sm.acc_empty[buf]);
            else tc::mbar_arrive_remote(&sm.acc_empty[buf], 0);
        }
        accph ^= 1u << buf;
        buf ^= 1;
    }
}

// RAW: the loader warps. A stage is 61 rows of 8 words; a lane copies word c of every eighth row
// (A rows first, then B rows), and 16 lanes a chunk of the digit rows. Rows of SNPs that are not
// there and words past the last one are left as they are: those pairs are masked in the epilogue,
// and individuals past the last one have zero digits and flags on the B side.
template <class C>
__device__ __forceinline__ void raw_loader(const ScanArgs &a, typename C::Smem &sm, uint32_t rank, int pair, int npairs)
{
    volatile int *abort = &sm.abort;
    const int t = threadIdx.x - 13 * 32, c = t & 7, rg = t >> 3;  // 64 lanes
    const int nks = a.Np / KS, npack1 = a.npack + (a.remain > 0);
    const long long stride8 = 8LL * npack1;
    uint32_t rs = 0, rph = 0;
    bool ok = true;
    for (Walker<C> un(a, pair, npairs); !un.done && ok; un.next()) {
        const int iA = un.i0 + TI * (int)rank, jB = un.j0 + C::TJH * (int)rank;
        const int nA = min(TI, un.bd.size1 - iA), nB = min(C::TJH, un.bd.size2 - jB);  // rows that are there
        const int32_t *pA = a.gpack + (long long)(un.bd.start1 + iA + rg) * npack1 + c;
        const int32_t *pB = a.gpack + (long long)(un.bd.start2 + jB + rg) * npack1 + c;
        for (int ks = 0; ks < nks; ++ks) {
            if (!tc::mbar_wait(&sm.raw_empty[rs], rph ^ 1u, abort, a.wait_ns)) {
                fail(a, sm, 14);
                ok = false;
                break;
            }
            uint8_t *const raw = sm.raw[rs];
            if (8 * ks + c < npack1) {
                const int32_t *src = pA;
#pragma unroll
                for (int x = 0; x < TI / 8; ++x, src += stride8)
                    if (rg + 8 * x < nA) tc::cp_async4(raw + (rg + 8 * x) * 32 + 4 * c, src);
                src = pB;
#pragma unroll
                for (int x = 0; x < (C::TJH + 7) / 8; ++x, src += stride8)
                    if (rg + 8 * x < nB) tc::cp_async4(raw + (TI + rg + 8 * x) * 32 + 4 * c, src);
            }
            pA += 8;
            pB += 8;
            if (t < 16)  // row t / 8 (D, w), chunk c
                tc::cp_async16(raw + PACKED_D + 16 * t, a.ydig + (size_t)(t >> 3) * a.Np + ks * KS + 16 * c);
            tc::cp_async_arrive(&sm.raw_full[rs]);
            advance<C::RSTAGES>(rs, rph);
        }
    }
    tc::cp_async_wait_all();
}

// RAW: one warp of a producer group: per thread one chunk c of 16 individuals (a packed word) of
// a few adjacent SNPs, whose rows in the operand tile follow each other. The first two warps build
// A, 8 threads by 5 SNPs and three genotype rows (15 stores of 16 bytes), the other two B, 7 by 3
// SNPs and six column types (18 stores). A word's 16 codes become byte-permute selectors, and every
// row is one table look-up per four individuals. With the rows' addresses as eight precomputed
// swizzled starts plus constants a stage is about 180 instructions; three groups give each three
// stage times for its latency.
template <class C>
__device__ __forceinline__ void raw_producers(const ScanArgs &a, typename C::Smem &sm, uint32_t rank, int pair,
                                              int npairs)
{
    constexpr int STAGES = C::STAGES, RSTAGES = C::RSTAGES, PW = C::PW;
    constexpr int SA = 5, SB = 3;  // SNPs per thread
    static_assert(8 * SA == TI && 7 * SB == C::TJH && 10 % SA == 0, "producer rows");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    volatile int *abort = &sm.abort;
    const int pg = warp < 8 ? 0 : (warp >> 2) - 3;  // warps 4-7, 16-19, 20-23
    const int t = threadIdx.x & 63, c = t & 7, rg = t >> 3;
    const bool sideA = (threadIdx.x & 64) == 0;
    const int nks = a.Np / KS;
    const long long total = a.seg_units > pair ? ((a.seg_units - 1 - pair) / npairs + 1) * nks : 0;  // stages
    int ks = pg % nks;  // of stage q
    uint32_t stage = pg % STAGES, phase = pg / STAGES & 1, rs = pg % RSTAGES, rph = pg / RSTAGES & 1;
    // tile rows nb, nb + 1, ..: A rows 32 (s / 10) + 3 (s % 10) + g of i-SNP s, B rows 6 s + 2 g + i; row
    // n's chunk c is at n 128 + ((c ^ (n & 7)) << 4)
    const int nb = sideA ? 32 * (SA * rg / 10) + 3 * (SA * rg % 10) : C::TY * SB * rg;
    const int word0 = sideA ? 32 * SA * rg + 4 * c : 32 * (TI + SB * rg) + 4 * c;  // its first word in a raw stage
    uint32_t at[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) at[k] = nb * 128 + ((c ^ ((nb + k) & 7)) << 4);
    for (long long q = pg; q < total; q += PW) {
        if (!tc::mbar_wait(&sm.raw_full[rs], rph, abort, a.wait_ns) ||
            !tc::mbar_wait(&sm.empty[stage], phase ^ 1u, abort, a.wait_ns)) {
            fail(a, sm, 13);
            return;
        }
        const uint8_t *const raw = sm.raw[rs];
        const bool tail = 8 * ks + c == a.npack && a.remain > 0;
        auto word = [&](int x) {
            const uint32_t w = *reinterpret_cast<const uint32_t *>(raw + word0 + 32 * x);
            return tail ? (w << (32 - 2 * a.remain)) | (0xFFFFFFFFu >> (2 * a.remain)) : w;
        };
        if (sideA) {
            uint8_t *const base = sm.a[stage];
#pragma unroll
            for (int x = 0; x < SA; ++x) {
                uint32_t sel[4];
                packed_selectors(word(x), sel);
#pragma unroll
                for (int g = 0; g < 3; ++g) {
                    constexpr uint32_t tables[3] = {PACKED_TABLE(1u, 0u, 0u, 0u), PACKED_TABLE(0u, 1u, 0u, 0u),
                                                    PACKED_TABLE(0u, 0u, 1u, 0u)};
                    const int i = 3 * x + g;
                    *reinterpret_cast<uint4 *>(base + at[i & 7] + 128 * i) = packed_lookup(tables[g], sel);
                }
            }
        } else if (rg < 7) {
            uint8_t *const base = sm.b[stage];
            const uint4 d[2] = {*reinterpret_cast<const uint4 *>(raw + PACKED_D + KS + 16 * c),  // w, D
                                *reinterpret_cast<const uint4 *>(raw + PACKED_D + 16 * c)};
#pragma unroll
            for (int x = 0; x < SB; ++x) {
                uint32_t sel[4];
                packed_selectors(word(x), sel);
#pragma unroll
                for (int g = 0; g < 3; ++g) {
                    constexpr uint32_t tables[3] = {PACKED_TABLE(0xFFu, 0u, 0u, 0u), PACKED_TABLE(0u, 0xFFu, 0u, 0u),
                                                    PACKED_TABLE(0u, 0u, 0xFFu, 0u)};
                    const uint4 M = packed_lookup(tables[g], sel);
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const int i = C::TY * x + 2 * g + k;
                        *reinterpret_cast<uint4 *>(base + at[i & 7] + 128 * i) =
                            make_uint4(M.x & d[k].x, M.y & d[k].y, M.z & d[k].z, M.w & d[k].w);
                    }
                }
            }
        }
        // (the raw slot is released after the stores, which consume every value loaded from it)
        tc::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
            tc::mbar_arrive(&sm.raw_empty[rs]);
            if (rank == 0) tc::mbar_arrive(&sm.full[stage]);
            else tc::mbar_arrive_remote(&sm.full[stage], 0);
        }
        ks += PW;
        while (ks >= nks) ks -= nks;
#pragma unroll
        for (int x = 0; x < PW; ++x) {
            advance<STAGES>(stage, phase);
            advance<RSTAGES>(rs, rph);
        }
    }
}

template <class C>
__global__ void __launch_bounds__(C::NTHREADS, 1) k_scan_mma(ScanArgs a, const __grid_constant__ MmaMaps maps)
{
    constexpr int STAGES = C::STAGES, RSTAGES = C::RSTAGES, EPW = C::EPW, PW = C::PW;
    using Smem = typename C::Smem;
    extern __shared__ uint8_t smem_raw[];
    // the operand stages need 1024-byte alignment (128-byte swizzle atoms); the offset is the
    // same in both CTAs of the pair, as the pair MMA and the remote arrivals require
    const uint32_t raw_s = tc::smem_u32(smem_raw);
    Smem &sm = *reinterpret_cast<Smem *>(smem_raw + (((raw_s + 1023u) & ~1023u) - raw_s));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = tc::cluster_rank();  // 0: issues the MMAs
    const int pair = (int)tc::cluster_id(), npairs = (int)tc::cluster_count();
    const int nks = a.Np / KS;
    // an earlier segment's candidates did not fit: the host scans again without the screen (the
    // flag is written between the segments' kernels only, so every thread reads the same)
    if (C::SCR && a.counters[CNT_OVERFLOW]) return;
    // the next segment's candidates: nothing else in this segment touches their counter
    if (C::SCR && !C::RAW && blockIdx.x == 0 && threadIdx.x == 0) a.counters[CNT_CAND + (a.segment + 1) % CAND_RING] = 0ull;

    if (warp == 12) {
        tc::tmem_alloc_pair(&sm.tmem_base, TMEM_COLS);
        tc::tmem_relinquish_pair();
    }
    // each CTA's B half holds six column types in rows 0-125: rows 126-127 stay zero
    constexpr int ZR = NH - TYH * TJ;
    for (int w = threadIdx.x; w < STAGES * ZR * 8; w += blockDim.x) {
        const int st = w / (ZR * 8), n = TYH * TJ + (w / 8) % ZR, c = w % 8;
        *reinterpret_cast<uint4 *>(sm.b[st] + (n >> 3) * 1024 + (n & 7) * 128 + c * 16) = make_uint4(0, 0, 0, 0);
    }
    tc::fence_proxy_async_smem();
    // maxima of F and F2 per trait: per CTA in shared memory (flushed to global memory once,
    // at the end) up to SMAX_TRAITS traits, else the global maxima directly
    // (the screen keeps none)
    const bool smax_local = !C::SCR && a.ntraits <= SMAX_TRAITS;
    unsigned int *smax = reinterpret_cast<unsigned int *>(reinterpret_cast<uint8_t *>(&sm) + sizeof(Smem));
    if (smax_local)
        for (int w = threadIdx.x; w < 2 * a.ntraits; w += blockDim.x) smax[w] = 0u;
    unsigned int *const mxf = smax_local ? smax : a.maxf;
    unsigned int *const mxf2 = smax_local ? smax + a.ntraits : a.maxf2;
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            tc::mbar_init(&sm.full[s], rank == 0 ? (C::XF ? 1 : C::RAW ? 8 : 10) : 1);
            tc::mbar_init(&sm.empty[s], 1);
        }
        for (int r = 0; r < RSTAGES; ++r) {
            tc::mbar_init(&sm.raw_full[r], C::RAW ? 64 : 1);
            tc::mbar_init(&sm.raw_empty[r], 4);
        }
        for (int b = 0; b < 2; ++b) {
            tc::mbar_init(&sm.acc_full[b], 1);
            tc::mbar_init(&sm.acc_empty[b], 8 * EPW);  // every epilogue warp of both CTAs
        }
        tc::mbar_init(&sm.drain, 1);
        tc::mbar_init(&sm.stall, 1);
        sm.abort = 0;
        tc::fence_barrier_init();
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::cluster_sync();  // both CTAs' barriers exist before any remote arrival
    tc::tc_fence_after();
    const uint32_t tmem = sm.tmem_base;
    volatile int *abort = &sm.abort;

    // epilogue warps: 0-3, 8-11 (and 16-19 with three per lane quarter, 4-7 too with four); producer warps: 4-7
    // (and 16-19 with two producer groups)
    const bool epi_warp = warp < 4 || (warp >= 8 && warp < 12) || (EPW >= 3 && warp >= 16) || (EPW == 4 && warp < 8);
    const bool prod_warp = !C::XF && ((warp >= 4 && warp < 8) || (PW >= 2 && warp >= 16));
    if constexpr (C::REBALANCE) {
        if (epi_warp) tc::setmaxnreg_inc<C::EPI_REGS>();
        else if (prod_warp) tc::setmaxnreg_dec<C::PROD_REGS>();
        else tc::setmaxnreg_dec<40>();
    }
    if (C::RAW && prod_warp) {
        if constexpr (C::RAW) raw_producers<C>(a, sm, rank, pair, npairs);
    } else if (prod_warp) {
        // ---------------- B producers: thread -> (j-SNP, 16-individual chunk) ----------------
        // items (jj, c) with jj < 16 for every thread, and (16 + t/8, c) for t < XTRA; with two
        // groups, group pg builds the stages whose sequence number is pg modulo 2 (and follows
        // the ring positions of the others without touching them)
        const int pg = warp >= 16 ? 1 : 0;
        const int t = threadIdx.x - (pg ? 512 : 128), jj = t >> 3, c = t & 7;
        const bool xtra = C::TJH > 16 && t < XTRA, mine = jj < C::TJH;
        constexpr int DG = C::SCR ? 1 + C::SCR : 2;  // digit rows of this CTA's half
        uint32_t stage = 0, phase = 0, rs = 0, rph = 0, seq = 0;
        bool ok = true;
        for (Walker<C> un(a, pair, npairs); !un.done && ok; un.next()) {
            for (int ks = 0; ks < nks; ++ks) {
                if ((int)(seq++ % (uint32_t)PW) != pg) {
                    advance<STAGES>(stage, phase);
                    advance<RSTAGES>(rs, rph);
                    continue;
                }
                if (!tc::mbar_wait(&sm.raw_full[rs], rph, abort, a.wait_ns) || !tc::mbar_wait(&sm.empty[stage], phase ^ 1u, abort, a.wait_ns)) {
                    fail(a, sm, 2);
                    ok = false;
                    break;
                }
                const uint8_t *raw = sm.raw[rs];
                uint8_t *base = sm.b[stage];
                // the digit rows of this CTA's half: all digits -- 2 rank and 2 rank + 1 of w, d2,
                // d1, d0; one digit -- w and D of the rows D, w; two -- w, d2, d1
                uint4 d[DG];
#pragma unroll
                for (int r = 0; r < DG; ++r)
                    d[r] = ld_sw128(raw + RAW_D, C::SCR == 0 ? 2 * (int)rank + r : C::SCR == 1 ? 1 - r : r, c);
                // local type q = DG b + r (genotype b, digit row r) of j-SNP jx at local row TY jx + q
                auto put = [&](int q, int jx, const uint4 &m) {
                    const int n = C::TY * jx + q;
                    const uint4 &dv = d[q % DG];
                    uint4 o;
                    o.x = m.x & dv.x;
                    o.y = m.y & dv.y;
                    o.z = m.z & dv.z;
                    o.w = m.w & dv.w;
                    *reinterpret_cast<uint4 *>(base + (n >> 3) * 1024 + (n & 7) * 128 + ((c ^ (n & 7)) << 4)) = o;
                };
                // byte mask of genotype b: one-hot bit b of each byte spread to 0xFF
                auto gmask = [](const uint4 &h, int b) {
                    uint4 m;
                    m.x = ((h.x >> b) & 0x01010101u) * 0xFFu;
                    m.y = ((h.y >> b) & 0x01010101u) * 0xFFu;
                    m.z = ((h.z >> b) & 0x01010101u) * 0xFFu;
                    m.w = ((h.w >> b) & 0x01010101u) * 0xFFu;
                    return m;
                };
                auto build = [&](int jx) {
                    const uint4 h = ld_sw128(raw + RAW_J, jx, c);
#pragma unroll
                    for (int b = 0; b < 3; ++b) {
                        const uint4 m = gmask(h, b);
#pragma unroll
                        for (int r = 0; r < DG; ++r) put(DG * b + r, jx, m);
                    }
                };
                if (mine) build(jj);
                if (xtra) build(16 + jj);
                // the raw slot is released only after the stores above, which consume every
                // value loaded from it (an arrive right after the loads can overtake them)
                tc::fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {
                    tc::mbar_arrive(&sm.raw_empty[rs]);
                    if (rank == 0) tc::mbar_arrive(&sm.full[stage]);
                    else tc::mbar_arrive_remote(&sm.full[stage], 0);
                }
                advance<STAGES>(stage, phase);
                advance<RSTAGES>(rs, rph);
            }
        }
    } else if (C::SCR && epi_warp) {
        if constexpr (C::GT > 1) group_epilogue<C>(a, sm, tmem, rank, pair, npairs);
        else if constexpr (C::SCR != 0) screen_epilogue<C>(a, sm, tmem, rank, pair, npairs);
    } else if (epi_warp) {
        // ---------------- epilogue: the j rounds split over the warps of each lane quarter ----------------
        // warps 0-3 (group 0), 8-11 (group 1), 16-19 (group 2): rounds [rb(g), rb(g + 1))
        const int e = warp & 3, grp = warp < 4 ? 0 : (warp < 12 ? 1 : 2);
        const int rho_begin = (grp * ROUNDS + EPW - 1) / EPW, rho_end = ((grp + 1) * ROUNDS + EPW - 1) / EPW;
        const int ii = 10 * e + lane / 3, ga = lane % 3, tbase = (lane / 3) * 3;
        const bool rowok = lane < 30;
        const uint32_t tl = tmem + ((uint32_t)(32 * e) << 16);
        uint32_t accph[2] = {0u, 0u};
        int buf = 0;
        for (Walker<C> un(a, pair, npairs); !un.done; un.next()) {
            const int t = un.trait;
            const double sc = a.yscale[t];
            const int di = un.i0 + TI * (int)rank + ii;  // this CTA's i-SNPs
            const bool ivalid = rowok && di < un.bd.size1;
            const int gi = un.bd.start1 + (ivalid ? di : 0);
            const size_t mi = (size_t)t * a.nsnp + gi;
            // sum of ytilde^2 over the valid individuals known at SNP i; and the quantities of
            // the individuals missing at i that the exact path needs
            const double pki = ivalid ? a.qtot[t] - a.qm[mi] : 0.0;
            const double smi = ivalid ? a.sm[mi] : 0.0, nmi_nv = ivalid ? a.nm[mi] - a.nvalid[t] : 0.0;
            const double ytot = a.ytot[t];
            if (!tc::mbar_wait(&sm.acc_full[buf], accph[buf], abort, a.wait_ns)) {
                fail(a, sm, 3);
                break;
            }
            tc::tc_fence_after();
            const uint32_t acc = tl + acc_col(buf);
            const bool report = a.report_trait < 0 || a.report_trait == t;
            const bool dumping = t == a.report_trait && (a.dump_counts || a.dump_F || a.dump_F2 || a.dump_df1 || a.dump_df2);
            const float t1c = screen_lo(a.t1), t2c = screen_lo(a.t2), scf = (float)sc;
            unsigned int fmx = 0u, f2mx = 0u;  // this thread's largest F, F2 of the tile (encoded)
            // screen against the CTA's maxima so far (exact values, a lower bound of the final
            // maxima): a pair that can raise a maximum always takes the exact path
            const unsigned int m1 = reinterpret_cast<volatile unsigned int *>(mxf)[t];
            const unsigned int m2 = reinterpret_cast<volatile unsigned int *>(mxf2)[t];
            float fmx_f = m1 ? ord2f(m1) : -INFINITY, f2mx_f = m2 ? ord2f(m2) : -INFINITY;
#pragma unroll 1
            for (int rho = rho_begin; rho < rho_end; ++rho) {
                const int jb = 3 * rho;
                const int jl = jb + ga;
                const int dj = un.j0 + jl;
                const bool valid = ivalid && (jl < TJ) && dj < un.bd.size2 &&
                                   (un.bd.start1 + di > un.bd.start2 + dj);
                const int gj = un.bd.start2 + (valid ? dj : 0);
                const size_t mj = (size_t)t * a.nsnp + gj;
                const double qmj = valid ? a.qm[mj] : 0.0;
                // the round's columns of both halves, then v[ty][c] = type ty of j-SNP jb + c
                uint32_t wv[2][RCOLS], v[NTYPE][3];
                auto load_round = [&]() {
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int k = 0; k < RCOLS / 4; ++k)
                            tc::tmem_ld4(acc + h * NH + 6 * jb + 4 * k, wv[h][4 * k], wv[h][4 * k + 1], wv[h][4 * k + 2],
                                         wv[h][4 * k + 3]);
                    tc::tmem_wait_ld();
#pragma unroll
                    for (int ty = 0; ty < NTYPE; ++ty)
#pragma unroll
                        for (int c = 0; c < 3; ++c) v[ty][c] = wv[(ty & 3) >> 1][6 * c + bq(ty)];
                };
                load_round();
                // this lane's accumulator row (SNP i, genotype ga) folded per column c of the round
                // (j-SNP jb + c): three counts and three FP32 phenotype sums. Up to 131,072
                // individuals every digit sum is below 2^24 in magnitude, so the conversions are
                // exact and the two fmas round once each (beyond, the conversions round too:
                // relative 2^-24, far inside the screen's margin).
                int cn[3][3];
                float cs[3][3];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
#pragma unroll
                    for (int b = 0; b < 3; ++b) {
                        cn[c][b] = (int)v[4 * b][c];
                        cs[c][b] = fmaf(65536.0f, (float)(int)v[4 * b + 1][c],
                                        fmaf(256.0f, (float)(int)v[4 * b + 2][c], (float)(int)v[4 * b + 3][c]));
                    }
                }
                // the pair (SNP i, j-SNP jb + ga) is this lane's: its own row directly, the rows of
                // the triplet's other two lanes by shuffle, each lane offering the column its reader
                // needs (the lane of genotype ga+1 offers its column (ga+1)+2 = ga, mod 3). Cells
                // row-major in this relative row order (own, ga+1, ga+2): F and F2 do not depend
                // on the order of the rows; only the count dump maps them back to genotypes.
                const int s1 = tbase + (ga + 1) % 3, s2 = tbase + (ga + 2) % 3;
                const int o1 = (ga + 2) % 3, o2 = (ga + 1) % 3;  // the columns this lane offers
                int n[9];
                float sfd[9];
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    n[b] = pick3(cn[0][b], cn[1][b], cn[2][b], ga);
                    n[3 + b] = __shfl_sync(0xffffffffu, pick3(cn[0][b], cn[1][b], cn[2][b], o1), s1);
                    n[6 + b] = __shfl_sync(0xffffffffu, pick3(cn[0][b], cn[1][b], cn[2][b], o2), s2);
                    sfd[b] = pick3(cs[0][b], cs[1][b], cs[2][b], ga);
                    sfd[3 + b] = __shfl_sync(0xffffffffu, pick3(cs[0][b], cs[1][b], cs[2][b], o1), s1);
                    sfd[6 + b] = __shfl_sync(0xffffffffu, pick3(cs[0][b], cs[1][b], cs[2][b], o2), s2);
                }
                PairStat s;
                s.nfac = s.d1 = s.d2 = 0;
                s.F = s.F2 = 0.0;
                int npair = 0;
                bool exact = false;
                if (valid) {
#pragma unroll
                    for (int c = 0; c < 9; ++c) npair += n[c];
                    // a lower bound of the pair's sum of squares (QMM_ij >= 0 left out), so the
                    // screened F and F2 bound the pair's values from above
                    const float Qf = (float)(pki - qmj);
                    float Ff, F2f;
                    pair_stat_f32(n, sfd, scf, Qf, a.test_int != 0, Ff, F2f);
                    exact = dumping || npair < 256 || !(Ff <= t1c) || !(Ff <= screen_lo(fmx_f)) ||
                            (a.test_int && (!(F2f <= t2c) || !(F2f <= screen_lo(f2mx_f))));
                    if (!exact) {
                        // below every threshold and both running maxima by more than the margin
                        int nfac = 0;
#pragma unroll
                        for (int c = 0; c < 9; ++c) nfac += n[c] > 0;
                        s.nfac = nfac;
                        s.d1 = nfac - 1;
                        s.d2 = npair - nfac;
                        s.F = Ff;
                        s.F2 = F2f;
                    }
                }
                if (__any_sync(0xffffffffu, exact)) {
                    // rare (pairs near a threshold or a running maximum, count dumps, small
                    // blocks): the exact digit sums of every cell, gathered again from the
                    // accumulator (still in TMEM until this warp releases it)
                    load_round();
                    uint32_t r1[NTYPE], r2[NTYPE];
#pragma unroll
                    for (int ty = 0; ty < NTYPE; ++ty) {
                        r1[ty] = __shfl_sync(0xffffffffu, sel3(v[ty], o1), s1);
                        r2[ty] = __shfl_sync(0xffffffffu, sel3(v[ty], o2), s2);
                    }
                    double si[9];  // digit sums as exact integers
                    double qmm = 0.0;
                    int nmm = 0;
                    if (exact) {
                        double st = 0.0;
#pragma unroll
                        for (int b = 0; b < 3; ++b) {
                            const uint32_t c3[3] = {sel3(v[4 * b + 1], ga), r1[4 * b + 1], r2[4 * b + 1]};
                            const uint32_t c2[3] = {sel3(v[4 * b + 2], ga), r1[4 * b + 2], r2[4 * b + 2]};
                            const uint32_t c1[3] = {sel3(v[4 * b + 3], ga), r1[4 * b + 3], r2[4 * b + 3]};
#pragma unroll
                            for (int r = 0; r < 3; ++r) {
                                si[3 * r + b] = fma(65536.0, (double)(int)c3[r],
                                                    fma(256.0, (double)(int)c2[r], (double)(int)c1[r]));
                                st += si[3 * r + b];
                            }
                        }
                        // the individuals missing at both SNPs: their number, and for a single
                        // one its y^2 from the Y sums (every term an exact integer below 2^53)
                        nmm = npair + (int)(nmi_nv + a.nm[mj]);
                        if (nmm == 1) {
                            const double ymm = (st - ytot + smi + a.sm[mj]) * sc;
                            qmm = ymm * ymm;
                        }
                    }
                    // two or more: the whole warp intersects the two SNPs' missing bits for each
                    // such pair in turn and sums ytilde^2 over the intersection
                    unsigned int need = __ballot_sync(0xffffffffu, exact && nmm >= 2);
                    while (need) {
                        const int src = __ffs(need) - 1;
                        need &= need - 1;
                        const int si_ = __shfl_sync(0xffffffffu, gi, src), sj_ = __shfl_sync(0xffffffffu, gj, src);
                        const double part = missing_both_q(a, t, si_, sj_);
                        if (lane == src) qmm = part;
                    }
                    if (exact) s = pair_stat_exact(n, si, sc, pki - qmj + qmm, a.test_int != 0);
                }
                if (valid && dumping) {
                    const size_t o = (size_t)di * un.bd.size2 + dj;
                    if (a.dump_counts)
#pragma unroll
                        for (int c = 0; c < 9; ++c)  // relative row c/3 is genotype (ga + c/3) mod 3
                            a.dump_counts[9 * o + 3 * ((ga + c / 3) % 3) + c % 3] = n[c];
                    if (a.dump_F) a.dump_F[o] = (float)s.F;
                    if (a.dump_F2) a.dump_F2[o] = (float)s.F2;
                    if (a.dump_df1) a.dump_df1[o] = s.d1;
                    if (a.dump_df2) a.dump_df2[o] = s.d2;
                }
                const bool hit = valid && report && is_hit(a, s);
                emit_hit(a, hit, un.bd.start1 + di, un.bd.start2 + dj, s, t, un.block);
                if (valid && s.F == s.F) {
                    fmx = max(fmx, f2ord((float)s.F));
                    fmx_f = fmaxf(fmx_f, (float)s.F);
                }
                if (valid && s.F2 == s.F2) {
                    f2mx = max(f2mx, f2ord((float)s.F2));
                    f2mx_f = fmaxf(f2mx_f, (float)s.F2);
                }
            }
            fold_max_enc(&mxf[t], fmx);
            if (a.test_int) fold_max_enc(&mxf2[t], f2mx);
            tc::tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if (rank == 0) tc::mbar_arrive(&sm.acc_empty[buf]);
                else tc::mbar_arrive_remote(&sm.acc_empty[buf], 0);
            }
            accph[buf] ^= 1u;
            buf ^= 1;
        }
    } else if (C::RAW && (warp == 13 || warp == 14)) {
        if constexpr (C::RAW) raw_loader<C>(a, sm, rank, pair, npairs);
    } else if (warp == 13 && !C::RAW) {
        // ---------------- A loader: this CTA's indicator rows, one slot per operand stage ----
        if (lane == 0) {
            uint32_t as = 0, aph = 0, issued_a = 0;
            bool ok = true;
            for (Walker<C> un(a, pair, npairs); !un.done && ok; un.next()) {
                const int arow = 3 * (un.bd.start1 + un.i0 + TI * (int)rank);
                const int xrow = C::SCR ? (un.trait * a.nsnp + un.bd.start2 + un.j0 + C::TJH * (int)rank) * C::TY
                                        : ((un.trait * 2 + (int)rank) * a.nsnp + un.bd.start2 + un.j0) * C::TY;
                for (int ks = 0; ks < nks; ++ks) {
                    if (!tc::mbar_wait(&sm.empty[as], aph ^ 1u, abort, a.wait_ns)) {
                        fail(a, sm, 7);
                        ok = false;
                        break;
                    }
                    if constexpr (C::XF) {
                        // both CTAs' loads complete on CTA 0's barrier, which expects the bytes of
                        // both (no forward through CTA 1); this CTA's half of the B stage: 126
                        // expanded rows
                        if (rank == 0) tc::mbar_arrive_expect_tx(&sm.full[as], 2 * (A_BYTES + XB_BYTES));
                        const uint32_t bar = tc::mapa(&sm.full[as], 0);
#pragma unroll
                        for (int w = 0; w < 4; ++w)
                            tc::tma_load_2d_pair(sm.a[as] + 32 * w * KS, &maps.hi, ks * KS, arow + A_BOX * w, bar);
                        tc::tma_load_2d_pair(sm.b[as], &maps.hx, ks * KS, xrow, bar);
                    } else {
                        tc::mbar_arrive_expect_tx(&sm.full[as], A_BYTES);
#pragma unroll
                        for (int w = 0; w < 4; ++w)
                            tc::tma_load_2d(sm.a[as] + 32 * w * KS, &maps.hi, ks * KS, arow + A_BOX * w, &sm.full[as]);
                    }
                    ++issued_a;
                    advance<STAGES>(as, aph);
                }
            }
            // no TMA write may still be landing in shared memory when the CTA exits: wait for
            // the last loads issued into every slot. A stages of CTA 1 complete on its local
            // barrier; CTA 0's also need CTA 1's forward, so CTA 0 waits for its own bytes only
            // through the phases it can observe (all its issued phases complete on the normal
            // path; after an abort the bounded wait ends). With streamed B CTA 0 waits for both
            // CTAs' loads, and CTA 1 for CTA 0 in the cluster barrier below.
            int no_abort = 0;
            for (uint32_t back = 1; back <= STAGES && back <= issued_a && !(C::XF && rank == 1); ++back) {
                const uint32_t slot = (as + STAGES - back) % STAGES, par = back > as ? (aph ^ 1u) : aph;
                if (!tc::mbar_wait(&sm.full[slot], par, &no_abort, a.wait_ns)) fail(a, sm, 8);
            }
        }
    } else if (warp == 14 && !C::XF && !C::RAW) {
        // ---------------- raw loader: j one-hot rows and trait digit rows ----------------
        // gated only by the B producers' consumption, so it runs up to RSTAGES stages ahead
        // of them (the j rows come from DRAM once per pair tile)
        if (lane == 0) {
            uint32_t rs = 0, rph = 0, issued_r = 0;
            bool ok = true;
            for (Walker<C> un(a, pair, npairs); !un.done && ok; un.next()) {
                for (int ks = 0; ks < nks; ++ks) {
                    if (!tc::mbar_wait(&sm.raw_empty[rs], rph ^ 1u, abort, a.wait_ns)) {
                        fail(a, sm, 10);
                        ok = false;
                        break;
                    }
                    uint8_t *raw = sm.raw[rs];
                    tc::mbar_arrive_expect_tx(&sm.raw_full[rs], C::RAW_BYTES);
                    tc::tma_load_2d(raw + RAW_J, C::SCR == 2 ? &maps.hj2 : &maps.hj, ks * KS,
                                    un.bd.start2 + un.j0 + (C::SCR ? C::TJH * (int)rank : 0), &sm.raw_full[rs]);
                    if constexpr (C::SCR == 0)
                        tc::tma_load_2d(raw + RAW_D, &maps.dg, ks * KS, DROWS * un.trait + 1, &sm.raw_full[rs]);
                    else if constexpr (C::SCR == 1)
                        tc::tma_load_2d(raw + RAW_D, &maps.ds, ks * KS, DROWS * un.trait, &sm.raw_full[rs]);
                    else
                        tc::tma_load_2d(raw + RAW_D, &maps.ds2, ks * KS, DROWS * un.trait + 1, &sm.raw_full[rs]);
                    ++issued_r;
                    advance<RSTAGES>(rs, rph);
                }
            }
            int no_abort = 0;
            for (uint32_t back = 1; back <= RSTAGES && back <= issued_r; ++back) {
                const uint32_t slot = (rs + RSTAGES - back) % RSTAGES, par = back > rs ? (rph ^ 1u) : rph;
                if (!tc::mbar_wait(&sm.raw_full[slot], par, &no_abort, a.wait_ns)) fail(a, sm, 11);
            }
        }
    } else if (warp == 12 && lane == 0 && rank == 1 && !C::XF && !C::RAW) {
        // ---------------- A forwarder (CTA 1, warp 12) ----------------
        // each of this CTA's A stages, once landed, counts as one arrival on CTA 0's full
        uint32_t as = 0, aph = 0;
        bool ok = true;
        for (long long u = pair; u < a.seg_units && ok; u += npairs) {
            for (int ks = 0; ks < nks; ++ks) {
                if (!tc::mbar_wait(&sm.full[as], aph, abort, a.wait_ns)) {
                    fail(a, sm, 9);
                    ok = false;
                    break;
                }
                tc::mbar_arrive_remote(&sm.full[as], 0);
                advance<STAGES>(as, aph);
            }
        }
    } else if (warp == 12 && lane == 0 && rank == 0) {
        // ---------------- MMA issuer (CTA 0, warp 12) ----------------
        // (it needs the number of this cluster's units only: walking them would cost it about 900
        // cycles between two units, and it is the critical path)
        uint32_t as = 0, aph = 0, accph[2] = {0u, 0u};
        int buf = 0;
        bool ok = true;
        // test hook: the first CTA pair's issuer waits on a barrier that nothing arrives at, so
        // the wait runs out after wait_ns and the scan ends with a timeout status
        if (a.debug_stall && pair == 0 && !tc::mbar_wait(&sm.stall, 0, abort, a.wait_ns)) {
            fail(a, sm, 12);
            ok = false;
        }
        for (long long u = pair; u < a.seg_units && ok; u += npairs) {
            if (!tc::mbar_wait_cluster(&sm.acc_empty[buf], accph[buf] ^ 1u, abort, a.wait_ns)) {
                fail(a, sm, 4);
                break;
            }
            tc::tc_fence_after();
            const uint32_t d = tmem + acc_col(buf);
            for (int ks = 0; ks < nks; ++ks) {
                if (!tc::mbar_wait_cluster(&sm.full[as], aph, abort, a.wait_ns)) {
                    fail(a, sm, 5);
                    ok = false;
                    break;
                }
                tc::tc_fence_after();
                const uint32_t asb = tc::smem_u32(sm.a[as]), bsb = tc::smem_u32(sm.b[as]);
#pragma unroll
                for (int kk = 0; kk < KS / 32; ++kk)
                    tc::mma_i8_pair(d, tc::smem_desc_sw128(asb + 32 * kk), tc::smem_desc_sw128(bsb + 32 * kk), IDESC,
                                    (ks | kk) != 0);
                tc::mma_commit_pair_mc(&sm.empty[as], 0x3);
                advance<STAGES>(as, aph);
            }
            if (!ok) break;
            tc::mma_commit_pair_mc(&sm.acc_full[buf], 0x3);
            accph[buf] ^= 1u;
            buf ^= 1;
        }
        // every MMA issued above has completed once `drain` flips (waited for even after an
        // abort: the accumulators and both CTAs' operands must be idle before the TMEM and
        // shared memory are released)
        tc::mma_commit_pair(&sm.drain);
        int no_abort = 0;
        if (!tc::mbar_wait(&sm.drain, 0, &no_abort, a.wait_ns)) fail(a, sm, 6);
    }

    tc::tc_fence_before();
    __syncthreads();
    tc::cluster_sync();  // CTA 0's MMAs (which read CTA 1's shared memory) have drained
    if (warp == 12) {
        tc::tc_fence_after();
        tc::tmem_dealloc_pair(tmem, TMEM_COLS);
    }
    if (smax_local)
        for (int w = threadIdx.x; w < 2 * a.ntraits; w += blockDim.x)
            if (smax[w]) atomicMax(w < a.ntraits ? &a.maxf[w] : &a.maxf2[w - a.ntraits], smax[w]);
}

}  // namespace mma

using Screen2Digits = mma::Rings<6, 6, 2, 1, false, 2>;
using GroupRings = mma::Rings<7, 1, 2, 1, true, 1, false, GROUP_TRAITS>;
struct GroupOf { using type = GroupRings; };

// Tensor maps of the tensor form's TMA loads: the genotype-indicator rows h3 [3 nsnp][Np]
// with 30-row boxes (A), the one-hot genotype bytes [nsnp][Np] with boxes of a half's j-SNPs (21; 14 for
// the screen with two digits) and the trait digit rows [5T][Np] with boxes of 4 (all digits), 2 and 3 rows
// (the screen with one digit and with two); all 128 bytes wide, 128-byte swizzled, out-of-range rows read
// as zero.
static cudaError_t encode_2d(CUtensorMap *m, const void *base, uint64_t inner, uint64_t rows, uint32_t box_rows)
{
    static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    if (!encode) {
        cudaDriverEntryPointQueryResult q;
        void *fn = nullptr;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
        if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !fn) return cudaErrorNotSupported;
        encode = (PFN_cuTensorMapEncodeTiled_v12000)fn;
    }
    const cuuint64_t dims[2] = {inner, rows};
    const cuuint64_t strides[1] = {inner};
    const cuuint32_t box[2] = {(cuuint32_t)mma::KS, box_rows};
    const cuuint32_t es[2] = {1, 1};
    CUresult r = encode(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(base), dims, strides, box, es,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

cudaError_t mma_encode_genotypes(MmaMaps *maps, const uint8_t *hcodes, const uint8_t *h3, int nsnp, int Np)
{
    cudaError_t e = encode_2d(&maps->hi, h3, (uint64_t)Np, 3 * (uint64_t)nsnp, mma::A_BOX);
    if (e == cudaSuccess) e = encode_2d(&maps->hj, hcodes, (uint64_t)Np, (uint64_t)nsnp, mma::TJ);
    if (e == cudaSuccess) e = encode_2d(&maps->hj2, hcodes, (uint64_t)Np, (uint64_t)nsnp, Screen2Digits::TJH);
    return e;
}

cudaError_t mma_encode_traits(MmaMaps *maps, const int8_t *ydig, int ntraits, int Np)
{
    const uint64_t rows = (uint64_t)mma::DROWS * ntraits;
    cudaError_t e = encode_2d(&maps->dg, ydig, (uint64_t)Np, rows, mma::ND);
    if (e == cudaSuccess) e = encode_2d(&maps->ds, ydig, (uint64_t)Np, rows, 2);
    if (e == cudaSuccess) e = encode_2d(&maps->ds2, ydig, (uint64_t)Np, rows, 3);
    return e;
}

// The streamed-B variant's expanded rows ([ntraits][2][nsnp][6][Np] with all digits, prep.cu: k_expand) go
// in boxes of one CTA half of a j tile (126 rows). Rows per SNP and set of them:
int mma_x_rows(int screen) { return screen == 3 ? 3 * (1 + GROUP_TRAITS) : screen ? 3 * (1 + screen) : mma::NTYPE; }
// and sets: one per trait, or per group of traits
int mma_x_sets(int screen, int ntraits) { return screen == 3 ? (ntraits + GROUP_TRAITS - 1) / GROUP_TRAITS : ntraits; }

cudaError_t mma_encode_x(MmaMaps *maps, const int8_t *x, int nsnp, int Np, int ntraits, int screen)
{
    return encode_2d(&maps->hx, x, (uint64_t)Np, (uint64_t)mma_x_rows(screen) * nsnp * mma_x_sets(screen, ntraits),
                     mma::TYH * mma::TJ);
}

bool mma_available() { return true; }
int mma_tile_i() { return mma::TIP; }  // the host tiles blocks by CTA-pair tiles
int mma_tile_j(int screen)
{
    return screen == 0 ? mma::TJ : screen == 1 ? 2 * mma::TJ : screen == 2 ? Screen2Digits::TJT : GroupRings::TJT;
}
// The automatic choice screens with this form from here on. Kernel time against the plain form, 8 df and
// 4 df, B200: N = 64 x 2,000 SNPs 64 us and 320, N = 150 x 240 22 and 88, N = 231 x 2,003 69 and
// 443, N = 126 x 30,000 6.3 ms and 61. With few individuals many pairs fit nearly perfectly and
// the screen settles none of them: at N = 20 both take 0.3 ms.
int mma_min_nid() { return 64; }
int mma_max_nid() { return 1 << 24; }  // digit sums stay within int32
// the screen's sums (127 per individual) stay below 2^22, its counts below 2^15
int mma_screen_max_nid() { return (1 << 15) - mma::KS; }

// The variants the autotuner chooses among -- operand slots and raw stages (each ~200-230 KB
// of shared memory) and epilogue warps per TMEM lane quarter:
//   0  6 slots / 6 raw, 2 epilogue warps   1  5 / 10, 2   2  6 / 4, 2   3  6 / 6, 3
//   4  6 / 6, 2 epilogue warps, two producer groups on alternate stages
//   5  6 slots, streamed B (expanded rows TMA-loaded from HBM; no producers, no raw ring)
// The screen needs half the expanded rows per pair, so streamed B is its fastest variant at every
// size and comes twice, with 7 slots: 5 with 2 epilogue warps per lane quarter, 2 with 4 (the
// faster one below about 1,500 individuals, where the epilogue bounds a unit: N = 500 x 4,000
// SNPs 130 us against 146; N = 4,000 x 20,000 SNPs 8.70 ms against 8.55).
constexpr int MMA_SHAPES = 6;

// variant v with SCR digits in the screen (0: all digits)
template <int V, int SCR>
struct VariantOf;
template <int SCR> struct VariantOf<0, SCR> { using type = mma::Rings<6, 6, 2, 1, false, SCR>; };
template <int SCR> struct VariantOf<1, SCR> { using type = mma::Rings<5, 10, 2, 1, false, SCR>; };
template <int SCR> struct VariantOf<2, SCR> { using type = mma::Rings<7, 1, 4, 1, true, SCR>; };
template <> struct VariantOf<2, 0> { using type = mma::Rings<6, 4, 2, 1, false, 0>; };
template <int SCR> struct VariantOf<3, SCR> { using type = mma::Rings<6, 6, 3, 1, false, SCR>; };
template <int SCR> struct VariantOf<4, SCR> { using type = mma::Rings<6, 6, 2, 2, false, SCR>; };
template <int SCR> struct VariantOf<5, SCR> { using type = mma::Rings<SCR ? 7 : 6, 1, 2, 1, true, SCR>; };

bool mma_needs_x(int v, int screen) { return v == 5 || (v == 2 && screen); }

int mma_shapes() { return MMA_SHAPES; }

void mma_shape(int v, int screen, const char **desc)
{
    static const char *names[MMA_SHAPES] = {"6 operand slots / 6 raw stages, 8 epilogue warps",
                                            "5 operand slots / 10 raw stages, 8 epilogue warps",
                                            "6 operand slots / 4 raw stages, 8 epilogue warps",
                                            "6 operand slots / 6 raw stages, 12 epilogue warps (setmaxnreg)",
                                            "6 operand slots / 6 raw stages, 8 epilogue warps, 2 producer groups (setmaxnreg)",
                                            "6 operand slots, B streamed from HBM, 8 epilogue warps"};
    if (desc) *desc = screen && v == 2   ? "7 operand slots, B streamed from HBM, 16 epilogue warps"
                      : screen && v == 5 ? "7 operand slots, B streamed from HBM, 8 epilogue warps"
                                         : names[v];
}

// Launch shape per (device, variant, dynamic shared memory size): the attribute set and the
// number of co-resident clusters, queried once (the occupancy query costs far more than a
// small scan's host work).
struct MmaShape {
    int device, variant;
    size_t smem;
    int clusters;
};

static std::mutex g_shape_mu;
static std::vector<MmaShape> g_shapes;

template <class C>
static cudaLaunchConfig_t mma_config(int ntraits, int grid, cudaStream_t stream, cudaLaunchAttribute *attr)
{
    cudaLaunchConfig_t cfg = {};
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)grid, 1, 1);
    cfg.blockDim = dim3(C::NTHREADS, 1, 1);
    // more than half of the SM's shared memory: one CTA per SM, which owns all 512 TMEM
    // columns; the tail holds the per-CTA maxima
    cfg.dynamicSmemBytes = sizeof(typename C::Smem) + 1024 + (C::SCR ? 0 : smax_bytes(ntraits));
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

template <class C>
static cudaError_t prepare(int v, int ntraits, int grid_request, int *grid)
{
    static_assert(sizeof(typename C::Smem) + 1024 > 116 * 1024, "one CTA per SM");
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = mma_config<C>(ntraits, std::max(2, (grid_request + 1) & ~1), nullptr, attr);
    int clusters = 0;
    {
        std::lock_guard<std::mutex> lock(g_shape_mu);
        for (const MmaShape &sh : g_shapes)
            if (sh.device == device && sh.variant == v && sh.smem == cfg.dynamicSmemBytes) clusters = sh.clusters;
        if (clusters == 0) {
            // the attribute admits the largest size any trait count asks for
            e = cudaFuncSetAttribute(mma::k_scan_mma<C>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(sizeof(typename C::Smem) + 1024 + (C::SCR ? 0 : smax_bytes(SMAX_TRAITS))));
            if (e != cudaSuccess) return e;
            e = cudaOccupancyMaxActiveClusters(&clusters, mma::k_scan_mma<C>, &cfg);
            if (e != cudaSuccess) return e;
            if (clusters < 1) return cudaErrorInvalidConfiguration;
            g_shapes.push_back({device, v, cfg.dynamicSmemBytes, clusters});
        }
    }
    *grid = std::min((int)cfg.gridDim.x, 2 * clusters);
    return cudaSuccess;
}

template <class C>
static cudaError_t enqueue(const ScanArgs &a, const MmaMaps &maps, int grid, cudaStream_t stream)
{
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = mma_config<C>(a.ntraits, grid, stream, attr);
    cudaError_t e = cudaLaunchKernelEx(&cfg, mma::k_scan_mma<C>, a, maps);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

// f(VariantOf<v, screen>())
template <int SCR, class F>
static cudaError_t with_rings(int v, F f)
{
    switch (v) {
    case 0: return f(VariantOf<0, SCR>());
    case 1: return f(VariantOf<1, SCR>());
    case 2: return f(VariantOf<2, SCR>());
    case 3: return f(VariantOf<3, SCR>());
    case 4: return f(VariantOf<4, SCR>());
    case 5: return f(VariantOf<5, SCR>());
    }
    return cudaErrorInvalidValue;
}

template <class F>
static cudaError_t with_variant(int v, int screen, F f)
{
    switch (screen) {
    case 0: return with_rings<0>(v, f);
    case 1: return with_rings<1>(v, f);
    case 2: return with_rings<2>(v, f);
    case 3: return f(GroupOf());  // one variant only
    }
    return cudaErrorInvalidValue;
}

using RawRings = mma::Rings<6, 8, 2, 3, false, 1, true>;

// The same for the kernel of epi_scan_block_noalloc.
cudaError_t mma_raw_prepare(int grid_request, int *grid) { return prepare<RawRings>(-1, 1, grid_request, grid); }
cudaError_t mma_raw_enqueue(const ScanArgs &a, int grid, cudaStream_t stream)
{
    static const MmaMaps none = {};
    return enqueue<RawRings>(a, none, grid, stream);
}

// The launch shape of a scan with variant v, resolved before any stream capture: the kernel's
// shared-memory attribute and the number of co-resident clusters, then whole clusters of two --
// at least one, never more than can be resident at once.
cudaError_t mma_prepare(int v, int screen, int ntraits, int grid_request, int *grid)
{
    return with_variant(v, screen, [&](auto c) {
        return prepare<typename decltype(c)::type>(v + MMA_SHAPES * screen, ntraits, grid_request, grid);
    });
}

// The launch itself (a stream operation only, so it can be captured into a CUDA graph).
cudaError_t mma_enqueue(int v, int screen, const ScanArgs &a, const MmaMaps &maps, int grid, cudaStream_t stream)
{
    return with_variant(v, screen,
                        [&](auto c) { return enqueue<typename decltype(c)::type>(a, maps, grid, stream); });
}

}  // namespace epi
