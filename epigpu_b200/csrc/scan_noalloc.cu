// scan_noalloc.cu -- the allocation-free entry point (epi_scan_block_noalloc): a scan that reads
// the reference's packed genotype words directly (src/readplink.c:1066-1102) and writes 24-byte
// result rows, with all of its working memory in one fixed device array.
//
// Two ways. The tensor form's one-digit screen (scan_mma.cu: its RAW
// variant builds both operands from the packed words; k_exact settles what it passes on) in parts
// of up to 3,072 x 3,072 SNPs (the fixed array holds what either side needs per SNP, and a list of 8,000
// candidates), a second time with a small first part where a list ran over that was expected to be near
// full; and, where the screen would pass on too much (low thresholds, many
// individuals) or its list runs over all the same, the plain kernel below. At 1,203 individuals x
// 2,502 SNPs the plain kernel takes 4.7 ms, ten FP32 operations per pair and individual.
//
// The plain kernel is the reference's per-individual method (src/EpiOpenCL.c:110-228: unpack two
// SNPs, count the 3x3 genotype cells, add the phenotype into its cell) on the CUDA cores.
// Persistent, one 512-thread CTA per SM, pulling 64 x 32 SNP-pair tiles from a queue. Per
// tile it walks the individuals in stages of 64:
//   * stage expansion: the i-tile's genotype bits become U_a = [g_i==a]*y and U_V = [g_i valid]
//     as floats in shared memory (read by the whole warp: broadcast loads);
//   * cell counts: AND + __popc of 32-bit plane words (phenotype mask folded into the
//     i side), 16-bit packed counters;
//   * cell sums: each lane turns its own j-SNP's plane bits into F_b = [g_j==b] and
//     F_Q = [g_j valid]*q in registers, then S_ab += U_a*F_b (9 FP32 FMAs per pair and
//     individual) and Q += U_V*F_Q (sum of y^2 over valid individuals, q = y^2 - mean y^2).
// Each thread owns 4 whole pairs (the warp's four i-SNPs x the lane's j-SNP).
// Epilogue: FP64 SSB/SSI/F/F2 per pair, warp-aggregated atomic row append, maximum F.
#include <algorithm>
#include <cmath>
#include <cstddef>

#include "epi_internal.cuh"
#include "epigpu.h"
#include "screen_rule.cuh"

namespace epi {
namespace popc_raw {

constexpr int TI = 64;   // i-SNPs per tile (16 warps x 4, shared by the warp's lanes)
constexpr int TJ = 32;   // j-SNPs per tile (one per lane)
constexpr int NT = 512;
constexpr int KI = 64;   // individuals per stage
constexpr int KW = 2;    // 32-individual words per stage
constexpr int KP = 32;   // individual pairs per stage

struct __align__(16) Smem {
    float4 u[KP][2][TI];  // [0] = (U0a, U0b, U1a, U1b), [1] = (U2a, U2b, UVa, UVb)
    uint4 pi[KW][TI];     // i-side planes AND phenotype mask
    uint4 pj[KW][TJ];     // j-side planes
    float2 q[KP];         // q of the two individuals of each pair
    long long tile;
};

__device__ __forceinline__ float bitf(uint32_t w, int b) { return ((w >> b) & 1u) ? 1.0f : 0.0f; }
__device__ __forceinline__ float bitsel(uint32_t w, int b, float v) { return ((w >> b) & 1u) ? v : 0.0f; }

__device__ __forceinline__ void count9(uint32_t c[5], const uint4 &p, const uint4 &r)
{
    c[0] += __popc(p.x & r.x) + (__popc(p.x & r.y) << 16);
    c[1] += __popc(p.x & r.z) + (__popc(p.y & r.x) << 16);
    c[2] += __popc(p.y & r.y) + (__popc(p.y & r.z) << 16);
    c[3] += __popc(p.z & r.x) + (__popc(p.z & r.y) << 16);
    c[4] += __popc(p.z & r.z);
}

// Genotype bit-planes of 32 individuals (word w) of one SNP, decoded from the reference's packed
// row (src/readplink.c:1066-1102: MSB-first words, right-aligned tail word).
__device__ __forceinline__ uint4 load_planes(const ScanArgs &a, int snp, int w)
{
    const int npack1 = a.remain ? a.npack + 1 : a.npack;
    const uint32_t *row = reinterpret_cast<const uint32_t *>(a.gpack) + (size_t)snp * npack1;
    uint32_t p0 = 0, p1 = 0, p2 = 0;
#pragma unroll 4
    for (int t = 0; t < 32; ++t) {
        const int k = 32 * w + t;
        uint32_t c = 3u;
        if (k < 16 * a.npack) c = (__ldg(row + (k >> 4)) >> (30 - 2 * (k & 15))) & 3u;
        else if (k < a.nid) c = (__ldg(row + a.npack) >> (2 * (a.remain - 1 - (k - 16 * a.npack)))) & 3u;
        p0 |= (uint32_t)(c == 0u) << t;
        p1 |= (uint32_t)(c == 1u) << t;
        p2 |= (uint32_t)(c == 2u) << t;
    }
    return make_uint4(p0, p1, p2, p0 | p1 | p2);
}

struct PairAcc {
    uint32_t C[5];
    float S[9];
    float Q;
};

// FP64 statistics of one pair from its packed counts, FP32 cell sums and y^2 sum. Kept out of
// line: the kernel's accumulators stay in registers and only this call's arguments go through
// the stack.
__device__ __noinline__ PairStat eval_pair(const ScanArgs &a, const PairAcc acc, double qc)
{
    int n[9];
    double Sd[9];
    int N = 0;
#pragma unroll
    for (int c = 0; c < 9; ++c) {
        n[c] = (int)((acc.C[c >> 1] >> (16 * (c & 1))) & 0xffffu);
        Sd[c] = (double)acc.S[c];
        N += n[c];
    }
    return pair_stat(n, Sd, (double)acc.Q + qc * (double)N, a.test_int != 0);
}

__global__ void __launch_bounds__(NT, 1) k_scan_popc(ScanArgs a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Smem &sm = *reinterpret_cast<Smem *>(smem_raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nstages = a.Wp / KW;
    // maxima of F and F2 per trait: per CTA in shared memory (flushed to global memory once,
    // at the end) up to SMAX_TRAITS traits, else the global maxima directly
    const bool smax_local = a.ntraits <= SMAX_TRAITS;
    unsigned int *smax = reinterpret_cast<unsigned int *>(smem_raw + sizeof(Smem));
    if (smax_local)
        for (int w = tid; w < 2 * a.ntraits; w += NT) smax[w] = 0u;
    unsigned int *const mxf = smax_local ? smax : a.maxf;
    unsigned int *const mxf2 = smax_local ? smax + a.ntraits : a.maxf2;

    for (;;) {
        if (tid == 0) sm.tile = (long long)atomicAdd(&a.counters[1], 1ull);
        __syncthreads();
        const long long tile = sm.tile;
        __syncthreads();
        if (tile >= a.ntiles) break;
        const int b = find_block(a.blocks, a.nblocks, tile);
        const BlockDesc bd = a.blocks[b];
        const long long lt = tile - bd.tile_base;
        const int i0 = (int)(lt / bd.tiles_j) * TI, j0 = (int)(lt % bd.tiles_j) * TJ;
        // no pair with snp1 > snp2 in this tile (upper part of a diagonal block)
        if (bd.start1 + min(i0 + TI, bd.size1) - 1 <= bd.start2 + j0) continue;

        for (int t = 0; t < a.ntraits; ++t) {
            const float *yt = a.y + (size_t)t * a.Np;
            const float *qt = a.q + (size_t)t * a.Np;
            const uint32_t *wt = a.wmask + (size_t)t * a.Wp;
            float S[4][9];
            float Q[4];
            uint32_t C[4][5];
#pragma unroll
            for (int ii = 0; ii < 4; ++ii) {
#pragma unroll
                for (int c = 0; c < 9; ++c) S[ii][c] = 0.0f;
                Q[ii] = 0.0f;
#pragma unroll
                for (int c = 0; c < 5; ++c) C[ii][c] = 0u;
            }

            for (int st = 0; st < nstages; ++st) {
                const int w0 = st * KW, k0 = st * KI;
                __syncthreads();
                {   // i side: thread -> (i, 8 individuals)
                    const int i = tid >> 3, part = tid & 7;
                    const int gi = i0 + i;
                    uint4 P = make_uint4(0, 0, 0, 0);
                    if (gi < bd.size1) P = load_planes(a, bd.start1 + gi, w0 + (part >> 2));
                    const float4 ya = *reinterpret_cast<const float4 *>(yt + k0 + 8 * part);
                    const float4 yb = *reinterpret_cast<const float4 *>(yt + k0 + 8 * part + 4);
                    const float yv[8] = {ya.x, ya.y, ya.z, ya.w, yb.x, yb.y, yb.z, yb.w};
                    const int bit0 = 8 * (part & 3);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int bA = bit0 + 2 * e, bB = bA + 1;
                        const float yA = yv[2 * e], yB = yv[2 * e + 1];
                        sm.u[part * 4 + e][0][i] = make_float4(bitsel(P.x, bA, yA), bitsel(P.x, bB, yB),
                                                               bitsel(P.y, bA, yA), bitsel(P.y, bB, yB));
                        sm.u[part * 4 + e][1][i] = make_float4(bitsel(P.z, bA, yA), bitsel(P.z, bB, yB),
                                                               bitf(P.w, bA), bitf(P.w, bB));
                    }
                }
                if (tid < KW * TI) {
                    const int w = tid / TI, i = tid % TI, gi = i0 + i;
                    uint4 P = make_uint4(0, 0, 0, 0);
                    if (gi < bd.size1) P = load_planes(a, bd.start1 + gi, w0 + w);
                    const uint32_t W = wt[w0 + w];
                    sm.pi[w][i] = make_uint4(P.x & W, P.y & W, P.z & W, 0u);
                } else if (tid < KW * TI + KW * TJ) {
                    const int idx = tid - KW * TI, w = idx / TJ, j = idx % TJ, gj = j0 + j;
                    uint4 P = make_uint4(0, 0, 0, 0);
                    if (gj < bd.size2) P = load_planes(a, bd.start2 + gj, w0 + w);
                    sm.pj[w][j] = P;
                } else if (tid < KW * TI + KW * TJ + KP) {
                    const int kp = tid - KW * TI - KW * TJ;
                    sm.q[kp] = *reinterpret_cast<const float2 *>(qt + k0 + 2 * kp);
                }
                __syncthreads();

#pragma unroll
                for (int w = 0; w < KW; ++w) {
                    const uint4 r = sm.pj[w][lane];
#pragma unroll
                    for (int ii = 0; ii < 4; ++ii) count9(C[ii], sm.pi[w][warp * 4 + ii], r);
                }
#pragma unroll
                for (int w = 0; w < KW; ++w) {
                    // this lane's j-SNP: indicator floats from its plane bits
                    const uint4 r = sm.pj[w][lane];
#pragma unroll 1
                    for (int h = 0; h < 16; ++h) {
                        const int kp = 16 * w + h, bA = 2 * h, bB = bA + 1;
                        const float2 qq = sm.q[kp];
                        const float F[3][2] = {{bitf(r.x, bA), bitf(r.x, bB)},
                                               {bitf(r.y, bA), bitf(r.y, bB)},
                                               {bitf(r.z, bA), bitf(r.z, bB)}};
                        const float FQa = bitsel(r.w, bA, qq.x), FQb = bitsel(r.w, bB, qq.y);
#pragma unroll
                        for (int ii = 0; ii < 4; ++ii) {
                            const float4 ua = sm.u[kp][0][warp * 4 + ii], ub = sm.u[kp][1][warp * 4 + ii];
                            const float U[3][2] = {{ua.x, ua.y}, {ua.z, ua.w}, {ub.x, ub.y}};
#pragma unroll
                            for (int x = 0; x < 3; ++x)
#pragma unroll
                                for (int y = 0; y < 3; ++y) {
                                    S[ii][3 * x + y] = fmaf(U[x][0], F[y][0], S[ii][3 * x + y]);
                                    S[ii][3 * x + y] = fmaf(U[x][1], F[y][1], S[ii][3 * x + y]);
                                }
                            Q[ii] = fmaf(ub.z, FQa, Q[ii]);
                            Q[ii] = fmaf(ub.w, FQb, Q[ii]);
                        }
                    }
                }
            }

            // epilogue
            const double qc = a.qc[t];
            const bool report = a.report_trait < 0 || a.report_trait == t;
#pragma unroll
            for (int ii = 0; ii < 4; ++ii) {
                const int gi = i0 + warp * 4 + ii, gj = j0 + lane;
                const bool valid = gi < bd.size1 && gj < bd.size2 && (bd.start1 + gi > bd.start2 + gj);
                PairStat s;
                s.nfac = s.d1 = s.d2 = 0;
                s.F = s.F2 = 0.0;
                if (valid) {
                    PairAcc acc;
#pragma unroll
                    for (int c = 0; c < 5; ++c) acc.C[c] = C[ii][c];
#pragma unroll
                    for (int c = 0; c < 9; ++c) acc.S[c] = S[ii][c];
                    acc.Q = Q[ii];
                    s = eval_pair(a, acc, qc);
                }
                const bool hit = valid && report && is_hit(a, s);
                emit_row(a, hit, bd.start1 + gi, bd.start2 + gj, s);
                fold_max(&mxf[t], valid, s.F);
                if (a.test_int) fold_max(&mxf2[t], valid, s.F2);
            }
        }
    }
    __syncthreads();
    if (smax_local)
        for (int w = tid; w < 2 * a.ntraits; w += NT)
            if (smax[w]) atomicMax(w < a.ntraits ? &a.maxf[w] : &a.maxf2[w - a.ntraits], smax[w]);
}

}  // namespace popc_raw

}  // namespace epi

// ---------------------------------------------------------------------------------------
// Allocation-free entry point (epi_scan_block_noalloc).
//
// Some callers cannot allocate GPU memory: code that must not call cudaMalloc while it runs
// (a latency-critical service or a real-time loop after start-up), or a host framework
// that hands out device memory only from its own pool. They pass device buffers for every
// input and output, and the scan's working memory -- counters, the block descriptor, the
// maxima, and what either way keeps of the phenotype -- lives in the fixed array below, sized
// for at most EPI_NOALLOC_MAX_NID individuals (about 520 KiB, held by every GPU that loads the
// library until the process exits).
// ---------------------------------------------------------------------------------------
namespace epi {
cudaError_t launch_traits(const float *yraw, const uint8_t *valid, int mode, int nid, int Np, int ntraits,
                          const TraitArrays &o, TraitInfo *info, cudaStream_t stream);
cudaError_t exact_enqueue(const ScanArgs &a, int sm_count, cudaStream_t stream);
cudaError_t mma_raw_prepare(int grid_request, int *grid);
cudaError_t mma_raw_enqueue(const ScanArgs &a, int grid, cudaStream_t stream);
int mma_tile_i();
int mma_tile_j(int screen);
int mma_screen_max_nid();

namespace noalloc {

constexpr int NP_MAX = 65536;        // individuals, padded to a multiple of 128
constexpr int NP_SCREEN_MAX = 32768; // of the screen (mma_screen_max_nid is a little below)

// What both ways keep; the counters' overflow flag ends the screen.
struct Head {
    unsigned long long counters[NCOUNTERS];
    unsigned int maxf[2], lowf[2];  // order-encoded max F and max F2; the screen's lower bounds of them
    double qc;                      // mean of the centred phenotype's square (plain kernel)
    BlockDesc block;
};

struct Scratch {  // plain kernel
    Head h;
    alignas(16) float y[NP_MAX];     // centred phenotype (0 where missing)
    alignas(16) float q[NP_MAX];     // y^2 - qc (0 where missing)
    uint32_t wmask[NP_MAX / 32];     // phenotype-valid bits
};

struct ScreenScratch {  // screen: layouts as in epi_internal.cuh, one trait, one part of the block
    Head h;
    TraitInfo info;
    double ysq, qtot, yscale[3];
    alignas(16) float4 tscr[2];
    uint32_t wmask[NP_SCREEN_MAX / 32];
    alignas(16) int8_t ydig[5 * NP_SCREEN_MAX];
    // per SNP of the part, i side then j side
    double qm[2 * RAW_SNPS], sm[2 * RAW_SNPS], nm[2 * RAW_SNPS];
    float qmf[2 * RAW_SNPS];
    Cand cand[RAW_CAND];
};
static_assert(sizeof(ScreenScratch) <= sizeof(Scratch), "both ways share the array");
// read in words of 16 bytes (k_scan_popc: y, q; the screen: tscr, ydig)
static_assert(offsetof(Scratch, y) % 16 == 0 && offsetof(Scratch, q) % 16 == 0 && offsetof(ScreenScratch, tscr) % 16 == 0 &&
                  offsetof(ScreenScratch, ydig) % 16 == 0,
              "alignment");

// The scratch: one copy per device, shared by every call on that device. In host code this
// name only stands for the array; the device address comes from cudaGetSymbolAddress.
static __device__ __align__(256) unsigned char g_scratch[sizeof(Scratch)];

__device__ __forceinline__ void block_sum(double &v, long long &n, double *sv, long long *sn)
{
    for (int o = 16; o > 0; o >>= 1) {
        v += __shfl_xor_sync(0xffffffffu, v, o);
        n += __shfl_xor_sync(0xffffffffu, n, o);
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) {
        sv[w] = v;
        sn[w] = n;
    }
    __syncthreads();
    v = 0.0;
    n = 0;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) {
        v += sv[i];
        n += sn[i];
    }
}

__device__ __forceinline__ double block_max(double v, double *sv)
{
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) sv[w] = v;
    __syncthreads();
    v = 0.0;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) v = fmax(v, sv[i]);
    return v;
}

// One block: resets the counters and maxima (every call starts from zero), writes the block
// descriptor, then the centred phenotype as k_traits (prep.cu) makes it for epi_set_traits:
// centred by the valid mean and scaled by the power of two that brings its largest magnitude
// into [0.5, 1) (exact, so F and F2 are unchanged, and a trait in units of 1e20 or 1e-20
// neither overflows nor underflows the single-precision squares).
__global__ void __launch_bounds__(1024) k_prep(Scratch *s, const float *__restrict__ phen, int nid, int Np, int Wp,
                                               int safe, BlockDesc bd)
{
    __shared__ double sv[32];
    __shared__ long long sn[32];
    const int tid = threadIdx.x;
    if (tid < 4) s->h.counters[tid] = 0ull;
    if (tid < 2) s->h.maxf[tid] = ENC_NEG_INF;
    if (tid == 0) s->h.block = bd;
    double sum = 0.0;
    long long n = 0;
    for (int k = tid; k < nid; k += blockDim.x) {
        const float y = phen[k];
        if (safe || y != -9.0f) {
            sum += (double)y;
            ++n;
        }
    }
    block_sum(sum, n, sv, sn);
    const double mu = n ? sum / (double)n : 0.0;
    double mx = 0.0;
    for (int k = tid; k < nid; k += blockDim.x) {
        const float y = phen[k];
        if (safe || y != -9.0f) mx = fmax(mx, fabs((double)y - mu));
    }
    const double maxabs = block_max(mx, sv);
    const double p2 = (maxabs > 0.0 && isfinite(maxabs)) ? ldexp(1.0, -(ilogb(maxabs) + 1)) : 1.0;
    double s2 = 0.0;
    long long dummy = 0;
    for (int k = tid; k < Np; k += blockDim.x) {
        const float y = k < nid ? phen[k] : -9.0f;
        const bool ok = k < nid && (safe || y != -9.0f);
        const float yc = ok ? (float)(((double)y - mu) * p2) : 0.0f;
        s->y[k] = yc;
        if (ok) s2 += (double)yc * (double)yc;
    }
    block_sum(s2, dummy, sv, sn);
    const double c = n ? s2 / (double)n : 0.0;
    if (tid == 0) s->h.qc = c;
    for (int k = tid; k < Np; k += blockDim.x) {
        const float y = k < nid ? phen[k] : -9.0f;
        const bool ok = k < nid && (safe || y != -9.0f);
        const double yc = s->y[k];
        s->q[k] = ok ? (float)(yc * yc - c) : 0.0f;
    }
    for (int w = tid; w < Wp; w += blockDim.x) {
        uint32_t bits = 0;
        for (int t = 0; t < 32; ++t) {
            const int k = 32 * w + t;
            if (k < nid && (safe || phen[k] != -9.0f)) bits |= 1u << t;
        }
        s->wmask[w] = bits;
    }
}

__global__ void k_finish(const Head *s, int64_t *nhits, float *maxf, int test_int)
{
    if (threadIdx.x != 0) return;
    *nhits = (int64_t)s->counters[0];
    if (maxf) {
        maxf[0] = ord2f(s->maxf[0]);
        maxf[1] = test_int ? ord2f(s->maxf[1]) : 0.0f;
    }
}

// The candidates expected of the first part of a block, and of the largest of the others: their pairs and
// the roots of the largest draws that the screen's lower bounds come from. In the first part these are
// R below the draws (screen_rule.cuh); from the second on k_exact has put them at the first part's own
// largest F.
struct PartSizes {
    double first, others, top8[2], top4[2];
};
__host__ __device__ inline double fullest_list(const PartSizes &p, int want_int, double t1, double t2, double r, double nv)
{
    double n[2];
    for (int k = 0; k < 2; ++k) {
        double share = screen_share_of(t1, true, 8, p.top8[k] + k * r, r, nv);
        if (want_int) share += screen_share_of(t2, true, 4, p.top4[k] + k * r, r, nv);
        n[k] = share * (k ? p.others : p.first);
    }
    return (n[0] > n[1] ? n[0] : n[1]) / RAW_CAND;
}

// Start of a pass over the parts: counters and maxima reset, and the overflow flag set, so that the
// parts' kernels return at once, where the lists are expected to be fuller than `most` (R = E / sigma
// is known on the device only). A candidate takes about as long as 110 pairs of the screen, the plain
// kernel 20 to 40 times as long as the screen: no share that the lists hold is too large.
__global__ void k_begin(ScreenScratch *s, int fresh, int want_int, float t1, float t2, PartSizes p, double most)
{
    const int tid = threadIdx.x;
    if (tid < NCOUNTERS) s->h.counters[tid] = 0ull;
    if (tid < 2) {
        s->h.maxf[tid] = ENC_NEG_INF;
        if (fresh) s->h.lowf[tid] = ENC_NEG_INF;  // (a pass that was given up has left bounds that hold)
    }
    __syncthreads();
    if (tid != 0) return;
    const double r = s->info.r1;
    if (!(isfinite(r) && fullest_list(p, want_int, t1, t2, r, s->info.nv) <= most)) s->h.counters[CNT_OVERFLOW] = 1ull;
}

// Start of a part of the block: its descriptor, an empty candidate list, and per SNP of either
// side, one warp each, the sums over the individuals missing at it (as k_qmiss, prep.cu) from the
// packed words and the digits.
__global__ void k_part(ScreenScratch *s, BlockDesc bd, const int32_t *__restrict__ gpack, int nid, int npack, int remain,
                       int Np)
{
    if (s->h.counters[CNT_OVERFLOW]) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        s->h.block = bd;
        s->h.counters[CNT_CAND] = 0ull;
    }
    const int q = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (q >= bd.size1 + bd.size2) return;
    const int snp = q < bd.size1 ? bd.start1 + q : bd.start2 + q - bd.size1;
    const uint32_t *row = reinterpret_cast<const uint32_t *>(gpack) + (size_t)snp * (npack + (remain > 0));
    const int8_t *dg = s->ydig;
    const double unit = s->yscale[0];
    double x = 0.0, r = 0.0;
    int cnt = 0;
    for (int w = lane; 16 * w < nid; w += 32) {
        const uint32_t v = packed_word(row, w, npack, remain);
        uint32_t m = v & (v >> 1) & 0x55555555u;
        while (m) {
            const int k = 16 * w + 15 - ((31 - __clz(m)) >> 1);
            m &= ~(0x80000000u >> __clz(m));
            if (k < nid && dg[Np + k]) {
                const int Y = dg[4 * Np + k] + 256 * dg[3 * Np + k] + 65536 * dg[2 * Np + k];
                const double yq = (double)Y * unit;
                x += yq * yq;
                r += (double)Y;
                ++cnt;
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        x += __shfl_xor_sync(0xffffffffu, x, o);
        r += __shfl_xor_sync(0xffffffffu, r, o);
    }
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (lane == 0) {
        const int o = q < bd.size1 ? q : RAW_SNPS + q - bd.size1;
        s->qm[o] = x;
        s->sm[o] = r;
        s->nm[o] = (double)cnt;
        s->qmf[o] = (float)x;
    }
}

constexpr int MAX_DEVICES = 64;
static int g_sms[MAX_DEVICES];  // per device: SM count, 0 until the device's set-up ran

}  // namespace noalloc
}  // namespace epi

extern "C" epi_status epi_scan_block_noalloc(const int32_t *d_gpack, int32_t nid, int32_t nsnp, const float *d_phen,
                                             const epi_block *block, const epi_scan_opts *opts, epi_hit *d_hits,
                                             int64_t cap, int64_t *d_nhits, float *d_maxf, void *stream)
{
    using namespace epi;
    if (!d_gpack || !d_phen || !block || !opts || !d_nhits || cap < 0 || (cap > 0 && !d_hits) || nsnp < 1 || nid < 1)
        return EPI_E_INVALID;
    if (nid > EPI_NOALLOC_MAX_NID) return EPI_E_UNSUPPORTED;  // beyond the fixed scratch
    if ((opts->test != 'f' && opts->test != 'i') || (opts->safe != 0 && opts->safe != 1)) return EPI_E_INVALID;
    if (block->start1 < 0 || block->start2 < 0 || block->size1 < 0 || block->size2 < 0 ||
        (int64_t)block->start1 + block->size1 > nsnp || (int64_t)block->start2 + block->size2 > nsnp)
        return EPI_E_INVALID;
    // an error left pending by the caller's earlier work is theirs: report it, do not clear it
    if (cudaPeekAtLastError() != cudaSuccess) return EPI_E_CUDA;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= noalloc::MAX_DEVICES) return EPI_E_NODEVICE;
    cudaStream_t st = (cudaStream_t)stream;
    const size_t smem = sizeof(popc_raw::Smem) + 8;  // + per-CTA maxima of one trait
    int screen_grid = 0;  // the screen's kernel: its attribute and launch shape (a look-up after the first call)

    // set-up, once per device with that device current: the device check, the SM count and
    // the kernel's shared-memory attribute
    if (noalloc::g_sms[dev] == 0) {
        int major = 0, sms = 0;
        if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev) != cudaSuccess || major != 10)
            return EPI_E_NODEVICE;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1)
            return EPI_E_CUDA;
        if (cudaFuncSetAttribute(popc_raw::k_scan_popc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
            cudaSuccess)
            return EPI_E_CUDA;
        noalloc::g_sms[dev] = sms;
    }
    if (mma_raw_prepare(noalloc::g_sms[dev], &screen_grid) != cudaSuccess) return EPI_E_CUDA;
    // The scratch array's device address. In host code g_scratch only stands for the array;
    // the address comes from the runtime, for the current device. It is looked up on every
    // call (a host-side table lookup once the module is loaded), so that a device reset
    // between calls, which reloads the module, cannot leave a stale address behind.
    void *ptr = nullptr;
    if (cudaGetSymbolAddress(&ptr, noalloc::g_scratch) != cudaSuccess || ptr == nullptr) return EPI_E_CUDA;
    noalloc::Scratch *scr = (noalloc::Scratch *)ptr;
    noalloc::ScreenScratch *ss = (noalloc::ScreenScratch *)ptr;

    const int Wp = ((nid + 31) / 32 + 3) / 4 * 4;
    const int Np = 32 * Wp;
    BlockDesc bd;
    bd.start1 = block->start1;
    bd.size1 = block->size1;
    bd.start2 = block->start2;
    bd.size2 = block->size2;
    bd.tiles_i = (block->size1 + popc_raw::TI - 1) / popc_raw::TI;
    bd.tiles_j = (block->size2 + popc_raw::TJ - 1) / popc_raw::TJ;
    bd.tile_base = 0;
    const long long ntiles = (long long)bd.tiles_i * bd.tiles_j;

    ScanArgs a;
    memset(&a, 0, sizeof(a));
    a.gpack = d_gpack;
    a.npack = nid / 16;
    a.remain = nid % 16;
    a.nid = nid;
    a.nsnp = nsnp;
    a.Wp = Wp;
    a.Np = Np;
    a.y = scr->y;
    a.q = scr->q;
    a.wmask = scr->wmask;
    a.qc = &scr->h.qc;
    a.ntraits = 1;
    a.blocks = &scr->h.block;
    a.nblocks = 1;
    a.ntiles = ntiles;
    a.test_int = opts->test == 'i';
    a.safe = opts->safe;
    a.report_trait = 0;
    a.t1 = opts->t1;
    a.t2 = opts->t2;
    a.rows = reinterpret_cast<HitRow *>(d_hits);
    a.cap = cap;
    a.counters = scr->h.counters;
    a.maxf = &scr->h.maxf[0];
    a.maxf2 = &scr->h.maxf[1];

    // hits, maxima and the end of the scan; the counters come to the host
    unsigned long long state[CNT_OVERFLOW + 1] = {0ull};  // hits, tile queue, error flag and site, overflow flag
    cudaError_t e = cudaSuccess;
    const auto finish = [&]() -> epi_status {
        noalloc::k_finish<<<1, 32, 0, st>>>(&scr->h, d_nhits, d_maxf, a.test_int);
        if (cudaGetLastError() != cudaSuccess || e != cudaSuccess) return EPI_E_CUDA;
        if (cudaMemcpyAsync(state, scr->h.counters, sizeof(state), cudaMemcpyDeviceToHost, st) != cudaSuccess)
            return EPI_E_CUDA;
        if (cudaStreamSynchronize(st) != cudaSuccess) return EPI_E_CUDA;
        return state[2] != 0 ? EPI_E_TIMEOUT : EPI_OK;
    };

    // The screen, in one of two passes over parts of the block: the first `head` SNPs of either side, then
    // 3,072 at a time.
    //   first pass   head = 3,072: while the lists are expected to be at most three times full. The
    //                expectation holds for unassociated SNPs; effects of 1% lift the bounds and leave a
    //                fifth of it
    //   second pass  after the first has run over: a head so small that its list should hold what its first
    //                wave of tiles (2.5e5 pairs) lets through, for a normal trait that reaches 4.2 standard
    //                deviations (R = 0.0097 sqrt(N)); the parts after it go by its largest F. Not where the
    //                first pass's lists should have been a quarter full: what ran over then (linkage)
    //                runs over again.
    // 8,000 individuals x 3,000 SNPs, 8 df, p = 1e-6, no effects: the first pass runs over at 9,400 candidates,
    // the second's parts have 4,700 and 600; without it the plain kernel took 38.7 ms.
    bool done = false;
    const bool screen = ntiles > 0 && Np <= mma_screen_max_nid();
    int heads[2] = {RAW_SNPS, RAW_SNPS};
    noalloc::PartSizes sizes[2];
    const double most[2] = {3.0, 0.9}, usual = 0.0097 * std::sqrt((double)nid);
    const auto fullest = [&](const noalloc::PartSizes &s, double r) {
        return noalloc::fullest_list(s, a.test_int, a.t1, a.t2, r, nid);
    };
    const auto sizes_of = [&](int head, double wave) {
        const auto pairs = [&](int i, int ni, int j, int nj) {
            return (double)pairs_below(bd.start1 + i, std::max(0, std::min(ni, bd.size1 - i)), bd.start2 + j,
                                       std::max(0, std::min(nj, bd.size2 - j)));
        };
        noalloc::PartSizes s;
        s.first = pairs(0, head, 0, head);
        s.others = std::max(std::max(pairs(head, RAW_SNPS, 0, head), pairs(0, head, head, RAW_SNPS)),
                            pairs(head, RAW_SNPS, head, RAW_SNPS));
        const double drawn[2] = {std::min(wave, s.first), s.first};
        for (int k = 0; k < 2; ++k) {
            s.top8[k] = chi_top(drawn[k], 8);
            s.top4[k] = chi_top(drawn[k], 4);
        }
        return s;
    };
    if (screen) {
        const TraitArrays out = {nullptr, ss->wmask, ss->ydig, nullptr, &ss->ysq, &ss->qtot, ss->yscale, ss->tscr};
        e = launch_traits(d_phen, nullptr, opts->safe ? VALID_ALL : VALID_NOT9, nid, Np, 1, out, &ss->info, st);
        sizes[0] = sizes_of(RAW_SNPS, 1e300);
    }
    bool fresh = true;  // no bounds of an earlier pass yet
    for (int pass = 0; screen && pass < 2 && !done; ++pass) {
        if (pass == 1) {
            if (fullest(sizes_of(RAW_SNPS, 2.5e5), usual) < 0.25) break;
            do {
                heads[1] = heads[1] * 3 / 4;
                sizes[1] = sizes_of(heads[1], 2.5e5);
            } while (fullest(sizes[1], usual) > 0.7 && heads[1] > 600);
        }
        if (fullest(sizes[pass], 0.0) > most[pass]) continue;  // too full for any trait
        noalloc::k_begin<<<1, 32, 0, st>>>(ss, fresh, a.test_int, a.t1, a.t2, sizes[pass], most[pass]);
        fresh = false;
        ScanArgs p = a;
        p.wmask = ss->wmask;
        p.ydig = ss->ydig;
        p.tscr = ss->tscr;
        p.yscale = ss->yscale;
        p.ytot = ss->yscale + 1;
        p.nvalid = ss->yscale + 2;
        p.qtot = &ss->qtot;
        p.qm = ss->qm;
        p.sm = ss->sm;
        p.nm = ss->nm;
        p.lowf = &ss->h.lowf[0];
        p.lowf2 = &ss->h.lowf[1];
        p.cand = ss->cand;
        p.cand_cap = RAW_CAND;
        p.wait_ns = opts->wait_limit_ms > 0 ? (unsigned long long)opts->wait_limit_ms * 1000000ull : 2000000000ull;
        p.debug_stall = opts->debug == EPI_DEBUG_STALL;
        p.xsi = 1;
        p.xsj = 1 << 30;
        p.seg1 = {1, 0, 0};
        const int TI = mma_tile_i(), TJ = mma_tile_j(1);
        const int head = heads[pass];
        for (int i = 0, ni = head; i < bd.size1; i += ni, ni = RAW_SNPS)
            for (int j = 0, nj = head; j < bd.size2; j += nj, nj = RAW_SNPS) {
                BlockDesc d;
                d.start1 = bd.start1 + i;
                d.size1 = std::min(ni, bd.size1 - i);
                d.start2 = bd.start2 + j;
                d.size2 = std::min(nj, bd.size2 - j);
                d.tiles_i = (d.size1 + TI - 1) / TI;
                d.tiles_j = (d.size2 + TJ - 1) / TJ;
                d.tile_base = 0;
                p.seg_units = 0;  // tiles that hold a pair (scan_mma.cu: Walker)
                for (int ti = 0; ti < d.tiles_i; ++ti) {
                    const long long end = (long long)d.start1 + ((ti + 1) * TI < d.size1 ? (ti + 1) * TI : d.size1);
                    const long long x = end - 1 - d.start2, n = x <= 0 ? 0 : (x + TJ - 1) / TJ;
                    p.seg_units += n < d.tiles_j ? n : d.tiles_j;
                }
                if (p.seg_units == 0) continue;  // no pair with snp1 > snp2
                // the per-SNP sums, indexed by SNP
                p.qmf = (const float *)((uintptr_t)ss->qmf - sizeof(float) * (uintptr_t)d.start1);
                p.qmf_j = (const float *)((uintptr_t)(ss->qmf + RAW_SNPS) - sizeof(float) * (uintptr_t)d.start2);
                const unsigned snps = (unsigned)(d.size1 + d.size2);
                noalloc::k_part<<<(snps + 7) / 8, 256, 0, st>>>(ss, d, d_gpack, nid, a.npack, a.remain, Np);
                const long long want = 2 * p.seg_units;
                if (e == cudaSuccess) e = mma_raw_enqueue(p, (int)(want < screen_grid ? want : screen_grid), st);
                if (e == cudaSuccess) e = exact_enqueue(p, noalloc::g_sms[dev], st);
            }
        const epi_status s = finish();
        if (s != EPI_OK) return s;
        done = state[CNT_OVERFLOW] == 0ull;
    }
    if (!done) {
        // the plain kernel
        noalloc::k_prep<<<1, 1024, 0, st>>>(scr, d_phen, nid, Np, Wp, opts->safe, bd);
        if (ntiles > 0) {
            const int grid = (int)(ntiles < noalloc::g_sms[dev] ? ntiles : noalloc::g_sms[dev]);
            popc_raw::k_scan_popc<<<grid, popc_raw::NT, smem, st>>>(a);
        }
        const epi_status s = finish();
        if (s != EPI_OK) return s;
    }
    const unsigned long long found = state[0];
    // as epi_scan: more hits than `cap` is reported (the first `cap` rows are written, and
    // *d_nhits holds the total)
    return (int64_t)found > cap ? EPI_E_OVERFLOW : EPI_OK;
}
