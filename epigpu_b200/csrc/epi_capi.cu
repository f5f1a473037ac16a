// epi_capi.cu -- the C ABI of libepigpu.so (include/epigpu.h).
//
// Host side of the scan: device selection, genotype and trait upload, the tile schedule
// over chromosome blocks, kernel dispatch (plain popcount form / tcgen05 tensor form),
// hit readback and ordering. It replaces the OpenCL host code of perform_scan
// (src/EpiOpenCL.c:1383-1627); the results file itself is written by the C host
// (epigpu_b200/host/scan_driver.c).
#include "epigpu.h"
#include "epi_internal.cuh"
#include "screen_rule.cuh"

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <numeric>
#include <string>
#include <vector>

namespace epi {
cudaError_t launch_unpack(const int32_t *raw, int nsnp, int nid, int npack, int remain, uint4 *planes, int Wp,
                          uint32_t *codes, int Wc, uint8_t *hcodes, uint8_t *h3, uint32_t *missbits,
                          cudaStream_t stream);
cudaError_t launch_qmiss(const uint32_t *missbits, int nsnp, int Wp, const uint32_t *wmask, const double *qd,
                        const double *qr, int Np, int ntraits, double *qm, double *rm, double *nm,
                        float *qmf, cudaStream_t stream);
cudaError_t launch_traits(const float *yraw, const uint8_t *valid, int mode, int nid, int Np, int ntraits,
                          const TraitArrays &o, TraitInfo *info, cudaStream_t stream);
cudaError_t launch_major(const uint4 *planes, int nsnp, int Wp, uint8_t *maj, cudaStream_t stream);
cudaError_t launch_marg(const uint4 *planes, int nsnp, int Wp, const float *y, const uint32_t *wmask, int Np,
                        int ntraits, double *pmC, int32_t *pmN, double *pmQ, cudaStream_t stream);
// plain form (scan_popc.cu)
int popc_shapes();
void popc_shape(int v, int *ti, int *tj, const char **desc);
cudaError_t popc_prepare(int v);
cudaError_t popc_enqueue(int v, const ScanArgs &a, const PopcMaps &maps, int grid, cudaStream_t stream);
cudaError_t popc_encode_planes(int v, PopcMaps *maps, const uint4 *planes, int nsnp, int Wp);
// tensor form (scan_mma.cu)
bool mma_available();
int mma_tile_i();
int mma_tile_j(int screen);
int mma_x_rows(int screen);
int mma_x_sets(int screen, int ntraits);
int mma_min_nid();
int mma_max_nid();
int mma_screen_max_nid();
int mma_shapes();
void mma_shape(int v, int screen, const char **desc);
cudaError_t mma_prepare(int v, int screen, int ntraits, int grid_request, int *grid);
cudaError_t mma_enqueue(int v, int screen, const ScanArgs &a, const MmaMaps &maps, int grid,
                        cudaStream_t stream);
cudaError_t exact_enqueue(const ScanArgs &a, int sm_count, cudaStream_t stream);
cudaError_t mma_encode_genotypes(MmaMaps *maps, const uint8_t *hcodes, const uint8_t *h3, int nsnp, int Np);
cudaError_t mma_encode_traits(MmaMaps *maps, const int8_t *ydig, int ntraits, int Np);
cudaError_t mma_encode_x(MmaMaps *maps, const int8_t *x, int nsnp, int Np, int ntraits, int screen);
bool mma_needs_x(int v, int screen);
cudaError_t launch_expand(const uint8_t *hcodes, const int8_t *ydig, int nsnp, int Np, int ntraits, int screen,
                          int8_t *x, cudaStream_t stream);
// Counters to zero, the per-trait maxima of F and F2 and the screen's lower bounds of them to the
// order-encoded -inf: before the first scan of a context, and after its number of traits changed.
__global__ void k_scan_init(unsigned long long *counters, unsigned int *maxf, int n)
{
    if (threadIdx.x < NCOUNTERS) counters[threadIdx.x] = 0ull;
    for (int i = threadIdx.x; i < n; i += blockDim.x) maxf[i] = ENC_NEG_INF;
}

// End of a scan, one block: the counters, the maxima and the first FINISH_HITS hits written
// straight into pinned host memory, then the counters and maxima reset for the next scan. Against
// a reset kernel before the scan, two copies after it and a third, with a second
// synchronisation, for the hits, a small scan's call is 15 us shorter (N = 500 x 2,000 SNPs).
constexpr int FINISH_HITS = 4096;
__global__ void __launch_bounds__(256) k_finish(unsigned long long *counters, unsigned int *maxf, int ntraits,
                                                const DevHit *__restrict__ hits, long long cap,
                                                unsigned long long *out_counters, DevHit *out_hits)
{
    static_assert(sizeof(DevHit) == 2 * sizeof(uint4), "copied in two words of 16 bytes");
    const unsigned long long found = counters[0];
    const int n = (int)min(min(found, (unsigned long long)cap), (unsigned long long)FINISH_HITS);
    for (int i = threadIdx.x; i < 2 * n; i += blockDim.x)
        reinterpret_cast<uint4 *>(out_hits)[i] = reinterpret_cast<const uint4 *>(hits)[i];
    unsigned int *const out_max = reinterpret_cast<unsigned int *>(out_counters + NCOUNTERS);
    for (int i = threadIdx.x; i < 4 * ntraits; i += blockDim.x) {
        if (i < 2 * ntraits) out_max[i] = maxf[i];
        maxf[i] = ENC_NEG_INF;
    }
    __syncthreads();  // counters[0] read by every thread
    if (threadIdx.x < NCOUNTERS) {
        out_counters[threadIdx.x] = counters[threadIdx.x];
        counters[threadIdx.x] = 0ull;
    }
}
}  // namespace epi

using epi::BlockDesc;
using epi::DevHit;

// The last screened scan whose candidates ran over their list (genotypes in linkage around a strong
// effect; the share expected of unassociated ones does not foresee it). No scan that asks for as much
// or more is screened again while the same genotypes and traits are loaded, nor, since the next trait of
// a panel is likely to be such another, for the next 1, 2, 4 .. 64 changes of them: a loop over such
// traits then spends under a twentieth of its time on screens that come to nothing, where each one's
// screen cost up to half as much again as the scan with all digits.
struct Overrun {
    bool on = false, changed = false, want_int = false;
    int report = 0, left = 0, next = 1;  // changes that it still holds for, and the next time
    float t1 = 0.0f, t2 = 0.0f;
    double tests = 0.0;

    // before a scan
    void begin()
    {
        if (changed && left-- == 0) on = false;
        if (!on) left = 0;
        changed = false;
    }
    void record(const epi_scan_opts *o, double tests_)
    {
        if (!on) {
            left = next;
            next = std::min(2 * next, 64);
        }
        on = true;
        want_int = o->test == 'i';
        report = o->report_trait;
        t1 = o->t1;
        t2 = o->t2;
        tests = tests_;
    }
    // as many tests or more, for the same trait or all, at the same or lower thresholds of the tests made
    bool as_hard(const epi_scan_opts *o, double tests_) const
    {
        return tests_ >= tests && (o->report_trait == report || o->report_trait < 0) && o->t1 <= t1 &&
               (!want_int || (o->test == 'i' && o->t2 <= t2));
    }
    bool covers(const epi_scan_opts *o, double tests_) const { return on && as_hard(o, tests_); }
    // after a screened scan whose list held
    void held(const epi_scan_opts *o, double tests_)
    {
        if (as_hard(o, tests_)) next = 1;
    }
};

struct epi_ctx {
    int device = -1;
    int sm_count = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    // genotypes
    int nid = 0, nsnp = 0, npack = 0, remain = 0;
    int Wp = 0, Wc = 0, Np = 0;
    int32_t *d_raw = nullptr;
    size_t raw_cap = 0;
    uint4 *d_planes = nullptr;
    uint8_t *d_hcodes = nullptr, *d_h3 = nullptr;
    uint32_t *d_missbits = nullptr;
    uint8_t *d_maj = nullptr;
    size_t planes_cap = 0, hcodes_cap = 0, h3_cap = 0, missbits_cap = 0, maj_cap = 0;
    epi::PopcMaps pmaps;
    // traits
    int ntraits = 0, traits_nid = 0;
    float *d_y = nullptr, *d_yraw = nullptr;  // centred, and as given
    uint8_t *d_yvalid = nullptr;
    uint32_t *d_wmask = nullptr;
    double *d_yscale = nullptr, *d_qd = nullptr, *d_qtot = nullptr, *d_qm = nullptr;
    int8_t *d_ydig = nullptr;
    size_t y_cap = 0, yraw_cap = 0, yvalid_cap = 0, ydig_cap = 0, qd_cap = 0, qm_cap = 0, wmask_cap = 0, qtot_cap = 0,
           yscale_cap = 0;
    bool qm_valid = false;
    epi::MmaMaps maps;
    // tensor form, streamed-B variant: the expanded B rows of every SNP and trait (12 bytes per
    // SNP, individual and trait), built on first use after each genotype or trait load
    int8_t *d_x = nullptr;  // (own_x below)
    size_t x_cap = 0;
    int x_valid = -1;  // -1: none, 0: of all digits, 1, 2: of the screen with that many digits
    // screened scan: constants per trait and per (trait, SNP), the candidate list; per trait
    // E / sigma of either screen and the number of valid individuals (pinned, written by k_traits;
    // screen_digits)
    float4 *d_tscr = nullptr;
    epi::Cand *d_cand = nullptr;
    size_t tscr_cap = 0, cand_cap = 0;
    epi::TraitInfo *h_info = nullptr;
    int h_info_cap = 0;
    Overrun overrun;
    // plain form: marginals per (trait, SNP) and the sum of y^2 per trait
    double *d_pmC = nullptr, *d_pmQ = nullptr, *d_ysq = nullptr;
    int32_t *d_pmN = nullptr;
    size_t pmC_cap = 0, pmQ_cap = 0, pmN_cap = 0, ysq_cap = 0;
    bool pm_valid = false;
    // scan scratch. The first scan of a context takes one allocation (d_slab) for its hits, its
    // candidates and, up to 256 MB, its expanded B rows: a cudaMalloc of a megabyte or more costs
    // about 0.35 ms, as much as a small scan's whole pass. What outgrows its part of it gets
    // memory of its own (own_*).
    void *d_slab = nullptr;
    bool own_hits = false, own_cand = false, own_x = false;
    DevHit *d_hits = nullptr;
    int64_t hit_cap = 0;
    unsigned long long *d_counters = nullptr;
    unsigned int *d_maxf = nullptr;
    int maxf_cap = 0;
    BlockDesc *d_blocks = nullptr;
    int blocks_cap = 0;
    // pinned host staging of the device part of a scan (parts of h_arena where they fit): the block schedule it uploads, the
    // counters and maxima it reads back
    BlockDesc *h_blocks = nullptr;
    int h_blocks_cap = 0;
    unsigned char *h_arena = nullptr;
    DevHit *h_hits = nullptr;  // its last part: the first hits of a scan, written by k_finish
    // what the device holds: counters and maxima as k_finish leaves them for this many traits (0: to
    // be initialised), and the block schedule
    int clean_traits = 0;
    std::vector<BlockDesc> dev_blocks;
    unsigned long long *h_state = nullptr;  // the counters, then 2 x ntraits encoded maxima
    size_t h_state_cap = 0;
    // the device part of the last scan, captured as a CUDA graph, and what it was captured for
    cudaGraphExec_t gexec = nullptr;
    std::vector<unsigned char> gkey;
    // last scan
    double last_ms = 0.0;
    int64_t last_pairs = 0;
    int last_launches = 0;
    int last_form = 0;
    std::string last_config;  // form, kernel variant and how it was chosen
    std::string err;
};

static epi_status set_err(epi_ctx *ctx, epi_status s, const char *fmt, ...)
{
    if (ctx) {
        char buf[1024];
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(buf, sizeof(buf), fmt, ap);
        va_end(ap);
        ctx->err = buf;
    }
    return s;
}

#define CK(call)                                                                                      \
    do {                                                                                              \
        cudaError_t e_ = (call);                                                                      \
        if (e_ != cudaSuccess) {                                                                      \
            cudaGetLastError(); /* a failed call must not surface again at the next launch check */  \
            return set_err(ctx, e_ == cudaErrorMemoryAllocation ? EPI_E_NOMEM : EPI_E_CUDA,          \
                           "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__);      \
        }                                                                                             \
    } while (0)

// ensure() for memory that may be a part of the context's slab: that is not freed by itself.
template <class T>
static cudaError_t ensure_own(T **p, size_t *cap_bytes, size_t bytes, bool *own)
{
    if (*p && *cap_bytes >= bytes) return cudaSuccess;
    if (*p && *own) cudaFree(*p);
    *p = nullptr;
    *cap_bytes = 0;
    cudaError_t e = cudaMalloc((void **)p, bytes ? bytes : 16);
    if (e == cudaSuccess) {
        *cap_bytes = bytes;
        *own = true;
    }
    return e;
}

// Pinned host memory of `count` elements: the arena's part for it, or an allocation of its own
// where that is too small.
constexpr size_t ARENA_STATE = 0, ARENA_INFO = 16384, ARENA_BLOCKS = 32768, ARENA_HITS = 65536,
                 ARENA_BYTES = ARENA_HITS + epi::FINISH_HITS * sizeof(DevHit);
template <class T, class N>
static cudaError_t ensure_pinned(epi_ctx *ctx, T **p, N *cap, size_t count, size_t at, size_t end)
{
    if (*p && (size_t)*cap >= count) return cudaSuccess;
    T *const part = reinterpret_cast<T *>(ctx->h_arena + at);
    if (*p && *p != part) cudaFreeHost(*p);
    *p = nullptr;
    *cap = 0;
    if (count <= (end - at) / sizeof(T)) {
        *p = part;
        *cap = (N)((end - at) / sizeof(T));
        return cudaSuccess;
    }
    cudaError_t e = cudaHostAlloc((void **)p, count * sizeof(T), cudaHostAllocDefault);
    if (e == cudaSuccess) *cap = (N)count;
    return e;
}

template <class T>
static cudaError_t ensure(T **p, size_t *cap_bytes, size_t bytes)
{
    if (*p && *cap_bytes >= bytes) return cudaSuccess;
    if (*p) cudaFree(*p);
    *p = nullptr;
    *cap_bytes = 0;
    cudaError_t e = cudaMalloc((void **)p, bytes ? bytes : 16);
    if (e == cudaSuccess) *cap_bytes = bytes;
    return e;
}

// The expanded rows that are not a part of the slab (up to 64 GiB), given back.
static void release_x(epi_ctx *ctx)
{
    if (!ctx->d_x || !ctx->own_x) return;
    cudaStreamSynchronize(ctx->stream);
    cudaFree(ctx->d_x);
    ctx->d_x = nullptr;
    ctx->own_x = false;
    ctx->x_cap = 0;
    ctx->x_valid = -1;
}

// f(), which allocates for new genotypes or traits; where memory runs out, once more without the
// expanded rows, which the new data have made useless.
template <class F>
static cudaError_t without_x(epi_ctx *ctx, F f)
{
    cudaError_t e = f();
    if (e != cudaErrorMemoryAllocation || !ctx->d_x || !ctx->own_x) return e;
    cudaGetLastError();
    release_x(ctx);
    return f();
}

extern "C" {

void epi_default_opts(epi_scan_opts *o)
{
    if (!o) return;
    memset(o, 0, sizeof(*o));
    o->test = 'f';
    o->safe = 0;
    o->chunk = 128;
    o->t1 = 6.5f;
    o->t2 = 10.5f;
    o->form = EPI_FORM_AUTO;
    o->report_trait = 0;
}

const char *epi_strerror(epi_status s)
{
    switch (s) {
    case EPI_OK: return "success";
    case EPI_E_INVALID: return "invalid argument";
    case EPI_E_CUDA: return "CUDA error";
    case EPI_E_NOMEM: return "out of device memory";
    case EPI_E_OVERFLOW: return "more hits than the output capacity";
    case EPI_E_STATE: return "genotypes or phenotypes not loaded";
    case EPI_E_TIMEOUT: return "device wait timed out";
    case EPI_E_NODEVICE: return "no suitable CUDA device";
    case EPI_E_UNSUPPORTED: return "unsupported option for this form";
    }
    return "unknown status";
}

const char *epi_last_error(const epi_ctx *ctx) { return ctx ? ctx->err.c_str() : ""; }

epi_status epi_open(int32_t device, epi_ctx **out)
{
    if (!out) return EPI_E_INVALID;
    *out = nullptr;
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) return EPI_E_NODEVICE;
    if (device < 0 || device >= n) return EPI_E_NODEVICE;
    // (single attributes: the whole property structure, with the name, takes 3 ms to fill)
    int major = 0, sms = 0;
    if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
        return EPI_E_NODEVICE;
    if (major != 10) return EPI_E_NODEVICE;  // the library carries sm_100a code only
    epi_ctx *ctx = new epi_ctx();
    ctx->device = device;
    ctx->sm_count = sms;
    cudaError_t e = cudaSetDevice(device);
    if (e == cudaSuccess) e = cudaHostAlloc((void **)&ctx->h_arena, ARENA_BYTES, cudaHostAllocDefault);
    if (e == cudaSuccess) ctx->h_hits = (DevHit *)(ctx->h_arena + ARENA_HITS);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreate(&ctx->ev0);
    if (e == cudaSuccess) e = cudaEventCreate(&ctx->ev1);
    if (e == cudaSuccess) e = cudaMalloc((void **)&ctx->d_counters, epi::NCOUNTERS * sizeof(unsigned long long));
    if (e != cudaSuccess) {
        epi_close(ctx);
        return EPI_E_CUDA;
    }
    *out = ctx;
    return EPI_OK;
}

epi_status epi_close(epi_ctx *ctx)
{
    if (!ctx) return EPI_OK;
    if (ctx->device >= 0) cudaSetDevice(ctx->device);
    if (ctx->stream) cudaStreamSynchronize(ctx->stream);
    void *bufs[] = {ctx->d_raw, ctx->d_planes, ctx->d_hcodes, ctx->d_h3, ctx->d_missbits, ctx->d_y, ctx->d_yraw, ctx->d_yvalid,
                    ctx->d_wmask, ctx->d_yscale, ctx->d_qd, ctx->d_qtot, ctx->d_qm, ctx->d_ydig,
                    ctx->d_slab, ctx->own_hits ? ctx->d_hits : nullptr, ctx->d_counters, ctx->d_maxf, ctx->d_blocks, ctx->d_maj, ctx->d_pmC,
                    ctx->d_pmQ, ctx->d_ysq, ctx->d_pmN, ctx->own_x ? ctx->d_x : nullptr, ctx->d_tscr,
                    ctx->own_cand ? ctx->d_cand : nullptr};
    for (void *p : bufs)
        if (p) cudaFree(p);
    if (ctx->gexec) cudaGraphExecDestroy(ctx->gexec);
    const auto inside = [&](const void *p) {
        return p >= ctx->h_arena && p < ctx->h_arena + ARENA_BYTES;
    };
    for (void *p : {(void *)ctx->h_blocks, (void *)ctx->h_state, (void *)ctx->h_info})
        if (p && !inside(p)) cudaFreeHost(p);
    if (ctx->h_arena) cudaFreeHost(ctx->h_arena);
    if (ctx->ev0) cudaEventDestroy(ctx->ev0);
    if (ctx->ev1) cudaEventDestroy(ctx->ev1);
    if (ctx->stream) cudaStreamDestroy(ctx->stream);
    delete ctx;
    return EPI_OK;
}

epi_status epi_device_info(const epi_ctx *ctx, char *name, int32_t name_len, int32_t *sm_count)
{
    if (!ctx) return EPI_E_INVALID;
    if (name && name_len > 0) {
        cudaDeviceProp prop;
        if (cudaGetDeviceProperties(&prop, ctx->device) != cudaSuccess) return EPI_E_CUDA;
        snprintf(name, (size_t)name_len, "%s", prop.name);
    }
    if (sm_count) *sm_count = ctx->sm_count;
    return EPI_OK;
}

epi_status epi_load_packed(epi_ctx *ctx, const int32_t *gpack, int32_t nid, int32_t nsnp, int32_t npack,
                           int32_t remain)
{
    if (!ctx) return EPI_E_INVALID;
    if (!gpack || nid < 1 || nsnp < 1)
        return set_err(ctx, EPI_E_INVALID, "epi_load_packed: need gpack, nid >= 1, nsnp >= 1");
    if (npack != nid / 16 || remain != nid % 16)
        return set_err(ctx, EPI_E_INVALID, "epi_load_packed: npack/remain (%d/%d) inconsistent with nid %d "
                       "(src/readplink.c:1071-1072)", npack, remain, nid);
    CK(cudaSetDevice(ctx->device));
    const int npack1 = remain ? npack + 1 : npack;
    const int Wp = ((nid + 31) / 32 + 3) / 4 * 4;  // multiple of 4 words = 128 individuals
    const int Wc = 2 * Wp;
    // no genotypes until the new ones are there: an allocation that fails below has freed the old ones
    ctx->nid = ctx->nsnp = 0;
    ctx->qm_valid = false;
    ctx->pm_valid = false;
    ctx->x_valid = -1;
    if (ctx->traits_nid != nid) ctx->overrun = Overrun();
    ctx->overrun.changed = true;
    CK(without_x(ctx, [&] {
        cudaError_t e = ensure(&ctx->d_raw, &ctx->raw_cap, (size_t)nsnp * npack1 * sizeof(int32_t));
        if (e == cudaSuccess) e = ensure(&ctx->d_planes, &ctx->planes_cap, (size_t)nsnp * Wp * sizeof(uint4));
        if (e == cudaSuccess) e = ensure(&ctx->d_hcodes, &ctx->hcodes_cap, (size_t)nsnp * Wp * 32);
        if (e == cudaSuccess) e = ensure(&ctx->d_h3, &ctx->h3_cap, 3 * (size_t)nsnp * Wp * 32);
        if (e == cudaSuccess) e = ensure(&ctx->d_missbits, &ctx->missbits_cap, (size_t)nsnp * Wp * sizeof(uint32_t));
        if (e == cudaSuccess) e = ensure(&ctx->d_maj, &ctx->maj_cap, (size_t)nsnp);
        return e;
    }));
    CK(cudaMemcpyAsync(ctx->d_raw, gpack, (size_t)nsnp * npack1 * sizeof(int32_t), cudaMemcpyHostToDevice,
                       ctx->stream));
    CK(epi::launch_unpack(ctx->d_raw, nsnp, nid, npack, remain, ctx->d_planes, Wp, nullptr, Wc, ctx->d_hcodes,
                          ctx->d_h3, ctx->d_missbits, ctx->stream));
    CK(epi::launch_major(ctx->d_planes, nsnp, Wp, ctx->d_maj, ctx->stream));
    CK(epi::mma_encode_genotypes(&ctx->maps, ctx->d_hcodes, ctx->d_h3, nsnp, 32 * Wp));
    if (ctx->traits_nid != nid) ctx->ntraits = 0;  // traits no longer match
    ctx->nid = nid;
    ctx->nsnp = nsnp;
    ctx->npack = npack;
    ctx->remain = remain;
    ctx->Wp = Wp;
    ctx->Wc = Wc;
    ctx->Np = 32 * Wp;
    return EPI_OK;
}

// The phenotype columns as given are uploaded and k_traits (prep.cu) makes all that the scans
// need of them on the device.
static epi_status set_traits(epi_ctx *ctx, const float *y, int32_t nid, int32_t ntraits, const uint8_t *valid, int mode)
{
    if (!ctx) return EPI_E_INVALID;
    if (!y || nid < 1 || ntraits < 1) return set_err(ctx, EPI_E_INVALID, "epi_set_traits: bad arguments");
    if (ctx->nid == 0) return set_err(ctx, EPI_E_STATE, "epi_set_traits: load genotypes first");
    if (nid != ctx->nid)
        return set_err(ctx, EPI_E_INVALID, "epi_set_traits: %d individuals, genotypes have %d", nid, ctx->nid);
    CK(cudaSetDevice(ctx->device));
    const int Np = ctx->Np, Wp = ctx->Wp;
    const size_t T = (size_t)ntraits, cells = T * nid;
    ctx->ntraits = 0;  // until the new ones are there
    // buffers are kept across calls while they are large enough: a cudaFree would
    // synchronise the device on every trait upload
    CK(without_x(ctx, [&] {
        cudaError_t e = ensure(&ctx->d_yraw, &ctx->yraw_cap, cells * sizeof(float));
        if (e == cudaSuccess && mode == epi::VALID_BYTES) e = ensure(&ctx->d_yvalid, &ctx->yvalid_cap, cells);
        if (e == cudaSuccess) e = ensure(&ctx->d_y, &ctx->y_cap, T * Np * sizeof(float));
        if (e == cudaSuccess) e = ensure(&ctx->d_wmask, &ctx->wmask_cap, T * Wp * sizeof(uint32_t));
        if (e == cudaSuccess) e = ensure(&ctx->d_ysq, &ctx->ysq_cap, T * sizeof(double));
        if (e == cudaSuccess) e = ensure(&ctx->d_ydig, &ctx->ydig_cap, 5 * T * Np);
        if (e == cudaSuccess) e = ensure(&ctx->d_qd, &ctx->qd_cap, 2 * T * Np * sizeof(double));
        if (e == cudaSuccess) e = ensure(&ctx->d_qtot, &ctx->qtot_cap, T * sizeof(double));
        if (e == cudaSuccess) e = ensure(&ctx->d_yscale, &ctx->yscale_cap, 3 * T * sizeof(double));
        if (e == cudaSuccess) e = ensure(&ctx->d_tscr, &ctx->tscr_cap, 2 * T * sizeof(float4));
        return e;
    }));
    CK(ensure_pinned(ctx, &ctx->h_info, &ctx->h_info_cap, T, ARENA_INFO, ARENA_BLOCKS));
    CK(epi::mma_encode_traits(&ctx->maps, ctx->d_ydig, ntraits, Np));
    CK(cudaMemcpyAsync(ctx->d_yraw, y, cells * sizeof(float), cudaMemcpyHostToDevice, ctx->stream));
    if (mode == epi::VALID_BYTES)
        CK(cudaMemcpyAsync(ctx->d_yvalid, valid, cells, cudaMemcpyHostToDevice, ctx->stream));
    const epi::TraitArrays out = {ctx->d_y,  ctx->d_wmask, ctx->d_ydig,   ctx->d_qd,
                                  ctx->d_ysq, ctx->d_qtot, ctx->d_yscale, ctx->d_tscr};
    CK(epi::launch_traits(ctx->d_yraw, ctx->d_yvalid, mode, nid, Np, ntraits, out, ctx->h_info, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    ctx->ntraits = ntraits;
    ctx->traits_nid = nid;
    ctx->qm_valid = false;
    ctx->pm_valid = false;
    ctx->x_valid = -1;
    ctx->overrun.changed = true;
    return EPI_OK;
}

epi_status epi_set_traits(epi_ctx *ctx, const float *y, int32_t nid, int32_t ntraits, const uint8_t *valid)
{
    return set_traits(ctx, y, nid, ntraits, valid, valid ? epi::VALID_BYTES : epi::VALID_NOT9);
}

epi_status epi_set_phenotype(epi_ctx *ctx, const float *phen, int32_t nid, int32_t safe)
{
    return set_traits(ctx, phen, nid, 1, nullptr, safe ? epi::VALID_ALL : epi::VALID_NOT9);
}

void epi_permute_phenotype(float *phen, int32_t nid, uint32_t seed)
{
    if (!phen) return;
    srand(seed);
    for (int i = nid; i > 1; i--) {
        const int r = rand() % i;
        const float t = phen[r];
        phen[r] = phen[i - 1];
        phen[i - 1] = t;
    }
}

}  // extern "C"

static int64_t block_pairs(const epi_block &b) { return epi::pairs_below(b.start1, b.size1, b.start2, b.size2); }

namespace {

struct ScanRun {
    epi::ScanArgs args;
    int form;
    int variant;  // the form's kernel variant (tile shape or ring depths)
    int screen;   // tensor form: the digits of the screened scan, 0: all digits
    int segments;
    // tensor form: units in all and of one trait, and where each row group begins (units of the
    // trait before it, block, group)
    struct Start {
        int64_t units;
        int block, group;
    };
    int64_t units, trait_units;
    int xsi, xsj;
    std::vector<Start> starts;
    // the first row group at or past `u` units, and the units before it
    epi::SegPos at(int64_t u, int ntraits, int64_t *before) const
    {
        *before = units;
        if (u >= units) return {ntraits, 0, 0};
        const auto it = std::lower_bound(starts.begin(), starts.end(), u % trait_units,
                                         [](const Start &x, int64_t y) { return x.units < y; });
        const int t = (int)(u / trait_units);
        *before = t * trait_units + (it == starts.end() ? trait_units : it->units);
        return it == starts.end() ? epi::SegPos{t + 1, 0, 0} : epi::SegPos{t, it->block, it->group};
    }
    int64_t ntiles;
    std::vector<BlockDesc> desc;
};

epi_status check_opts(epi_ctx *ctx, const epi_scan_opts *o)
{
    if (!o) return set_err(ctx, EPI_E_INVALID, "null options");
    if (o->test != 'f' && o->test != 'i') return set_err(ctx, EPI_E_INVALID, "test must be 'f' or 'i'");
    if (o->safe != 0 && o->safe != 1) return set_err(ctx, EPI_E_INVALID, "safe must be 0 or 1");
    if (o->chunk < 1) return set_err(ctx, EPI_E_INVALID, "chunk must be >= 1");
    if (o->form < EPI_FORM_AUTO || o->form > EPI_FORM_TENSOR) return set_err(ctx, EPI_E_INVALID, "bad form");
    if (o->report_trait < -1 || o->report_trait >= ctx->ntraits)
        return set_err(ctx, EPI_E_INVALID, "report_trait %d out of range", o->report_trait);
    if (o->wait_limit_ms < 0) return set_err(ctx, EPI_E_INVALID, "wait_limit_ms must be >= 0");
    if (o->debug != 0 && o->debug != EPI_DEBUG_STALL) return set_err(ctx, EPI_E_INVALID, "bad debug flags");
    if (o->no_graph != 0 && o->no_graph != 1) return set_err(ctx, EPI_E_INVALID, "no_graph must be 0 or 1");
    if (o->tile_config < 0) return set_err(ctx, EPI_E_INVALID, "tile_config must be >= 0");
    return EPI_OK;
}

// The form of a scan without a screen. The automatic choice is the plain one below 256 individuals: it
// keeps y in 32 bits, which the tensor form's digits do not.
int pick_form(const epi_ctx *ctx, const epi_scan_opts *o)
{
    if (o->form != EPI_FORM_AUTO) return o->form;
    return epi::mma_available() && ctx->nid >= 256 && ctx->Np <= epi::mma_max_nid() ? EPI_FORM_TENSOR : EPI_FORM_POPC;
}

// Whether the automatic choice of the plain form may be screened by the tensor form, whose candidates are
// then evaluated from y (and no kernel variant of the plain form is asked for).
bool screens_plain(const epi_ctx *ctx, const epi_scan_opts *o)
{
    return o->form == EPI_FORM_AUTO && pick_form(ctx, o) == EPI_FORM_POPC && o->tile_config == 0 && epi::mma_available() &&
           ctx->nid >= epi::mma_min_nid();
}

// Builds the kernel arguments and tile schedule for `blocks` and uploads the schedule.
// Bytes of the streamed-B variant's expanded rows, and whether they may be allocated: at most
// 64 GiB and half the device's free memory (beyond, that variant is not a candidate).
static size_t x_bytes(const epi_ctx *ctx, int screen)
{
    return (size_t)epi::mma_x_rows(screen) * ctx->nsnp * ctx->Np * epi::mma_x_sets(screen, ctx->ntraits);
}
static bool x_usable(const epi_ctx *ctx, int screen)
{
    const size_t need = x_bytes(ctx, screen);
    if (need <= ctx->x_cap) return true;
    size_t fr = 0, tot = 0;
    if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) return false;
    return need <= (64ull << 30) && need <= fr / 2 + (ctx->own_x ? ctx->x_cap : 0);  // (the slab's part stays)
}

// The streamed-B variant as an autotuner candidate: only up to 6,144 padded individuals. Its
// expanded rows are 12 bytes per SNP and individual, and the DRAM traffic of its super-tiles
// grows with N per second of scanning; at N = 10,000 a full scan then runs into the 1 kW power
// cap (SM clock ~1,350 MHz against ~1,935 MHz for the shared-memory producers) and ends 12%
// slower, although the autotuner's short sample, run before the cap bites, ranks it 15% faster.
// At N = 4,000 it is 10-14% faster at full clock. tile_config can still force it.
// The screen needs half the rows per pair: there it is the fastest at every size, also at
// N = 10,000 under the power cap (605 ms at 1,567 MHz against 640 ms for two producer groups).
static bool x_candidate(const epi_ctx *ctx, int screen) { return (screen || ctx->Np <= 6144) && x_usable(ctx, screen); }

// The share of a scan's pair tests that the screen with `digits` phenotype digits (1 or 2,
// scan_mma.cu) is expected to pass on (screen_rule.cuh).
static double screen_share(const epi_ctx *ctx, const epi_scan_opts *o, double pairs, int digits)
{
    const double top8 = epi::chi_top(pairs, 8), top4 = epi::chi_top(pairs, 4);
    double share = 0.0;
    for (int t = 0; t < ctx->ntraits; ++t) {
        const double r = digits == 1 ? ctx->h_info[t].r1 : ctx->h_info[t].r2, nv = ctx->h_info[t].nv;
        if (!std::isfinite(r)) return INFINITY;
        const bool report = o->report_trait < 0 || o->report_trait == t;
        share += epi::screen_share_of(o->t1, report, 8, top8, r, nv);
        if (o->test == 'i') share += epi::screen_share_of(o->t2, report, 4, top4, r, nv);
    }
    return share / ctx->ntraits;
}

// Capacity of the candidate list of a segment: one percent of its pair tests (where the screen stops
// paying), 2^16 to 2^22 entries (100 MB); a longer list ends the screened scan.
constexpr double CAND_MAX = 4194304.0;
static int64_t cand_capacity(double tests)
{
    return (int64_t)std::min(CAND_MAX, std::max(65536.0, tests / 100.0));
}

// Segments that keep the candidates expected of the largest list at half of it (a list of one percent
// holds twice what the screen is chosen for, 1 in 250). A segment boundary costs 30 us; at 1 in 250 a
// segment is 5e8 tests, 0.05 s at N = 10,000.
constexpr int MAX_SEGMENTS = 1024;
static double segments_for(double tests, double share) { return 2.0 * share * tests / CAND_MAX; }

// Whether the one-digit screen takes the traits in groups of five that share their counts (screen
// 3): all have the same valid individuals, their groups take fewer tiles (a tile is 14 j-SNPs by
// five traits against 42 by one: not for 1 to 3 or 6 traits), the expanded rows fit, and no other
// kernel variant is asked for.
static bool group_traits(const epi_ctx *ctx, const epi_scan_opts *o)
{
    const int T = ctx->ntraits, G = epi::GROUP_TRAITS;
    if (o->tile_config != 0 && o->tile_config != 6) return false;
    if (T <= 3 * ((T + G - 1) / G)) return false;
    for (int t = 0; t < T; ++t)
        if (ctx->h_info[t].same_mask == 0.0) return false;
    return x_usable(ctx, 3);
}

// The digits of the screen for a scan of `pairs` pairs (3: one digit, grouped traits), or 0 for all digits without a screen. A
// candidate costs about as much as 110 pairs of the one-digit screen (11 ns against 0.1 ns at
// N = 10,000, both in proportion to N), a pair with two digits 1.5 and with all digits 2 of them:
// so one digit up to a share of 1 in 250 (0.72 of the time with all digits there), two up to 1 in
// 400, or where that is at most 1,024 candidates in all (fewer than the exact kernel's warps). For
// a normal trait R is 0.0092 sqrt(N) with one digit: the rule turns to two at 10,000 to 14,000
// individuals at p = 1e-6, and to all digits at thresholds that let one pair in 400 through.
// `share` is the share expected of the chosen screen; more than its lists would hold refuses it.
static int screen_digits(const epi_ctx *ctx, const epi_scan_opts *o, double pairs, double *share)
{
    *share = 0.0;
    const double tests = pairs * ctx->ntraits;
    if (ctx->overrun.covers(o, tests)) return 0;
    if (!(pairs >= 1.0) || ctx->Np > epi::mma_screen_max_nid()) return 0;
    const double most = (double)MAX_SEGMENTS / segments_for(tests, 1.0);
    const double one = screen_share(ctx, o, pairs, 1);
    if ((one <= 1.0 / 250.0 || one * tests <= 1024.0) && one <= most) {
        *share = one;
        return group_traits(ctx, o) ? 3 : 1;
    }
    const double two = screen_share(ctx, o, pairs, 2);
    if ((two > 1.0 / 400.0 && two * tests > 1024.0) || two > most) return 0;
    *share = two;
    return 2;
}

// share: of the pair tests that the screen is expected to pass on
epi_status setup_run(epi_ctx *ctx, const epi_block *blocks, int nblocks, const epi_scan_opts *o, ScanRun &r, int form,
                     int variant, int screen, double share = 0.0)
{
    r.form = form;
    r.variant = variant;
    r.screen = screen;
    r.segments = 1;
    if (r.form == EPI_FORM_TENSOR && !epi::mma_available())
        return set_err(ctx, EPI_E_UNSUPPORTED, "tensor form not available in this library");
    if (r.form == EPI_FORM_TENSOR && ctx->Np > epi::mma_max_nid())
        return set_err(ctx, EPI_E_UNSUPPORTED, "tensor form: at most %d individuals", epi::mma_max_nid());
    if (r.form == EPI_FORM_POPC && ctx->nid > 65535)
        return set_err(ctx, EPI_E_UNSUPPORTED, "popcount form counts in 16 bits: at most 65535 individuals "
                       "(the reference's unsigned short counts, EpiOpenCL.c:68)");
    const bool needs_x = r.form == EPI_FORM_TENSOR && epi::mma_needs_x(variant, screen);
    if (needs_x && !x_usable(ctx, screen))
        return set_err(ctx, EPI_E_UNSUPPORTED, "tensor variant %d: its %zu bytes of expanded B rows do not fit",
                       variant + 1, x_bytes(ctx, screen));
    int TI = epi::mma_tile_i(), TJ = epi::mma_tile_j(screen);
    if (r.form == EPI_FORM_POPC) {
        epi::popc_shape(variant, &TI, &TJ, nullptr);
        CK(epi::popc_encode_planes(variant, &ctx->pmaps, ctx->d_planes, ctx->nsnp, ctx->Wp));
    }
    r.desc.resize(nblocks);
    int64_t base = 0;
    for (int b = 0; b < nblocks; ++b) {
        const epi_block &e = blocks[b];
        if (e.size1 < 0 || e.size2 < 0 || e.start1 < 0 || e.start2 < 0 ||
            (int64_t)e.start1 + e.size1 > ctx->nsnp || (int64_t)e.start2 + e.size2 > ctx->nsnp)
            return set_err(ctx, EPI_E_INVALID, "block %d out of range", b);
        BlockDesc &d = r.desc[b];
        d.start1 = e.start1;
        d.size1 = e.size1;
        d.start2 = e.start2;
        d.size2 = e.size2;
        d.tiles_i = (e.size1 + TI - 1) / TI;
        d.tiles_j = (e.size2 + TJ - 1) / TJ;
        d.tile_base = base;
        base += (int64_t)d.tiles_i * d.tiles_j;
    }
    r.ntiles = base;
    size_t bcap = (size_t)ctx->blocks_cap * sizeof(BlockDesc);
    if (bcap < (size_t)std::max(nblocks, 1) * sizeof(BlockDesc)) ctx->dev_blocks.clear();
    CK(ensure(&ctx->d_blocks, &bcap, (size_t)std::max(nblocks, 1) * sizeof(BlockDesc)));
    ctx->blocks_cap = (int)(bcap / sizeof(BlockDesc));
    CK(ensure_pinned(ctx, &ctx->h_blocks, &ctx->h_blocks_cap, (size_t)nblocks, ARENA_BLOCKS, ARENA_HITS));
    CK(ensure_pinned(ctx, &ctx->h_state, &ctx->h_state_cap, epi::NCOUNTERS + (size_t)ctx->ntraits, ARENA_STATE,
                     ARENA_INFO));
    if (ctx->maxf_cap < 4 * ctx->ntraits) {  // maxima, then the screen's lower bounds of them
        if (ctx->d_maxf) cudaFree(ctx->d_maxf);
        ctx->d_maxf = nullptr;
        ctx->maxf_cap = 0;
        ctx->clean_traits = 0;
        CK(cudaMalloc((void **)&ctx->d_maxf, 4 * (size_t)ctx->ntraits * sizeof(unsigned int)));
        ctx->maxf_cap = 4 * ctx->ntraits;
    }
    // the tensor form's order of units (scan_mma.cu: Walker): super-tiles of about 40 MB of A rows
    // (3 bytes per SNP and individual) and expanded B rows for the streamed-B variant, equal
    // sides in pair tiles; row by row over all j-tiles otherwise
    r.xsi = 1;
    r.xsj = 1 << 30;
    r.starts.clear();
    r.units = base * ctx->ntraits;
    if (r.form == EPI_FORM_TENSOR) {
        if (epi::mma_needs_x(variant, screen)) {
            const double per = (3.0 * TI + (double)epi::mma_x_rows(screen) * TJ) * ctx->Np;
            r.xsi = r.xsj = std::max(1, (int)(40e6 / per));
        }
        r.units = 0;
        for (const BlockDesc &d : r.desc)
            for (int ti = 0; ti < d.tiles_i; ++ti) {
                if (ti % r.xsi == 0) r.starts.push_back({r.units, (int)(&d - r.desc.data()), ti / r.xsi});
                const int64_t x = (int64_t)d.start1 + std::min((ti + 1) * TI, d.size1) - 1 - d.start2;
                r.units += x <= 0 ? 0 : std::min<int64_t>(d.tiles_j, (x + TJ - 1) / TJ);
            }
        r.trait_units = r.units;
        r.units *= epi::mma_x_sets(screen, ctx->ntraits);
        if (r.units == 0) r.ntiles = 0;  // no pair at all
    }
    size_t cand = 0;  // bytes of the candidate list
    if (screen) {
        double tests = 0.0;
        for (int b = 0; b < nblocks; ++b) tests += (double)block_pairs(blocks[b]) * ctx->ntraits;
        // Segments: the list of each is worked off before the next begins, so the list stays
        // short, the exact maxima of the first ones tighten the screen of the later ones and a
        // list that runs over costs a part of the scan only. A segment boundary idles the GPU for
        // about 30 us, so a segment lasts 5 ms or more (600 cycles a stage, two SMs a unit).
        // More than eight only where their lists would run over.
        const double ms = (double)r.units / (ctx->sm_count / 2) * (ctx->Np / 128) * 600.0 / 1.9e6;
        r.segments = (int)std::max(std::min(8.0, std::max(1.0, ms / 5.0)),
                                   std::min((double)MAX_SEGMENTS, std::ceil(segments_for(tests, share))));
        cand = (size_t)cand_capacity(tests / r.segments) * sizeof(epi::Cand);
    }
    if (!ctx->d_slab) {
        // the first scan's memory in one piece: hits (2^20), candidates, expanded B rows; the hits alone
        // where that is too much
        const size_t hits = sizeof(DevHit) << 20, cand_part = (cand + 255) & ~(size_t)255;
        const size_t x = needs_x && x_bytes(ctx, screen) <= (256u << 20) ? x_bytes(ctx, screen) : 0;
        bool whole = true;
        cudaError_t e = cudaMalloc(&ctx->d_slab, hits + cand_part + x);
        if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            whole = false;
            e = cudaMalloc(&ctx->d_slab, hits);
        }
        if (e != cudaSuccess) ctx->d_slab = nullptr;
        CK(e);
        unsigned char *const p = (unsigned char *)ctx->d_slab;
        ctx->d_hits = (DevHit *)p;
        ctx->hit_cap = 1 << 20;
        if (cand && whole) {
            ctx->d_cand = (epi::Cand *)(p + hits);
            ctx->cand_cap = cand;
        }
        if (x && whole) {
            ctx->d_x = (int8_t *)(p + hits + cand_part);
            ctx->x_cap = x;
        }
    }
    if (cand) CK(ensure_own(&ctx->d_cand, &ctx->cand_cap, cand, &ctx->own_cand));
    if (needs_x && ctx->x_valid != screen) {
        ctx->x_valid = -1;  // until the rows are there: the old ones may be gone when the allocation fails
        CK(ensure_own(&ctx->d_x, &ctx->x_cap, x_bytes(ctx, screen), &ctx->own_x));
        CK(epi::launch_expand(ctx->d_hcodes, ctx->d_ydig, ctx->nsnp, ctx->Np, ctx->ntraits, screen, ctx->d_x,
                              ctx->stream));
        CK(epi::mma_encode_x(&ctx->maps, ctx->d_x, ctx->nsnp, ctx->Np, ctx->ntraits, screen));
        ctx->x_valid = screen;
    }
    if (r.form == EPI_FORM_TENSOR && !ctx->qm_valid) {
        const size_t tn = (size_t)ctx->ntraits * ctx->nsnp;
        CK(ensure(&ctx->d_qm, &ctx->qm_cap, tn * (3 * sizeof(double) + sizeof(float))));
        CK(epi::launch_qmiss(ctx->d_missbits, ctx->nsnp, ctx->Wp, ctx->d_wmask, ctx->d_qd,
                             ctx->d_qd + (size_t)ctx->ntraits * ctx->Np, ctx->Np, ctx->ntraits, ctx->d_qm,
                             ctx->d_qm + tn, ctx->d_qm + 2 * tn, (float *)(ctx->d_qm + 3 * tn), ctx->stream));
        ctx->qm_valid = true;
    }
    if (r.form == EPI_FORM_POPC && !ctx->pm_valid) {
        const size_t tn = (size_t)ctx->ntraits * ctx->nsnp;
        CK(ensure(&ctx->d_pmC, &ctx->pmC_cap, 3 * tn * sizeof(double)));
        CK(ensure(&ctx->d_pmN, &ctx->pmN_cap, 3 * tn * sizeof(int32_t)));
        CK(ensure(&ctx->d_pmQ, &ctx->pmQ_cap, tn * sizeof(double)));
        CK(epi::launch_marg(ctx->d_planes, ctx->nsnp, ctx->Wp, ctx->d_y, ctx->d_wmask, ctx->Np, ctx->ntraits,
                            ctx->d_pmC, ctx->d_pmN, ctx->d_pmQ, ctx->stream));
        ctx->pm_valid = true;
    }
    epi::ScanArgs &a = r.args;
    memset(&a, 0, sizeof(a));
    a.planes = ctx->d_planes;
    a.hcodes = ctx->d_hcodes;
    a.missbits = ctx->d_missbits;
    a.Wp = ctx->Wp;
    a.Wc = ctx->Wc;
    a.nid = ctx->nid;
    a.nsnp = ctx->nsnp;
    a.yscale = ctx->d_yscale;
    a.ytot = ctx->d_yscale + ctx->ntraits;
    a.nvalid = ctx->d_yscale + 2 * (size_t)ctx->ntraits;
    a.qd = ctx->d_qd;
    a.qtot = ctx->d_qtot;
    a.qm = ctx->d_qm;
    a.sm = ctx->d_qm + (size_t)ctx->ntraits * ctx->nsnp;
    a.nm = ctx->d_qm + 2 * (size_t)ctx->ntraits * ctx->nsnp;
    a.ydig = ctx->d_ydig;
    a.maj = ctx->d_maj;
    a.pmC = ctx->d_pmC;
    a.pmN = ctx->d_pmN;
    a.pmQ = ctx->d_pmQ;
    a.ysq = ctx->d_ysq;
    a.y = ctx->d_y;
    a.wmask = ctx->d_wmask;
    a.Np = ctx->Np;
    a.ntraits = ctx->ntraits;
    a.blocks = ctx->d_blocks;
    a.nblocks = nblocks;
    a.ntiles = r.ntiles;
    a.test_int = o->test == 'i';
    a.safe = o->safe;
    a.report_trait = o->report_trait;
    a.t1 = o->t1;
    a.t2 = o->t2;
    a.wait_ns = o->wait_limit_ms > 0 ? (unsigned long long)o->wait_limit_ms * 1000000ull : 2000000000ull;
    a.debug_stall = o->debug == EPI_DEBUG_STALL;
    a.xsi = r.xsi;
    a.xsj = r.xsj;
    a.seg1 = {ctx->ntraits, 0, 0};
    a.seg_units = r.units;
    a.tscr = ctx->d_tscr;
    a.qmf = (const float *)(ctx->d_qm + 3 * (size_t)ctx->ntraits * ctx->nsnp);
    a.qmf_j = a.qmf;
    a.cand = ctx->d_cand;
    a.cand_cap = (int64_t)(ctx->cand_cap / sizeof(epi::Cand));
    a.lowf = ctx->d_maxf + 2 * (size_t)ctx->ntraits;
    a.lowf2 = ctx->d_maxf + 3 * (size_t)ctx->ntraits;
    a.counters = ctx->d_counters;
    a.maxf = ctx->d_maxf;
    a.maxf2 = ctx->d_maxf + ctx->ntraits;
    return EPI_OK;
}

// The device part of a scan, on the context's stream and nothing but stream operations (so it
// can be captured): the selected form's kernels between the timing events, and k_finish, which
// hands counters, maxima and the first hits to the host and resets them. What it expects on the
// device (clean counters and maxima, the block schedule) launch_run has put there.
cudaError_t enqueue_scan(epi_ctx *ctx, const ScanRun &r, int grid, bool capturing)
{
    cudaStream_t s = ctx->stream;
    // under stream capture the timing events are recorded as external records, which become
    // event nodes of the graph (so they time every replay); a direct launch records them plainly
    const unsigned int ev_flags = capturing ? cudaEventRecordExternal : cudaEventRecordDefault;
    cudaError_t e = cudaEventRecordWithFlags(ctx->ev0, s, ev_flags);
    if (e == cudaSuccess && r.ntiles > 0) {
        if (r.form != EPI_FORM_TENSOR) e = epi::popc_enqueue(r.variant, r.args, ctx->pmaps, grid, s);
        else if (!r.screen) e = epi::mma_enqueue(r.variant, 0, r.args, ctx->maps, grid, s);
        else {
            epi::ScanArgs a = r.args;
            a.segment = -1;
            for (int k = 0; k < r.segments && e == cudaSuccess; ++k) {
                int64_t u0 = 0, u1 = 0;
                const int sets = epi::mma_x_sets(r.screen, ctx->ntraits);
                a.seg0 = r.at(r.units / r.segments * k, sets, &u0);
                a.seg1 = r.at(k + 1 == r.segments ? r.units : r.units / r.segments * (k + 1), sets, &u1);
                a.seg_units = u1 - u0;
                if (a.seg_units == 0) continue;
                a.segment = (a.segment + 1) % epi::CAND_RING;
                e = epi::mma_enqueue(r.variant, r.screen, a, ctx->maps, grid, s);
                if (e == cudaSuccess) e = epi::exact_enqueue(a, ctx->sm_count, s);
            }
        }
    }
    if (e == cudaSuccess) e = cudaEventRecordWithFlags(ctx->ev1, s, ev_flags);
    if (e == cudaSuccess) {
        epi::k_finish<<<1, 256, 0, s>>>(ctx->d_counters, ctx->d_maxf, ctx->ntraits, r.args.hits, r.args.cap, ctx->h_state,
                                        ctx->h_hits);
        e = cudaGetLastError();
    }
    return e;
}

template <class T>
static void key_add(std::vector<unsigned char> &k, const T &v)
{
    const unsigned char *p = reinterpret_cast<const unsigned char *>(&v);
    k.insert(k.end(), p, p + sizeof(T));
}

// Runs the device part of a scan. With use_graph, a repeat of the previous scan's shape (same
// kernel arguments, tensor maps, schedule and launch shape) replays the CUDA graph captured for
// it with one launch; any other scan is captured anew first. Without, the operations are
// launched one by one.
epi_status launch_run(epi_ctx *ctx, ScanRun &r, int nblocks, bool use_graph)
{
    int grid = 0;
    if (r.ntiles > 0) {
        const int64_t units = r.units;
        if (r.form == EPI_FORM_TENSOR) {
            // one CTA pair per unit (tile x trait) up to every SM
            CK(epi::mma_prepare(r.variant, r.screen, ctx->ntraits, (int)std::min<int64_t>(2 * units, ctx->sm_count), &grid));
        } else {
            // one CTA per unit up to every SM
            CK(epi::popc_prepare(r.variant));
            grid = (int)std::min<int64_t>(units, ctx->sm_count);
        }
    }
    if ((int)ctx->dev_blocks.size() < nblocks ||
        memcmp(ctx->dev_blocks.data(), r.desc.data(), nblocks * sizeof(BlockDesc)) != 0) {
        ctx->dev_blocks.clear();
        memcpy(ctx->h_blocks, r.desc.data(), nblocks * sizeof(BlockDesc));
        CK(cudaMemcpyAsync(ctx->d_blocks, ctx->h_blocks, nblocks * sizeof(BlockDesc), cudaMemcpyHostToDevice,
                           ctx->stream));
        ctx->dev_blocks = r.desc;
    }
    if (ctx->clean_traits != ctx->ntraits) {
        epi::k_scan_init<<<1, 256, 0, ctx->stream>>>(ctx->d_counters, ctx->d_maxf, 4 * ctx->ntraits);
        CK(cudaGetLastError());
    }
    ctx->clean_traits = 0;  // until the launch below has succeeded
    // the scan kernel, or the screen and the exact kernel of every segment, and k_finish
    ctx->last_launches = 1 + (r.ntiles > 0 ? (r.screen ? 2 * r.segments : 1) : 0);
    ctx->last_form = r.form;
    if (!use_graph) {
        CK(enqueue_scan(ctx, r, grid, false));
        ctx->clean_traits = ctx->ntraits;
        return EPI_OK;
    }
    std::vector<unsigned char> key;
    key_add(key, r.args);
    key_add(key, r.form);
    key_add(key, r.variant);
    key_add(key, r.screen);
    key_add(key, r.segments);
    key_add(key, ctx->h_state);
    key_add(key, ctx->h_blocks);
    key_add(key, grid);
    key_add(key, ctx->ntraits);
    if (r.form == EPI_FORM_TENSOR) key_add(key, ctx->maps);
    else key_add(key, ctx->pmaps);
    key.insert(key.end(), reinterpret_cast<const unsigned char *>(r.desc.data()),
               reinterpret_cast<const unsigned char *>(r.desc.data() + nblocks));
    if (!ctx->gexec || key != ctx->gkey) {
        if (ctx->gexec) cudaGraphExecDestroy(ctx->gexec);
        ctx->gexec = nullptr;
        ctx->gkey.clear();
        CK(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
        const cudaError_t e = enqueue_scan(ctx, r, grid, true);
        cudaGraph_t g = nullptr;
        const cudaError_t e2 = cudaStreamEndCapture(ctx->stream, &g);  // ends the capture in any case
        if (e != cudaSuccess || e2 != cudaSuccess) {
            if (g) cudaGraphDestroy(g);
            CK(e != cudaSuccess ? e : e2);
        }
        const cudaError_t e3 = cudaGraphInstantiate(&ctx->gexec, g, 0);
        cudaGraphDestroy(g);
        if (e3 != cudaSuccess) ctx->gexec = nullptr;
        CK(e3);
        ctx->gkey = std::move(key);
    }
    CK(cudaGraphLaunch(ctx->gexec, ctx->stream));
    ctx->clean_traits = ctx->ntraits;
    return EPI_OK;
}

// ---- autotuner: the kernel variant per (device, form, padded individuals, traits) ----
//
// Every candidate of the form's table (tile shapes of the plain form, ring depths of the
// tensor form) scans a sample block of the loaded genotypes and traits -- large enough for a
// few waves of tiles over every SM -- once to warm up and once timed with CUDA events; the
// fastest is kept for the process. The reference has one such knob, the chunk size of its
// launches (src/main.c:115-130, src/EpiOpenCL.c:1353-1362), set by hand.
struct TuneEntry {
    int device, form, Np, ntraits, variant;
    int screen;
    std::string how;
};
static std::mutex g_tune_mu;
static std::vector<TuneEntry> g_tune;

int form_variants(int form) { return form == EPI_FORM_TENSOR ? epi::mma_shapes() : epi::popc_shapes(); }

std::string variant_desc(int form, int v, int screen)
{
    const char *d = nullptr;
    int ti = 0, tj = 0;
    if (form == EPI_FORM_TENSOR) epi::mma_shape(v, screen, &d);
    else epi::popc_shape(v, &ti, &tj, &d);
    return std::string(form == EPI_FORM_TENSOR ? "tensor form, " : "plain form, ") + d;
}

epi_status pick_variant(epi_ctx *ctx, const epi_scan_opts *o, int form, int screen, int *v, std::string *how)
{
    const int nv = form_variants(form);
    if (o->tile_config > 0) {
        if (o->tile_config > nv)
            return set_err(ctx, EPI_E_INVALID, "tile_config %d: this form has %d candidates", o->tile_config, nv);
        *v = o->tile_config - 1;
        *how = "requested";
        return EPI_OK;
    }
    {
        std::lock_guard<std::mutex> lock(g_tune_mu);
        // (a kept choice of the streamed-B variant holds only while this context's expanded rows
        // would fit: another context of the same shape may hold more SNPs)
        for (const TuneEntry &t : g_tune)
            if (t.device == ctx->device && t.form == form && t.Np == ctx->Np && t.ntraits == ctx->ntraits &&
                t.screen == screen && !(form == EPI_FORM_TENSOR && epi::mma_needs_x(t.variant, screen) && !x_candidate(ctx, screen))) {
                *v = t.variant;
                *how = t.how;
                return EPI_OK;
            }
    }
    if (nv == 1) {
        *v = 0;
        *how = "only candidate";
        return EPI_OK;
    }
    if (screen == 3) {  // grouped traits have one kernel
        *v = 5;
        *how = "8-bit screen, traits in groups";
        return EPI_OK;
    }
    // sample: an off-diagonal s x s block (every pair valid) when the genome holds one, with
    // enough tiles for about sixteen waves over the SMs at this trait count, at least 1,024
    // SNPs a side (a smaller block ranked the tensor variants wrongly at 64 traits) unless that
    // makes more than 2^28 pair tests, and at most 2,048
    const int T = ctx->ntraits;
    int s = (int)std::ceil(std::sqrt(16.0 * ctx->sm_count * 4096.0 / T));
    const int lo = std::max(256, std::min(1024, (int)std::sqrt(268435456.0 / T)));
    s = std::max(lo, std::min(s, 2048));
    epi_block blk;
    if (ctx->nsnp >= 2 * s) blk = {s, s, 0, s};
    else blk = {0, ctx->nsnp, 0, ctx->nsnp};
    epi_scan_opts o2 = *o;
    o2.report_trait = 0;
    std::vector<float> ms(nv, 0.0f);
    for (int c = 0; c < nv; ++c) {
        // the streamed-B variant is no candidate where its expanded rows would not fit or would
        // run into the power cap (x_candidate)
        if (form == EPI_FORM_TENSOR && epi::mma_needs_x(c, screen) && !x_candidate(ctx, screen)) {
            ms[c] = INFINITY;
            continue;
        }
        ScanRun r;
        epi_status st = setup_run(ctx, &blk, 1, &o2, r, form, c, screen);
        if (st != EPI_OK) return st;
        r.args.hits = ctx->d_hits;
        r.args.cap = ctx->hit_cap;
        for (int rep = 0; rep < 2; ++rep) {
            st = launch_run(ctx, r, 1, false);
            if (st != EPI_OK) return st;
        }
        CK(cudaStreamSynchronize(ctx->stream));
        if (ctx->h_state[2] != 0)
            return set_err(ctx, EPI_E_TIMEOUT, "a bounded device wait gave up while tuning (site %llu)",
                           ctx->h_state[3]);
        CK(cudaEventElapsedTime(&ms[c], ctx->ev0, ctx->ev1));
    }
    const int best = (int)(std::min_element(ms.begin(), ms.end()) - ms.begin());
    char buf[256];
    int len = snprintf(buf, sizeof(buf), "autotuned on a %d x %d-SNP block%s:", blk.size1, blk.size2,
                       screen == 1 ? ", 8-bit screen" : screen == 2 ? ", 16-bit screen" : "");
    for (int c = 0; c < nv && len < (int)sizeof(buf); ++c)
        len += std::isfinite(ms[c]) ? snprintf(buf + len, sizeof(buf) - len, "%s %.3f ms", c ? " /" : "", ms[c])
                                    : snprintf(buf + len, sizeof(buf) - len, "%s n/a", c ? " /" : "");
    *v = best;
    *how = buf;
    // the streamed-B candidate's expanded rows (up to 64 GiB) are released when it lost
    if (form == EPI_FORM_TENSOR && !epi::mma_needs_x(best, screen)) release_x(ctx);
    std::lock_guard<std::mutex> lock(g_tune_mu);
    g_tune.push_back({ctx->device, form, ctx->Np, ctx->ntraits, best, screen, *how});
    return EPI_OK;
}

// Output order of hits: (trait,) block, result slot, chunk k, chunk l, gx, gy
// (src/EpiOpenCL.c:1576-1627). The fields of a scan's hits nearly always fit one 64-bit key --
// inside chunk k only gx's remainder is left of gx -- so the hits are ordered by (key, index)
// pairs: std::sort up to 4,096, above that a radix sort over the key's bytes in use (211,000
// hits: 3 ms; seven-field comparisons took 20 ms). Wider keys go by the fields themselves.
struct HitKey {
    uint64_t key;
    uint32_t idx;
};

int bits_of(uint64_t largest)
{
    int n = 0;
    while (largest >> n) ++n;
    return n;
}

std::vector<uint32_t> output_order(const DevHit *h, size_t n, const epi_block *blocks, int nblocks, int ntraits,
                                   const epi_scan_opts *o)
{
    const uint32_t L = o->safe ? 8 : 16, chunk = (uint32_t)o->chunk;
    uint32_t size1 = 1, size2 = 1;
    for (int b = 0; b < nblocks; ++b) {
        size1 = std::max(size1, (uint32_t)blocks[b].size1);
        size2 = std::max(size2, (uint32_t)blocks[b].size2);
    }
    const int wr1 = bits_of(std::min(chunk, size1) - 1), wr2 = bits_of(std::min(chunk, size2) - 1);
    const int wk = bits_of((size1 - 1) / chunk), wl = bits_of((size2 - 1) / chunk);
    const int wb = bits_of((uint64_t)std::max(nblocks, 1) - 1), wt = o->report_trait < 0 ? bits_of((uint64_t)ntraits - 1) : 0;
    const int width = wt + wb + 8 + wk + wl + wr1 + wr2;
    std::vector<uint32_t> order(n);
    if (width > 64) {
        for (size_t i = 0; i < n; ++i) order[i] = (uint32_t)i;
        std::sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) {
            const DevHit &p = h[x], &q = h[y];
            if (o->report_trait < 0 && p.trait != q.trait) return p.trait < q.trait;
            if (p.block != q.block) return p.block < q.block;
            const epi_block &b = blocks[p.block];
            const uint32_t px = p.snp1 - b.start1, py = p.snp2 - b.start2, qx = q.snp1 - b.start1, qy = q.snp2 - b.start2;
            const uint32_t ps = (px % L) * L + py % L, qs = (qx % L) * L + qy % L;
            if (ps != qs) return ps < qs;
            if (px / chunk != qx / chunk) return px / chunk < qx / chunk;
            if (py / chunk != qy / chunk) return py / chunk < qy / chunk;
            return px != qx ? px < qx : py < qy;
        });
        return order;
    }
    std::vector<HitKey> keys(n);
    for (size_t i = 0; i < n; ++i) {
        const epi_block &b = blocks[h[i].block];
        const uint32_t gx = (uint32_t)(h[i].snp1 - b.start1), gy = (uint32_t)(h[i].snp2 - b.start2);
        uint64_t k = wt ? (uint64_t)(uint32_t)h[i].trait : 0;
        k = k << wb | (uint32_t)h[i].block;
        k = k << 8 | ((gx % L) * L + gy % L);
        k = k << wk | gx / chunk;
        k = k << wl | gy / chunk;
        k = k << wr1 | gx % chunk;
        k = k << wr2 | gy % chunk;
        keys[i] = {k, (uint32_t)i};
    }
    if (n <= 4096) {
        std::sort(keys.begin(), keys.end(), [](const HitKey &x, const HitKey &y) { return x.key < y.key; });
    } else {
        std::vector<HitKey> other(n);
        for (int shift = 0; shift < width; shift += 8) {
            size_t at[257] = {0};
            for (const HitKey &k : keys) ++at[(k.key >> shift & 255) + 1];
            for (int d = 0; d < 256; ++d) at[d + 1] += at[d];
            for (const HitKey &k : keys) other[at[k.key >> shift & 255]++] = k;
            keys.swap(other);
        }
    }
    for (size_t i = 0; i < n; ++i) order[i] = keys[i].idx;
    return order;
}

}  // namespace

extern "C" epi_status epi_scan(epi_ctx *ctx, const epi_block *blocks, int32_t nblocks, const epi_scan_opts *opts,
                               epi_hit *hits, int64_t cap, int64_t *nhits, int32_t *hit_block, int32_t *hit_trait,
                               float *max_f, float *max_f2)
{
    if (!ctx) return EPI_E_INVALID;
    ctx->err.clear();
    if (ctx->nid == 0 || ctx->ntraits == 0)
        return set_err(ctx, EPI_E_STATE, "epi_scan: load genotypes and traits first");
    if (nblocks < 0 || (nblocks > 0 && !blocks)) return set_err(ctx, EPI_E_INVALID, "epi_scan: bad blocks");
    if (cap < 0 || (cap > 0 && !hits)) return set_err(ctx, EPI_E_INVALID, "epi_scan: bad hit buffer");
    epi_status s = check_opts(ctx, opts);
    if (s != EPI_OK) return s;
    CK(cudaSetDevice(ctx->device));
    int variant = 0;
    std::string how;
    int64_t pairs = 0;
    for (int b = 0; b < nblocks; ++b) {
        const epi_block &e = blocks[b];
        if (e.size1 < 0 || e.size2 < 0 || e.start1 < 0 || e.start2 < 0 || (int64_t)e.start1 + e.size1 > ctx->nsnp ||
            (int64_t)e.start2 + e.size2 > ctx->nsnp)
            return set_err(ctx, EPI_E_INVALID, "block %d out of range", b);
        pairs += block_pairs(e);
    }
    double share = 0.0;
    ctx->overrun.begin();
    const bool plain = screens_plain(ctx, opts);
    int form = 0;
    int screen = plain || pick_form(ctx, opts) == EPI_FORM_TENSOR ? screen_digits(ctx, opts, (double)pairs, &share) : 0;
    ScanRun r;
    const auto prepare = [&]() {
        form = plain && screen ? EPI_FORM_TENSOR : pick_form(ctx, opts);
        epi_status st = pick_variant(ctx, opts, form, screen, &variant, &how);
        if (st == EPI_OK) st = setup_run(ctx, blocks, nblocks, opts, r, form, variant, screen, share);
        r.args.from_y = plain && screen;
        return st;
    };
    s = prepare();
    if ((s == EPI_E_NOMEM || s == EPI_E_UNSUPPORTED) && screen) {
        // no room for the candidates' list or the expanded rows: without a screen there is need of neither
        // (the variant that is asked for may stream B under the screen only)
        screen = 0;
        ctx->err.clear();
        s = prepare();
    }
    if (s != EPI_OK) return s;
    unsigned long long found = 0;
    bool again = false;
    for (int attempt = 0; attempt < 2; ++attempt) {
        r.args.hits = ctx->d_hits;
        r.args.cap = ctx->hit_cap;
        // the rescans, after a regrow or a list that ran over, are launched directly (one-off shapes)
        s = launch_run(ctx, r, nblocks, !opts->no_graph && !again);
        again = true;
        if (s != EPI_OK) return s;
        CK(cudaStreamSynchronize(ctx->stream));
        const unsigned long long *cnt = ctx->h_state;
        if (cnt[2] != 0)
            return set_err(ctx, EPI_E_TIMEOUT, "a bounded device wait of the scan kernel gave up (site %llu)",
                           cnt[3]);
        if (screen && cnt[epi::CNT_OVERFLOW] != 0) {
            // more candidates than the list holds: once more without a screen
            ctx->overrun.record(opts, (double)pairs * ctx->ntraits);
            screen = 0;
            s = prepare();
            if (s != EPI_OK) return s;
            attempt = -1;
            continue;
        }
        if (screen) ctx->overrun.held(opts, (double)pairs * ctx->ntraits);
        found = cnt[0];
        if ((int64_t)found <= ctx->hit_cap) break;
        // every hit is needed to put the first `cap` in output order: grow and rescan
        size_t hits_bytes = (size_t)ctx->hit_cap * sizeof(DevHit);
        ctx->hit_cap = 0;
        CK(ensure_own(&ctx->d_hits, &hits_bytes, (size_t)found * sizeof(DevHit), &ctx->own_hits));
        ctx->hit_cap = (int64_t)found;
    }
    float ms = 0.0f;
    CK(cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
    ctx->last_ms = ms;
    ctx->last_config = variant_desc(form, variant, screen) + " (" + how + ")";
    ctx->last_pairs = pairs * ctx->ntraits;

    const unsigned int *mx = reinterpret_cast<const unsigned int *>(ctx->h_state + epi::NCOUNTERS);
    // k_finish has brought the first hits; more come by a copy
    std::vector<DevHit> copied;
    const DevHit *dh = ctx->h_hits;
    if (found > epi::FINISH_HITS) {
        copied.resize((size_t)found);
        dh = copied.data();
        CK(cudaMemcpyAsync(copied.data(), ctx->d_hits, (size_t)found * sizeof(DevHit), cudaMemcpyDeviceToHost,
                           ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
    }
    for (int t = 0; t < ctx->ntraits; ++t) {
        if (max_f) max_f[t] = epi::ord2f(mx[t]);
        if (max_f2) max_f2[t] = opts->test == 'i' ? epi::ord2f(mx[ctx->ntraits + t]) : 0.0f;
    }

    const std::vector<uint32_t> order = output_order(dh, (size_t)found, blocks, nblocks, ctx->ntraits, opts);
    const int64_t nout = std::min<int64_t>((int64_t)found, cap);
    for (int64_t i = 0; i < nout; ++i) {
        const DevHit &h = dh[order[(size_t)i]];
        hits[i].snp1 = h.snp1;
        hits[i].snp2 = h.snp2;
        hits[i].df1 = h.df1;
        hits[i].df2 = h.df2;
        hits[i].F = h.F;
        hits[i].F2 = h.F2;
        if (hit_block) hit_block[i] = h.block;
        if (hit_trait) hit_trait[i] = h.trait;
    }
    if (nhits) *nhits = (int64_t)found;
    if ((int64_t)found > cap) return set_err(ctx, EPI_E_OVERFLOW, "%llu hits, capacity %lld", found, (long long)cap);
    return EPI_OK;
}

extern "C" epi_status epi_scan_dump(epi_ctx *ctx, const epi_block *block, const epi_scan_opts *opts, int32_t trait,
                                    int32_t *counts, float *F, float *F2, int32_t *df1, int32_t *df2)
{
    if (!ctx) return EPI_E_INVALID;
    ctx->err.clear();
    if (ctx->nid == 0 || ctx->ntraits == 0) return set_err(ctx, EPI_E_STATE, "epi_scan_dump: nothing loaded");
    if (!block) return set_err(ctx, EPI_E_INVALID, "epi_scan_dump: null block");
    if (trait < 0 || trait >= ctx->ntraits) return set_err(ctx, EPI_E_INVALID, "trait out of range");
    epi_scan_opts o = *opts;
    o.report_trait = trait;
    epi_status s = check_opts(ctx, &o);
    if (s != EPI_OK) return s;
    CK(cudaSetDevice(ctx->device));
    const int form = pick_form(ctx, &o);
    int variant = 0;
    std::string how;
    s = pick_variant(ctx, &o, form, 0, &variant, &how);
    if (s != EPI_OK) return s;
    ScanRun r;
    s = setup_run(ctx, block, 1, &o, r, form, variant, 0);
    if (s != EPI_OK) return s;
    const size_t np = (size_t)block->size1 * block->size2;
    int32_t *dc = nullptr, *dd1 = nullptr, *dd2 = nullptr;
    float *dF = nullptr, *dF2 = nullptr;
    struct Out { void *host; void **dev; size_t bytes; };
    Out outs[] = {{counts, (void **)&dc, np * 9 * sizeof(int32_t)}, {F, (void **)&dF, np * sizeof(float)},
                  {F2, (void **)&dF2, np * sizeof(float)}, {df1, (void **)&dd1, np * sizeof(int32_t)},
                  {df2, (void **)&dd2, np * sizeof(int32_t)}};
    epi_status st = EPI_OK;
    for (Out &x : outs) {
        if (!x.host || !np) continue;
        cudaError_t e = cudaMalloc(x.dev, x.bytes);
        if (e == cudaSuccess) e = cudaMemcpyAsync(*x.dev, x.host, x.bytes, cudaMemcpyHostToDevice, ctx->stream);
        if (e != cudaSuccess) { st = set_err(ctx, EPI_E_CUDA, "dump buffers: %s", cudaGetErrorString(e)); break; }
    }
    if (st == EPI_OK) {
        r.args.dump_counts = dc;
        r.args.dump_F = dF;
        r.args.dump_F2 = dF2;
        r.args.dump_df1 = dd1;
        r.args.dump_df2 = dd2;
        r.args.hits = ctx->d_hits;
        r.args.cap = 0;
        st = launch_run(ctx, r, 1, false);
    }
    if (st == EPI_OK) {
        cudaError_t e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) st = set_err(ctx, EPI_E_CUDA, "dump: %s", cudaGetErrorString(e));
        else if (ctx->h_state[2] != 0)
            st = set_err(ctx, EPI_E_TIMEOUT, "a bounded device wait gave up (site %llu)", ctx->h_state[3]);
    }
    if (st == EPI_OK) {
        for (Out &x : outs) {
            if (!x.host || !*x.dev) continue;
            cudaError_t e = cudaMemcpyAsync(x.host, *x.dev, x.bytes, cudaMemcpyDeviceToHost, ctx->stream);
            if (e != cudaSuccess) { st = set_err(ctx, EPI_E_CUDA, "dump readback: %s", cudaGetErrorString(e)); break; }
        }
        cudaError_t e = cudaStreamSynchronize(ctx->stream);
        if (st == EPI_OK && e != cudaSuccess) st = set_err(ctx, EPI_E_CUDA, "dump: %s", cudaGetErrorString(e));
    }
    for (Out &x : outs)
        if (*x.dev) cudaFree(*x.dev);
    return st;
}

extern "C" epi_status epi_scan_config(const epi_ctx *ctx, char *desc, int32_t len)
{
    if (!ctx || !desc || len < 1) return EPI_E_INVALID;
    snprintf(desc, (size_t)len, "%s", ctx->last_config.c_str());
    return EPI_OK;
}

extern "C" epi_status epi_get_stream(const epi_ctx *ctx, void **stream)
{
    if (!ctx || !stream) return EPI_E_INVALID;
    *stream = (void *)ctx->stream;
    return EPI_OK;
}

extern "C" epi_status epi_last_timing(const epi_ctx *ctx, double *kernel_ms, int64_t *pairs, int32_t *launches,
                                      int32_t *form)
{
    if (!ctx) return EPI_E_INVALID;
    if (form) *form = ctx->last_form;
    if (kernel_ms) *kernel_ms = ctx->last_ms;
    if (pairs) *pairs = ctx->last_pairs;
    if (launches) *launches = ctx->last_launches;
    return EPI_OK;
}
