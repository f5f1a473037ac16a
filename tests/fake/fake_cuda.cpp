// fake_cuda.cpp -- a CUDA runtime and a set of kernels that do nothing, for CPU tests of the
// library's host side (epi_capi.cu): device memory is a list of address ranges with a limit, any
// allocation can be made to fail, and every launch checks that the memory its arguments and tensor
// maps name is allocated and, for the expanded rows, holds what the kernel expects. A scan's
// outcome (the candidates it lists, overflows) is set by the test.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <cstring>
#include <algorithm>
#include <cstdlib>
#include <map>
#include <string>
#include <vector>

// names that the header's device functions use; none of them runs here
namespace epi {
static const struct { unsigned x; } threadIdx = {0};
using std::max;
using std::min;
template <class T> T __ldg(const T *p) { return *p; }
template <class T> T __shfl_sync(unsigned, T v, int) { return v; }
template <class T> T __shfl_xor_sync(unsigned, T v, int) { return v; }
template <class T, class U> T atomicAdd(T *p, U) { return *p; }
template <class T> T atomicMax(T *p, T) { return *p; }
inline unsigned __ballot_sync(unsigned, bool) { return 0; }
inline unsigned __brev(unsigned x) { return x; }
inline unsigned __byte_perm(unsigned x, unsigned, unsigned) { return x; }
inline unsigned __float_as_uint(float) { return 0; }
inline int __ffs(unsigned) { return 0; }
inline int __popc(unsigned) { return 0; }
}  // namespace epi
#include "epi_internal.cuh"

using epi::MmaMaps;
using epi::PopcMaps;
using epi::ScanArgs;

namespace {
std::map<uintptr_t, size_t> g_live;
std::map<uintptr_t, int> g_rows;  // expanded rows at this address: of which screen
uintptr_t g_next = 0x100000000ull;
size_t g_used = 0, g_limit = (size_t)180 << 30;
int g_fail_from = -1, g_mallocs = 0;  // allocations from this one on fail (-1: none)
std::string g_error;
double g_r1 = 0.5, g_r2 = 0.002, g_same = 1.0;
double g_rate = 0.0;  // share of a screened launch's pairs that it lists
int g_scans[4], g_exact, g_plain, g_captures;
double g_units[4];
std::map<const void *, std::string> &names()  // (filled while the library is being loaded)
{
    static std::map<const void *, std::string> m;
    return m;
}

void fault(const char *what, const void *p)
{
    char buf[160];
    snprintf(buf, sizeof(buf), "%s: %p is not allocated", what, p);
    if (g_error.empty()) g_error = buf;
}

void need(const char *what, const void *p, size_t bytes)
{
    auto it = g_live.upper_bound((uintptr_t)p);
    if (it == g_live.begin()) return fault(what, p);
    --it;
    if ((uintptr_t)p + bytes > it->first + it->second) fault(what, p);
}

struct Op {
    int kind;  // 0 scan, 1 exact, 2 finish, 3 plain
    int variant, screen;
    ScanArgs a;
    MmaMaps m;
    unsigned long long *counters;
    unsigned int *maxf;
    int ntraits;
    unsigned long long *out;
};
std::vector<Op> g_captured;
bool g_capturing = false, g_overflow = false;

int x_rows(int screen) { return screen == 3 ? 18 : screen ? 3 * (1 + screen) : 12; }
int x_sets(int screen, int t) { return screen == 3 ? (t + 4) / 5 : t; }
int tile_j(int screen) { return screen == 0 ? 21 : screen == 1 ? 42 : screen == 2 ? 28 : 14; }
bool needs_x(int v, int screen) { return v == 5 || (v == 2 && screen); }

const void *base(const CUtensorMap &m)
{
    const void *p;
    memcpy(&p, &m, sizeof(p));
    return p;
}

void run(const Op &o)
{
    const ScanArgs &a = o.a;
    const size_t T = a.ntraits, M = a.nsnp;
    if (o.kind == 0) {
        ++g_scans[o.screen];
        g_units[o.screen] += (double)a.seg_units;
        need("one-hot rows", a.hcodes, M * a.Np);
        need("indicator rows", base(o.m.hi), 3 * M * a.Np);
        need("missing bits", a.missbits, M * a.Wp * 4);
        need("digits", a.ydig, 5 * T * a.Np);
        need("missing sums", a.qm, T * M * 28);
        need("squares", a.qd, 2 * T * a.Np * 8);
        need("screen constants", a.tscr, 2 * T * 16);
        need("blocks", a.blocks, a.nblocks * sizeof(epi::BlockDesc));
        need("maxima", a.maxf, 4 * T * 4);
        if (a.cap) need("hits", a.hits, a.cap * sizeof(epi::DevHit));
        if (o.screen) need("candidates", a.cand, a.cand_cap * sizeof(epi::Cand));
        if (needs_x(o.variant, o.screen)) {
            need("expanded rows", base(o.m.hx), (size_t)x_rows(o.screen) * M * a.Np * x_sets(o.screen, a.ntraits));
            const auto it = g_rows.find((uintptr_t)base(o.m.hx));
            if ((it == g_rows.end() || it->second != o.screen) && g_error.empty()) g_error = "expanded rows of another screen";
        }
        const double per = o.screen == 3 ? 5.0 : 1.0;
        if (o.screen && g_rate * (double)a.seg_units * 80.0 * tile_j(o.screen) * per > (double)a.cand_cap) g_overflow = true;
    } else if (o.kind == 1) {
        ++g_exact;
    } else if (o.kind == 3) {
        ++g_plain;
        need("planes", a.planes, M * a.Wp * 16);
        need("marginals", a.pmC, 3 * T * M * 8);
        need("maxima", a.maxf, 4 * T * 4);
        need("blocks", a.blocks, a.nblocks * sizeof(epi::BlockDesc));
    } else {
        need("counters", o.counters, epi::NCOUNTERS * 8);
        need("maxima", o.maxf, 4 * (size_t)o.ntraits * 4);
        memset(o.out, 0, epi::NCOUNTERS * 8 + 8 * (size_t)o.ntraits);
        o.out[epi::CNT_OVERFLOW] = g_overflow;
        g_overflow = false;
    }
}

cudaError_t submit(const Op &o)
{
    if (g_capturing) g_captured.push_back(o);
    else run(o);
    return cudaSuccess;
}
}  // namespace

// ---- the test's side ----
extern "C" {
void fake_reset()
{
    g_limit = (size_t)180 << 30;
    g_fail_from = -1;
    g_error.clear();
    g_r1 = 0.5;
    g_r2 = 0.002;
    g_same = 1.0;
    g_rate = 0.0;
}
void fake_limit(size_t bytes) { g_limit = bytes; }
size_t fake_used() { return g_used; }
void fake_fail_after(int n)  // the next n allocations succeed, those after them fail (-1: none fails)
{
    g_fail_from = n < 0 ? -1 : g_mallocs + n;
}
void fake_traits(double r1, double r2, double same) { g_r1 = r1, g_r2 = r2, g_same = same; }
void fake_rate(double rate) { g_rate = rate; }
const char *fake_error() { return g_error.c_str(); }
void fake_count(int *out)  // launches since the last call: per screen 0-3, exact, plain, graph captures
{
    for (int k = 0; k < 4; ++k) out[k] = g_scans[k], g_scans[k] = 0;
    out[4] = g_exact, out[5] = g_plain, out[6] = g_captures;
    g_exact = g_plain = g_captures = 0;
}

// ---- runtime ----
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int)
{
    *v = a == cudaDevAttrComputeCapabilityMajor ? 10 : 148;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp *, int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaMalloc(void **p, size_t bytes)
{
    const int n = g_mallocs++;
    if ((g_fail_from >= 0 && n >= g_fail_from) || g_used + bytes > g_limit) return cudaErrorMemoryAllocation;
    *p = (void *)g_next;
    g_live[g_next] = bytes;
    g_next += (bytes + 0xfffff) & ~(size_t)0xfffff;
    g_next += 0x100000;
    g_used += bytes;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p)
{
    if (!p) return cudaSuccess;
    const auto it = g_live.find((uintptr_t)p);
    if (it == g_live.end()) {
        fault("cudaFree", p);
        return cudaErrorInvalidValue;
    }
    g_used -= it->second;
    g_live.erase(it);
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t *fr, size_t *tot)
{
    *tot = g_limit;
    *fr = g_limit > g_used ? g_limit - g_used : 0;
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t)
{
    if (k == cudaMemcpyHostToDevice) need("copy to the device", d, n);
    else {
        need("copy from the device", s, n);
        memset(d, 0, n);
    }
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode)
{
    g_capturing = true;
    g_captured.clear();
    ++g_captures;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g)
{
    g_capturing = false;
    *g = (cudaGraph_t) new std::vector<Op>(g_captured);
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long)
{
    *x = (cudaGraphExec_t) new std::vector<Op>(*(std::vector<Op> *)g);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete (std::vector<Op> *)g; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t g) { delete (std::vector<Op> *)g; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t g, cudaStream_t)
{
    for (const Op &o : *(std::vector<Op> *)g) run(o);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3, dim3, void **args, size_t, cudaStream_t)
{
    const std::string &name = names()[f];
    if (name.find("k_finish") != std::string::npos) {
        Op o = {};
        o.kind = 2;
        o.counters = *(unsigned long long **)args[0];
        o.maxf = *(unsigned int **)args[1];
        o.ntraits = *(int *)args[2];
        o.out = *(unsigned long long **)args[5];
        return submit(o);
    }
    if (name.find("k_scan_init") != std::string::npos)
        need("maxima", *(unsigned int **)args[1], 4 * (size_t) * (int *)args[2]);
    else if (g_error.empty()) g_error = "unknown kernel " + name;
    return cudaSuccess;
}

// (what nvcc's host code calls to register and to launch kernels)
static dim3 s_grid, s_block;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t, cudaStream_t)
{
    s_grid = g, s_block = b;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *sh, void *st)
{
    *g = s_grid, *b = s_block, *sh = 0, *(void **)st = nullptr;
    return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *, int *)
{
    names()[host] = name;
}
}

// ---- kernels ----
namespace epi {
cudaError_t launch_unpack(const int32_t *raw, int nsnp, int nid, int, int, uint4 *planes, int Wp, uint32_t *, int,
                          uint8_t *hcodes, uint8_t *h3, uint32_t *missbits, cudaStream_t)
{
    need("packed words", raw, (size_t)nsnp * ((nid + 15) / 16) * 4);
    need("planes", planes, (size_t)nsnp * Wp * 16);
    need("one-hot rows", hcodes, (size_t)nsnp * Wp * 32);
    need("indicator rows", h3, 3 * (size_t)nsnp * Wp * 32);
    need("missing bits", missbits, (size_t)nsnp * Wp * 4);
    return cudaSuccess;
}
cudaError_t launch_qmiss(const uint32_t *, int nsnp, int, const uint32_t *wmask, const double *, const double *, int, int T,
                        double *qm, double *, double *, float *qmf, cudaStream_t)
{
    need("valid bits", wmask, 4);
    need("missing sums", qm, (size_t)T * nsnp * 8);
    need("missing sums", qmf, (size_t)T * nsnp * 4);
    return cudaSuccess;
}
cudaError_t launch_traits(const float *y, const uint8_t *, int, int nid, int, int T, const TraitArrays &, TraitInfo *info,
                          cudaStream_t)
{
    need("phenotypes", y, (size_t)T * nid * 4);
    for (int t = 0; t < T; ++t) info[t] = {(double)nid, g_r1, g_r2, t == 0 ? 1.0 : g_same};
    return cudaSuccess;
}
cudaError_t launch_major(const uint4 *, int nsnp, int, uint8_t *maj, cudaStream_t)
{
    need("most frequent genotypes", maj, nsnp);
    return cudaSuccess;
}
cudaError_t launch_marg(const uint4 *planes, int nsnp, int Wp, const float *, const uint32_t *, int, int T, double *pmC,
                        int32_t *, double *, cudaStream_t)
{
    need("planes", planes, (size_t)nsnp * Wp * 16);
    need("marginals", pmC, 3 * (size_t)T * nsnp * 8);
    return cudaSuccess;
}
int popc_shapes() { return 3; }
void popc_shape(int, int *ti, int *tj, const char **desc)
{
    *ti = 32, *tj = 64;
    if (desc) *desc = "fake";
}
cudaError_t popc_prepare(int) { return cudaSuccess; }
cudaError_t popc_enqueue(int v, const ScanArgs &a, const PopcMaps &, int, cudaStream_t)
{
    Op o = {};
    o.kind = 3, o.variant = v, o.a = a;
    return submit(o);
}
cudaError_t popc_encode_planes(int, PopcMaps *, const uint4 *, int, int) { return cudaSuccess; }
bool mma_available() { return true; }
int mma_tile_i() { return 80; }
int mma_tile_j(int screen) { return tile_j(screen); }
int mma_x_rows(int screen) { return x_rows(screen); }
int mma_x_sets(int screen, int t) { return x_sets(screen, t); }
int mma_min_nid() { return 64; }
int mma_max_nid() { return 1 << 24; }
int mma_screen_max_nid() { return 32640; }
int mma_shapes() { return 6; }
void mma_shape(int, int, const char **desc) { if (desc) *desc = "fake"; }
cudaError_t mma_prepare(int, int, int, int g, int *grid) { *grid = g; return cudaSuccess; }
cudaError_t mma_enqueue(int v, int screen, const ScanArgs &a, const MmaMaps &m, int, cudaStream_t)
{
    Op o = {};
    o.kind = 0, o.variant = v, o.screen = screen, o.a = a, o.m = m;
    return submit(o);
}
cudaError_t exact_enqueue(const ScanArgs &, int, cudaStream_t)
{
    Op o = {};
    o.kind = 1;
    return submit(o);
}
static cudaError_t set(CUtensorMap &m, const void *p) { memset(&m, 0, sizeof(m)); memcpy(&m, &p, sizeof(p)); return cudaSuccess; }
cudaError_t mma_encode_genotypes(MmaMaps *m, const uint8_t *hcodes, const uint8_t *h3, int, int)
{
    set(m->hj, hcodes);
    return set(m->hi, h3);
}
cudaError_t mma_encode_traits(MmaMaps *m, const int8_t *ydig, int, int) { return set(m->dg, ydig); }
cudaError_t mma_encode_x(MmaMaps *m, const int8_t *x, int, int, int, int) { return set(m->hx, x); }
bool mma_needs_x(int v, int screen) { return needs_x(v, screen); }
cudaError_t launch_expand(const uint8_t *hcodes, const int8_t *, int nsnp, int Np, int T, int screen, int8_t *x, cudaStream_t)
{
    need("one-hot rows", hcodes, (size_t)nsnp * Np);
    need("expanded rows", x, (size_t)x_rows(screen) * nsnp * Np * x_sets(screen, T));
    g_rows[(uintptr_t)x] = screen;
    return cudaSuccess;
}
}  // namespace epi
