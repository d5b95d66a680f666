/* Test driver for the library's host code without a GPU: the library's own
 * objects linked against the CUDA runtime below, which keeps device memory on
 * the host, records function attributes per device, can make a chosen call
 * fail, and in place of the freezeout kernels does what the host code sees of
 * them (the header, the crossed-cube counter, the rows).  One scenario per
 * process, named on the command line; exits 0 where every expectation holds. */
#define __CUDADEVRT_INTERNAL__     /* no declarations of the device-side runtime */
#include <cuda_runtime.h>
#include <algorithm>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <thread>
#include <vector>
#include "vh_b200.h"
#include "vh_kernels.h"

#ifndef __CUDA_ARCH__
namespace {
std::mutex mu;
std::map<const void *, std::string> names;                  /* host stub -> kernel name */
std::map<std::pair<int, const void *>, int> smem_limit;     /* (device, kernel) -> opt-in bytes */
thread_local int device = 0;
thread_local cudaError_t last = cudaSuccess;
int launches = 0;
/* fail the call number fail_at (from 0) of those counted, if counting */
bool counting = false;
int fail_at = -1, counted = 0;
std::string fail_kernel;                                     /* the next launch of a kernel of this name fails */
std::string small_attr;                                      /* opt-ins of kernels of this name to 48-56 KB are slow */
/* the freezeout stand-ins */
int block_total = 0, block_value = 0;
int *hdr = nullptr;                                          /* the last block's header */
bool null_store = false, list_overrun = false;
std::set<void *> live;                                       /* allocations not yet freed */

cudaError_t ret(cudaError_t e) { if (e != cudaSuccess) last = e; return e; }
bool refuse() { std::lock_guard<std::mutex> lk(mu); return counting && counted++ == fail_at; }
cudaError_t grab(void **p, size_t n)
{
    if (refuse()) return ret(cudaErrorMemoryAllocation);
    *p = calloc(n ? n : 1, 1);
    std::lock_guard<std::mutex> lk(mu);
    live.insert(*p);
    return cudaSuccess;
}
cudaError_t drop(void *p)
{
    std::lock_guard<std::mutex> lk(mu);
    live.erase(p);
    free(p);
    return cudaSuccess;
}

cudaError_t launch(const void *f, size_t smem, void **args)
{
    std::lock_guard<std::mutex> lk(mu);
    const std::string &n = names[f];
    auto is = [&](const char *k) { return n.find(k) != std::string::npos; };
    ++launches;
    auto it = smem_limit.find({device, f});
    if (smem > 48 * 1024 && (it == smem_limit.end() || (size_t)it->second < smem)) return ret(cudaErrorInvalidValue);
    if (!fail_kernel.empty() && is(fail_kernel.c_str())) { fail_kernel.clear(); return ret(cudaErrorLaunchOutOfResources); }
    if (is("fo_open_kernel")) {
        const vh::FoArgs &a = *(const vh::FoArgs *)args[0];
        if (!a.counts || !a.slab_cur) { null_store = true; return cudaSuccess; }
        hdr = a.counts + vh::freezeout_scratch_ints(a.nx, a.ny, a.nz) - vh::kFoHeaderInts;
        const int cubes = (a.nx - 1) * (a.ny - 1) * (a.nz > 1 ? a.nz - 1 : 1);
        hdr[0] += cubes;                                     /* every cube is crossed */
        if (hdr[0] > cubes) list_overrun = true;
    } else if (is("fo_offsets_kernel")) {
        int *host = *(int **)args[1];
        if (!host || !hdr) { null_store = true; return cudaSuccess; }
        host[0] = 1;
        host[1] = block_total;
        hdr[0] = hdr[1] = 0;
    } else if (is("fo_emit_kernel")) {
        const vh::FoArgs &a = *(const vh::FoArgs *)args[0];
        if (!a.elems || !a.host_elems || (!a.slots && a.slot_cap > 0)) { null_store = true; return cudaSuccess; }
        for (int i = 0; i < block_total * VH_FO_COLUMNS; ++i) {
            if (i < a.cap * VH_FO_COLUMNS) a.elems[i] = block_value;
            if (i < std::min(a.cap, a.host_cap) * VH_FO_COLUMNS) a.host_elems[i] = block_value;
        }
    }
    return cudaSuccess;
}

struct Config { dim3 g, b; size_t smem; cudaStream_t s; };
thread_local std::vector<Config> configs;
} // namespace

extern "C" {
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *, int *)
{
    names[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st *s)
{
    configs.push_back({g, b, smem, s});
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *s)
{
    const Config c = configs.back();
    configs.pop_back();
    *g = c.g; *b = c.b; *smem = c.smem; *(cudaStream_t *)s = c.s;
    return cudaSuccess;
}
cudaError_t CUDARTAPI cudaLaunchKernel(const void *f, dim3, dim3, void **args, size_t smem, cudaStream_t) { return launch(f, smem, args); }
cudaError_t CUDARTAPI cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args) { return launch(f, c->dynamicSmemBytes, args); }
cudaError_t CUDARTAPI cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v)
{
    if (a != cudaFuncAttributeMaxDynamicSharedMemorySize) return cudaSuccess;
    bool late;
    {
        std::lock_guard<std::mutex> lk(mu);
        late = !small_attr.empty() && v > 48 * 1024 && v < 56 * 1024 && names[f].find(small_attr) != std::string::npos;
    }
    if (late) std::this_thread::sleep_for(std::chrono::milliseconds(200));
    {
        std::lock_guard<std::mutex> lk(mu);
        smem_limit[{device, f}] = v;
    }
    if (late) std::this_thread::sleep_for(std::chrono::milliseconds(200));
    return cudaSuccess;
}
cudaError_t CUDARTAPI cudaFuncGetAttributes(cudaFuncAttributes *a, const void *) { memset(a, 0, sizeof *a); return cudaSuccess; }
cudaError_t CUDARTAPI cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) { *n = 2; return cudaSuccess; }
cudaError_t CUDARTAPI cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
cudaError_t CUDARTAPI cudaSetDevice(int d) { device = d; return cudaSuccess; }
cudaError_t CUDARTAPI cudaGetDeviceCount(int *n) { *n = 2; return cudaSuccess; }
cudaError_t CUDARTAPI cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t CUDARTAPI cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char *CUDARTAPI cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t CUDARTAPI cudaMalloc(void **p, size_t n) { return grab(p, n); }
cudaError_t CUDARTAPI cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t, cudaStream_t) { return grab(p, n); }
cudaError_t CUDARTAPI cudaHostAlloc(void **p, size_t n, unsigned) { return grab(p, n); }
cudaError_t CUDARTAPI cudaMallocHost(void **p, size_t n) { return grab(p, n); }
cudaError_t CUDARTAPI cudaFree(void *p) { return drop(p); }
cudaError_t CUDARTAPI cudaFreeAsync(void *p, cudaStream_t) { return drop(p); }
cudaError_t CUDARTAPI cudaFreeHost(void *p) { return drop(p); }
cudaError_t CUDARTAPI cudaMemGetInfo(size_t *f, size_t *t) { *f = *t = (size_t)1 << 34; return cudaSuccess; }
cudaError_t CUDARTAPI cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps *) { *p = nullptr; return cudaSuccess; }
cudaError_t CUDARTAPI cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t CUDARTAPI cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t)
{
    if (!d || !s) return ret(cudaErrorInvalidValue);
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t CUDARTAPI cudaMemset(void *p, int v, size_t n) { memset(p, v, n); return cudaSuccess; }
cudaError_t CUDARTAPI cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t)
{
    if (refuse()) return ret(cudaErrorInvalidValue);
    memset(p, v, n);
    return cudaSuccess;
}
cudaError_t CUDARTAPI cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = (cudaStream_t)&live; return cudaSuccess; }
cudaError_t CUDARTAPI cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { *g = nullptr; return cudaSuccess; }
cudaError_t CUDARTAPI cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) { *e = nullptr; return cudaSuccess; }
cudaError_t CUDARTAPI cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)&live; return cudaSuccess; }
cudaError_t CUDARTAPI cudaEventCreateWithFlags(cudaEvent_t *e, unsigned)
{
    if (refuse()) return ret(cudaErrorMemoryAllocation);
    *e = (cudaEvent_t)&live;
    return cudaSuccess;
}
cudaError_t CUDARTAPI cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaEventElapsedTime(float *t, cudaEvent_t, cudaEvent_t) { *t = 0; return cudaSuccess; }
cudaError_t CUDARTAPI cudaGetSymbolAddress(void **p, const void *) { static int mem[1 << 19]; *p = mem; return cudaSuccess; }
cudaError_t CUDARTAPI cudaGetDriverEntryPoint(const char *, void **, unsigned long long, cudaDriverEntryPointQueryResult *) { return ret(cudaErrorInvalidValue); }
}

namespace {
int failures = 0;
void expect(bool ok, const char *what)
{
    if (ok) return;
    ++failures;
    printf("FAILED: %s (%s)\n", what, vh_last_error());
}

vh_event *make(int nx, int ny, int nz)
{
    vh_config c = {};
    c.nx = nx; c.ny = ny; c.nz = nz;
    c.dx = c.dy = 0.3; c.dz = 0.3; c.dt = 0.02; c.t0 = 0.6; c.etabar = 0.1;
    c.T_freezeout_GeV = 0.15; c.T_reg_GeV = 0.1; c.fo_factor = 2; c.theta = 1.8;
    c.eos_kind = VH_EOS_TABLE; c.bulk = 1; c.precision = VH_PREC_FP64;
    std::vector<double> rows;                                /* e, p, s, T */
    for (int i = 0; i < 200; ++i) {
        const double e = 0.05 * i;
        rows.insert(rows.end(), {e, e / 3.0, 0.0, 0.1 + 0.01 * i});
    }
    vh_event *ev = nullptr;
    expect(vh_event_create(&c, rows.data(), 200, &ev) == VH_OK, "create");
    const size_t N = (size_t)nx * ny * nz;
    std::vector<double> e(N, 1.0), u(4 * N, 0.0);
    for (size_t i = 0; i < N; ++i) u[i] = 1.0;
    expect(vh_event_set_initial(ev, e.data(), e.data(), u.data(), nullptr, nullptr) == VH_OK, "set_initial");
    return ev;
}

/* a block of n rows of this value, fetched */
void good_block(vh_event *ev, int n, int value)
{
    block_total = n;
    block_value = value;
    int got = -1, above = -1;
    expect(vh_event_freezeout(ev, &got, &above) == VH_OK, "block");
    expect(got == n, "the block's count");
    std::vector<double> rows((size_t)n * VH_FO_COLUMNS, -1.0);
    expect(vh_event_fetch_surface(ev, rows.data(), n, &got) == VH_OK && got == n, "fetch");
    for (double r : rows)
        if (r != value) { expect(false, "the block's rows"); break; }
}

/* a failed call is reported once: the next one, which succeeds, does not
 * report it again */
void error_cleared()
{
    vh_event *ev = make(9, 8, 1);
    auto fails = [&](const char *what, auto call) {
        counting = true; counted = 0; fail_at = 0;
        const int rc = call();
        counting = false;
        expect(rc != VH_OK, what);
        expect(vh_event_step(ev, 1) == VH_OK, what);
    };
    fails("regulation factors", [&] { return vh_event_keep_regulation(ev, 1); });
    fails("vorticity", [&] { return vh_event_vorticity(ev, 1); });
    fails("another event", [&] {
        vh_config c = {};
        c.nx = c.ny = 5; c.nz = 1; c.dx = c.dy = c.dz = c.dt = c.t0 = 0.5; c.theta = 1; c.eos_kind = VH_EOS_TABLE;
        const double rows[8] = {0, 0, 0, 0.1, 1, 0.3, 0, 0.2};
        vh_event *x = nullptr;
        return vh_event_create(&c, rows, 2, &x);
    });
    fails("batch", [&] { vh_batch *b = nullptr; return vh_batch_create(&ev, 1, &b); });
    fails("Cornelius service", [&] {
        const double cube[8] = {0, 1, 0, 1, 0, 1, 0, 1}, dx[3] = {1, 1, 1};
        double el[60];
        int n = 0, count = 0;
        return vh_cornelius_surfaces(3, cube, 1, 0.5, dx, el, 10, &count, &n);
    });
    vh_event_destroy(ev);
}

/* a first block whose set-up fails at its k-th step launches nothing and
 * leaves nothing allocated; the next call sets up again */
void setup_rollback()
{
    for (int k = 0; k < 64; ++k) {
        vh_event *ev = make(9, 8, 1);
        const size_t before = live.size();
        const int l0 = launches;
        counting = true; counted = 0; fail_at = k;
        block_total = 3; block_value = 7;
        const int rc = vh_event_freezeout(ev, nullptr, nullptr);
        counting = false;
        if (rc == VH_OK) {
            expect(k >= 8, "every step of the set-up was failed once");
            expect(counted <= k, "a failed step was reported");
            vh_event_destroy(ev);
            break;
        }
        expect(launches == l0, "no kernel after a failed set-up");
        expect(live.size() == before, "a failed set-up gives its memory back");
        good_block(ev, 5, k + 1);
        expect(!null_store, "kernels get every buffer");
        expect(!list_overrun, "the crossed-cube counter starts at zero");
        vh_event_destroy(ev);
    }
}

/* the element buffer cannot grow: neither that block nor the one before it
 * can be read any more, and later blocks are whole again */
void regrow_failure()
{
    setenv("VH_FO_INITIAL_CAP", "4", 1);
    vh_event *ev = make(9, 8, 1);
    good_block(ev, 3, 1);
    block_total = 10; block_value = 2;
    expect(vh_event_freezeout_launch(ev) == VH_OK, "launch");
    counting = true; counted = 0; fail_at = 0;
    expect(vh_event_freezeout_finish(ev, nullptr, nullptr) != VH_OK, "the failed growth is reported");
    counting = false;
    std::vector<double> rows(20 * VH_FO_COLUMNS, -1.0);
    int n = 0;
    expect(vh_event_fetch_surface(ev, rows.data(), 20, &n) != VH_OK, "lost rows are not handed out");
    good_block(ev, 2, 3);
    good_block(ev, 12, 4);
    expect(!null_store, "kernels get every buffer");
    vh_event_destroy(ev);
}

/* a block of whose four kernels one cannot be launched reports it, and the
 * next block starts from a clean header */
void chain_failure()
{
    for (const char *k : {"fo_open_kernel", "fo_count3_kernel", "fo_offsets_kernel", "fo_emit_kernel"}) {
        vh_event *ev = make(9, 8, 1);
        good_block(ev, 3, 1);
        fail_kernel = k;
        expect(vh_event_freezeout_launch(ev) != VH_OK, "the failed launch is reported");
        good_block(ev, 4, 2);
        expect(!list_overrun, "the crossed-cube counter starts at zero");
        vh_event_destroy(ev);
    }
}

void step(vh_event *ev, const char *what) { expect(vh_event_step(ev, 2) == VH_OK, what); }

/* short lines need more than 48 KB: on every device, in any order of lengths */
void opt_in_devices()
{
    for (int d : {0, 1}) {
        cudaSetDevice(d);
        vh_event *a = make(41, 37, 5), *b = make(41, 37, 9), *c = make(21, 19, 4);
        step(b, "longer lines");
        step(a, "short lines");
        step(b, "longer lines again");
        block_total = 2;
        expect(vh_event_freezeout(c, nullptr, nullptr) == VH_OK, "3+1D block");
        for (vh_event *e : {a, b, c}) vh_event_destroy(e);
    }
}

/* the smaller of two first opt-ins, made at the same time, takes effect last */
void opt_in_threads()
{
    vh_event *a = make(41, 37, 5), *b = make(41, 37, 9);
    small_attr = "kt_flux_lines_kernel";
    std::thread tb([&] { step(b, "longer lines"); });
    std::this_thread::sleep_for(std::chrono::milliseconds(100));
    step(a, "short lines");
    std::this_thread::sleep_for(std::chrono::milliseconds(200));
    step(a, "short lines again");
    tb.join();
    small_attr.clear();
    step(b, "longer lines again");
    vh_event_destroy(a);
    vh_event_destroy(b);
}

/* a batch created later with longer lines leaves the earlier one's opt-in */
void opt_in_batches()
{
    vh_event *a = make(41, 37, 5), *b = make(41, 37, 20);
    vh_batch *ba = nullptr, *bb = nullptr;
    expect(vh_batch_create(&a, 1, &ba) == VH_OK, "batch of short lines");
    expect(vh_batch_create(&b, 1, &bb) == VH_OK, "batch of longer lines");
    expect(vh_batch_step(bb, 1) == VH_OK, "longer lines");
    expect(vh_batch_step(ba, 1) == VH_OK, "short lines");
    vh_batch_destroy(ba);
    vh_batch_destroy(bb);
    vh_event_destroy(a);
    vh_event_destroy(b);
}
} // namespace

int main(int argc, char **argv)
{
    const std::map<std::string, void (*)()> all = {
        {"error_cleared", error_cleared},
        {"setup_rollback", setup_rollback}, {"regrow_failure", regrow_failure}, {"chain_failure", chain_failure},
        {"opt_in_devices", opt_in_devices}, {"opt_in_threads", opt_in_threads}, {"opt_in_batches", opt_in_batches}};
    auto it = argc > 1 ? all.find(argv[1]) : all.end();
    if (it == all.end()) return 2;
    it->second();
    return failures ? 1 : 0;
}
#endif
