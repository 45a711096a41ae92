// extern "C" entry points of the displacement backend (include/disco_b200.h):
// device queries, plans (tables built and uploaded once), the resident
// execute and the host-buffer drop-in that replaces kroupaGPU
// (Code/backend_cuda.cu:568-722).
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <exception>
#include <mutex>
#include <string>
#include <vector>

#include <cuda.h>
#include <cuda_runtime.h>

#include "common.cuh"
#include "field.cuh"
#include "tree.cuh"

namespace disco {
int choose_split(int64_t n, int nimg, int resident_ctas);
int launch_field_fp32(const FieldArgs& a, int kind, int sm_count, int split_hint,
                      cudaStream_t stream, std::string& err);
}

struct disco_plan {
    int device = 0;
    int sm_count = 0;
    double box[3] = { 0., 0., 0. };
    disco_options opt;
    int nimg = 1;
    int nloops = 0;
    disco::HostTable tables[2];              // line, loopon
    // one block of device memory: the image (status word, tables, chunk lists;
    // plan_image) and behind it the FP32 line form's list of atoms with near-cut
    // pairs
    size_t table_at[2] = { 0, 0 }, chunks_at[2] = { 0, 0 }, image_bytes = 0, near_at = 0, bytes = 0;
    unsigned char* block = nullptr;          // owned where `own`: cudaMalloc'd, or from the
    bool own = false, pooled = false;        // scratch pool in the order of `stream`
    cudaStream_t stream = nullptr;
    unsigned char* d_table[2] = { nullptr, nullptr };
    disco::Chunk* d_chunks[2] = { nullptr, nullptr };
    int* d_status = nullptr;
    int32_t* d_near = nullptr;
    unsigned int* d_near_count = nullptr;
    int32_t near_cap = 0;
    std::vector<double> loop_evals;          // per input loop: segments or loopons
    disco_plan_stats stats;
    // the sum by cells: its shape for the last atom count, and the context
    // whose scratch pool this plan holds (0: none); both set by execute
    std::mutex tree_mutex;
    int64_t tree_n[2] = { -1, -1 };
    disco::TreeShape tree[2];
    unsigned long long tree_pool = 0;
};

namespace {

// Last error message of the calling thread: a fixed buffer, so that setting it
// never allocates.
thread_local char g_last_error[512];

void store_error(const char* msg)
{
    std::snprintf(g_last_error, sizeof(g_last_error), "%s", msg);
}

int fail(int code, const std::string& msg)
{
    store_error(msg.c_str());
    return code;
}

int cuda_fail(cudaError_t e, const char* what)
{
    return fail(e == cudaErrorMemoryAllocation ? DISCO_ENOMEM : DISCO_ECUDA,
                std::string(what) + ": " + cudaGetErrorString(e));
}

#define DISCO_TRY_CUDA(call, what)                     \
    do {                                               \
        cudaError_t e_ = (call);                       \
        if (e_ != cudaSuccess) return cuda_fail(e_, what); \
    } while (0)

int check_options(const disco_options& o)
{
    if (o.precision != DISCO_FP64 && o.precision != DISCO_FP32C)
        return fail(DISCO_EINVAL, "precision must be DISCO_FP64 or DISCO_FP32C");
    if (o.images < 0 || o.images > 8) return fail(DISCO_EINVAL, "images must be in 0..8");
    if (o.image_min < 0 || o.image_min > o.images) return fail(DISCO_EINVAL, "image_min must be in 0..images");
    if (!(o.nu > -1.0 && o.nu < 0.5)) return fail(DISCO_EINVAL, "nu must be in (-1, 0.5)");
    if (!(o.near_plane >= 0.0) || !(o.near_rim >= 0.0))
        return fail(DISCO_EINVAL, "near_plane and near_rim must be >= 0");
    if (o.stage_kb != 0 && (o.stage_kb < 16 || o.stage_kb > 100))
        return fail(DISCO_EINVAL, "stage_kb must be 0 or in 16..100");
    if (o.image_split != 0 && (o.image_split < 1 || o.image_split > 32 ||
                               (o.image_split & (o.image_split - 1))))
        return fail(DISCO_EINVAL, "image_split must be 0 or a power of two up to 32");
    return DISCO_OK;
}

void free_plan(disco_plan* p)
{
    if (!p) return;
    if (p->own && p->block && p->pooled) cudaFreeAsync(p->block, p->stream);
    else if (p->own && p->block) cudaFree(p->block);
    if (p->tree_pool) disco::scratch_release(p->device, p->tree_pool);
    delete p;
}

// The shape of the sum by cells for n atoms; use = false: sum directly.  A
// caller's own image split names the direct kernel, a stream under capture
// keeps to it (its launches allocate nothing), and so does a sum over far
// shells alone (image_min > 0): that is the term-by-term sum the learned form
// is measured and tested against, in error and in time.
disco::TreeShape plan_shape(disco_plan* p, int k, int64_t n)
{
    disco::TreeShape none;
    if (!p->tables[k].aux_tree || p->opt.image_split != 0 || p->opt.image_min > 0) return none;
    std::lock_guard<std::mutex> lock(p->tree_mutex);
    if (p->tree_n[k] != n) {
        try {
            p->tree[k] = disco::tree_shape(p->tables[k], n, p->box, p->opt.images, p->sm_count);
        } catch (const std::exception&) {        // no host memory for the choice: the plain kernel needs none
            return none;
        }
        p->tree_n[k] = n;
    }
    return p->tree[k];
}

disco::TreeShape plan_tree(disco_plan* p, int k, int64_t n, cudaStream_t s)
{
    disco::TreeShape none;
    if (!p->tables[k].aux_tree) return none;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap) != cudaSuccess) { cudaGetLastError(); return none; }
    if (cap != cudaStreamCaptureStatusNone) return none;
    const disco::TreeShape shape = plan_shape(p, k, n);
    if (shape.use) {
        std::lock_guard<std::mutex> lock(p->tree_mutex);
        if (!p->tree_pool) p->tree_pool = disco::scratch_retain(p->device);
    }
    return shape;
}

double now_s()
{
    using C = std::chrono::steady_clock;
    return std::chrono::duration<double>(C::now().time_since_epoch()).count();
}

} // namespace

namespace {

constexpr uint64_t kScratchKeep = 32ull << 20, kScratchKeepPlans = 1024ull << 20;

// The scratch pools, one per device and context (two contexts of a device do
// not share one; the memory of a context that is gone went with it, and its
// entry stays).
struct ScratchPool { int device; unsigned long long ctx; cudaMemPool_t pool; int plans; };
std::mutex g_scratch_mutex;
std::vector<ScratchPool> g_scratch;

// Idle non-blocking streams of host calls, at most four: making and destroying
// one costs 0.12 ms, more than such a call's copies.
struct IdleStream { cudaStream_t stream; int device; unsigned long long ctx; };
constexpr size_t kIdleStreams = 4;
std::mutex g_idle_mutex;
std::vector<IdleStream> g_idle;

using CtxGetCurrentFn = CUresult (*)(CUcontext*);
using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long*);

void scratch_keep(cudaMemPool_t pool, uint64_t bytes)
{
    if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &bytes) != cudaSuccess) cudaGetLastError();
}

// Identifier of the calling thread's context; a thread that has none yet gets
// the device's primary one.
unsigned long long bound_context_id()
{
    unsigned long long id = disco::current_context_id();
    if (id == 0 && cudaFree(nullptr) == cudaSuccess) id = disco::current_context_id();
    return id;
}

// The entry of the calling thread's context, made if there is none (null when
// that fails); the mutex is held.
ScratchPool* scratch_entry(int device)
{
    const unsigned long long ctx = bound_context_id();
    if (ctx == 0) return nullptr;
    for (ScratchPool& p : g_scratch)
        if (p.device == device && p.ctx == ctx) return &p;
    cudaMemPoolProps props;
    std::memset(&props, 0, sizeof(props));
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    cudaMemPool_t pool = nullptr;
    if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    scratch_keep(pool, kScratchKeep);
    try {
        g_scratch.push_back({ device, ctx, pool, 0 });
    } catch (const std::exception&) {
        cudaMemPoolDestroy(pool);
        return nullptr;
    }
    return &g_scratch.back();
}

cudaError_t take_stream(int device, IdleStream& out)
{
    out = { nullptr, device, disco::current_context_id() };
    {
        std::lock_guard<std::mutex> lock(g_idle_mutex);
        for (size_t k = 0; k < g_idle.size(); ++k)
            if (g_idle[k].device == device && g_idle[k].ctx == out.ctx && out.ctx != 0) {
                out.stream = g_idle[k].stream;
                g_idle.erase(g_idle.begin() + k);
                return cudaSuccess;
            }
    }
    return cudaStreamCreateWithFlags(&out.stream, cudaStreamNonBlocking);
}

void give_stream(const IdleStream& s, bool healthy)
{
    if (!s.stream) return;
    if (healthy && s.ctx != 0) {
        std::lock_guard<std::mutex> lock(g_idle_mutex);
        // streams of a context that is gone are gone with it
        for (size_t k = g_idle.size(); k-- > 0;)
            if (g_idle[k].device == s.device && g_idle[k].ctx != s.ctx) g_idle.erase(g_idle.begin() + k);
        if (g_idle.size() < kIdleStreams) {
            try {
                g_idle.push_back(s);
                return;
            } catch (const std::exception&) {}
        }
    }
    cudaStreamDestroy(s.stream);
}

} // namespace

// The driver's cuCtxGetId, reached through the runtime without linking libcuda.
unsigned long long disco::current_context_id()
{
    static CtxGetCurrentFn get_current = nullptr;
    static CtxGetIdFn get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_current = reinterpret_cast<CtxGetCurrentFn>(f);
        f = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = reinterpret_cast<CtxGetIdFn>(f);
    });
    CUcontext c = nullptr;
    unsigned long long id = 0;
    if (get_current && get_id && get_current(&c) == CUDA_SUCCESS && c && get_id(c, &id) == CUDA_SUCCESS) return id;
    return 0;
}

cudaMemPool_t disco::scratch_pool(int device)
{
    OutsideCapture relaxed;
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    const ScratchPool* p = scratch_entry(device);
    return p ? p->pool : nullptr;
}

cudaError_t disco::scratch_alloc(void** p, size_t bytes, cudaStream_t s)
{
    OutsideCapture relaxed;
    int dev = 0;
    cudaMemPool_t pool = cudaGetDevice(&dev) == cudaSuccess ? scratch_pool(dev) : nullptr;
    if (pool && cudaMallocFromPoolAsync(p, bytes, pool, s) == cudaSuccess) return cudaSuccess;
    cudaGetLastError();
    return cudaMallocAsync(p, bytes, s);
}

unsigned long long disco::scratch_retain(int device)
{
    OutsideCapture relaxed;
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    ScratchPool* p = scratch_entry(device);
    if (!p) return 0;
    if (++p->plans == 1) scratch_keep(p->pool, kScratchKeepPlans);
    return p->ctx;
}

void disco::scratch_release(int device, unsigned long long ctx)
{
    OutsideCapture relaxed;
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    for (ScratchPool& p : g_scratch) {
        if (p.device != device || p.ctx != ctx || --p.plans > 0) continue;
        // a pool of a context that is gone must not be touched; the plan's device
        // need not be the current one
        int current = device;
        const bool other = cudaGetDevice(&current) == cudaSuccess && current != device;
        if (other) cudaSetDevice(device);
        if (bound_context_id() == ctx) {
            scratch_keep(p.pool, kScratchKeep);
            if (cudaMemPoolTrimTo(p.pool, kScratchKeep) != cudaSuccess) cudaGetLastError();
        }
        if (other) cudaSetDevice(current);
    }
}

void disco::set_last_error(const std::string& msg) { store_error(msg.c_str()); }
void disco::set_last_error(const char* msg) { store_error(msg); }

extern "C" {

const char* disco_b200_last_error(void) { return g_last_error; }

const char* disco_b200_strerror(int s)
{
    switch (s) {
    case DISCO_OK:       return "ok";
    case DISCO_EINVAL:   return "invalid argument";
    case DISCO_ENODEV:   return "no usable CUDA device";
    case DISCO_ECUDA:    return "CUDA error";
    case DISCO_ENOMEM:   return "out of memory";
    case DISCO_ELIMIT:   return "size above a limit or capacity";
    case DISCO_ETIMEOUT: return "bounded device wait gave up";
    case DISCO_EPLANES:  return "|b.n| is not a whole number of plane spacings";
    default:             return "unknown status";
    }
}

int disco_b200_available(void)
{
    int count = 0;
    return (cudaGetDeviceCount(&count) == cudaSuccess && count > 0) ? 1 : 0;
}

int disco_b200_line_fp64(void) { return 1; }

// printGpuInfo (Code/backend_cuda.cu:543-553): same banner lines.
int disco_b200_device_info(char* buf, size_t len)
{
    if (!buf || len == 0) return fail(DISCO_EINVAL, "null buffer");
    if (!disco_b200_available()) return fail(DISCO_ENODEV, "no CUDA device");
    int dev = 0;
    DISCO_TRY_CUDA(cudaGetDevice(&dev), "cudaGetDevice");
    cudaDeviceProp p;
    DISCO_TRY_CUDA(cudaGetDeviceProperties(&p, dev), "cudaGetDeviceProperties");
    std::snprintf(buf, len,
                  "\n--- GPU: %s ---\n  SMs              : %d\n  Global memory    : %zu MB\n"
                  "  Shared mem/block : %zu KB\n\n",
                  p.name, p.multiProcessorCount, (size_t)(p.totalGlobalMem >> 20),
                  (size_t)(p.sharedMemPerBlock / 1024));
    return DISCO_OK;
}

void disco_b200_options_default(disco_options* o)
{
    if (!o) return;
    std::memset(o, 0, sizeof(*o));
    o->precision = DISCO_FP64;
    o->images = 1;                // Code/backend_cpu.cpp:51-53
    o->nu = 0.35;                 // Code/kroupa.hpp:24
    o->chunk_pairs = -1.0;        // GpuOptions default (Code/backend.hpp:55)
}

} // extern "C"

namespace {

// A plan without its device memory: checks, tables, and the block's layout.
int plan_build(const disco_loop* loops, int32_t nloops, const double box[3], const disco_options* opt,
               int64_t max_atoms, disco_plan** out)
{
    if (!out) return fail(DISCO_EINVAL, "null plan pointer");
    *out = nullptr;
    if (nloops < 0 || (nloops > 0 && !loops)) return fail(DISCO_EINVAL, "bad loop array");
    if (!box || !(box[0] > 0.) || !(box[1] > 0.) || !(box[2] > 0.))
        return fail(DISCO_EINVAL, "box lengths must be positive");
    disco_options o;
    if (opt) o = *opt; else disco_b200_options_default(&o);
    int st = check_options(o);
    if (st) return st;
    if (max_atoms < 0) return fail(DISCO_EINVAL, "max_atoms < 0");
    if (!disco_b200_available()) return fail(DISCO_ENODEV, "no CUDA device");

    disco_plan* p = new disco_plan();
    p->opt = o;
    p->nloops = nloops;
    for (int i = 0; i < 3; ++i) p->box[i] = box[i];
    const int W = 2 * o.images + 1;
    p->nimg = W * W * W;
    cudaError_t e = cudaGetDevice(&p->device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&p->sm_count, cudaDevAttrMultiProcessorCount, p->device);
    if (e != cudaSuccess) { free_plan(p); return cuda_fail(e, "device query"); }

    std::memset(&p->stats, 0, sizeof(p->stats));
    p->stats.n_loops = nloops;
    p->stats.n_images = p->nimg;
    p->loop_evals.assign((size_t)nloops, 0.0);
    for (int l = 0; l < nloops; ++l) {
        if (loops[l].line) p->stats.n_line_loops++; else p->stats.n_loopon_loops++;
    }
    for (int k = 0; k < 2; ++k) {
        std::string err;
        const int kind = k == 0 ? disco::kLineKind : disco::kLooponKind;
        const uint32_t cap = o.stage_kb > 0 ? (uint32_t)o.stage_kb * 1024u : 0u;
        st = o.precision == DISCO_FP32C
                 ? disco::build_table_fp32(loops, nloops, kind, o.nu, p->tables[k], err, cap)
                 : disco::build_table(loops, nloops, kind, o.precision, o.nu, p->tables[k], err, cap, true);
        if (st) { free_plan(p); return fail(st, err); }
        disco::append_tree_pieces(p->tables[k]);
        const disco::HostTable& T = p->tables[k];
        for (int l = 0; l < nloops; ++l) p->loop_evals[l] += T.loop_evals[l];
        p->stats.n_segments += T.n_segments;
        p->stats.n_loopons += T.n_loopons;
    }
    {
        const int inner = o.image_min > 0 ? 2 * o.image_min - 1 : 0;
        p->stats.n_images = p->nimg - inner * inner * inner;
    }
    p->stats.evals_per_atom = (double)(p->stats.n_segments + p->stats.n_loopons) * p->stats.n_images;
    size_t at = 256;                                     // the status word
    auto take = [&](size_t bytes) { const size_t o = at; at += (bytes + 255) & ~size_t(255); return o; };
    for (int k = 0; k < 2; ++k) {
        if (p->tables[k].chunks.empty()) continue;
        p->table_at[k] = take(p->tables[k].bytes.size());
        p->chunks_at[k] = take(p->tables[k].chunks.size() * sizeof(disco::Chunk));
    }
    p->image_bytes = at;
    if (o.precision == DISCO_FP32C && !p->tables[0].chunks.empty()) {
        // the list of atoms with near-cut pairs: up to 2^21 (a longer list
        // overflows and the FP64 pass visits every atom)
        p->near_cap = (int32_t)std::min<int64_t>(std::max<int64_t>(max_atoms, 1 << 16), 1 << 21);
        p->near_at = take(256 + (size_t)p->near_cap * sizeof(int32_t));
    }
    p->bytes = at;
    *out = p;
    return DISCO_OK;
}

// Copies the parts of a plan's image by copy(offset in the image, source, bytes)
// until one fails.
template <class Copy>
cudaError_t plan_image(const disco_plan* p, Copy copy)
{
    static const unsigned char zero[256] = {};
    cudaError_t e = copy((size_t)0, static_cast<const void*>(zero), sizeof(zero));       // the status word
    for (int k = 0; k < 2; ++k) {
        const disco::HostTable& T = p->tables[k];
        if (T.chunks.empty()) continue;
        if (e == cudaSuccess) e = copy(p->table_at[k], static_cast<const void*>(T.bytes.data()), T.bytes.size());
        if (e == cudaSuccess)
            e = copy(p->chunks_at[k], static_cast<const void*>(T.chunks.data()), T.chunks.size() * sizeof(disco::Chunk));
    }
    return e;
}

// The image on the host, behind `at` bytes of other data.
std::vector<unsigned char> plan_packed(const disco_plan* p, size_t at)
{
    std::vector<unsigned char> pack(at + p->image_bytes, 0);
    plan_image(p, [&](size_t o, const void* src, size_t bytes) {
        std::memcpy(pack.data() + at + o, src, bytes);
        return cudaSuccess;
    });
    return pack;
}

// The image of a plan that has its block, on `s`: small ones in one copy.
cudaError_t plan_upload(const disco_plan* p, cudaStream_t s)
{
    if (p->image_bytes <= (size_t)64 << 10) {
        const std::vector<unsigned char> pack = plan_packed(p, 0);
        return cudaMemcpyAsync(p->block, pack.data(), pack.size(), cudaMemcpyHostToDevice, s);
    }
    return plan_image(p, [&](size_t o, const void* src, size_t bytes) {
        return cudaMemcpyAsync(p->block + o, src, bytes, cudaMemcpyHostToDevice, s);
    });
}

// Gives a plan its block (p->bytes, 256-byte aligned; the image still has to be
// copied to its start).
void plan_place(disco_plan* p, unsigned char* block)
{
    p->block = block;
    p->d_status = reinterpret_cast<int*>(block);
    for (int k = 0; k < 2; ++k) {
        if (p->tables[k].chunks.empty()) continue;
        p->d_table[k] = block + p->table_at[k];
        p->d_chunks[k] = reinterpret_cast<disco::Chunk*>(block + p->chunks_at[k]);
    }
    if (p->near_at) {
        p->d_near_count = reinterpret_cast<unsigned int*>(block + p->near_at);
        p->d_near = reinterpret_cast<int32_t*>(block + p->near_at + 256);
    }
}

} // namespace

// A plan for one call inside the library: its block comes from the scratch pool
// in the order of `s` (cudaMalloc without one), and the caller has waited for
// its last kernel before it destroys the plan.
int disco::plan_create_on(const disco_loop* loops, int32_t nloops, const double box[3], const disco_options* opt,
                          int64_t max_atoms, cudaStream_t s, disco_plan** out)
{
    int st = plan_build(loops, nloops, box, opt, max_atoms, out);
    if (st) return st;
    disco_plan* p = *out;
    *out = nullptr;
    unsigned char* block = nullptr;
    cudaMemPool_t pool = scratch_pool(p->device);
    p->pooled = pool && cudaMallocFromPoolAsync(reinterpret_cast<void**>(&block), p->bytes, pool, s) == cudaSuccess;
    cudaError_t e = cudaSuccess;
    if (!p->pooled) {
        cudaGetLastError();
        block = nullptr;
        e = cudaMalloc(&block, p->bytes);
    }
    if (e != cudaSuccess) { free_plan(p); return cuda_fail(e, "plan memory"); }
    plan_place(p, block);
    p->own = true;
    p->stream = s;
    e = plan_upload(p, s);
    if (e != cudaSuccess) { free_plan(p); return cuda_fail(e, "loop table upload"); }
    *out = p;
    return DISCO_OK;
}

int disco::plan_execute_counted(disco_plan* p, const disco_atoms* a, cudaStream_t s, int* launches)
{
    *launches = 0;
    if (!p || !a) return fail(DISCO_EINVAL, "null plan or atoms");
    if (a->n < 0) return fail(DISCO_EINVAL, "negative atom count");
    if (a->n == 0) return DISCO_OK;
    if (!a->x || !a->y || !a->z || !a->ux || !a->uy || !a->uz) return fail(DISCO_EINVAL, "null atom array");
    for (int k = 0; k < 2; ++k) {
        const disco::HostTable& T = p->tables[k];
        if (T.chunks.empty()) continue;
        disco::FieldArgs fa;
        std::memset(&fa, 0, sizeof(fa));
        fa.x = a->x; fa.y = a->y; fa.z = a->z;
        fa.ux = a->ux; fa.uy = a->uy; fa.uz = a->uz;
        fa.n = a->n;
        fa.table = p->d_table[k];
        fa.chunks = p->d_chunks[k];
        fa.nchunks = (int32_t)T.chunks.size();
        fa.stage_bytes = T.stage_bytes;
        fa.resident = T.resident ? 1 : 0;
        fa.images = p->opt.images;
        fa.nimg = p->nimg;
        fa.image_min = p->opt.image_min;
        fa.Lx = p->box[0]; fa.Ly = p->box[1]; fa.Lz = p->box[2];
        const double pi = 3.14159265358979323846;
        const double c3 = 1.0 / (8.0 * pi * (1.0 - p->opt.nu));      // Code/barnett.hpp:51
        fa.cJ = c3 - 1.0 / (4.0 * pi);
        fa.cK = c3;
        fa.c2 = 1.0 - 2.0 * p->opt.nu;                              // Code/kroupa.hpp:66
        fa.status = p->d_status;
        fa.near_h = (float)p->opt.near_plane;
        fa.near_r = (float)p->opt.near_rim;
        if (k == 0 && T.aux_raw)
            fa.raw = reinterpret_cast<const double*>(p->d_table[k] + T.aux_raw);
        if (T.fp32 && k == 0 && T.aux_pieces) {
            fa.pieces64 = reinterpret_cast<const disco::LinePiece*>(p->d_table[k] + T.aux_pieces);
            fa.segs64 = reinterpret_cast<const disco::LineSeg*>(p->d_table[k] + T.aux_segs);
            fa.near_list = p->d_near;
            fa.near_count = p->d_near_count;
            fa.near_cap = p->near_cap;
        }
        std::string err;
        const int kind = k == 0 ? disco::kLineKind : disco::kLooponKind;
        const disco::TreeShape shape = plan_tree(p, k, a->n, s);
        if (shape.use) {
            int queued = 0;
            const int st = disco::launch_tree(fa, T, shape, p->sm_count, s, &queued, err);
            if (st) return fail(st, err);
            *launches += queued;
            if (queued) continue;
        }
        const int st = T.fp32
            ? disco::launch_field_fp32(fa, kind, p->sm_count, p->opt.image_split, s, err)
            : disco::launch_field(fa, kind, false, p->sm_count, p->opt.threads_per_block,
                                  p->opt.image_split, s, err);
        if (st) return fail(st, err);
        *launches += T.fp32 && k == 0 ? 2 : 1;               // FP32 lines: the near-cut pairs' pass
    }
    return DISCO_OK;
}

extern "C" {

int disco_b200_plan_create(const disco_loop* loops, int32_t nloops, const double box[3],
                           const disco_options* opt, int64_t max_atoms, disco_plan** out)
{
    int st = plan_build(loops, nloops, box, opt, max_atoms, out);
    if (st) return st;
    disco_plan* p = *out;
    *out = nullptr;
    unsigned char* block = nullptr;
    cudaError_t e = cudaMalloc(&block, p->bytes);
    if (e != cudaSuccess) { free_plan(p); return cuda_fail(e, "plan memory"); }
    plan_place(p, block);
    p->own = true;
    e = plan_upload(p, nullptr);
    if (e == cudaSuccess) e = cudaStreamSynchronize(nullptr);
    if (e != cudaSuccess) { free_plan(p); return cuda_fail(e, "loop table upload"); }
    for (disco::HostTable& T : p->tables) std::vector<unsigned char>().swap(T.bytes);
    *out = p;
    return DISCO_OK;
}

int disco_b200_plan_execute(disco_plan* p, const disco_atoms* a, void* stream)
{
    int launches;
    return disco::plan_execute_counted(p, a, static_cast<cudaStream_t>(stream), &launches);
}

int disco_b200_plan_sync(disco_plan* p, void* stream)
{
    if (!p) return fail(DISCO_EINVAL, "null plan");
    DISCO_TRY_CUDA(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)), "stream synchronize");
    int st = 0;
    DISCO_TRY_CUDA(cudaMemcpy(&st, p->d_status, sizeof(int), cudaMemcpyDeviceToHost), "status read");
    if (st) {
        cudaMemset(p->d_status, 0, sizeof(int));
        return fail(st, "a kernel reported: " + std::string(disco_b200_strerror(st)));
    }
    return DISCO_OK;
}

int disco_b200_plan_stats(const disco_plan* p, disco_plan_stats* s)
{
    if (!p || !s) return fail(DISCO_EINVAL, "null argument");
    *s = p->stats;
    return DISCO_OK;
}

int disco_b200_plan_cells(disco_plan* p, int64_t n)
{
    if (!p || n <= 0) return 0;
    int levels = 0;
    for (int k = 0; k < 2; ++k) {
        const disco::TreeShape shape = plan_shape(p, k, n);
        if (shape.use) levels += shape.levels;
    }
    return levels;
}

int disco_b200_plan_destroy(disco_plan* p)
{
    free_plan(p);
    return DISCO_OK;
}

// kroupaGPU on host buffers (Code/backend_cuda.cu:568-722): allocate, upload,
// one launch per loop kind, download, free.  The displacement arrays are
// uploaded too, so the call accumulates into them exactly like the CPU backend.
int disco_b200_displace(const disco_atoms* atoms, const disco_loop* loops, int32_t nloops,
                        const double box[3], const disco_options* opt, disco_timing* timing)
{
    if (!atoms) return fail(DISCO_EINVAL, "null atoms");
    const int64_t n = atoms->n;
    if (n < 0) return fail(DISCO_EINVAL, "negative atom count");
    if (n > 0 && (!atoms->x || !atoms->y || !atoms->z || !atoms->ux || !atoms->uy || !atoms->uz))
        return fail(DISCO_EINVAL, "null atom array");
    disco_options o;
    if (opt) o = *opt; else disco_b200_options_default(&o);

    const double t0 = now_s();
    disco_plan* plan = nullptr;
    int st = plan_build(loops, nloops, box, &o, n, &plan);
    if (st) return st;
    if (o.verbose) {
        std::printf("Precision: %s\n", o.precision == DISCO_FP32C
                    ? "single (fp32 pair term, compensated sums)" : "double");
    }
    // one block of device memory: x, y, z, ux, uy, uz, then the plan's (its
    // status word first), from the scratch pool or, without one, cudaMalloc
    const size_t bytes = (size_t)n * sizeof(double), atoms_at = (6 * bytes + 255) & ~size_t(255);
    unsigned char* block = nullptr;
    bool pooled = false, healthy = false;
    IdleStream is = { nullptr, 0, 0 };
    cudaEvent_t ev[2] = { nullptr, nullptr };
    auto cleanup = [&]() {
        if (block && pooled) cudaFreeAsync(block, is.stream);
        else if (block) cudaFree(block);
        // the pool gives back what it holds above its 32 MB when it is waited for
        // or trimmed (by the plan's end): a large call leaves neither to its caller
        if (pooled && atoms_at + plan->bytes > (8ull << 20)) cudaStreamSynchronize(is.stream);
        disco_b200_plan_destroy(plan);
        give_stream(is, healthy);
        for (auto& x : ev) if (x) cudaEventDestroy(x);
    };
    cudaError_t e = cudaFree(nullptr);                    // the primary context, before its identifier is read
    if (e == cudaSuccess) e = take_stream(plan->device, is);
    cudaStream_t s = is.stream;
    if (e == cudaSuccess) e = cudaEventCreate(&ev[0]);
    if (e == cudaSuccess) e = cudaEventCreate(&ev[1]);
    if (e == cudaSuccess) {
        cudaMemPool_t pool = disco::scratch_pool(plan->device);
        pooled = pool && cudaMallocFromPoolAsync(reinterpret_cast<void**>(&block), atoms_at + plan->bytes, pool, s) ==
                             cudaSuccess;
        if (!pooled) {
            cudaGetLastError();
            block = nullptr;
            e = cudaMalloc(&block, atoms_at + plan->bytes);
        }
    }
    if (e != cudaSuccess) { cleanup(); return cuda_fail(e, "atom allocation"); }
    plan_place(plan, block + atoms_at);
    // small calls: one copy each way through a packed host buffer
    std::vector<unsigned char> pack;
    const bool small = atoms_at + plan->image_bytes <= (size_t)128 << 10;
    const double* src[6] = { atoms->x, atoms->y, atoms->z, atoms->ux, atoms->uy, atoms->uz };
    if (small) {
        pack = plan_packed(plan, atoms_at);
        for (int k = 0; k < 6 && n > 0; ++k) std::memcpy(pack.data() + k * bytes, src[k], bytes);
        e = cudaMemcpyAsync(block, pack.data(), pack.size(), cudaMemcpyHostToDevice, s);
    } else {
        for (int k = 0; k < 6 && e == cudaSuccess && n > 0; ++k)
            e = cudaMemcpyAsync(block + k * bytes, src[k], bytes, cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess)
            e = plan_upload(plan, s);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) { cleanup(); return cuda_fail(e, "atom upload"); }
    const double t1 = now_s();

    if (o.verbose) std::printf("Running GPU kernels...\n");
    double* d = reinterpret_cast<double*>(block);
    disco_atoms da;
    da.x = d; da.y = d + n; da.z = d + 2 * n;
    da.ux = d + 3 * n; da.uy = d + 4 * n; da.uz = d + 5 * n;
    da.n = n;
    e = cudaEventRecord(ev[0], s);
    if (e != cudaSuccess) { cleanup(); return cuda_fail(e, "event"); }
    st = disco_b200_plan_execute(plan, &da, s);
    if (st) { std::string m = g_last_error; cleanup(); return fail(st, m); }
    e = cudaEventRecord(ev[1], s);
    if (e == cudaSuccess) e = cudaEventSynchronize(ev[1]);
    if (e != cudaSuccess) { cleanup(); return cuda_fail(e, "displacement kernels"); }
    float ms = 0.f;
    cudaEventElapsedTime(&ms, ev[0], ev[1]);
    const double t2 = now_s();
    if (o.verbose) std::printf("\nGPU kernel time: %g ms\n\n", (double)ms);

    // the status word first (small calls: behind uz in the same copy)
    int status = 0;
    if (small) {
        e = cudaMemcpyAsync(pack.data(), block + 3 * bytes, atoms_at - 3 * bytes + sizeof(int), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e == cudaSuccess) std::memcpy(&status, pack.data() + atoms_at - 3 * bytes, sizeof(int));
    } else {
        e = cudaMemcpyAsync(&status, plan->d_status, sizeof(int), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    }
    if (e == cudaSuccess && status) {
        cleanup();
        return fail(status, "a kernel reported: " + std::string(disco_b200_strerror(status)));
    }
    double* dst[3] = { atoms->ux, atoms->uy, atoms->uz };
    if (small) {
        for (int k = 0; k < 3 && e == cudaSuccess && n > 0; ++k) std::memcpy(dst[k], pack.data() + k * bytes, bytes);
    } else {
        for (int k = 0; k < 3 && e == cudaSuccess && n > 0; ++k)
            e = cudaMemcpyAsync(dst[k], block + (3 + k) * bytes, bytes, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    }
    if (e != cudaSuccess) { cleanup(); return cuda_fail(e, "displacement download"); }
    healthy = true;
    std::vector<double> evals = plan->loop_evals;
    cleanup();
    const double t3 = now_s();
    if (timing) {
        timing->upload = t1 - t0;
        timing->kernels = t2 - t1;
        timing->download = t3 - t2;
        if (timing->loop_sec) {
            double tot = 0.0;
            for (double v : evals) tot += v;
            for (int l = 0; l < nloops; ++l)
                timing->loop_sec[l] = tot > 0.0 ? (ms * 1e-3) * evals[l] / tot : 0.0;
        }
    }
    return DISCO_OK;
}

} // extern "C"
