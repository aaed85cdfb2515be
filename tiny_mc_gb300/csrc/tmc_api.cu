// tmc_api.cu — the C ABI (include/tmc.h): validation, per-device resources,
// the drop-in photon_batch entry points and the FP64 finalisation kernel.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>

#include "tmc_device.cuh"
#include "tmc_internal.h"

namespace tmc {

namespace {
std::mutex g_mutex;
thread_local std::string g_error;   // per thread, like errno
DeviceCtx g_ctx[64];
int g_plain_block = 0;
int g_plain_blocks_per_sm = 0;
int g_plain_max_blocks = 0;
}  // namespace

std::mutex &api_mutex() { return g_mutex; }

void set_error_text(const std::string &s) { g_error = s; }

int set_cuda_error(cudaError_t e, const char *where)
{
    char buf[256];
    std::snprintf(buf, sizeof buf, "%s: %s (%s)", where, cudaGetErrorString(e), cudaGetErrorName(e));
    g_error = buf;
    if (e == cudaErrorMemoryAllocation)
        return TMC_E_NOMEM;
    if (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver ||
        e == cudaErrorNoKernelImageForDevice)
        return TMC_E_NODEVICE;
    return TMC_E_CUDA;
}

int validate(const tmc_params *p)
{
    auto invalid = [](const char *why) {
        set_error_text(std::string("invalid parameters: ") + why);
        return TMC_E_INVALID;
    };
    if (!p)
        return invalid("null tmc_params");
    if (p->shells == 0 || p->shells > (1u << 24))
        return invalid("shells must be 1 .. 2^24");
    // MU_A "!!non-zero!!" (params.h:14): with mu_a = 0 the weight never
    // decays and a photon never dies.
    if (!(p->mu_a > 0.0f) || !std::isfinite(p->mu_a))
        return invalid("mu_a must be finite and > 0");
    if (!(p->mu_s >= 0.0f) || !std::isfinite(p->mu_s))
        return invalid("mu_s must be finite and >= 0");
    if (!(p->microns_per_shell > 0.0f) || !std::isfinite(p->microns_per_shell))
        return invalid("microns_per_shell must be finite and > 0");
    if (p->math != TMC_MATH_EXACT && p->math != TMC_MATH_FAST)
        return invalid("math must be TMC_MATH_EXACT or TMC_MATH_FAST");
    if (p->reserved != 0)
        return invalid("reserved must be 0");
    // If mu_a is so small against mu_s that the float albedo rounds to 1, the
    // weight never decays (photon.c:32) and no photon would ever die.
    if (!(p->mu_s / (p->mu_s + p->mu_a) < 1.0f))
        return invalid("mu_a too small against mu_s: the float albedo rounds to 1");
    return TMC_OK;
}

Derived derive(float mu_a, float mu_s, float microns_per_shell, uint32_t shells)
{
    Derived d;
    d.albedo = mu_s / (mu_s + mu_a);                                      // photon.c:8
    d.spm = (float)(1e4 / (double)microns_per_shell / (double)(mu_a + mu_s));  // photon.c:9
    d.c = 1.0f - d.albedo;
    d.last = (float)(shells - 1);
    d.shells = shells;
    return d;
}

DeviceCtx *current_ctx(int *status)
{
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        *status = set_cuda_error(e, "cudaGetDevice");
        return nullptr;
    }
    if (dev < 0 || dev >= 64) {
        *status = TMC_E_NODEVICE;
        return nullptr;
    }
    DeviceCtx &c = g_ctx[dev];
    if (c.device < 0) {
        cudaDeviceProp prop;
        e = cudaGetDeviceProperties(&prop, dev);
        if (e != cudaSuccess) {
            *status = set_cuda_error(e, "cudaGetDeviceProperties");
            return nullptr;
        }
        c.sms = prop.multiProcessorCount;
        c.cc_major = prop.major;
        c.cc_minor = prop.minor;
        c.smem_optin = prop.sharedMemPerBlockOptin;
        e = cudaMalloc(&c.workspace, WORKSPACE_BYTES);
        if (e != cudaSuccess) {
            *status = set_cuda_error(e, "cudaMalloc(workspace)");
            return nullptr;
        }
        e = cudaMallocHost(&c.pinned, PINNED_BYTES);
        if (e != cudaSuccess) {
            *status = set_cuda_error(e, "cudaMallocHost");
            return nullptr;
        }
        e = cudaStreamCreateWithFlags(&c.stream, cudaStreamNonBlocking);
        if (e != cudaSuccess) {
            *status = set_cuda_error(e, "cudaStreamCreate");
            return nullptr;
        }
        e = cudaEventCreateWithFlags(&c.ws_done, cudaEventDisableTiming);
        if (e != cudaSuccess) {
            *status = set_cuda_error(e, "cudaEventCreate");
            return nullptr;
        }
        c.device = dev;
    }
    *status = TMC_OK;
    return &c;
}

static bool capturing(cudaStream_t stream)
{
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(stream, &cs) == cudaSuccess && cs != cudaStreamCaptureStatusNone;
}

cudaError_t ws_acquire(DeviceCtx &c, cudaStream_t stream)
{
    if (capturing(stream))
        return cudaSuccess;
    return cudaStreamWaitEvent(stream, c.ws_done, 0);
}

cudaError_t ws_release(DeviceCtx &c, cudaStream_t stream)
{
    if (capturing(stream))
        return cudaSuccess;
    return cudaEventRecord(c.ws_done, stream);
}

// All of a context's calls use its one stream, so its device scratch is ordered by
// that stream and growing or freeing it waits for no other work on the device.
cudaError_t CallBuffers::device(size_t bytes, size_t keep)
{
    if (bytes > keep) {
        const cudaError_t e = cudaMallocAsync(&dev, bytes, ctx.stream);
        own_dev = e == cudaSuccess;
        return e;
    }
    if (bytes > ctx.scratch_cap) {
        if (ctx.scratch)
            cudaFreeAsync(ctx.scratch, ctx.stream);
        ctx.scratch = nullptr;
        ctx.scratch_cap = 0;
        const size_t want = std::min(keep, std::max<size_t>(bytes + bytes / 2, 16384));
        const cudaError_t e = cudaMallocAsync(&ctx.scratch, want, ctx.stream);
        if (e != cudaSuccess)
            return e;
        ctx.scratch_cap = want;
    }
    dev = static_cast<char *>(ctx.scratch);
    return cudaSuccess;
}

CallBuffers::~CallBuffers()
{
    if (own_dev)
        cudaFreeAsync(dev, ctx.stream);
}

// n results from device memory through pinned memory, from its byte 64 on, in
// pieces of which one is copied while the one before is taken: take(first, count,
// data).  The stream's earlier work has ended before the first is taken.
template <class T, class Take>
static cudaError_t read_back(DeviceCtx &c, const T *d, size_t n, Take take)
{
    size_t piece = (PINNED_BYTES - 64) / sizeof(T);
    if (n > piece)
        piece /= 2;
    T *const half[2] = {reinterpret_cast<T *>(c.pinned + 64), reinterpret_cast<T *>(c.pinned + 64) + piece};
    auto copy = [&](size_t at, int h) {
        return cudaMemcpyAsync(half[h], d + at, sizeof(T) * std::min(piece, n - at), cudaMemcpyDeviceToHost, c.stream);
    };
    cudaError_t e = copy(0, 0);
    int h = 0;
    for (size_t at = 0; at < n; at += piece, h ^= 1) {
        if (e == cudaSuccess)
            e = cudaStreamSynchronize(c.stream);
        if (e == cudaSuccess && at + piece < n)
            e = copy(at + piece, h ^ 1);
        if (e != cudaSuccess)
            return e;
        take(at, std::min(piece, n - at), half[h]);
    }
    return e;
}

__global__ void tally_to_heat_kernel(const tmc_tally *t, uint32_t shells, double c, double *heat,
                                     double *heat2)
{
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= shells)
        return;
    const tmc_tally q = t[s];
    const double sw = (double)q.w_hi * 0x1p24 + (double)q.w_lo * 0x1p-40;
    const double sw2 = (double)q.w2_hi * 0x1p24 + (double)q.w2_lo * 0x1p-40;
    heat[s] = c * sw;
    heat2[s] = (c * c) * sw2;
}

// tiny_mc.c:60-66 in FP64 from exact tallies: t = 4 pi MPS^3 N / 1e12 (cm^3),
// density[i] = heat[i] / t / (i^2 + i + 1/3), error[i] = sqrt(heat2[i] -
// heat[i]^2 / N) / t / (i^2 + i + 1/3) (NaN where the per-deposit variance
// estimate goes negative, as the reference's does), extra = heat[S-1] / N.
__global__ void report_fp64_kernel(const tmc_tally *t, uint32_t shells, double c, double mps,
                                   double photons, double *density, double *error, double *extra)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= shells)
        return;
    const tmc_tally q = t[i];
    const double heat = c * ((double)q.w_hi * 0x1p24 + (double)q.w_lo * 0x1p-40);
    const double heat2 = (c * c) * ((double)q.w2_hi * 0x1p24 + (double)q.w2_lo * 0x1p-40);
    const double vol = 4.0 * 3.14159265358979323846 * mps * mps * mps * photons / 1e12;
    const double shell = (double)i * (double)i + (double)i + 1.0 / 3.0;
    if (i + 1 < shells) {
        density[i] = heat / vol / shell;
        error[i] = sqrt(heat2 - heat * heat / photons) / vol / shell;
    } else {
        *extra = heat / photons;
    }
}

cudaError_t launch_report_fp64(const tmc_tally *d_tally, uint32_t shells, double c, double mps,
                               double photons, double *d_out, cudaStream_t stream)
{
    report_fp64_kernel<<<(shells + 255) / 256, 256, 0, stream>>>(d_tally, shells, c, mps, photons, d_out,
                                                                  d_out + shells, d_out + 2 * shells);
    return cudaGetLastError();
}

cudaError_t launch_tally_to_heat(const tmc_tally *d_tally, uint32_t shells, double c,
                                 double *d_heat, double *d_heat2, cudaStream_t stream)
{
    const int bs = 256;
    tally_to_heat_kernel<<<(shells + bs - 1) / bs, bs, 0, stream>>>(d_tally, shells, c, d_heat,
                                                                   d_heat2);
    return cudaGetLastError();
}

// Shared part of the host-array entry points.  Device scratch: claim and step
// counters (WORKSPACE_BYTES), the tallies, then FP64 heat and heat2; the walk
// fills the tallies and the step counter.
struct HostWalk {
    tmc_tally *tally;
    unsigned long long *steps;
    double *heat;
};

static int walk_into(CallBuffers &buf, DeviceCtx &c, uint64_t n, const tmc_params *p, const Derived &d, bool steps,
                     HostWalk &w)
{
    const size_t S = p->shells;
    cudaError_t e = buf.device(WORKSPACE_BYTES + (sizeof(tmc_tally) + 2 * sizeof(double)) * S, WALK_KEEP);
    if (e != cudaSuccess)
        return set_cuda_error(e, "host-array call's scratch");
    w.tally = reinterpret_cast<tmc_tally *>(buf.dev + WORKSPACE_BYTES);
    w.steps = reinterpret_cast<unsigned long long *>(buf.dev) + 1;
    w.heat = reinterpret_cast<double *>(buf.dev + WORKSPACE_BYTES + sizeof(tmc_tally) * S);
    e = cudaMemsetAsync(buf.dev, 0, WORKSPACE_BYTES + sizeof(tmc_tally) * S, c.stream);
    if (e != cudaSuccess)
        return set_cuda_error(e, "cudaMemsetAsync");
    if (n == 0)
        return TMC_OK;
    PlainLaunch L{};
    L.p = p;
    L.d = d;
    L.n_photons = n;
    L.d_tally = w.tally;
    L.d_work = reinterpret_cast<unsigned long long *>(buf.dev);
    L.d_steps = steps ? w.steps : nullptr;
    L.block = g_plain_block;
    L.blocks_per_sm = g_plain_blocks_per_sm;
    L.max_blocks = g_plain_max_blocks;
    e = launch_plain(L, c, c.stream);
    if (e != cudaSuccess)
        return set_cuda_error(e, "walk_plain launch");
    return TMC_OK;
}

static int check_sizes(uint64_t n, const tmc_params *p)
{
    if (n > (1ull << 62) || p->photon_id_base > ~0ull - n) {
        set_error_text("photon count or photon_id_base + count overflows 64-bit photon ids");
        return TMC_E_OVERFLOW;
    }
    return TMC_OK;
}

__global__ void debug_rand_kernel(PhiloxKeys keys, uint32_t pid_lo, uint32_t pid_hi, uint32_t n,
                                  int32_t *out)
{
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;   // Philox block index
    if (4 * b >= n)
        return;
    const uint4 r = philox4x32_10(b, 0u, pid_lo, pid_hi, keys);
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
    for (uint32_t j = 0; j < 4 && 4 * b + j < n; ++j)
        out[4 * b + j] = (int32_t)rand31(w[j]);
}

}  // namespace tmc

using namespace tmc;

extern "C" {

void tmc_params_default(tmc_params *p)
{
    if (!p)
        return;
    std::memset(p, 0, sizeof *p);
    p->shells = 101;             // params.h:6
    p->microns_per_shell = 50;   // params.h:22
    p->mu_a = 2.0f;              // params.h:14
    p->mu_s = 20.0f;             // params.h:18
    p->seed = 1;
    p->photon_id_base = 0;
    p->math = TMC_MATH_EXACT;
}

size_t tmc_workspace_bytes(void) { return WORKSPACE_BYTES; }

int tmc_photon_batch_fx(tmc_tally *tally, uint64_t n_photons, const tmc_params *p,
                        uint64_t *photon_steps)
{
    tmc::NvtxRange nvtx_range("tmc_photon_batch_fx");
    int st = validate(p);
    if (st)
        return st;
    if (!tally)
        return TMC_E_INVALID;
    std::lock_guard<std::mutex> lk(api_mutex());
    DeviceCtx *c = current_ctx(&st);
    if (!c)
        return st;
    if ((st = check_sizes(n_photons, p)))
        return st;
    const Derived d = derive(p->mu_a, p->mu_s, p->microns_per_shell, p->shells);
    CallBuffers buf(*c);
    HostWalk w{};
    if ((st = walk_into(buf, *c, n_photons, p, d, true, w)))
        return st;
    cudaError_t e = cudaMemcpyAsync(c->pinned, w.steps, sizeof(uint64_t), cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess)
        e = read_back(*c, w.tally, p->shells, [&](size_t first, size_t count, const tmc_tally *h) {
            tmc_tally *t = tally + first;
            for (size_t s = 0; s < count; ++s) {
                unsigned __int128 a = ((unsigned __int128)t[s].w_hi << 64) | t[s].w_lo;
                unsigned __int128 b = ((unsigned __int128)t[s].w2_hi << 64) | t[s].w2_lo;
                a += ((unsigned __int128)h[s].w_hi << 64) | h[s].w_lo;
                b += ((unsigned __int128)h[s].w2_hi << 64) | h[s].w2_lo;
                t[s].w_lo = (uint64_t)a;
                t[s].w_hi = (uint64_t)(a >> 64);
                t[s].w2_lo = (uint64_t)b;
                t[s].w2_hi = (uint64_t)(b >> 64);
            }
        });
    if (e != cudaSuccess)
        return set_cuda_error(e, "tmc_photon_batch_fx");
    if (photon_steps)
        *photon_steps += *reinterpret_cast<const uint64_t *>(c->pinned);
    return TMC_OK;
}

int tmc_photon_batch(float *heat, float *heat2, uint64_t n_photons, const tmc_params *p)
{
    tmc::NvtxRange nvtx_range("tmc_photon_batch");
    int st = validate(p);
    if (st)
        return st;
    if (!heat || !heat2)
        return TMC_E_INVALID;
    std::lock_guard<std::mutex> lk(api_mutex());
    DeviceCtx *c = current_ctx(&st);
    if (!c)
        return st;
    if ((st = check_sizes(n_photons, p)))
        return st;
    const Derived d = derive(p->mu_a, p->mu_s, p->microns_per_shell, p->shells);
    const size_t S = p->shells;
    CallBuffers buf(*c);
    HostWalk w{};
    if ((st = walk_into(buf, *c, n_photons, p, d, false, w)))
        return st;
    cudaError_t e = launch_tally_to_heat(w.tally, p->shells, (double)d.c, w.heat, w.heat + S, c->stream);
    auto add = [](float *to, const double *h, size_t count) {
        for (size_t s = 0; s < count; ++s)
            to[s] = (float)((double)to[s] + h[s]);
    };
    if (e == cudaSuccess)   // S values of heat, then S of heat2
        e = read_back(*c, w.heat, 2 * S, [&](size_t first, size_t count, const double *h) {
            const size_t one = first < S ? std::min(count, S - first) : 0;
            if (one)
                add(heat + first, h, one);
            if (count > one)
                add(heat2 + (first + one - S), h + one, count - one);
        });
    if (e != cudaSuccess)
        return set_cuda_error(e, "tmc_photon_batch");
    return TMC_OK;
}

int tmc_photon_batch_device(tmc_tally *d_tally, uint64_t n_photons, const tmc_params *p,
                            uint64_t *d_steps, void *d_workspace, void *stream)
{
    tmc::NvtxRange nvtx_range("tmc_photon_batch_device");
    int st = validate(p);
    if (st)
        return st;
    if (!d_tally)
        return TMC_E_INVALID;
    std::lock_guard<std::mutex> lk(api_mutex());
    DeviceCtx *c = current_ctx(&st);
    if (!c)
        return st;
    if ((st = check_sizes(n_photons, p)))
        return st;
    if (n_photons == 0)
        return TMC_OK;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    void *ws = d_workspace ? d_workspace : c->workspace;
    cudaError_t e = d_workspace ? cudaSuccess : ws_acquire(*c, s);
    if (e == cudaSuccess)
        e = cudaMemsetAsync(ws, 0, sizeof(unsigned long long), s);
    if (e != cudaSuccess)
        return set_cuda_error(e, "cudaMemsetAsync(workspace)");
    PlainLaunch L{};
    L.p = p;
    L.d = derive(p->mu_a, p->mu_s, p->microns_per_shell, p->shells);
    L.n_photons = n_photons;
    L.d_tally = d_tally;
    L.d_work = reinterpret_cast<unsigned long long *>(ws);
    L.d_steps = reinterpret_cast<unsigned long long *>(d_steps);
    L.block = g_plain_block;
    L.blocks_per_sm = g_plain_blocks_per_sm;
    L.max_blocks = g_plain_max_blocks;
    e = launch_plain(L, *c, s);
    if (e == cudaSuccess && !d_workspace)
        e = ws_release(*c, s);
    if (e != cudaSuccess)
        return set_cuda_error(e, "walk_plain launch");
    return TMC_OK;
}

int tmc_report_fp64_device(const tmc_tally *d_tally, const tmc_params *p, uint64_t photons, double *d_out,
                           void *stream)
{
    int st = validate(p);
    if (st)
        return st;
    if (!d_tally || !d_out || photons == 0)
        return TMC_E_INVALID;
    const Derived d = derive(p->mu_a, p->mu_s, p->microns_per_shell, p->shells);
    cudaError_t e = launch_report_fp64(d_tally, p->shells, (double)d.c, (double)p->microns_per_shell,
                                       (double)photons, d_out, reinterpret_cast<cudaStream_t>(stream));
    return e == cudaSuccess ? TMC_OK : set_cuda_error(e, "tmc_report_fp64_device");
}

int tmc_report_fp64(const tmc_tally *tally, const tmc_params *p, uint64_t photons, double *density,
                    double *error, double *extra)
{
    int st = validate(p);
    if (st)
        return st;
    if (!tally || !density || !error || !extra || photons == 0)
        return TMC_E_INVALID;
    std::lock_guard<std::mutex> lk(api_mutex());
    DeviceCtx *c = current_ctx(&st);
    if (!c)
        return st;
    const uint32_t S = p->shells;
    CallBuffers buf(*c);
    cudaError_t e = buf.device(sizeof(tmc_tally) * (size_t)S + sizeof(double) * (2 * (size_t)S + 1), WALK_KEEP);
    if (e != cudaSuccess)
        return set_cuda_error(e, "tmc_report_fp64");
    tmc_tally *d_tally = reinterpret_cast<tmc_tally *>(buf.dev);
    double *d_out = reinterpret_cast<double *>(buf.dev + sizeof(tmc_tally) * (size_t)S);
    e = cudaMemcpyAsync(d_tally, tally, sizeof(tmc_tally) * S, cudaMemcpyHostToDevice, c->stream);
    const Derived d = derive(p->mu_a, p->mu_s, p->microns_per_shell, S);
    if (e == cudaSuccess)
        e = launch_report_fp64(d_tally, S, (double)d.c, (double)p->microns_per_shell, (double)photons, d_out,
                               c->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(density, d_out, sizeof(double) * (S - 1), cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(error, d_out + S, sizeof(double) * (S - 1), cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(extra, d_out + 2 * S, sizeof(double), cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(c->stream);
    return e == cudaSuccess ? TMC_OK : set_cuda_error(e, "tmc_report_fp64");
}

int tmc_tally_to_heat(const tmc_tally *tally, const tmc_params *p, double *heat, double *heat2)
{
    int st = validate(p);
    if (st)
        return st;
    if (!tally)
        return TMC_E_INVALID;
    const Derived d = derive(p->mu_a, p->mu_s, p->microns_per_shell, p->shells);
    const double c = (double)d.c;
    for (uint32_t s = 0; s < p->shells; ++s) {
        const double sw = (double)tally[s].w_hi * 0x1p24 + (double)tally[s].w_lo * 0x1p-40;
        const double sw2 = (double)tally[s].w2_hi * 0x1p24 + (double)tally[s].w2_lo * 0x1p-40;
        if (heat)
            heat[s] = c * sw;
        if (heat2)
            heat2[s] = (c * c) * sw2;
    }
    return TMC_OK;
}

int tmc_set_plain_launch(int block, int blocks_per_sm, int max_blocks)
{
    if (block != 0 && block != 128 && block != 256 && block != 512)
        return TMC_E_INVALID;
    if (blocks_per_sm < 0 || blocks_per_sm > 32 || max_blocks < 0)
        return TMC_E_INVALID;
    std::lock_guard<std::mutex> lk(api_mutex());
    g_plain_block = block;
    g_plain_blocks_per_sm = blocks_per_sm;
    g_plain_max_blocks = max_blocks;
    return TMC_OK;
}

int tmc_debug_rand(uint64_t seed, uint64_t photon, uint32_t n, int32_t *out)
{
    if (!out || n == 0 || n > (1u << 24))
        return TMC_E_INVALID;
    std::lock_guard<std::mutex> lk(api_mutex());
    int st = TMC_OK;
    DeviceCtx *c = current_ctx(&st);
    if (!c)
        return st;
    int32_t *d = nullptr;
    cudaError_t e = cudaMallocAsync(&d, sizeof(int32_t) * n, c->stream);
    if (e != cudaSuccess)
        return set_cuda_error(e, "cudaMallocAsync(debug)");
    const uint32_t blocks = (n + 3) / 4;
    debug_rand_kernel<<<(blocks + 127) / 128, 128, 0, c->stream>>>(
        make_philox_keys(seed), (uint32_t)photon, (uint32_t)(photon >> 32), n, d);
    e = cudaGetLastError();
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(out, d, sizeof(int32_t) * n, cudaMemcpyDeviceToHost, c->stream);
    cudaFreeAsync(d, c->stream);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess)
        return set_cuda_error(e, "tmc_debug_rand");
    return TMC_OK;
}

const char *tmc_strerror(int status)
{
    switch (status) {
    case TMC_OK: return "ok";
    case TMC_E_INVALID: return "invalid parameter";
    case TMC_E_CUDA: return "CUDA error";
    case TMC_E_NOMEM: return "out of memory";
    case TMC_E_TIMEOUT: return "wait timed out";
    case TMC_E_OVERFLOW: return "count overflow";
    case TMC_E_NODEVICE: return "no usable CUDA device";
    case TMC_E_BUSY: return "admission refused";
    case TMC_E_STATE: return "invalid state";
    default: return "unknown status";
    }
}

const char *tmc_last_error(void) { return g_error.c_str(); }

}  // extern "C"
