// tmc_plain.cu — the plain photon-walk kernel: one problem, n photons.
//
// Reference path: tiny_mc.c:47-49 calls photon() (photon.c:6-51) once per
// photon.  Here a persistent grid walks all n photons with the loop in
// tmc_walk.cuh.  Deposits go into a block's shared-memory histogram of the
// problem's shells, added into the 128-bit global tally every flush_steps
// iterations (2^23 / threads) and at the end.
// Short walks over not too many shells (params.h's among them) take
// walk_counts: one count per (step, shell) and block instead of the sums.
// Shell counts whose histogram leaves no room for the SM's blocks (params.h's
// SHELLS is any size in the reference) take the split form: a histogram of the
// shells nearest to the source and of the last one, and 64-bit atomics on the
// 128-bit global tally between them; or, with shells so thin that most deposits
// land beyond it, of the last one alone.  The sums are the same integers in every form.
#include <algorithm>
#include <cmath>

#include "tmc_internal.h"
#include "tmc_walk.cuh"

namespace tmc {

// Photon ids a warp claims per atomic.
//
// Large launches: a quarter of an even share, 32 to 256, so that every
// resident warp has photons and the last claims are short.  A lane walks its
// warp's photons one after another, so a claim of 256 is eight photons in a
// row per lane whatever else is idle: with it fixed at 256, 2^19 high-albedo
// photons kept 2048 of 7296 warps busy (53.7 ms against 40.5) and 32768
// photons ran on 8 of 152 SMs (695 us against 167).
//
// Small launches: one photon, which the whole warp then walks (warp_steps).
// With k steps to the first roulette that costs about n (k / 32 + 1.4) rounds
// on the launch's schedulers, while on lanes it takes the latency of k
// iterations whatever n (exact arithmetic's are the longer).  Measured equal at
// about 11000 photons of params.h optics (k = 73) in fast arithmetic and 14000
// in exact, 17500 and 22000 at k = 342, 18000 and 24000 of high albedo (k =
// 6905); at half of that one to a warp takes 0.7 of the time (6000 photons of
// params.h optics 45 us against 61, 9000 of high albedo 1.8 ms against 3.1).
constexpr unsigned MIN_CHUNK = 32, MAX_CHUNK = 256;

static unsigned claim_chunk(unsigned long long n_photons, unsigned long long warps, int sms, float albedo,
                            bool exact)
{
    const double k = albedo > 0.0f ? std::log(0.001) / std::log((double)albedo) : 0.0;
    if ((double)n_photons < (exact ? 38.0 : 30.0) * 4 * sms * k / (k + 45.0))
        return 1;
    const unsigned long long share = n_photons / (4 * warps) / MIN_CHUNK * MIN_CHUNK;
    return (unsigned)std::max<unsigned long long>(MIN_CHUNK, std::min<unsigned long long>(MAX_CHUNK, share));
}

struct PlainArgs {
    PhiloxKeys keys;
    WalkConsts c;
    unsigned long long n_photons;
    unsigned long long id_base;
    unsigned long long *tally;   // [shells][4]: w lo, w hi, w2 lo, w2 hi
    unsigned long long *work;    // photon claim counter, zero at launch
    unsigned long long *steps;   // += photon steps, may be null
    unsigned chunk;              // photon ids per claim
    uint32_t rows;               // walk_counts: steps with counts
};

// Cells of the split form's histogram: what 1024 threads per SM (two blocks of
// 512) leave of its 228 KB beside the rings and each block's own 1 KB.
__host__ __device__ constexpr uint32_t split_cells(int block)
{
    return ((228 * 1024) / (1024 / block) - 1024 - 4 * SLOTS * block) / 16;
}
__host__ __device__ constexpr uint32_t split_near(int block, uint32_t shells)   // shells nearest to the source in it
{
    return split_cells(block) - LAST_CELLS < shells - 1 ? split_cells(block) - LAST_CELLS : shells - 1;
}
static_assert(split_cells(512) == 4544 && split_cells(128) % 4 == 0, "whole 16-byte rows of the ring behind it");

// 1024 threads per SM.  Where each deposit waits for the L2 (200000 shells of 0.1
// um) 1536 at 40 registers spill in the whole warp's walk: 2^20 photons 1.31 ms
// against 1.21, 2^24 19.43 against 18.10.
template <int BLOCK, class M, Hist H>
__global__ void __launch_bounds__(BLOCK, 1024 / BLOCK) walk_plain(const PlainArgs a)
{
    extern __shared__ __align__(16) uint32_t smem[];
    const uint32_t S = a.c.shells;
    const uint32_t near = H == Hist::Split ? split_near(BLOCK, S) : 0;   // (the whole form counts on S alone)
    // words per histogram
    const uint32_t hist = 4 * (H == Hist::Split ? split_cells(BLOCK) : hist_cells(H == Hist::Far ? 1 : S));
    for (uint32_t s = threadIdx.x; s < hist; s += BLOCK)
        smem[s] = 0;
    __syncthreads();

    GlobalSource src;
    src.counter = a.work;
    src.n = a.n_photons;
    src.id_base = a.id_base;
    src.chunk = a.chunk;
    uint32_t *my = smem + hist + threadIdx.x;   // ring slot k: my[k * BLOCK]
    // (a body of four iterations where each deposit waits: 2^24 photons of three steps
    // over 200000 shells, exact arithmetic, 0.97 ms with eight, 0.81 with four)
    const uint32_t steps = walk_loop<BLOCK, M, GlobalSource, H, H == Hist::Far ? SHORT_TRIP : TRIP>(
        a.c, src, a.keys, smem, a.tally, my, near);

    __syncthreads();
    flush_tally<BLOCK, H>(smem, near, a.c.shells, a.tally);
    if (a.steps) {
        const unsigned long long tot = warp_sum_u64(steps);
        if ((threadIdx.x & 31u) == 0 && tot)
            atomicAdd(a.steps, tot);
    }
}

// One count per (step, shell): see CountTable.  Rows end behind a roulette.
constexpr int COUNT_BLOCK = 512;

__host__ __device__ constexpr uint32_t count_words(uint32_t rows, uint32_t shells)
{
    return ((rows + 1) * (hist_cells(shells) + 2) + 3) / 4 * 4;
}

template <class M, int TRIP>
__global__ void __launch_bounds__(COUNT_BLOCK, 2) walk_counts(const PlainArgs a)
{
    extern __shared__ __align__(16) uint32_t smem[];
    const uint32_t S = a.c.shells, C = hist_cells(S), stride = C + 2, rows = a.rows;
    const uint32_t words = count_words(rows, S);
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(smem);
    const CountTable table{base, base + 4 * rows * stride, 4 * stride, 4 * C};
    for (uint32_t s = threadIdx.x; s < words; s += COUNT_BLOCK)
        smem[s] = 0;
    __syncthreads();
    // each row's weight and the row behind the next roulette, photon.c:32, 45-49
    for (uint32_t n = threadIdx.x; n <= rows; n += COUNT_BLOCK) {
        float weight = WEIGHT_ONE;
        for (uint32_t k = 0;; ++k) {
            if (k == n)
                smem[n * stride + C] = __float_as_uint(weight);
            weight = M::mul(weight, a.c.albedo);
            const bool low = weight < 0.001f * WEIGHT_ONE;
            if (k >= n && (low || k >= rows)) {
                smem[n * stride + C + 1] = base + 4 * (k + 1) * stride;
                break;
            }
            if (low)
                weight = __fdiv_rn(weight, 0.1f);
        }
    }
    __syncthreads();

    GlobalSource src;
    src.counter = a.work;
    src.n = a.n_photons;
    src.id_base = a.id_base;
    src.chunk = a.chunk;
    const float beyond = a.c.last + (float)(threadIdx.x & 31u);
    CountTally<M, COUNT_BLOCK> tally{table, S - 1, a.tally, table.base};
    auto add_steps = [&](unsigned long long n) {
        if (a.steps) {
            n = warp_sum_u64(n);
            if ((threadIdx.x & 31u) == 0 && n)
                atomicAdd(a.steps, n);
        }
    };
    // a warp adds at most 2^27 to a count between its flushes: 2^31 for a block
    walk_photons<COUNT_BLOCK, M, true, (1u << 22), TRIP>(
        a.c, beyond, src, a.keys, smem + words + threadIdx.x, tally, [&] {
            const unsigned long long n = flush_counts<true>(smem, rows, S, threadIdx.x & 31u, 32, 0, 1, a.tally);
            add_steps(n + ((threadIdx.x & 31u) == 0 ? atomicExch(smem + rows * stride, 0u) : 0u));
        });

    __syncthreads();
    // the last shell's cells into its first, then shells x row groups
    for (uint32_t n = threadIdx.x / 32; n < rows; n += COUNT_BLOCK / 32) {
        uint32_t *at = smem + n * stride + S - 1;
        uint32_t v = at[threadIdx.x & 31u];
        v = __reduce_add_sync(FULL_MASK, v);
        if ((threadIdx.x & 31u) == 0)
            *at = v;
    }
    __syncthreads();
    const uint32_t across = min((S + 31) / 32 * 32, (uint32_t)COUNT_BLOCK), groups = COUNT_BLOCK / across;
    unsigned long long counted = threadIdx.x == 0 ? smem[rows * stride] : 0u;
    if (threadIdx.x < groups * across)
        counted += flush_counts<false>(smem, rows, S, threadIdx.x % across, across, threadIdx.x / across, groups,
                                       a.tally);
    add_steps(counted);
}

// Rows up to the fourth, third or second roulette, whichever count table still
// leaves two blocks per SM; 0 if none does.
static uint32_t count_rows(const Derived &d, size_t smem_optin)
{
    const size_t most = (smem_optin + 1024) / 2 - 1024;   // of an SM's shared memory, less a block's own 1 KB
    uint32_t rows = 0;
    float weight = WEIGHT_ONE;
    int roulettes = 0;
    for (uint32_t n = 1; roulettes < 4; ++n) {
        if (4 * (size_t)(count_words(n, d.shells) + SLOTS * COUNT_BLOCK) > most)
            break;
        weight *= d.albedo;
        if (weight < 0.001f * WEIGHT_ONE) {
            weight /= 0.1f;
            if (++roulettes >= 2)
                rows = n;
        }
    }
    return rows;
}

static size_t plain_smem_bytes(uint32_t shells, int block, Hist h)
{
    const uint32_t cells = h == Hist::Split ? split_cells(block) : hist_cells(h == Hist::Far ? 1 : shells);
    return (size_t)16 * cells + (size_t)4 * SLOTS * block;
}

template <int BLOCK, class M, Hist H>
static cudaError_t set_smem(size_t smem)
{
    return cudaFuncSetAttribute(walk_plain<BLOCK, M, H>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

// Blocks of walk_plain<BLOCK, M, H> resident per SM with `smem` bytes (0 if
// it does not fit).
template <int BLOCK, class M, Hist H>
static cudaError_t occupancy(const DeviceCtx &ctx, size_t smem, int &per_sm)
{
    per_sm = 0;
    const size_t cap = ctx.smem_optin ? ctx.smem_optin : 48 * 1024;
    if (smem > cap)
        return cudaSuccess;
    cudaError_t e = set_smem<BLOCK, M, H>(smem);
    if (e != cudaSuccess)
        return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, walk_plain<BLOCK, M, H>, BLOCK, smem);
}

// Grid and arguments of a launch of `block`-thread blocks, per_sm resident.
static unsigned plain_args(const PlainLaunch &L, const DeviceCtx &ctx, int block, int per_sm, PlainArgs &a)
{
    if (L.blocks_per_sm > 0)
        per_sm = std::min(per_sm, L.blocks_per_sm);
    unsigned long long grid = (unsigned long long)ctx.sms * per_sm;
    // no more blocks than there are photon chunks to hand out
    a.chunk = claim_chunk(L.n_photons, grid * (block / 32), ctx.sms, L.d.albedo, L.p->math == TMC_MATH_EXACT);
    const unsigned long long warps_needed = (L.n_photons + a.chunk - 1) / a.chunk;
    const unsigned long long blocks_needed = (warps_needed + block / 32 - 1) / (block / 32);
    grid = std::max(1ull, std::min(grid, blocks_needed));
    if (L.max_blocks > 0)
        grid = std::min(grid, (unsigned long long)L.max_blocks);
    a.keys = make_philox_keys(L.p->seed);
    a.c.albedo = L.d.albedo;
    a.c.spm = L.d.spm;
    a.c.last = L.d.last;
    a.c.shells = L.d.shells;
    a.n_photons = L.n_photons;
    a.id_base = L.p->photon_id_base;
    a.tally = reinterpret_cast<unsigned long long *>(L.d_tally);
    a.work = L.d_work;
    a.steps = L.d_steps;
    a.rows = 0;
    return (unsigned)grid;
}

template <int BLOCK, class M, Hist H>
static cudaError_t launch_t(const PlainLaunch &L, const DeviceCtx &ctx, int per_sm, cudaStream_t stream)
{
    const size_t smem = plain_smem_bytes(L.d.shells, BLOCK, H);
    cudaError_t e = set_smem<BLOCK, M, H>(smem);
    if (e != cudaSuccess)
        return e;
    if (per_sm < 1)
        return cudaErrorInvalidConfiguration;
    PlainArgs a;
    const unsigned grid = plain_args(L, ctx, BLOCK, per_sm, a);
    walk_plain<BLOCK, M, H><<<grid, BLOCK, smem, stream>>>(a);
    return cudaGetLastError();
}

template <class M, int TRIP>
static cudaError_t launch_counts_t(const PlainLaunch &L, const DeviceCtx &ctx, uint32_t rows, cudaStream_t stream)
{
    const size_t smem = 4 * (size_t)(count_words(rows, L.d.shells) + SLOTS * COUNT_BLOCK);
    cudaError_t e =
        cudaFuncSetAttribute(walk_counts<M, TRIP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int per_sm = 0;
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, walk_counts<M, TRIP>, COUNT_BLOCK, smem);
    if (e != cudaSuccess)
        return e;
    if (per_sm < 1)
        return cudaErrorInvalidConfiguration;
    PlainArgs a;
    const unsigned grid = plain_args(L, ctx, COUNT_BLOCK, per_sm, a);
    a.rows = rows;
    walk_counts<M, TRIP><<<grid, COUNT_BLOCK, smem, stream>>>(a);
    return cudaGetLastError();
}

static cudaError_t launch_counts(const PlainLaunch &L, const DeviceCtx &ctx, uint32_t rows, cudaStream_t stream)
{
    if (L.p->math == TMC_MATH_FAST)
        return L.d.albedo < SHORT_ALBEDO ? launch_counts_t<FastMath, SHORT_TRIP>(L, ctx, rows, stream)
                                         : launch_counts_t<FastMath, TRIP>(L, ctx, rows, stream);
    return L.d.albedo < SHORT_ALBEDO ? launch_counts_t<ExactMath, SHORT_TRIP>(L, ctx, rows, stream)
                                     : launch_counts_t<ExactMath, TRIP>(L, ctx, rows, stream);
}

// The split form pays where its histogram reaches far enough: a walk of k steps
// of about a mean free path ends about sqrt(k) of them out.  512-thread blocks (4512
// shells), 2^20 photons over 20000 shells at params.h optics (k = 73): 0.34 um (a
// reach of 0.4) 1.70 ms split, 1.22 far; 0.52 um (0.6) 1.49, 1.34; 0.60 um (0.7)
// 1.33, 1.46; 0.86 um (1.0) 0.93, 1.55; 1.7 um 0.65, 1.67.  At albedo 0.09 (k = 3)
// either within 20%: 0.24 um (0.6) 0.088, 0.074; 0.8 um (2.0) 0.078, 0.091.
static bool reaches(uint32_t shells, const Derived &d)
{
    const double k = d.albedo > 0.0f ? std::log(0.001) / std::log((double)d.albedo) : 0.0;
    return shells >= 0.6 * d.spm * std::sqrt(1.0 + k);
}

template <int BLOCK, class M, Hist H>
static cudaError_t try_launch(const PlainLaunch &L, const DeviceCtx &ctx, cudaStream_t stream)
{
    int per_sm = 0;
    const cudaError_t e = occupancy<BLOCK, M, H>(ctx, plain_smem_bytes(L.d.shells, BLOCK, H), per_sm);
    return e == cudaSuccess ? launch_t<BLOCK, M, H>(L, ctx, per_sm, stream) : e;
}

// A histogram per block where it leaves the SM its 1024 threads, else the split
// form where it reaches (8000 shells of 12.5 um, 2^21 photons of params.h
// optics: one block per SM 1.26 ms, split 1.02; but of 0.86 um, 2^20 photons, 0.66
// and 0.90), else a block's histogram at any occupancy (8000 shells of 0.35 um: one
// block per SM 0.66 ms, far 1.13), else far.
template <int BLOCK, class M>
static cudaError_t launch_m(const PlainLaunch &L, const DeviceCtx &ctx, cudaStream_t stream)
{
    const uint32_t S = L.d.shells;
    int block_sm = 0;
    const cudaError_t e = occupancy<BLOCK, M, Hist::Block>(ctx, plain_smem_bytes(S, BLOCK, Hist::Block), block_sm);
    if (e != cudaSuccess)
        return e;
    if (block_sm >= 1024 / BLOCK)
        return launch_t<BLOCK, M, Hist::Block>(L, ctx, block_sm, stream);
    if (reaches(split_near(BLOCK, S), L.d))
        return try_launch<BLOCK, M, Hist::Split>(L, ctx, stream);
    if (block_sm >= 1)
        return launch_t<BLOCK, M, Hist::Block>(L, ctx, block_sm, stream);
    return try_launch<BLOCK, M, Hist::Far>(L, ctx, stream);
}

template <int BLOCK>
static cudaError_t launch_b(const PlainLaunch &L, const DeviceCtx &ctx, cudaStream_t stream)
{
    return L.p->math == TMC_MATH_FAST ? launch_m<BLOCK, FastMath>(L, ctx, stream)
                                      : launch_m<BLOCK, ExactMath>(L, ctx, stream);
}

template <class M>
static cudaError_t load_kernels()
{
    const void *kernels[] = {
        (const void *)walk_plain<128, M, Hist::Block>, (const void *)walk_plain<128, M, Hist::Split>,
        (const void *)walk_plain<128, M, Hist::Far>,   (const void *)walk_plain<512, M, Hist::Block>,
        (const void *)walk_plain<512, M, Hist::Split>, (const void *)walk_plain<512, M, Hist::Far>,
        (const void *)walk_counts<M, TRIP>, (const void *)walk_counts<M, SHORT_TRIP>};
    for (const void *k : kernels) {
        cudaFuncAttributes attr;
        const cudaError_t e = cudaFuncGetAttributes(&attr, k);
        if (e != cudaSuccess)
            return e;
    }
    return cudaSuccess;
}

cudaError_t launch_plain(const PlainLaunch &L, const DeviceCtx &ctx, cudaStream_t stream)
{
    // Counts instead of sums wherever their table fits and the launch fills the
    // device: 2^24 photons of params.h optics 7.63 -> 6.72 ms, 2^25 in exact
    // arithmetic 20.0 -> 18.2 ms, 2^22 at albedo 0.09 0.25 -> 0.15 ms.  In smaller
    // launches setting the table up and adding it costs more: 100000 photons 125
    // us against 100, 131072 127 against 118, 155000 128 against 130; at albedo
    // 0.09 70000 photons 38 against 64.
    const unsigned long long per_sm = L.n_photons / (unsigned)ctx.sms;
    const bool fill = per_sm >= (L.d.albedo < SHORT_ALBEDO ? 256 : 900);
    // Sums take blocks of 128 threads where eight histograms fit an SM: they
    // spread small launches over more SMs (32768 photons on 64 blocks of 512
    // took 114 us, 84 on 256 of 128) and end one by one (2^18 high-albedo
    // photons 13.3 -> 12.5 ms).  More shells take them below 512 photons per SM:
    // with walks of 73 steps, of the time of 512-thread blocks, 0.8 - 1.1 at 1100 ..
    // 2500 shells and 100 - 300 photons per SM, 1.2 - 1.3 at 500 (past 2900 shells,
    // where fewer than four blocks fit an SM, 1.0 - 2).  Short walks take 512: setting
    // a small block's histogram up and adding it is most of their time (75000 photons
    // at 10/cm and 1/cm: 7000 shells 61 us against 29, 12000 of 0.3 um 83 against 29).
    const bool blocks128 = hist_cells(L.d.shells) <= split_cells(128) ||
                           (per_sm < 512 && L.d.albedo >= SHORT_ALBEDO);
    // a launch of no photons is a caller's set-up call: it loads every kernel
    // a call of its arithmetic may take
    if (L.n_photons == 0 && !L.block) {
        const cudaError_t e = L.p->math == TMC_MATH_FAST ? load_kernels<FastMath>() : load_kernels<ExactMath>();
        if (e != cudaSuccess)
            return e;
    }
    if (L.block == 0 && fill) {
        const uint32_t rows = count_rows(L.d, ctx.smem_optin);
        if (rows)
            return launch_counts(L, ctx, rows, stream);
    }
    switch (L.block ? L.block : blocks128 ? 128 : 512) {
    case 128: return launch_b<128>(L, ctx, stream);
    case 256: return launch_b<256>(L, ctx, stream);
    case 512: return launch_b<512>(L, ctx, stream);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace tmc
