// tmc_walk.cuh — the photon-walk loop shared by the plain and batched kernels.
//
// Reference path: tiny_mc.c:47-49 calls photon() (photon.c:6-51) once per
// photon.  Here every thread of a persistent grid carries one photon at a
// time and warps refill dead lanes with new photon ids:
//
//  * when a photon dies in the roulette (photon.c:45-49) its lane takes the
//    next photon id from a chunk its warp claimed from a PhotonSource (a
//    global counter for the plain kernel, a shared-memory counter over one
//    work item for the batched kernel), so lanes never idle while work
//    remains;
//  * the rejection loop of photon.c:36-40 is folded into the main loop: each
//    iteration evaluates the next two rejection tries from the buffered
//    stream and consumes only the words photon.c would (two if the first try
//    is accepted, four otherwise).  A photon whose two tries both failed
//    (p = 0.046) skips the move/absorb part on the next iteration, so lanes
//    of a warp stay in lock-step instead of waiting for the lane with the
//    most retries;
//  * random words come, as floats, from a per-thread ring of 16 slots in shared
//    memory; slots 16..20 mirror 0..4, so the <= 6 words one iteration reads (step,
//    four for two tries, roulette) are fixed offsets from one base.  Every
//    second iteration each lane computes two Philox blocks and stores them if
//    its ring has room for eight words.  No vote decides on a refill: an
//    iteration uses 3.4 words on average and a refill brings four per
//    iteration, so a vote would save 6% of the Philox work and cost more
//    than that; without it the loop is straight-line code whose Philox
//    multiplies overlap the walk's arithmetic;
//  * the two tallies of photon.c:30-31 go into a shared-memory histogram of
//    64-bit fixed-point sums (sum of w and of w^2, 2^-40 units), each kept as
//    two 32-bit words updated with native 32-bit shared atomics (a 64-bit
//    shared atomicAdd is a compare-and-swap loop, 4x slower here), or, for
//    short walks over not too many shells, into one 32-bit count per step
//    number and shell (CountTable).  A warp adds the block's histogram into the
//    128-bit global tally and clears it every flush_steps iterations, which
//    keeps the sums from wrapping, so a deposit needs no wrap check;
//  * the last few photons of a warp, whose lanes would each take a step in
//    turns that nobody else shares, are walked by all 32 lanes (warp_steps).
//
// What bounds it: instruction issue.  2^25 photons of params.h optics in fast
// arithmetic: 226 thread-instructions per photon step before the loop took this
// form (8.34 warp-instructions, 3.28 per clock per SM), 159 with sums (5.86,
// 3.03), 136 with counts (4.89, 2.97); shared-memory wavefronts 69% of peak
// with sums, 34% with counts; ALU pipe 53%, heavy FMA pipe (Philox multiplies)
// 42%.  Exact arithmetic 194 (6.97, 3.13).  What the loop's parts were worth, 2^26 such
// photons with sums: 41.1 ms with voted single-block refills, 35.1 with one
// unvoted block per iteration, 33.8 with the loop body unrolled twice, 32.1 with
// two blocks every second iteration (which share the round-key loads), 31.2
// with four iterations per check for finished photons; with counts and eight
// iterations 26.9.  Occupancy does not matter at this point: 48 warps per SM
// (40 registers) measured the same as 32.
#pragma once

#include "tmc_device.cuh"

namespace tmc {

constexpr int RING = 16;        // random words buffered per thread
constexpr int MIRROR = 5;       // slots 16..20 repeat slots 0..4
constexpr int SLOTS = RING + MIRROR;

// Iterations of the unrolled loop body, between checks for finished photons.  A
// check is ~60 warp-instructions when a photon has ended, a lane whose photon
// ended waits half a body, and every pass through the loop moves the lane's
// state between registers (5 instructions per step with a body of 4).  2^26
// photons of params.h optics: 27.8 ms with 4, 27.3 with 6, 26.9 with 8; 2^20
// high-albedo 44.1, 42.5, 42.3; 2^22 photons of three steps (albedo 0.09)
// 0.152, 0.169, 0.175 ms.  (Two passes through a body of 4 per check: 27.9.)
// walk_counts and walk_batch (brief_walk) have a kernel of each length.  (Both loops
// in one kernel, or one that leaves a body of 8 in its middle: 1.5% slower for long
// walks.)
constexpr int TRIP = 8, SHORT_TRIP = 4;
constexpr float SHORT_ALBEDO = 0.8f;   // below: walks of under 31 steps to the first roulette

// The whole warp walks its photons one after another (warp_steps) once the
// source has no more and at most this many are left.  A lane-loop iteration is
// ~190 warp-instructions however few lanes walk, a photon's step by the whole
// warp ~23, so 8 is where the issue slots break even.  4096-problem sweep at a
// reduced scale: 788 ms without, 608 (6), 619 (10), 615 (16), 812 ms (24).
// A round of the whole warp costs the same however few of its 32 steps are walked,
// so short walks, whose last photons have about k / 2 steps to go (k to the first
// roulette), go on in lanes: one photon per 8 steps of k.  Batches of short walks
// (albedo 0.01, exact arithmetic), with four iterations per check as well: 4000
// problems of 200 photons 260 -> 115 us in 512-thread blocks, 500 of 100000 2.34 ->
// 1.47 ms.  The kernels for long walks keep the constant: read from a register it
// costs them 1%.
constexpr int WARP_WALK_MAX = 8;
__device__ __forceinline__ int warp_walk_most(float albedo)
{
    const float a2 = albedo * albedo, a4 = a2 * a2, a8 = a4 * a4;   // the weight after 8 steps
    int most = 0;
    for (float weight = a8; most < WARP_WALK_MAX && weight >= 0.001f; weight *= a8)
        ++most;
    return most;
}

// Where a walk keeps its tallies.  Block: a shared histogram per block (one per
// warp measured the same from 2^18 photons on and costs small launches more
// flushes: 75000 photons 127 us against 96).  Split: a block's histogram holds
// the shells nearest to the source, where nearly all deposits of a point source
// land, and the last one, and a deposit between them is a 64-bit atomic add into
// the 128-bit global tally (shell counts whose histogram does not fit in shared
// memory).  Far: the last one alone (shells so thin that most deposits land beyond
// such a histogram).  Counts have a tally of their own (CountTally).
enum class Hist { Block, Split, Far };

// A warp adds its block's histogram, of `lanes` lanes, into the global tally and
// clears it every flush_steps(lanes) of its iterations.  A lane deposits at most once per
// iteration, so between two flushes, whichever warps make them, every lane
// deposits at most flush_steps times (its warp would have flushed).  A deposit
// adds at most 2^8 + 1 to a high word (w <= 1, plus the low word's carry), so
// a high word stays below lanes * 257 * (2^23 / lanes + 1) < 2^32: the 64-bit
// sums never wrap.
__host__ __device__ constexpr uint32_t flush_steps(uint32_t lanes)
{
    return (1u << 23) / lanes;
}
static_assert(512ull * 257ull * ((1ull << 23) / 512 + 1) < (1ull << 32), "high word bound");

// Cells of a shared histogram or row of counts.  Every photon beyond the last
// shell deposits into it (photon.c:27-29): in an optically thin problem nearly all
// lanes of a warp at once, and shared atomics on one word take their turns.  So the
// last shell has 32 cells, one per lane, which the flushes add up.  2^20 high-albedo
// photons (1001 shells of 10 um, many walks leave): 46.8 -> 44.8 ms; the reduced
// 4096-problem sweep 609 -> 555 ms.
// They stand in the last shell's place, in the split forms before shell 0, and those
// use the one at -1 alone: as global atomics on one address 2^21 photons of params.h
// optics over 4600 shells of 0.53 um took 128.7 ms, 1.65 so, 1.16 with a cell per lane;
// but where few photons leave (2000003 photons, 20000 shells of 5 um) 1.007 ms so, 1.023
// with a lane's own constant held through the loop, 1.045 with the cells behind the near
// shells (a second compare and a branch's join).  (Before shell 0 in a whole histogram:
// 7% slower in walk_batch's 256-thread blocks at albedo 0.99.)
constexpr uint32_t LAST_CELLS = 32;
__host__ __device__ constexpr uint32_t hist_cells(uint32_t shells) { return shells + LAST_CELLS - 1; }
// Index of shell 0's cell, and of the last shell's first, in a histogram of `near`
// shells and the last.
template <Hist H>
__device__ __forceinline__ uint32_t shell0_cell()
{
    return H == Hist::Block ? 0 : LAST_CELLS;
}
template <Hist H>
__device__ __forceinline__ uint32_t last_cell(uint32_t near)
{
    return H == Hist::Block ? near : 0;
}

// Take the 64-bit sum of a cell, by atomic exchanges against zero.
__device__ __forceinline__ unsigned long long take_cell(uint32_t *lo, uint32_t *hi)
{
    const uint32_t l = atomicExch(lo, 0u), h = atomicExch(hi, 0u);
    return ((unsigned long long)h << 32) | l;
}

// Add a histogram of the first `near` shells (H = Block: all) and the last of S into
// the 128-bit global tally and clear it, by one warp while the others keep
// depositing: every word is taken with an atomic exchange against zero.  Sums stay
// exact: a deposit's low-word overflow is carried into a high word by the
// depositing lane, whichever side of an exchange either add lands on, and every
// word's content reaches the global tally at one flush or the next.  probe_acc /
// probe_hi (shared, may be null): the 128-bit running sum of the w words taken from
// shell probe_shell.  Warp-collective.  The last shell's cells are added up first
// (their total obeys the bound above, so it fits 64 bits).  (Block's shell count is
// not passed: a register held for it through the loop costs 0.5 - 4%.)
template <Hist H>
__device__ __forceinline__ void warp_flush_tally(uint32_t *tally, uint32_t near, uint32_t S, unsigned long long *g,
                                                 unsigned long long *probe_acc = nullptr,
                                                 uint32_t *probe_hi = nullptr, uint32_t probe_shell = 0)
{
    if constexpr (H == Hist::Block)
        near = S - 1;
    const uint32_t C = hist_cells(near + 1), lane = threadIdx.x & 31u;
    __syncwarp();
    uint32_t *const first = tally + shell0_cell<H>(), *const last = tally + last_cell<H>(near);
    for (uint32_t s = lane; s < near; s += 32) {
        const unsigned long long v = take_cell(&first[s], &first[C + s]);
        flush128(&g[4 * s + 0], &g[4 * s + 1], v);
        if (probe_acc && s == probe_shell && v) {
            const unsigned long long old = atomicAdd(probe_acc, v);
            if (old + v < old)
                atomicAdd(probe_hi, 1u);
        }
        flush128(&g[4 * s + 2], &g[4 * s + 3], take_cell(&first[2 * C + s], &first[3 * C + s]));
    }
    __syncwarp();
    const unsigned long long v = warp_sum_u64(take_cell(&last[lane], &last[C + lane]));
    const unsigned long long v2 = warp_sum_u64(take_cell(&last[2 * C + lane], &last[3 * C + lane]));
    if (lane == 0) {
        unsigned long long *gl = g + 4 * (size_t)(S - 1);
        flush128(&gl[0], &gl[1], v);
        if (probe_acc && S - 1 == probe_shell && v) {
            const unsigned long long old = atomicAdd(probe_acc, v);
            if (old + v < old)
                atomicAdd(probe_hi, 1u);
        }
        flush128(&gl[2], &gl[3], v2);
    }
    __syncwarp();
}

// ------------------------------------------- counts per step and shell
// A photon's weight is a function of the number of its steps alone: it decays
// by one multiplication a step, and whether a roulette follows, and what
// survivors are multiplied by, depends on the weight only.  So instead of two
// 64-bit sums per shell (four atomics, two conversions and two carries a step),
// a block can keep one 32-bit count per (step number, shell) and multiply by the
// step's tally units at the end: the same integers, one atomic a step and no
// weight in the loop.  It takes rows for the steps up to the second, third or
// fourth roulette; a photon that survives that one (1 in 100 .. 10^4) is walked
// to its end by the whole warp and tallied with 64-bit global atomics.
//
// A row is hist_cells counts, the weight (times 2^20) its deposits have, and
// the address just behind the next roulette's row; one more row holds the
// weight behind the last and, in its first word, the number of steps outside the
// table.  Addresses are shared-memory bytes.
struct CountTable {
    uint32_t base, end, stride;
    uint32_t weight_at;   // of a row's weight; the roulette address follows
};

__device__ __forceinline__ uint32_t ld_shared(uint32_t addr)
{
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}

// Add a 128-bit value into a 128-bit global tally.
__device__ __forceinline__ void flush128(unsigned long long *g_lo, unsigned long long *g_hi, unsigned long long lo,
                                         unsigned long long hi)
{
    if (lo | hi) {
        const unsigned long long old = atomicAdd(g_lo, lo);
        hi += old + lo < old ? 1ull : 0ull;
        if (hi)
            atomicAdd(g_hi, hi);
    }
}

// Add the counts of shells s0, s0 + ds, ... over rows n0, n0 + dn, ... into the
// global tally; returns the sum of the counts.  EXCHANGE: take and clear them by
// atomic exchanges while other warps deposit, the last shell's cells included;
// else shell S-1's first cell holds the sum of its cells.
template <bool EXCHANGE>
__device__ __forceinline__ unsigned long long flush_counts(uint32_t *table, uint32_t rows, uint32_t S, uint32_t s0,
                                                           uint32_t ds, uint32_t n0, uint32_t dn,
                                                           unsigned long long *g)
{
    const uint32_t C = hist_cells(S), stride = C + 2;
    unsigned long long total = 0;
    for (uint32_t s = s0; s < S; s += ds) {
        unsigned long long lo = 0, hi = 0, lo2 = 0, hi2 = 0;
        for (uint32_t n = n0; n < rows; n += dn) {
            uint32_t *row = table + n * stride;
            uint32_t count = 0;
            if constexpr (EXCHANGE) {
                for (uint32_t c = s; c < (s + 1 < S ? s + 1 : C); ++c)
                    count += atomicExch(row + c, 0u);
            } else {
                count = row[s];
            }
            if (count == 0)
                continue;
            total += count;
            const float weight = __uint_as_float(row[C]);
            uint32_t l, h;
            units_split(weight_units(weight), l, h);
            const unsigned long long u = ((unsigned long long)(h - UNITS_HI_BIAS) << 32) | l;
            units_split(weight2_units(weight), l, h);
            const unsigned long long u2 = ((unsigned long long)(h - UNITS_HI_BIAS) << 32) | l;
            lo += u * count;
            hi += __umul64hi(u, count) + (lo < u * count ? 1ull : 0ull);
            lo2 += u2 * count;
            hi2 += __umul64hi(u2, count) + (lo2 < u2 * count ? 1ull : 0ull);
        }
        unsigned long long *gs = g + 4 * (size_t)s;
        flush128(&gs[0], &gs[1], lo, hi);
        flush128(&gs[2], &gs[3], lo2, hi2);
    }
    return total;
}

// Per-problem constants of photon.c:8-9 (computed on the host in float,
// exactly as photon.c does) plus the shell count.
struct WalkConsts {
    float albedo;
    float spm;     // shells_per_mfp
    float last;    // (float)(shells - 1)
    uint32_t shells;
};

// Photon ids from a global 64-bit counter over [0, n): each warp claims
// `chunk` ids per atomic.
struct GlobalSource {
    unsigned long long *counter;
    unsigned long long n;
    unsigned long long id_base;
    unsigned chunk;   // below 32: lanes a claim leaves without a photon get none
    unsigned long long next_id = 0;   // of the ids claimed and not handed out,
    unsigned left = 0;                // and how many there are
    bool exhausted = false;

    // Warp-collective.  need = ballot of lanes wanting a photon, rank = this
    // lane's index among them.  Returns true and the photon id if this lane
    // got one (only meaningful for wanting lanes).
    __device__ __forceinline__ bool next(unsigned need, unsigned rank, unsigned lane,
                                         unsigned long long &pid)
    {
        const unsigned n_need = __popc(need);
        unsigned long long id = next_id + rank;
        bool got = rank < left;
        if (n_need > left) {
            const unsigned had = left;
            unsigned long long base = 0;
            if (!exhausted) {
                if (lane == 0)
                    base = atomicAdd(counter, (unsigned long long)chunk);
                base = __shfl_sync(FULL_MASK, base, 0);
                exhausted = base >= n;
            }
            const unsigned fresh = exhausted ? 0u : (unsigned)min((unsigned long long)chunk, n - base);
            const unsigned used = min(n_need - had, fresh);
            if (!got) {
                id = base + (rank - had);
                got = rank - had < fresh;
            }
            next_id = base + used;
            left = fresh - used;
        } else {
            next_id += n_need;
            left -= n_need;
        }
        pid = id_base + id;
        return got;
    }
};

// Photon ids from a shared-memory 32-bit counter over one work item of
// `count` photons starting at id `first`.
struct SharedSource {
    uint32_t *counter;   // shared memory, zero at the start of the item
    uint32_t count;
    unsigned long long first;
    uint32_t chunk;      // ids per claim (as GlobalSource's)
    uint32_t cnext = 0, cend = 0;
    bool exhausted = false;

    __device__ __forceinline__ bool next(unsigned need, unsigned rank, unsigned lane,
                                         unsigned long long &pid)
    {
        const unsigned n_need = __popc(need);
        uint32_t id = cnext + rank;
        bool got = rank < cend - cnext;
        if (n_need > cend - cnext) {
            const unsigned take0 = cend - cnext;
            uint32_t base = 0;
            if (!exhausted) {
                if (lane == 0)
                    base = atomicAdd(counter, chunk);
                base = __shfl_sync(FULL_MASK, base, 0);
                exhausted = base >= count;
            }
            if (exhausted) {
                cnext = cend;
            } else {
                cend = min(base + chunk, count);
                if (!got) {
                    id = base + (rank - take0);
                    got = id < cend;
                }
                cnext = min(base + (n_need - take0), cend);
            }
        } else {
            cnext += n_need;
        }
        pid = first + id;
        return got;
    }
};

// A lane's photon.  Ring positions are in bytes (slot x the W bytes between a
// thread's slots) modulo 2^32: blk * 4 W is the end of the words produced,
// cur the next word to use; their difference is the fill, and a lane without
// a photon is kept at a fill of -W.
struct LanePhoton {
    PhotonKey key;
    uint32_t blk = 0, cur = 0;
    float x = 0.f, y = 0.f, z = 0.f, u = 0.f, v = 0.f, w = 0.f;
    float weight = 0.f;   // times 2^20 (an exact scaling)
    // Norm of the last try; above 1 the direction is still sought, and cur is
    // one word before the next try's (where a step's own word would be), so
    // that tries are always words 1 .. 4 from cur.
    float t = 0.f;
};

template <int BLOCK>
struct Ring {
    static constexpr uint32_t W = BLOCK * 4;
    static constexpr uint32_t MASK = RING * W - 1;
    static constexpr uint32_t NO_PHOTON = W;   // cur - blk * 4 W of a lane without one

    __device__ static __forceinline__ int fill(const LanePhoton &p) { return (int)(p.blk * (4 * W) - p.cur); }
    __device__ static __forceinline__ bool walking(const LanePhoton &p) { return fill(p) >= 0; }
    __device__ static __forceinline__ void drop(LanePhoton &p) { p.cur = p.blk * (4 * W) + NO_PHOTON; }
    // A photon its lane cannot go on with: kept at a fill below -W until the
    // whole warp walks it.
    static constexpr uint32_t ASIDE = 4 * RING * W;
    __device__ static __forceinline__ void set_aside(LanePhoton &p) { p.cur += ASIDE; }
    __device__ static __forceinline__ bool aside(const LanePhoton &p) { return fill(p) < -(int)W; }
    __device__ static __forceinline__ float real(const char *at, int slot)
    {
        return *reinterpret_cast<const float *>(at + slot * W);
    }

    // Two Philox blocks into the ring where it has room for them (a lane
    // without a photon, or set aside, has a negative fill: no room).
    __device__ static __forceinline__ void refill(LanePhoton &p, char *ring, const PhiloxKeys &keys)
    {
        const uint4 r = philox_block(p.blk, p.key, keys);
        const uint4 q = philox_block(p.blk + 1, p.key, keys);
        const uint32_t off = (p.blk * (4 * W)) & MASK;
        const uint32_t filled = (uint32_t)fill(p);
        const uint32_t at = (uint32_t)__cvta_generic_to_shared(ring) + off;
        // predicated stores: branches around them cost more than the stores
        asm volatile("{\n\t.reg .pred p, q;\n\t"
                     "setp.le.u32 p, %0, %11;\n\tsetp.eq.and.u32 q, %1, 0, p;\n\t"
                     "@p st.shared.f32 [%2], %3;\n\t@p st.shared.f32 [%2+%12], %4;\n\t"
                     "@p st.shared.f32 [%2+%13], %5;\n\t@p st.shared.f32 [%2+%14], %6;\n\t"
                     "@p st.shared.f32 [%2+%15], %7;\n\t@p st.shared.f32 [%2+%16], %8;\n\t"
                     "@p st.shared.f32 [%2+%17], %9;\n\t@p st.shared.f32 [%2+%18], %10;\n\t"
                     "@q st.shared.f32 [%2+%19], %3;\n\t@q st.shared.f32 [%2+%20], %4;\n\t"
                     "@q st.shared.f32 [%2+%21], %5;\n\t@q st.shared.f32 [%2+%22], %6;\n\t"
                     "@q st.shared.f32 [%2+%23], %7;\n\t}" ::"r"(filled),
                     "r"(off), "r"(at), "f"(rand_float(r.x)), "f"(rand_float(r.y)), "f"(rand_float(r.z)),
                     "f"(rand_float(r.w)), "f"(rand_float(q.x)), "f"(rand_float(q.y)), "f"(rand_float(q.z)),
                     "f"(rand_float(q.w)), "n"((RING - 8) * W), "n"(W), "n"(2 * W), "n"(3 * W), "n"(4 * W),
                     "n"(5 * W), "n"(6 * W), "n"(7 * W), "n"(RING * W), "n"((RING + 1) * W), "n"((RING + 2) * W),
                     "n"((RING + 3) * W), "n"((RING + 4) * W)
                     : "memory");
        static_assert(MIRROR == 5, "the mirror stores above");
        if (filled <= (RING - 8) * W)
            p.blk += 2;
    }

    // Words of the photon's stream used so far, as whole blocks and a rest.
    __device__ static __forceinline__ void position(const LanePhoton &p, uint32_t &block, uint32_t &rest)
    {
        const uint32_t words = (uint32_t)fill(p) / W;
        block = p.blk - (words + 3) / 4;
        rest = (0u - words) & 3u;
    }
    // Continue from a position with nothing buffered.
    __device__ static __forceinline__ void restart(LanePhoton &p, uint32_t block, uint32_t rest, char *ring,
                                                   const PhiloxKeys &keys)
    {
        const uint32_t even = block & ~1u;   // refills fill half a ring
        p.blk = even;
        p.cur = even * (4 * W);
        refill(p, ring, keys);
        p.cur += (4 * (block - even) + rest) * W;
    }
};

// Photon launch, photon.c:12-18.
template <class M>
__device__ __forceinline__ void launch_photon(LanePhoton &p, unsigned long long pid, const PhiloxKeys &keys)
{
    p.key = photon_key(pid, keys);
    p.blk = 0;
    p.cur = 0;
    p.x = p.y = p.z = 0.f;
    p.u = p.v = 0.f;
    p.w = M::ONE;
    p.weight = WEIGHT_ONE;
    p.t = 0.f;
}

// One iteration of a lane's photon if six words are buffered (else it waits
// for the next refill): move, deposit and decay unless its direction is still
// sought, then two tries for the next direction and the roulette.
// A radius below `last` shells goes to its shell's cell, any other (NaN too) to
// cell `beyond`, which may be negative.  The tally keeps the photon's weight:
// step(p, cell) deposits and decays it, low(p) says whether it is below the
// roulette's threshold, survived(p) and died(p) are the roulette's outcomes.
template <int BLOCK, class M, class Tally>
__device__ __forceinline__ void step_photon(LanePhoton &p, const char *ring, float spm, float last, float beyond,
                                            Tally &tally)
{
    using R = Ring<BLOCK>;
    if (R::fill(p) < (int)(6 * R::W))
        return;
    const char *rd = ring + (p.cur & R::MASK);
    if (!(p.t > 1.0f)) {
        // move, photon.c:21-24
        const float t = M::step_length(uniform01(R::real(rd, 0)));
        p.x = M::move(p.x, t, p.u);
        p.y = M::move(p.y, t, p.v);
        p.z = M::move(p.z, t, p.w);
        // absorb, photon.c:26-32 (clamp in float: same shell for every radius
        // below 2^32 shells)
        const float r = M::radius_shells(p.x, p.y, p.z, spm);
        tally.step(p, (uint32_t)__float2int_rz(r < last ? r : beyond));
    }
    // the next two tries of the rejection method, photon.c:36-40; the second
    // one's words are consumed only if the first is rejected
    const float xa1 = uniform_pm1(R::real(rd, 1)), xa2 = uniform_pm1(R::real(rd, 2));
    const float xb1 = uniform_pm1(R::real(rd, 3)), xb2 = uniform_pm1(R::real(rd, 4));
    const float ta = M::norm2(xa1, xa2), tb = M::norm2(xb1, xb2);
    const bool first = !(1.0f < ta);
    const float xi1 = first ? xa1 : xb1;
    const float xi2 = first ? xa2 : xb2;
    p.t = first ? ta : tb;
    const bool sought = p.t > 1.0f;
    p.cur += first ? 3 * R::W : sought ? 4 * R::W : 5 * R::W;
    // new direction, photon.c:41-43 (that of a rejected try is not used; where
    // it costs little it is computed all the same, without a branch)
    if (M::CHEAP_DIRECTION || !sought)
        M::direction(p.t, xi1, xi2, p.u, p.v, p.w);
    // roulette, photon.c:45-49
    if (!sought && tally.low(p)) {
        const float U = uniform01(R::real(ring + (p.cur & R::MASK), 0));
        p.cur += R::W;
        if (U > 0.1f) {
            R::drop(p);
            tally.died(p);
        } else {
            tally.survived(p);
        }
    }
}

// ------------------------------------------------- one photon, whole warp
// A photon's steps are a serial chain only through its position in the random
// stream and the sums x += t u; everything else of a step follows from its
// words.  With few photons left in a warp, all 32 lanes therefore walk ONE
// photon, up to 32 steps at a time, in the same arithmetic and order:
//
//  * lane l computes Philox block l of the next 32 (128 words) and the
//    outcome of a rejection try at each of its four word positions; ballots
//    give, for a step starting at any position, where the next one starts;
//  * lane k finds the k-th step's start by applying that map k times
//    (doubling it by shuffles), then step k's length and new direction;
//  * the sums run over the steps in order, x, y and z in a lane each and the
//    repeatedly multiplied weight in a fourth: the only serial part;
//  * radius and deposit are again one step per lane.  A roulette ends a round.
//
// A round is ~730 warp-instructions (exact arithmetic) for 32 steps, bound by
// latency on an idle SM and by issue on a full one.  One high-albedo photon
// (7168 steps): 2.31 ms on its lane, 0.29 ms here.  4099 of them, one to a warp
// at a time: 4.2 -> 1.0 ms.  Groups of eight lanes with a photon each, 16 steps
// a round, measured slower: 0.64 and 1.6 ms.
struct WarpPhoton {   // the same in every lane
    PhotonKey key;
    uint32_t block, rest;   // words used: 4 block + rest
    float x, y, z, u, v, w, weight;
};

// Scratch of the warp: four rows of 32 words, `stride` bytes apart.
struct WarpScratch {
    char *rows;
    uint32_t stride;
    __device__ __forceinline__ char *row(uint32_t r) const { return rows + r * stride; }
    __device__ __forceinline__ uint32_t word(uint32_t p) const
    {
        return *reinterpret_cast<const uint32_t *>(rows + (p >> 5) * stride + (p & 31u) * 4);
    }
};

// Where a step starting at word 127 would end: not within the round, like any
// step whose successor is not below 127.  The map sends those to 127, which it
// sends to itself, so looking a position up needs no bounds check.
constexpr uint32_t NO_STEP = 127;

// next[p], p < 128, of a map packed four positions to a lane.
__device__ __forceinline__ uint32_t map_at(uint32_t packed, uint32_t p)
{
    return __byte_perm(__shfl_sync(FULL_MASK, packed, (int)(p >> 2)), 0u, 0x4440u | (p & 3u));
}

// Start of the step after one whose tries are bit 0 of c, then of d, then
// bit 1 of c, ...: at_c / at_d is the position of the first try of either.
__device__ __forceinline__ uint32_t after_try(uint32_t c, uint32_t d, uint32_t at_c, uint32_t at_d)
{
    const uint32_t any = c | d;
    const uint32_t k = __ffs((int)any) - 1;
    const uint32_t at = ((c >> (k & 31u)) & 1u) ? at_c : at_d;
    return any ? min(at + 4 * k + 2, NO_STEP) : NO_STEP;
}

// Word `at` of the photon's stream, counted from block p.block.
__device__ __forceinline__ uint32_t stream_word(const WarpPhoton &p, uint32_t at, const PhiloxKeys &keys)
{
    const uint4 q = philox_block(p.block + (at >> 2), p.key, keys);
    const uint32_t i = at & 3u;
    return i == 0u ? q.x : i == 1u ? q.y : i == 2u ? q.z : q.w;
}

// Up to 32 steps of the photon; returns their number n >= 1.  Lanes below n
// hold a step each: the cell it deposits into and the weight.  dead is set when
// the roulette ended the photon.
template <class M>
__device__ __forceinline__ uint32_t warp_steps(WarpPhoton &p, bool &dead, const WarpScratch &sc, const WalkConsts &c,
                                               const PhiloxKeys &keys, float beyond, uint32_t &cell_out,
                                               float &weight_out)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint4 r = philox_block(p.block + lane, p.key, keys);
    __syncwarp();   // the rows' earlier contents are read
    *reinterpret_cast<uint4 *>(sc.row(lane >> 3) + (lane & 7u) * 16) = r;

    // tries at this lane's four positions, then the map
    const float f0 = uniform_pm1(rand_float(r.x)), f1 = uniform_pm1(rand_float(r.y));
    const float f2 = uniform_pm1(rand_float(r.z)), f3 = uniform_pm1(rand_float(r.w));
    const float f4 = __shfl_down_sync(FULL_MASK, f0, 1);
    const uint32_t a0 = __ballot_sync(FULL_MASK, !(1.0f < M::norm2(f0, f1)));
    const uint32_t a1 = __ballot_sync(FULL_MASK, !(1.0f < M::norm2(f1, f2)));
    const uint32_t a2 = __ballot_sync(FULL_MASK, !(1.0f < M::norm2(f2, f3)));
    const uint32_t a3 = __ballot_sync(FULL_MASK, lane < 31u && !(1.0f < M::norm2(f3, f4)));
    const uint32_t b0 = a0 >> lane, b1 = a1 >> lane, b2 = a2 >> lane, b3 = a3 >> lane;
    const uint32_t at = 4 * lane;
    uint32_t map = after_try(b1, b3, at + 1, at + 3);                 // step at 4l: tries at 4l+1, 4l+3, ...
    map |= after_try(b2, b0 >> 1, at + 2, at + 4) << 8;
    map |= after_try(b3, b1 >> 1, at + 3, at + 5) << 16;
    map |= after_try(b0 >> 1, b2 >> 1, at + 4, at + 6) << 24;

    // step `lane` starts at the lane-fold image of the first step's start
    uint32_t start = p.rest, power = map;
#pragma unroll
    for (int b = 0; b < 5; ++b) {
        const uint32_t to = map_at(power, start);
        if ((lane >> b) & 1u)
            start = to;
        if (b < 4) {
            const uint32_t q0 = map_at(power, power & 255u), q1 = map_at(power, (power >> 8) & 255u);
            const uint32_t q2 = map_at(power, (power >> 16) & 255u), q3 = map_at(power, power >> 24);
            power = __byte_perm(__byte_perm(q0, q1, 0x0040u), __byte_perm(q2, q3, 0x0040u), 0x5410u);
        }
    }
    uint32_t next = map_at(map, start);
    const bool whole = next != NO_STEP;
    uint32_t n = __popc(__ballot_sync(FULL_MASK, whole));   // a prefix of the lanes
    __syncwarp();
    uint32_t w_step = sc.word(start), w_xi1 = sc.word(next - 2), w_xi2 = sc.word(next - 1);
    if (n == 0) {   // the first step alone needs more words than a round has
        next = p.rest;
        w_step = stream_word(p, next++, keys);
#pragma unroll 1
        for (bool second = false;; second = !second) {
            w_xi1 = w_xi2;
            w_xi2 = stream_word(p, next++, keys);
            if (second && !(1.0f < M::norm2(uniform_pm1(rand_float(w_xi1)), uniform_pm1(rand_float(w_xi2)))))
                break;
        }
        n = 1;
    }

    // step length, new direction
    const float t = M::step_length(uniform01(rand_float(w_step)));
    const float xi1 = uniform_pm1(rand_float(w_xi1)), xi2 = uniform_pm1(rand_float(w_xi2));
    float nu, nv, nw;
    M::direction(M::norm2(xi1, xi2), xi1, xi2, nu, nv, nw);
    float u = __shfl_up_sync(FULL_MASK, nu, 1), v = __shfl_up_sync(FULL_MASK, nv, 1);
    float w = __shfl_up_sync(FULL_MASK, nw, 1);
    if (lane == 0) {
        u = p.u;
        v = p.v;
        w = p.w;
    }
    __syncwarp();
    reinterpret_cast<float *>(sc.row(0))[lane] = t;
    reinterpret_cast<float *>(sc.row(1))[lane] = u;
    reinterpret_cast<float *>(sc.row(2))[lane] = v;
    reinterpret_cast<float *>(sc.row(3))[lane] = w;
    __syncwarp();

    // the moves in order: lanes 0..2 sum x, y and z, lane 3 decays the weight,
    // and leave what step j deposits with in word j of the rows (weight in 0)
    float sum = lane == 0 ? p.x : lane == 1 ? p.y : p.z, decay = p.weight;
    float *const along = reinterpret_cast<float *>(sc.row(min(lane + 1, 3u)));
    float *const out = lane == 3 ? reinterpret_cast<float *>(sc.row(0)) : along;
    const float *const lengths = reinterpret_cast<const float *>(sc.row(0));
#pragma unroll 2
    for (uint32_t j = 0; j < 32; j += 4) {
        const float4 t4 = *reinterpret_cast<const float4 *>(lengths + j);
        const float4 d4 = *reinterpret_cast<const float4 *>(along + j);
        float4 r4;
        r4.x = sum = M::move(sum, t4.x, d4.x);
        r4.y = sum = M::move(sum, t4.y, d4.y);
        r4.z = sum = M::move(sum, t4.z, d4.z);
        r4.w = sum = M::move(sum, t4.w, d4.w);
        const float w1 = M::mul(decay, c.albedo), w2 = M::mul(w1, c.albedo), w3 = M::mul(w2, c.albedo);
        if (lane == 3)
            r4 = make_float4(decay, w1, w2, w3);
        decay = M::mul(w3, c.albedo);
        __syncwarp();
        if (lane < 4)
            *reinterpret_cast<float4 *>(out + j) = r4;
    }
    __syncwarp();
    const float weight = reinterpret_cast<const float *>(sc.row(0))[lane];
    const float x = reinterpret_cast<const float *>(sc.row(1))[lane];
    const float y = reinterpret_cast<const float *>(sc.row(2))[lane];
    const float z = reinterpret_cast<const float *>(sc.row(3))[lane];
    const float decayed = M::mul(weight, c.albedo);
    const uint32_t low = __ballot_sync(FULL_MASK, lane < n && decayed < 0.001f * WEIGHT_ONE);
    if (low)
        n = __ffs((int)low);   // the steps up to the first roulette
    const float radius = M::radius_shells(x, y, z, c.spm);
    cell_out = (uint32_t)__float2int_rz(radius < c.last ? radius : beyond);
    weight_out = weight;

    const int l = (int)n - 1;
    p.x = __shfl_sync(FULL_MASK, x, l);
    p.y = __shfl_sync(FULL_MASK, y, l);
    p.z = __shfl_sync(FULL_MASK, z, l);
    p.u = __shfl_sync(FULL_MASK, nu, l);
    p.v = __shfl_sync(FULL_MASK, nv, l);
    p.w = __shfl_sync(FULL_MASK, nw, l);
    p.weight = __shfl_sync(FULL_MASK, decayed, l);
    uint32_t to = __shfl_sync(FULL_MASK, next, l);
    dead = false;
    if (low) {
        // roulette, photon.c:45-49; its word may lie behind the round's
        const float U = uniform01(rand_float(stream_word(p, to, keys)));
        ++to;
        dead = U > 0.1f;
        p.weight = __fdiv_rn(p.weight, 0.1f);
    }
    p.block += to >> 2;
    p.rest = to & 3u;
    return n;
}

// While the whole warp walks a photon, the lanes' photons are put away in the
// ring rows behind the scratch, a column per lane (what the rings hold is
// drawn again afterwards).  Kept in registers they and warp_steps' values
// exceed 64, and the compiler spills in the lane loop: 4.6 local-memory
// accesses per photon step.
enum SavedWord { S_KEY, S_BLOCK = 4, S_REST, S_X, S_Y, S_Z, S_U, S_V, S_W, S_WEIGHT, S_T, S_ROW, SAVED_WORDS };
constexpr int SAVED_ROW = 4;
static_assert(SAVED_ROW + SAVED_WORDS <= SLOTS, "saved photons fit in the ring");

template <int BLOCK>
struct SavedPhotons {
    char *rows;   // the warp's ring columns
    __device__ __forceinline__ uint32_t &word(int l, int k) const
    {
        return *reinterpret_cast<uint32_t *>(rows + (SAVED_ROW + k) * Ring<BLOCK>::W + 4 * l);
    }
    __device__ __forceinline__ float real(int l, int k) const { return __uint_as_float(word(l, k)); }
    __device__ __forceinline__ void put(int l, int k, float v) const { word(l, k) = __float_as_uint(v); }

    __device__ __forceinline__ void save(int l, const LanePhoton &p, float weight, uint32_t row) const
    {
        uint32_t block, rest;
        Ring<BLOCK>::position(p, block, rest);
        word(l, S_KEY) = p.key.a;
        word(l, S_KEY + 1) = p.key.b;
        word(l, S_KEY + 2) = p.key.c;
        word(l, S_KEY + 3) = p.key.d;
        put(l, S_T, p.t);
        put_walk(l, WarpPhoton{{}, block, rest, p.x, p.y, p.z, p.u, p.v, p.w, weight}, row);
    }
    __device__ __forceinline__ void put_walk(int l, const WarpPhoton &q, uint32_t row) const
    {
        word(l, S_BLOCK) = q.block;
        word(l, S_REST) = q.rest;
        put(l, S_X, q.x);
        put(l, S_Y, q.y);
        put(l, S_Z, q.z);
        put(l, S_U, q.u);
        put(l, S_V, q.v);
        put(l, S_W, q.w);
        put(l, S_WEIGHT, q.weight);
        word(l, S_ROW) = row;
    }
    __device__ __forceinline__ WarpPhoton get(int l) const
    {
        return WarpPhoton{{word(l, S_KEY), word(l, S_KEY + 1), word(l, S_KEY + 2), word(l, S_KEY + 3)},
                          word(l, S_BLOCK), word(l, S_REST),
                          real(l, S_X), real(l, S_Y), real(l, S_Z), real(l, S_U), real(l, S_V), real(l, S_W),
                          real(l, S_WEIGHT)};
    }
};

// Tally objects of step_photon: `whole` deposits a step of a photon that the
// whole warp walks.
struct Optics {
    WalkConsts c;
    float beyond;   // cell of a radius beyond the last shell, this lane's
};

template <class M, Hist H>
struct WeightTally {
    uint32_t hist;            // shared address of the histogram's shell 0
    uint32_t plane;           // bytes between a cell's words
    unsigned long long *g;    // global tally (H = Split, Far)
    float albedo;
    int near;                 // H = Split: shells nearest to the source in the histogram
    uint32_t steps = 0;

    __device__ __forceinline__ void deposit(int cell, float weight)
    {
        uint32_t lo, hi;
        if (H != Hist::Block && cell >= (H == Hist::Far ? 0 : near)) {
            deposit_global(g + 4 * (size_t)cell, weight);
        } else {
            const uint32_t at = hist + 4 * cell;
            units_split(weight_units(weight), lo, hi);
            tally_add_nowrap(at, at + plane, lo, hi);
            units_split(weight2_units(weight), lo, hi);
            tally_add_nowrap(at + 2 * plane, at + 3 * plane, lo, hi);
        }
        ++steps;
    }
    __device__ __forceinline__ void launched() {}
    __device__ __forceinline__ void step(LanePhoton &p, uint32_t cell)
    {
        deposit((int)cell, p.weight);
        p.weight = M::mul(p.weight, albedo);
    }
    __device__ __forceinline__ bool low(const LanePhoton &p) const { return p.weight < 0.001f * WEIGHT_ONE; }
    __device__ __forceinline__ void survived(LanePhoton &p) { p.weight = __fdiv_rn(p.weight, 0.1f); }
    __device__ __forceinline__ void died(LanePhoton &) {}
    // for the whole warp's walk: the weight, and the table's row (counts only)
    __device__ __forceinline__ float weight(const LanePhoton &p) const { return p.weight; }
    __device__ __forceinline__ uint32_t row_of(const LanePhoton &) const { return 0; }
    __device__ __forceinline__ uint32_t row_after(uint32_t, uint32_t) const { return 0; }
    __device__ __forceinline__ void resume(LanePhoton &, uint32_t) {}
    __device__ __forceinline__ void whole(uint32_t, uint32_t cell, float weight) { deposit((int)cell, weight); }
    __device__ __forceinline__ void walked(int, uint32_t) {}
};

template <class M, int BLOCK>
struct CountTally {
    CountTable table;
    uint32_t last;            // index of the last shell
    unsigned long long *g;
    uint32_t row;             // of the photon's next deposit, from table.base
    uint32_t roulette = 0;    // row behind its next roulette

    __device__ __forceinline__ void launched()
    {
        row = table.base;
        roulette = ld_shared(table.base + table.weight_at + 4);
    }
    __device__ __forceinline__ void step(LanePhoton &, uint32_t cell)
    {
        red_shared_add(row + 4 * cell, 1u);
        row += table.stride;
    }
    __device__ __forceinline__ bool low(const LanePhoton &) const { return row == roulette; }
    __device__ __forceinline__ void survived(LanePhoton &p)
    {
        if (row == table.end)
            Ring<BLOCK>::set_aside(p);
        else
            roulette = ld_shared(row + table.weight_at + 4);
    }
    __device__ __forceinline__ void died(LanePhoton &) {}
    __device__ __forceinline__ float weight(const LanePhoton &) const
    {
        return __uint_as_float(ld_shared(row + table.weight_at));
    }
    __device__ __forceinline__ void walked(int, uint32_t) {}
    __device__ __forceinline__ uint32_t row_of(const LanePhoton &) const { return row; }
    __device__ __forceinline__ uint32_t row_after(uint32_t at, uint32_t steps) const
    {
        return min(at + steps * table.stride, table.end);
    }
    __device__ __forceinline__ void resume(LanePhoton &p, uint32_t at)
    {
        row = at;
        if (p.t > 1.0f)   // the roulette behind its last deposit may be yet to come
            return;
        if (at == table.end)
            Ring<BLOCK>::set_aside(p);
        else
            roulette = ld_shared(at + table.weight_at + 4);
    }
    __device__ __forceinline__ void whole(uint32_t at, uint32_t cell, float weight)
    {
        if (at < table.end) {
            red_shared_add(at + 4 * cell, 1u);
            return;
        }
        deposit_global(g + 4 * (size_t)min(cell, last), weight);
        red_shared_add(table.end, 1u);   // counts such steps
    }
};

// The whole warp walks the photons of the lanes in `todo` one by one to their
// ends, or until `trips`, counted up once per round, reaches MAX_TRIPS (0: no
// bound).  Every lane's ring is used as scratch and filled again.  Returns the
// lanes whose photons ended.  optics(l) gives the constants of lane l's
// photon, tally.whole(..) deposits a step of it, tally.walked(l, n) counts n,
// tally.died is called on lane l at its end.
template <int BLOCK, class M, uint32_t MAX_TRIPS, class Tally, class Of>
__device__ __forceinline__ unsigned walk_whole(LanePhoton &p, unsigned todo, uint32_t &trips, char *ring,
                                               const PhiloxKeys &keys, Tally &tally, Of optics)
{
    using R = Ring<BLOCK>;
    const unsigned lane = threadIdx.x & 31u;
    const WarpScratch sc{ring - 4 * lane, R::W};
    unsigned left = __ballot_sync(FULL_MASK, R::walking(p));   // lanes with a photon
    const unsigned had = left;
    const SavedPhotons<BLOCK> saved{sc.rows};
    __syncwarp();
    saved.save((int)lane, p, tally.weight(p), tally.row_of(p));
    __syncwarp();
    while (todo && (MAX_TRIPS == 0 || trips < MAX_TRIPS)) {
        const int l = __ffs((int)todo) - 1;
        todo &= todo - 1;
        const Optics o = optics(l);
        WarpPhoton q = saved.get(l);
        uint32_t row = saved.word(l, S_ROW);
        bool over = false;
        do {
            uint32_t cell;
            float weight;
            const uint32_t n = warp_steps<M>(q, over, sc, o.c, keys, o.beyond, cell, weight);
            if (lane < n)
                tally.whole(tally.row_after(row, lane), cell, weight);
            row = tally.row_after(row, n);
            tally.walked(l, n);
            ++trips;
        } while (!over && (MAX_TRIPS == 0 || trips < MAX_TRIPS));
        if (over)
            left &= ~(1u << l);
        else if ((int)lane == l)   // a flush is due first: back to its lane
            saved.put_walk(l, q, row);
    }
    // back to the lanes, with fresh rings
    __syncwarp();
    const WarpPhoton q = saved.get((int)lane);
    const uint32_t row = saved.word((int)lane, S_ROW);
    p.t = saved.real((int)lane, S_T);
    __syncwarp();
    p.key = q.key;
    p.x = q.x; p.y = q.y; p.z = q.z;
    p.u = q.u; p.v = q.v; p.w = q.w;
    p.weight = q.weight;
    if ((left >> lane) & 1u) {
        R::restart(p, q.block, q.rest, ring, keys);
        tally.resume(p, row);
    } else {
        R::drop(p);
        if ((had >> lane) & 1u)
            tally.died(p);
    }
    return had & ~left;
}

// Walk photons from `src` until it is exhausted and every lane's photon has
// died.  Warp-collective: all 32 lanes of every warp call it.  flush() empties
// the shared tallies into the global one; it is called at the latest every
// FLUSH iterations.
template <int BLOCK, class M, bool COUNTS, uint32_t FLUSH, int TRIP, class Source, class Tally, class Flush>
__device__ __forceinline__ void walk_photons(const WalkConsts &c, float beyond, Source &src, const PhiloxKeys &keys,
                                             uint32_t *my, Tally &tally, Flush flush)
{
    using R = Ring<BLOCK>;
    constexpr uint32_t FLUSH_TRIPS = FLUSH / TRIP;
    const unsigned lane = threadIdx.x & 31u;
    const unsigned lt_mask = (1u << lane) - 1u;
    const int few = TRIP == SHORT_TRIP ? warp_walk_most(c.albedo) : WARP_WALK_MAX;
    char *ring = reinterpret_cast<char *>(my);

    LanePhoton p{};
    R::drop(p);
    uint32_t trips = 0;
    unsigned idle = 0;   // lanes that get no more photons

    for (;;) {
        // -------- hand new photon ids to lanes whose photon died
        const unsigned dead = __ballot_sync(FULL_MASK, !R::walking(p));
        unsigned todo = 0;   // photons for the whole warp
        if (dead != idle) {
            if constexpr (COUNTS)
                todo = __ballot_sync(FULL_MASK, R::aside(p));
            const unsigned need = dead & ~idle & ~todo;
            if (need) {
                unsigned long long pid = 0;
                const bool got = src.next(need, __popc(need & lt_mask), lane, pid) && ((need >> lane) & 1u);
                if (got) {
                    launch_photon<M>(p, pid, keys);
                    tally.launched();
                }
                idle = dead & ~todo & ~__ballot_sync(FULL_MASK, got);
                if (idle == FULL_MASK)
                    break;
            }
        }
        // -------- few photons left: the whole warp walks them one by one
        if (idle && 32 - __popc(idle) <= few) {
            // (a photon whose direction is still sought waits for the lane loop)
            todo |= __ballot_sync(FULL_MASK, R::walking(p) && !(p.t > 1.0f));
        }
        if (todo) {
            if (COUNTS && R::aside(p))
                p.cur -= R::ASIDE;
            if (walk_whole<BLOCK, M, FLUSH_TRIPS>(p, todo, trips, ring, keys, tally,
                                                  [&](int) { return Optics{c, beyond}; }))
                continue;
        }
        if (trips == FLUSH_TRIPS) {   // a trip stands for TRIP deposits of a lane at most
            trips = 0;
            flush();
        }
        ++trips;
#pragma unroll
        for (int k = 0; k < TRIP; ++k) {
            if (k % 2 == 0)
                R::refill(p, ring, keys);
            step_photon<BLOCK, M>(p, ring, c.spm, c.last, beyond, tally);
        }
    }
}

// walk_photons with a block's histogram of 64-bit sums, 4 * hist_cells words
// (low and high of sum w, then of sum w^2), flushed into g, the problem's global
// 128-bit tally [shells][4], every flush_steps iterations (the caller flushes
// what is left).  H = Split, Far: of 4 * hist_cells(near + 1) words, for the first
// `near` (Far: no) shells and the last.  probe_acc / probe_hi (Block only, may be
// null): receive the w sums those flushes take from shell probe_shell.  Returns
// this thread's photon steps.
template <int BLOCK, class M, class Source, Hist H, int BODY = TRIP>
__device__ __forceinline__ uint32_t walk_loop(const WalkConsts c, Source &src,
                                              const PhiloxKeys &keys, uint32_t *tally,
                                              unsigned long long *g, uint32_t *my, uint32_t near = 0,
                                              unsigned long long *probe_acc = nullptr,
                                              uint32_t *probe_hi = nullptr,
                                              uint32_t probe_shell = 0)
{
    constexpr uint32_t FLUSH = flush_steps((uint32_t)BLOCK);
    const float beyond = H != Hist::Block ? -1.0f : c.last + (float)(threadIdx.x & 31u);
    const uint32_t cells = hist_cells(H == Hist::Block ? c.shells : near + 1);
    WeightTally<M, H> t{(uint32_t)__cvta_generic_to_shared(tally + shell0_cell<H>()), 4 * cells, g, c.albedo,
                        (int)near};
    walk_photons<BLOCK, M, false, FLUSH, BODY>(c, beyond, src, keys, my, t, [&] {
        warp_flush_tally<H>(tally, near, c.shells, g, probe_acc, probe_hi, probe_shell);
    });
    return t.steps;
}

// Add what is left in a block's histogram (of the first `near` shells, H = Block:
// all, and the last of S) to a 128-bit global tally [shells][4], after a barrier.
// Block-collective.
template <int BLOCK, Hist H>
__device__ __forceinline__ void flush_tally(uint32_t *tally, uint32_t near, uint32_t S, unsigned long long *g)
{
    if constexpr (H == Hist::Block)
        near = S - 1;
    const uint32_t C = hist_cells(near + 1);
    const uint32_t *const first = tally + shell0_cell<H>();
    for (uint32_t s = threadIdx.x; s < near; s += BLOCK) {
        flush128(&g[4 * s + 0], &g[4 * s + 1], ((unsigned long long)first[C + s] << 32) | first[s]);
        flush128(&g[4 * s + 2], &g[4 * s + 3], ((unsigned long long)first[3 * C + s] << 32) | first[2 * C + s]);
    }
    if (threadIdx.x < 32) {
        const uint32_t s = last_cell<H>(near) + threadIdx.x;
        const unsigned long long v = warp_sum_u64(((unsigned long long)tally[C + s] << 32) | tally[s]);
        const unsigned long long v2 = warp_sum_u64(((unsigned long long)tally[3 * C + s] << 32) | tally[2 * C + s]);
        if (threadIdx.x == 0) {
            flush128(&g[4 * (size_t)(S - 1) + 0], &g[4 * (size_t)(S - 1) + 1], v);
            flush128(&g[4 * (size_t)(S - 1) + 2], &g[4 * (size_t)(S - 1) + 3], v2);
        }
    }
}

// The 64-bit sum of w that a block's histogram holds for shell s.  Called by
// the first warp.
__device__ __forceinline__ unsigned long long shell_sum(const uint32_t *tally, uint32_t S, uint32_t s)
{
    const uint32_t C = hist_cells(S);
    if (s + 1 < S)
        return ((unsigned long long)tally[C + s] << 32) | tally[s];
    const uint32_t at = s + (threadIdx.x & 31u);
    return warp_sum_u64(((unsigned long long)tally[C + at] << 32) | tally[at]);
}

}  // namespace tmc
