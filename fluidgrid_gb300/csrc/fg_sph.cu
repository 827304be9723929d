/* SPH density, forces and integration on GB300.
 *
 * Semantics follow GPU_Kernels/K_FluidSim.cu:
 *   density   CalculateMassDensityK + ProcessMassDensityGridD (:46-79, :210-254)
 *   forces    SPHCalculateForcesK / SPHCalculateForcesWithSRBK with
 *             CalculateFluidInternalForcesD, SPHCalculatePressureForceD,
 *             SPHCalculateViscosityForceD (:85-205, :260-413), walls from
 *             K_Boundaries_Walls.cu, rigid contact ProcessCollisionForcesD
 *             (K_DeviceFunctions.cu:32-159)
 *   integrate SPHIntegrateK (:418-438)
 * The 27 neighbour buckets are visited exactly as the reference visits them
 * (z-y-x order, same hashed buckets, a bucket reached twice is summed twice);
 * bucket indices are bit-exact.  Pair arithmetic is reorganised for the
 * GPU: squared-distance tests, rsqrt/rcp instead of divides, compensated
 * density sums (each term's rounding error added up beside); the results
 * agree with the reference arithmetic to the tolerances the parity tests
 * state.
 *
 * In the world pipeline the density pass is the only one that looks at the
 * ~216 candidates of the 27 buckets (~1,000 once the block compresses): it
 * records each particle's in-range visits (in visit order, duplicates and
 * the particle itself included) in the particle's own list, together with a
 * packed 32-byte record per particle.  The force pass then loops over the
 * ~30-110 listed neighbours per particle with all lanes busy, one 256-bit
 * record load each, instead of going over the candidates again. */
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>
#include "fg_device.cuh"
#include "fg_kernels.h"
#include "fg_sph_common.cuh"
#include "fg_stage.cuh"

namespace fg {

/* The density pass, by warp: fg_stage.cuh's staging, then a lane per target
 * over its staged candidates, two candidates an instruction where the sums'
 * order allows.  Bound by instruction issue (about 167 warp instructions a
 * target at 0.5 h spacing, of which 100 are staging, and 583 at 0.32 h; the
 * walk by thread took 237 and 700).  With lists, walk by thread -> staged, one
 * candidate at a time -> here: 1M particles at 0.5 h 351 -> 243 -> 229 us, 1M
 * compressed 922 -> 782 -> 725, 4M 1788 -> 1182 -> 1094, 262,144 at 0.45 h
 * (cells of 8 to 27 targets fill a warp badly) 138 -> 136 -> 126; 16,384, where
 * a thread's chain of 216 candidate loads was the pass, 37 -> 14.  64 worlds of
 * 1.23M particles that have splashed apart, whose warps lie in more and smaller
 * groups: 379 -> 378 after 20 steps, 504 -> 511 after 400 (a warp of more than
 * nine groups walking by thread instead: 415 and 547).
 *
 * Staged candidates of a warp: its targets lie in four or five groups of some
 * 90 (60-100 candidates kept of a cell's 216).  384 and ten CTAs an SM leave
 * the L1 60 KB: nine CTAs with 448, whose shared memory is no more, take 1395
 * us at 4M, ten with 320, more rounds, 1265, eleven 1480. */
#define FG_DENSITY_STAGE 384u
#define FG_DENSITY_CTAS 10
#define FG_STAGE_GROUPS 9u /* staged together; a warp of more takes them nine by nine */
#define FG_DENSITY_THREADS 64u

struct DensityShared {
    /* candidates, by component: four candidates a load, in pairs */
    float4 x[FG_DENSITY_STAGE / 4], y[FG_DENSITY_STAGE / 4], z[FG_DENSITY_STAGE / 4];
    uint4 j[FG_DENSITY_STAGE / 4]; /* sorted index */
    uint32_t idx[FG_STAGE_WINDOW];
};

/* One lane's list entries on their way to its list: collected in a ring of
 * sixteen in shared memory, stored a sector of eight at a time.  Lists are far
 * apart, so every store is a wavefront of its own a lane; and written in range
 * or not, kept by the count, an entry costs no divergent branch (0.32 h, 1M:
 * 855 us with two entries a store in a branch, 767 us so). */
struct ListRing {
    /* 16 entries of a word a thread; at = 256 times the count, plus the
     * thread's byte in an entry, so that one AND gives a push its address */
    uint32_t *ring;
    uint32_t at, done; /* done: entries stored, a multiple of 8 */

    __device__ __forceinline__ explicit ListRing(uint32_t *shared) : ring(shared), at(4u * threadIdx.x), done(0u) {}
    __device__ __forceinline__ uint32_t count() const { return at >> 8; }
    __device__ __forceinline__ uint32_t &slot(uint32_t a) const
    {
        return *(uint32_t *)((char *)ring + (a & (16u * 256u - 4u)));
    }
    /* j if it is in range */
    __device__ __forceinline__ void push(uint32_t j, bool in)
    {
        slot(at) = j;
        at += in ? 256u : 0u;
    }
    __device__ __forceinline__ uint4 four(uint32_t k) const
    {
        const uint32_t a = 256u * k + 4u * threadIdx.x; /* k: a multiple of 4 */
        return make_uint4(slot(a), slot(a + 256u), slot(a + 512u), slot(a + 768u));
    }
    /* after at most eight pushes since the last call */
    __device__ __forceinline__ void spill(uint32_t *lp, uint32_t cap)
    {
        if (count() - done >= 8u) {
            if (done + 8u <= cap)
                fg_st_list8(lp + done, four(done), four(done + 4u));
            else if (done + 4u <= cap)
                fg_st_list4(lp + done, four(done));
            done += 8u;
        }
    }
    /* the rest, padded to a whole group of four with the target itself, which
     * the force pass skips, so it reads only whole groups */
    __device__ __forceinline__ void finish(uint32_t *lp, uint32_t cap, uint32_t self)
    {
        const uint32_t cnt = count();
        if (cnt > cap) return;
        for (uint32_t a = at; a & 768u; a += 256u) slot(a) = self;
        for (; done < cnt; done += 4u) fg_st_list4(lp + done, four(done));
    }
};
static_assert(FG_DENSITY_THREADS == 64u, "a ring entry is a word of each of 64 threads");

/* Replacements for the scene's constants (the launchers'). */
struct DensityConst {
    float gas, rest, mass;
    int use;
};

/* A thread's counts over its targets. */
struct DensityTally {
    unsigned long long pairs = 0; /* in-range visits, the target itself included */
    uint32_t most = 0;            /* largest list count */
    uint32_t overflow = 0;        /* targets with more entries than slots */

    template <bool LIST>
    __device__ __forceinline__ void add(uint32_t cnt, uint32_t cap)
    {
        pairs += cnt;
        most = max(most, cnt);
        overflow += (LIST && cnt > cap) ? 1u : 0u;
    }
    /* once per warp: in-range pair visits for reporting, and the largest list
     * count for the capacity check */
    template <bool LIST, bool COUNT>
    __device__ __forceinline__ void flush(const NbrList &list, unsigned long long *out)
    {
        const uint32_t lane = threadIdx.x & 31u;
        if (COUNT && out) {
#pragma unroll
            for (int o = 16; o; o >>= 1) pairs += __shfl_xor_sync(FG_FULL, pairs, o);
            if (lane == 0 && pairs) atomicAdd(out, pairs);
        }
        if (LIST && list.max_count) {
            most = __reduce_max_sync(FG_FULL, most);
            if (lane == 0 && most) atomicMax(list.max_count, most);
        }
        if (LIST && list.overflow) {
            overflow = __reduce_add_sync(FG_FULL, overflow);
            if (lane == 0 && overflow) atomicAdd(list.overflow, (unsigned long long)overflow);
        }
    }
};

/* Density, pressure, record and list count of sorted target i at p. */
template <bool LIST>
__device__ __forceinline__ void density_store(const DensityAcc &acc, const FgScene *S, uint32_t i, float4 p,
                                              bool active, const float4 *__restrict__ svel, float2 *__restrict__ dp,
                                              const DensityConst &C, const NbrList &list)
{
    float2 d = make_float2(0.f, 0.f);
    if (active) {
        d = fg_density_out(C.use ? C.mass : S->mass, S->kpoly6, C.use ? C.gas : S->gas, C.use ? C.rest : S->rest,
                           acc.sum());
        dp[i] = d;
    } else if (LIST) {
        d = dp[i]; /* inactive particles stay neighbours with their stale density */
    }
    if (LIST) {
        const float4 v = __ldg(svel + i);
        list.rec[2 * i] = make_float4(p.x, p.y, p.z, d.x);
        list.rec[2 * i + 1] = make_float4(v.x, v.y, v.z, d.y);
        list.cnt[i] = acc.cnt;
    }
}

/* The density sum and list of sorted target i by a walk, and its visits. */
template <bool LIST, bool COUNT>
__device__ __forceinline__ void density_walk(DensityAcc &acc, const FgScene *S, uint32_t i, float4 p,
                                             const float4 *__restrict__ spos, const uint32_t *__restrict__ start,
                                             const uint32_t *__restrict__ end, uint32_t *lp, uint32_t cap)
{
    const float scale = S->scale, h2 = S->h2;
    const float px = p.x * scale, py = p.y * scale, pz = p.z * scale;
    fg_walk27_rows(p.x, p.y, p.z, S, start, end, [&](uint32_t j) {
        acc.visit<LIST, COUNT>(__ldg(spos + j), j, px, py, pz, scale, h2, lp, cap);
    });
    if (LIST) acc.flush(lp, cap, i);
}

/* The same out of line, for the staging kernel: inlined, it cost the staging 4%. */
template <bool LIST, bool COUNT>
__device__ __noinline__ uint2 density_walk_aside(const FgScene *S, uint32_t i, const float4 *spos,
                                                 const uint32_t *start, const uint32_t *end, uint32_t *lp,
                                                 uint32_t cap)
{
    DensityAcc acc;
    acc.init();
    density_walk<LIST, COUNT>(acc, S, i, __ldg(spos + i), spos, start, end, lp, cap);
    return make_uint2(__float_as_uint(acc.sum()), acc.cnt);
}

/* What a pass does with its dispersed ranges: those of more than `most`
 * buckets, whose targets share too little for a lookup and a cull a cell. */
enum { DISPERSED_STAGED, DISPERSED_WALKED, DISPERSED_ASIDE /* another kernel has them */ };

template <bool LIST, bool COUNT>
__global__ void __launch_bounds__(FG_DENSITY_THREADS, FG_DENSITY_CTAS) k_density(
    const FgWork *__restrict__ work, uint32_t nwork, uint32_t n_single, const FgScene *__restrict__ table,
    const __grid_constant__ FgScene single, uint32_t range, uint32_t most, int dispersed,
    const float4 *__restrict__ spos, const float4 *__restrict__ svel, const uint32_t *__restrict__ start,
    const uint32_t *__restrict__ end, float2 *__restrict__ dp, const __grid_constant__ DensityConst C,
    const __grid_constant__ NbrList list, unsigned long long *__restrict__ pairs)
{
    __shared__ DensityShared shared[FG_DENSITY_THREADS / 32];
    __shared__ uint32_t s_ring[LIST ? 16 * FG_DENSITY_THREADS : 1];
    DensityShared &sm = shared[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t cap = LIST ? __ldg(list.cap) : 0u;
    DensityTally tally;
    const uint32_t per = FG_CHUNK / range; /* warps per work item */
    for (uint32_t warp = blockIdx.x * (FG_DENSITY_THREADS / 32u) + (threadIdx.x >> 5); warp < nwork * per;
         warp += gridDim.x * (FG_DENSITY_THREADS / 32u)) {
        const FgWork it = fg_work(work, warp / per, n_single);
        const uint32_t q0 = (warp % per) * range;
        if (q0 >= it.count) continue; /* uniform over the warp */
        const FgScene *S = fg_scene(table, &single, it.scene);
        const uint32_t lo = table ? S->pbase : 0u, hi = table ? S->pbase + S->n : n_single;
        const float scale = S->scale, h2 = S->h2;
        const StageGrid G(S);
        uint32_t next, stop;
        const bool walk = fg_stage_range(it.first + q0, range, lo, hi, most, dispersed == DISPERSED_ASIDE, G, spos,
                                         next, stop);
        if (walk && dispersed == DISPERSED_ASIDE) continue;
        while (next < stop) {
            const uint32_t i = next + lane; /* sorted index */
            uint32_t n = min(32u, stop - next);
            float4 p = lane < n ? spos[i] : make_float4(0.f, 0.f, 0.f, 0.f);
            const StageSig sig = fg_stage_sig(p, G);
            if (stop - next > 32u) n = fg_stage_trim(sig, __ldg(spos + next + 32u), G);
            next += n;
            const bool valid = lane < n;
            const bool active = valid && p.w > 0.0f; /* inactive: density not written */
            const float px = p.x * scale, py = p.y * scale, pz = p.z * scale;
            DensityAcc acc;
            acc.init();
            ListRing ring(s_ring);
            uint32_t count = 0u; /* without a list */
            /* lists by sorted index: the force pass may visit the targets in another order */
            uint32_t *lp = LIST ? list.idx + (size_t)i * list.stride : nullptr;
            uint32_t lead, leads;
            if (!walk && !__any_sync(FG_FULL, active && sig.odd)) {
                fg_stage_groups(sig, __ballot_sync(FG_FULL, active), lead, leads);
                while (leads) {
                    /* the first FG_STAGE_GROUPS of the groups left */
                    uint32_t later = leads;
                    for (uint32_t k = 0u; k < FG_STAGE_GROUPS; k++) later &= later - 1u;
                    const uint32_t batch = leads ^ later;
                    leads = later;
                    fg_stage_rounds<FG_DENSITY_STAGE, FG_STAGE_GROUPS>(
                        sig, lead, batch, px, py, pz, G, spos, start, end, sm.idx,
                        [&](uint32_t slot, uint32_t j, float4 c) {
                            ((float *)sm.x)[slot] = c.x;
                            ((float *)sm.y)[slot] = c.y;
                            ((float *)sm.z)[slot] = c.z;
                            ((uint32_t *)sm.j)[slot] = j;
                        },
                        [&](uint32_t first, uint32_t stop, uint32_t) {
                            const F2 px2 = fg_pack(px, px), py2 = fg_pack(py, py), pz2 = fg_pack(pz, pz);
                            const F2 ns2 = fg_pack(-scale, -scale), hh2 = fg_pack(h2, h2);
                            for (uint32_t k = first >> 2; k < stop >> 2; k += 2u) {
#pragma unroll
                                for (uint32_t e = 0; e < 2u; e++) {
                                    const float4 x = sm.x[k + e], y = sm.y[k + e], z = sm.z[k + e];
                                    const uint4 j = LIST ? sm.j[k + e] : make_uint4(0u, 0u, 0u, 0u);
                                    bool in[4];
                                    acc.term2(fg_pack(x.x, x.y), fg_pack(y.x, y.y), fg_pack(z.x, z.y), px2, py2, pz2,
                                              ns2, hh2, h2, in[0], in[1]);
                                    acc.term2(fg_pack(x.z, x.w), fg_pack(y.z, y.w), fg_pack(z.z, z.w), px2, py2, pz2,
                                              ns2, hh2, h2, in[2], in[3]);
                                    if (LIST) {
                                        ring.push(j.x, in[0]);
                                        ring.push(j.y, in[1]);
                                        ring.push(j.z, in[2]);
                                        ring.push(j.w, in[3]);
                                    } else if (COUNT) {
#pragma unroll
                                        for (int u = 0; u < 4; u++) count += in[u] ? 1u : 0u;
                                    }
                                }
                                if (LIST) ring.spill(lp, cap);
                            }
                        });
                }
                if (LIST && active) ring.finish(lp, cap, i);
                acc.cnt = LIST ? ring.count() : count;
            } else if (active) {
                const uint2 r = density_walk_aside<LIST, COUNT>(S, i, spos, start, end, lp, cap);
                acc.s = __uint_as_float(r.x);
                acc.cnt = r.y;
            }
            if (valid) density_store<LIST>(acc, S, i, p, active, svel, dp, C, list);
            tally.add<LIST>(acc.cnt, cap);
        }
    }
    tally.flush<LIST, COUNT>(list, pairs);
}

/* The dispersed ranges (most = 0: every range), a thread a target.  Bound by
 * the L1's and L2's sectors (54 bucket words a target) and their latency, for
 * which it wants the L1 and the warps that the staging kernel's shared memory
 * takes: the same walk there takes 270 us where this takes 226, at 1,048,576
 * targets 1.2 h apart (staged: 477).  Eight CTAs an SM, 62 registers, without
 * lists (sixteen of 32, which spill: 262 us), ten with them.  A wave of CTAs;
 * the next range's positions are on their way while one walks or is passed
 * over. */
#define FG_WALK_CTAS(LIST) ((LIST) ? 10 : 8)
template <bool LIST, bool COUNT>
__global__ void __launch_bounds__(FG_CHUNK, FG_WALK_CTAS(LIST)) k_density_dispersed(
    const FgWork *__restrict__ work, uint32_t nwork, uint32_t n_single, const FgScene *__restrict__ table,
    const __grid_constant__ FgScene single, uint32_t most, const float4 *__restrict__ spos,
    const float4 *__restrict__ svel, const uint32_t *__restrict__ start, const uint32_t *__restrict__ end,
    float2 *__restrict__ dp, const __grid_constant__ DensityConst C, const __grid_constant__ NbrList list,
    unsigned long long *__restrict__ pairs)
{
    const uint32_t cap = LIST ? __ldg(list.cap) : 0u;
    DensityTally tally;
    auto load = [&](uint32_t w) {
        const FgWork it = fg_work(work, w, n_single);
        const FgScene *S = fg_scene(table, &single, it.scene);
        return __ldg(spos + min(it.first + threadIdx.x, (table ? S->pbase + S->n : n_single) - 1u));
    };
    uint32_t w = blockIdx.x;
    float4 ahead = w < nwork ? load(w) : make_float4(0.f, 0.f, 0.f, 0.f);
    for (; w < nwork; w += gridDim.x) {
        const FgWork it = fg_work(work, w, n_single);
        const FgScene *S = fg_scene(table, &single, it.scene);
        const float4 p = ahead;
        if (w + gridDim.x < nwork) ahead = load(w + gridDim.x);
        if ((threadIdx.x & ~31u) >= it.count) continue; /* uniform over the warp */
        if (most) {
            const StageGrid G(S);
            if (!fg_stage_dispersed(fg_stage_cell(p, G), G, 32u, most)) continue;
        }
        if (threadIdx.x < it.count) {
            const uint32_t i = it.first + threadIdx.x;
            const bool active = p.w > 0.0f;
            DensityAcc acc;
            acc.init();
            if (active)
                density_walk<LIST, COUNT>(acc, S, i, p, spos, start, end,
                                          LIST ? list.idx + (size_t)i * list.stride : nullptr, cap);
            density_store<LIST>(acc, S, i, LIST ? __ldg(spos + i) : p, active, svel, dp, C, list);
            tally.add<LIST>(acc.cnt, cap);
        }
        __syncwarp();
    }
    tally.flush<LIST, COUNT>(list, pairs);
}

/* out[0] += the buckets of every sixteenth range of 32, out[1] += 1 for each. */
__global__ void __launch_bounds__(FG_CHUNK) k_spread(const FgWork *__restrict__ work, uint32_t nwork, uint32_t n_single,
                                                     const FgScene *__restrict__ table,
                                                     const __grid_constant__ FgScene single,
                                                     const float4 *__restrict__ spos, uint32_t *out)
{
    for (uint32_t w = 4u * (blockIdx.x * (FG_CHUNK / 32u) + (threadIdx.x >> 5)); w < nwork;
         w += 4u * gridDim.x * (FG_CHUNK / 32u)) {
        const FgWork it = fg_work(work, w, n_single);
        const FgScene *S = fg_scene(table, &single, it.scene);
        const uint32_t hi = table ? S->pbase + S->n : n_single, lane = threadIdx.x & 31u;
        const StageGrid G(S);
        const uint32_t b = fg_stage_buckets(fg_stage_cell(__ldg(spos + min(it.first + lane, hi - 1u)), G), G, 32u);
        if (lane == 0u) {
            atomicAdd(out, b);
            atomicAdd(out + 1, 1u);
        }
    }
}

void launch_spread(const Launch &L, const float4 *spos, uint32_t *out)
{
    if (!L.nwork) return;
    k_spread<<<grid_for((L.nwork + 15u) / 16u, 16), FG_CHUNK, 0, L.stream>>>(L.work, L.nwork, L.n, L.table, *L.single,
                                                                             spos, out);
}

/* Targets of a warp: 32, or fewer where that leaves the SMs short of warps
 * (16 each): a group's lookups and staging are a chain of some ten memory
 * latencies, and a warp goes through its groups one after another. */
static uint32_t stage_range(uint32_t nwork)
{
    const uint64_t want = 16ull * (uint64_t)sm_count();
    uint32_t range = 32u;
    while (range > 8u && (uint64_t)nwork * (FG_CHUNK / range) < want) range >>= 1;
    return range;
}

/* What becomes of a pass's dispersed ranges, and beyond how many buckets a
 * range is one (32: none is).  Density without lists, 1,048,576 random targets,
 * staged -> walked: 0.5 h apart (four or five cells a range) 312 -> 315 us, 0.8
 * h (14) 362 -> 235, 1.2 h 477 -> 226, 3 h 543 -> 241; 262,144, 1.7 h: 147 ->
 * 67.  Nine parts the first two: with eight, the few ranges of the first that
 * walk take it to 326; with twelve, the second stays at 326.  With L.side the
 * walk is a kernel beside the staging one (3 us where no range walks); warps
 * of fewer targets, of which the GPU is not full, walk themselves.  A world with
 * lists chooses for all its ranges at once (World::check_list_cap): there the
 * walk of a few ranges, 27 rows and a list one after another, lasts as long as
 * the whole pass (32 uneven splashed scenes, an eighth of the ranges dispersed:
 * 298 us a step staged, 354 with those walked). */
static int dispersed_ranges(const Launch &L, uint32_t range, uint32_t &most)
{
    most = 32u;
    if (!L.side.stream) return DISPERSED_STAGED;
    most = range == 32u ? 9u : range - range / 4u;
    return range == 32u ? DISPERSED_ASIDE : DISPERSED_WALKED;
}

bool density_ranges_wide(uint32_t nwork) { return stage_range(nwork) == 32u; }

uint32_t density_launches(const Launch &L)
{
    uint32_t most;
    return dispersed_ranges(L, stage_range(L.nwork), most) == DISPERSED_ASIDE ? 2u : 1u;
}

/* L.side's stream, if it is used: forked from L's until the end of the scope.
 * Where that fails (a context made anew under the process) one kernel takes
 * every range. */
struct SideLaunch {
    const Launch &L;
    bool use;
    SideLaunch(const Launch &launch, int &dispersed) : L(launch), use(dispersed == DISPERSED_ASIDE)
    {
        if (!use || (cudaEventRecord(L.side.fork, L.stream) == cudaSuccess &&
                     cudaStreamWaitEvent(L.side.stream, L.side.fork, 0) == cudaSuccess))
            return;
        cudaGetLastError();
        use = false;
        dispersed = DISPERSED_WALKED;
    }
    ~SideLaunch()
    {
        if (!use) return;
        cudaEventRecord(L.side.join, L.side.stream);
        cudaStreamWaitEvent(L.stream, L.side.join, 0);
    }
};

void launch_density(const Launch &L, const float4 *spos, const uint32_t *start, const uint32_t *end, float2 *dp,
                    float gas_o, float rest_o, float mass_o, int use_o, const float4 *svel, const NbrList *list,
                    unsigned long long *pairs)
{
    if (!L.nwork) return;
    NbrList none;
    memset(&none, 0, sizeof(none));
    const NbrList &nl = list ? *list : none;
    const DensityConst C = {gas_o, rest_o, mass_o, use_o};
    if (list && L.walk) {
        k_density_dispersed<true, true><<<grid_for(L.nwork, FG_WALK_CTAS(true)), FG_CHUNK, 0, L.stream>>>(
            L.work, L.nwork, L.n, L.table, *L.single, 0u, spos, svel, start, end, dp, C, nl, pairs);
        return;
    }
    const uint32_t range = stage_range(L.nwork);
    uint32_t most;
    int dispersed = dispersed_ranges(L, range, most);
    /* ctas_per_sm counts CTAs of FG_CHUNK threads for 32 targets a warp */
    const uint32_t per = FG_CHUNK / range * 32u / FG_DENSITY_THREADS;
    const uint32_t g = grid_for(L.nwork * per, (int)((L.ctas_per_sm ? L.ctas_per_sm : 64u) * per));
#define FG_DENSITY(LI, CO)                                                                                          \
    k_density<LI, CO><<<g, FG_DENSITY_THREADS, 0, L.stream>>>(L.work, L.nwork, L.n, L.table, *L.single, range, most, \
                                                              dispersed, spos, svel, start, end, dp, C, nl, pairs)
    if (list) {
        FG_DENSITY(true, true);
        return;
    }
    const SideLaunch side(L, dispersed);
#define FG_DISPERSED(CO)                                                                                            \
    k_density_dispersed<false, CO><<<grid_for(L.nwork, FG_WALK_CTAS(false)), FG_CHUNK, 0, L.side.stream>>>(         \
        L.work, L.nwork, L.n, L.table, *L.single, most, spos, svel, start, end, dp, C, nl, pairs)
    if (pairs) {
        if (side.use) FG_DISPERSED(true);
        FG_DENSITY(false, true);
    } else {
        if (side.use) FG_DISPERSED(false);
        FG_DENSITY(false, false);
    }
#undef FG_DISPERSED
#undef FG_DENSITY
}

/* Work items are FG_CHUNK particles whatever the block size: a CTA of
 * BLOCK < FG_CHUNK threads takes an item in FG_CHUNK / BLOCK passes, one of
 * BLOCK > FG_CHUNK threads takes BLOCK / FG_CHUNK items at once.  Every
 * particle's arithmetic is the same for every block size. */
#define FG_ITEMS_PER_CTA(B) ((B) >= FG_CHUNK ? (B) / FG_CHUNK : 1u)
#define FG_PASSES(B) ((B) >= FG_CHUNK ? 1u : FG_CHUNK / (B))

struct RigidArgs {
    RigidGrid dyn;
    RigidGrid sta;
    int use_dyn, use_sta;
};

/* A world particle's contact with the bodies: stored by the contact pass, or
 * walked here. */
__device__ __forceinline__ float3 force_contact(const FgScene *S, uint32_t scene, float4 p, float4 v, uint32_t oi,
                                                const RigidArgs &R)
{
    if (!R.use_dyn || !(S->flags & FG_SCENE_HAS_RB)) return make_float3(0.f, 0.f, 0.f);
    if (!R.dyn.pre) return fg_fluid_rigid_contact(S, scene, p, v, R.dyn, true);
    if (fg_contact_outside(S, scene, p, R.dyn) || !fg_contact_marked(S, scene, p, R.dyn))
        return make_float3(0.f, 0.f, 0.f);
    const float4 q = R.dyn.pre[oi];
    return make_float3(q.x, q.y, q.z);
}

/* The contact that the contact pass stored for particle oi, if it is marked. */
__device__ __forceinline__ float3 force_contact_stored(const FgScene *S, bool active, float4 p, const RigidGrid &G,
                                                       uint32_t oi)
{
    if (!active || !fg_contact_marked(S, 0u, p, G)) return make_float3(0.f, 0.f, 0.f);
    const float4 q = __ldcg(G.pre + oi); /* the output's memory */
    return make_float3(q.x, q.y, q.z);
}

/* The contact of a warp's particles (whole warp, converged) with a grid whose
 * near cells are marked, one particle after another by the whole warp. */
__device__ __forceinline__ float3 force_contact_warp(const FgScene *S, bool active, float4 p, float4 v,
                                                     const RigidGrid &G, bool dynamic)
{
    float3 c = make_float3(0.f, 0.f, 0.f);
    const ContactShape C(S);
    for (uint32_t m = __ballot_sync(FG_FULL, active && fg_contact_marked(S, 0u, p, G)); m; m &= m - 1u) {
        const int b = __ffs((int)m) - 1;
        const float4 pb = make_float4(__shfl_sync(FG_FULL, p.x, b), __shfl_sync(FG_FULL, p.y, b),
                                      __shfl_sync(FG_FULL, p.z, b), 1.f);
        const float4 vb = make_float4(__shfl_sync(FG_FULL, v.x, b), __shfl_sync(FG_FULL, v.y, b),
                                      __shfl_sync(FG_FULL, v.z, b), 0.f);
        const float3 r = fg_contact_warp(S, C, pb, vb, G, dynamic);
        if ((int)(threadIdx.x & 31u) == b) c = r;
    }
    return c;
}

/* The launchers' contact: one grid's from the contact pass, and the static
 * one's searched here where that was the dynamic's. */
__device__ __forceinline__ void force_contacts(const FgScene *S, bool active, float4 p, float4 v, uint32_t oi,
                                               const RigidArgs &R, float3 &sta, float3 &dyn)
{
    sta = dyn = make_float3(0.f, 0.f, 0.f);
    if (R.use_dyn) dyn = force_contact_stored(S, active, p, R.dyn, oi);
    if (R.use_sta)
        sta = R.use_dyn ? force_contact_warp(S, active, p, v, R.sta, false)
                        : force_contact_stored(S, active, p, R.sta, oi);
}

/* Pair terms of one target by a walk over its 27 buckets. */
__device__ __forceinline__ void walk_terms(const FgScene *S, uint32_t i, float4 p, float4 v, float kv,
                                           const float4 *__restrict__ spos, const float4 *__restrict__ svel,
                                           const float2 *__restrict__ dp, const uint32_t *__restrict__ start,
                                           const uint32_t *__restrict__ end, float &fx, float &fy, float &fz)
{
    const float scale = S->scale, h = S->h, h2 = S->h2, kspiky = S->kspiky;
    const float px = p.x * scale, py = p.y * scale, pz = p.z * scale;
    const float2 di = dp[i];
    fg_walk27_rows(p.x, p.y, p.z, S, start, end, [&](uint32_t j) {
        if (j == i) return;
        const float4 q = __ldg(spos + j);
        const float dx = fmaf(-q.x, scale, px), dy = fmaf(-q.y, scale, py), dz = fmaf(-q.z, scale, pz);
        const float r2 = fmaf(dx, dx, fmaf(dy, dy, __fmul_rn(dz, dz)));
        if (r2 <= h2) {
            const float4 vj = __ldg(svel + j);
            const float2 dj = __ldg(dp + j);
            fg_pair(fx, fy, fz, dx, dy, dz, r2, h, kspiky, kv, di.x, di.y, v, dj.x, dj.y, vj);
        }
    });
}

/* The same out of line, for the search kernel's few. */
__device__ __noinline__ float3 walk_terms_aside(const FgScene *S, uint32_t i, float kv, const float4 *spos,
                                                const float4 *svel, const float2 *dp, const uint32_t *start,
                                                const uint32_t *end)
{
    float3 f = make_float3(0.f, 0.f, 0.f);
    walk_terms(S, i, __ldg(spos + i), __ldg(svel + i), kv, spos, svel, dp, start, end, f.x, f.y, f.z);
    return f;
}

/* From the summed pair terms to the particle's new velocity (and, fused, its
 * position): F = internal * mass + gravity + rigid contact, walls, force clamp
 * (K_FluidSim.cu:287-307, 389-411), newVel[id] = vel + F dt. */
__device__ __forceinline__ void force_finish(const FgScene *S, float4 p, float4 v, float fx, float fy, float fz,
                                             float mass, float3 sta, float3 dyn, uint32_t oi,
                                             float4 *__restrict__ vel_out, float4 *__restrict__ pos_out)
{
    float3 F = make_float3(0.f, 0.f, 0.f);
    if (p.w > 0.0f) {
        F = make_float3(fx * mass + S->gravity[0], fy * mass + S->gravity[1], fz * mass + S->gravity[2]);
        F.x += sta.x; F.y += sta.y; F.z += sta.z;
        F.x += dyn.x; F.y += dyn.y; F.z += dyn.z;
        const float3 wl = fg_walls(*S, make_float3(p.x, p.y, p.z), make_float3(v.x, v.y, v.z));
        F.x += wl.x; F.y += wl.y; F.z += wl.z;
        const float sp2 = F.x * F.x + F.y * F.y + F.z * F.z;
        const float speed = sqrtf(sp2);
        if (speed > S->vlimit) {
            const float t = S->vlimit / speed;
            F.x *= t; F.y *= t; F.z *= t;
        }
    }
    const float dt = S->dt;
    float4 nv;
    nv.x = v.x + F.x * dt;
    nv.y = v.y + F.y * dt;
    nv.z = v.z + F.z * dt;
    nv.w = v.w + 0.0f;
    vel_out[oi] = nv;
    if (pos_out && p.w > 0.0f) {
        /* SPHIntegrateK fused: pos += vel * (dt / scale), unfused rounding */
        const float c = S->dt_over_scale;
        float4 np;
        np.x = __fadd_rn(p.x, __fmul_rn(nv.x, c));
        np.y = __fadd_rn(p.y, __fmul_rn(nv.y, c));
        np.z = __fadd_rn(p.z, __fmul_rn(nv.z, c));
        np.w = __fadd_rn(p.w, __fmul_rn(nv.w, c));
        pos_out[oi] = np;
    }
}

/* The list form of the force pass (kernel 1). */
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK, 768 / BLOCK) k_forces(const FgWork *__restrict__ work, uint32_t nwork,
                                                    uint32_t n_single, const FgScene *__restrict__ table,
                                                    const __grid_constant__ FgScene single,
                                                    const float4 *__restrict__ spos, const float4 *__restrict__ svel,
                                                    const uint32_t *__restrict__ start,
                                                    const uint32_t *__restrict__ end,
                                                    const uint32_t *__restrict__ ids, float4 *__restrict__ vel_out,
                                                    float4 *__restrict__ pos_out,
                                                    const __grid_constant__ RigidArgs R,
                                                    const __grid_constant__ NbrList list, TargetOrder ord)
{
    constexpr uint32_t IPC = FG_ITEMS_PER_CTA(BLOCK), PASSES = FG_PASSES(BLOCK);
    const uint32_t sub = IPC > 1u ? threadIdx.x / FG_CHUNK : 0u;
    const uint32_t lt = IPC > 1u ? threadIdx.x % FG_CHUNK : threadIdx.x;
    for (uint32_t w = blockIdx.x * IPC + sub; w < nwork; w += gridDim.x * IPC)
#pragma unroll 1
    for (uint32_t ps = 0; ps < PASSES; ps++) {
        const uint32_t tid = lt + ps * BLOCK;
        FgWork it = fg_work(work, w, n_single);
        if (tid >= it.count) continue;
        const FgScene *S = fg_scene(table, &single, it.scene);
        const uint32_t tpos = it.first + tid; /* target slot */
        const uint32_t pid = ord.tord ? __ldg(ord.tord + tpos) : 0u;
        const uint32_t i = ord.tord ? __ldg(ord.inv + pid) : tpos;
        const float4 p = spos[i];
        const float4 v = svel[i];
        float fx = 0.f, fy = 0.f, fz = 0.f;
        float3 dyn = make_float3(0.f, 0.f, 0.f);
        const uint32_t oi = ord.tord ? pid : __ldg(ids + i);
        if (p.w > 0.0f) {
            const float scale = S->scale, h = S->h, h2 = S->h2;
            const float kspiky = S->kspiky, kv = S->kvisc * S->visc;
            const float px = p.x * scale, py = p.y * scale, pz = p.z * scale;
            const float4 r0 = list.rec[2 * i], r1 = list.rec[2 * i + 1];
            const float rho_i = r0.w, P_i = r1.w;
            const uint32_t c = list.cnt[i];
            if (c <= __ldg(list.cap)) {
                /* in-range visits in walk order (the target's own
                 * entries skipped) */
                const uint32_t *nl = list.idx + (size_t)i * list.stride;
                /* the list is padded with i to whole groups of four */
                const uint32_t c4 = (c + 3u) & ~3u;
                /* four 32-byte records in flight, one 256-bit load each,
                 * their target's own entries skipped */
                auto group = [&](const uint4 q) {
                    const uint32_t jj[4] = {q.x, q.y, q.z, q.w};
                    float4 a[4], b[4];
#pragma unroll
                    for (int e = 0; e < 4; e++) fg_ld_rec(list.rec + 2 * jj[e], a[e], b[e]);
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        if (jj[e] != i) {
                            const float dx = fmaf(-a[e].x, scale, px), dy = fmaf(-a[e].y, scale, py),
                                        dz = fmaf(-a[e].z, scale, pz);
                            const float r2 = fmaf(dx, dx, fmaf(dy, dy, __fmul_rn(dz, dz)));
                            fg_pair(fx, fy, fz, dx, dy, dz, r2, h, kspiky, kv, rho_i, P_i, v, a[e].w, b[e].w,
                                    b[e]);
                        }
                    }
                };
                /* eight indices (one sector, 32-byte aligned: the stride
                 * is a multiple of 8) per load, the next eight loading
                 * while these records do */
                uint4 qa = make_uint4(0u, 0u, 0u, 0u), qb = qa;
                if (c4) fg_ld_idx8(nl, qa, qb);
                for (uint32_t k = 0; k < c4; k += 8) {
                    const uint4 ca = qa, cb = qb;
                    if (k + 8u < c4) fg_ld_idx8(nl + k + 8u, qa, qb);
                    group(ca);
                    if (k + 4u < c4) group(cb);
                }
            } else {
                /* more in-range visits than list slots: walk the buckets */
                fg_walk27(p.x, p.y, p.z, S, start, end, [&](uint32_t j) {
                    if (j == i) return;
                    const float4 q0 = __ldg(list.rec + 2 * j);
                    const float dx = fmaf(-q0.x, scale, px), dy = fmaf(-q0.y, scale, py),
                                dz = fmaf(-q0.z, scale, pz);
                    const float r2 = fmaf(dx, dx, fmaf(dy, dy, __fmul_rn(dz, dz)));
                    if (r2 <= h2) {
                        const float4 q1 = __ldg(list.rec + 2 * j + 1);
                        fg_pair(fx, fy, fz, dx, dy, dz, r2, h, kspiky, kv, rho_i, P_i, v, q0.w, q1.w, q1);
                    }
                });
            }
            dyn = force_contact(S, it.scene, p, v, oi, R);
        }
        force_finish(S, p, v, fx, fy, fz, S->mass, make_float3(0.f, 0.f, 0.f), dyn, oi, vel_out, pos_out);
    }
}

/* The walking form (kernel 0), each thread over its target's 27 buckets: the
 * same terms in the same order as the list form. */
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK, 768 / BLOCK) k_forces_walk(
    const FgWork *__restrict__ work, uint32_t nwork, uint32_t n_single, const FgScene *__restrict__ table,
    const __grid_constant__ FgScene single, const float4 *__restrict__ spos, const float4 *__restrict__ svel,
    const float2 *__restrict__ dp, const uint32_t *__restrict__ start, const uint32_t *__restrict__ end,
    const uint32_t *__restrict__ ids, float4 *__restrict__ vel_out, float4 *__restrict__ pos_out,
    const __grid_constant__ RigidArgs R, TargetOrder ord)
{
    constexpr uint32_t IPC = FG_ITEMS_PER_CTA(BLOCK), PASSES = FG_PASSES(BLOCK);
    const uint32_t sub = IPC > 1u ? threadIdx.x / FG_CHUNK : 0u;
    const uint32_t lt = IPC > 1u ? threadIdx.x % FG_CHUNK : threadIdx.x;
    for (uint32_t w = blockIdx.x * IPC + sub; w < nwork; w += gridDim.x * IPC)
#pragma unroll 1
    for (uint32_t ps = 0; ps < PASSES; ps++) {
        const uint32_t tid = lt + ps * BLOCK;
        const FgWork it = fg_work(work, w, n_single);
        if (tid >= it.count) continue;
        const FgScene *S = fg_scene(table, &single, it.scene);
        const uint32_t tpos = it.first + tid; /* target slot */
        const uint32_t pid = ord.tord ? __ldg(ord.tord + tpos) : 0u;
        const uint32_t i = ord.tord ? __ldg(ord.inv + pid) : tpos;
        const uint32_t oi = ord.tord ? pid : __ldg(ids + i);
        const float4 p = spos[i];
        const float4 v = svel[i];
        float fx = 0.f, fy = 0.f, fz = 0.f;
        float3 dyn = make_float3(0.f, 0.f, 0.f);
        if (p.w > 0.0f) {
            walk_terms(S, i, p, v, S->kvisc * S->visc, spos, svel, dp, start, end, fx, fy, fz);
            dyn = force_contact(S, it.scene, p, v, oi, R);
        }
        force_finish(S, p, v, fx, fy, fz, S->mass, make_float3(0.f, 0.f, 0.f), dyn, oi, vel_out, pos_out);
    }
}

/* The form without lists (the reference-named launchers).  A warp takes its
 * targets' cells one after another: it stages a cell's candidates as in the
 * density pass, with velocity, density and pressure, then tests them for two
 * targets at a time, a candidate a lane, and compacts the hits, so that the
 * pair terms, four times a test's work for one candidate in four, run with all
 * lanes busy; a shuffle tree adds them.  (A walk by thread takes the pair
 * branch on nearly every candidate for a few of its lanes, and waits there for
 * the neighbour's velocity and density: 83 us at 33,333 particles of 0.5 h
 * spacing, 1381 us at 1,048,576 of 0.4 h; here 30 and 917.  Hits queued per
 * thread and drained together, 1923: lanes of a cell lose the loads that they
 * share while they walk in step.  Hits taken by a lane per target, 1268: their
 * numbers differ by lane and round.)  Dispersed ranges walk by thread: in
 * k_forces_dispersed, or here where a warp has fewer than 32 targets.  192
 * staged candidates leave twelve CTAs an SM: 256, 991 us; 128, 1073.  The rigid
 * contact follows by warp, for the particles in cells marked near a sphere,
 * where both grids are given: else it is read from the contact pass. */
#define FG_FORCE_STAGE 192u
#define FG_FORCE_CTAS 12
#define FG_FORCE_THREADS 64u
struct ForceShared {
    float4 a[FG_FORCE_STAGE];         /* x, y, z, rho */
    float4 b[FG_FORCE_STAGE];         /* vx, vy, vz, P */
    uint32_t j[FG_FORCE_STAGE];       /* sorted index */
    uint16_t hit[2][FG_FORCE_STAGE];  /* two targets' slots in range */
    uint32_t idx[FG_STAGE_WINDOW];
};

__global__ void __launch_bounds__(FG_FORCE_THREADS, FG_FORCE_CTAS) k_forces_search(
    uint32_t n_all, const __grid_constant__ FgScene scene, uint32_t range, uint32_t most, int dispersed,
    const float4 *__restrict__ spos, const float4 *__restrict__ svel, const float2 *__restrict__ dp,
    const uint32_t *__restrict__ start, const uint32_t *__restrict__ end, const uint32_t *__restrict__ ids,
    float4 *__restrict__ vel_out, float4 *__restrict__ pos_out, const __grid_constant__ RigidArgs R, float mass,
    float visc)
{
    __shared__ ForceShared shared[FG_FORCE_THREADS / 32];
    ForceShared &sm = shared[threadIdx.x >> 5];
    const FgScene *S = &scene;
    const StageGrid G(S);
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t lt = (1u << lane) - 1u;
    const float scale = S->scale, h = S->h, h2 = S->h2;
    const float kspiky = S->kspiky, kv = S->kvisc * visc;
    for (uint32_t b0 = (blockIdx.x * (FG_FORCE_THREADS / 32u) + (threadIdx.x >> 5)) * range; b0 < n_all;
         b0 += gridDim.x * (FG_FORCE_THREADS / 32u) * range) {
        uint32_t next, stop;
        const bool walk = fg_stage_range(b0, range, 0u, n_all, most, dispersed == DISPERSED_ASIDE, G, spos, next,
                                         stop);
        if (walk && dispersed == DISPERSED_ASIDE) continue;
        while (next < stop) {
            const uint32_t i0 = next, i = next + lane; /* sorted index */
            uint32_t n = min(32u, stop - next);
            const float4 p = lane < n ? spos[i] : make_float4(0.f, 0.f, 0.f, 0.f);
            const StageSig sig = fg_stage_sig(p, G);
            if (stop - next > 32u) n = fg_stage_trim(sig, __ldg(spos + next + 32u), G);
            next += n;
            const bool valid = lane < n;
            const bool active = valid && p.w > 0.0f;
            const float4 v = valid ? svel[i] : make_float4(0.f, 0.f, 0.f, 0.f);
            const float2 di = active ? dp[i] : make_float2(1.f, 0.f);
            const float px = p.x * scale, py = p.y * scale, pz = p.z * scale;
            float fx = 0.f, fy = 0.f, fz = 0.f;
            uint32_t lead, leads;
            fg_stage_groups(sig, __ballot_sync(FG_FULL, active && !sig.odd && !walk), lead, leads);
            for (; leads; leads &= leads - 1u) {
                const uint32_t l = (uint32_t)__ffs((int)leads) - 1u;
                const uint32_t group = __ballot_sync(FG_FULL, lead == l);
                fg_stage_rounds<FG_FORCE_STAGE, 1u>(
                    sig, lead, 1u << l, px, py, pz, G, spos, start, end, sm.idx,
                    [&](uint32_t slot, uint32_t j, float4 c) {
                        sm.a[slot] = c;
                        sm.j[slot] = j;
                    },
                    [&](uint32_t, uint32_t, uint32_t used) {
#pragma unroll 4
                        for (uint32_t s = lane; s < used; s += 32u) {
                            const uint32_t j = sm.j[s];
                            const float4 w = __ldg(svel + j);
                            const float2 d = __ldg(dp + j);
                            sm.b[s] = make_float4(w.x, w.y, w.z, d.y);
                            sm.a[s].w = d.x;
                        }
                        __syncwarp();
                        for (uint32_t g = group; g;) {
                            int t[2];
                            float tx[2], ty[2], tz[2];
                            uint32_t cnt[2] = {0u, 0u};
                            t[0] = __ffs((int)g) - 1;
                            g &= g - 1u;
                            const bool two = g != 0u;
                            t[1] = two ? __ffs((int)g) - 1 : t[0];
                            if (two) g &= g - 1u;
#pragma unroll
                            for (int u = 0; u < 2; u++) {
                                tx[u] = __shfl_sync(FG_FULL, px, t[u]);
                                ty[u] = __shfl_sync(FG_FULL, py, t[u]);
                                tz[u] = __shfl_sync(FG_FULL, pz, t[u]);
                            }
                            for (uint32_t s0 = 0u; s0 < used; s0 += 32u) {
                                const uint32_t s = s0 + lane;
                                const float4 q = sm.a[min(s, FG_FORCE_STAGE - 1u)];
                                const uint32_t j = s < used ? sm.j[s] : 0xffffffffu;
#pragma unroll
                                for (int u = 0; u < 2; u++) {
                                    const float dx = fmaf(-q.x, scale, tx[u]), dy = fmaf(-q.y, scale, ty[u]),
                                                dz = fmaf(-q.z, scale, tz[u]);
                                    const float r2 = fmaf(dx, dx, fmaf(dy, dy, __fmul_rn(dz, dz)));
                                    const bool in = r2 <= h2 && s < used && j != i0 + (uint32_t)t[u] && (u == 0 || two);
                                    const uint32_t m = __ballot_sync(FG_FULL, in);
                                    if (in) sm.hit[u][cnt[u] + (uint32_t)__popc(m & lt)] = (uint16_t)s;
                                    cnt[u] += (uint32_t)__popc(m);
                                }
                            }
                            __syncwarp();
                            float f[2][3];
#pragma unroll
                            for (int u = 0; u < 2; u++) {
                                f[u][0] = f[u][1] = f[u][2] = 0.f;
                                const float rho_t = __shfl_sync(FG_FULL, di.x, t[u]),
                                            P_t = __shfl_sync(FG_FULL, di.y, t[u]);
                                const float4 vt = make_float4(__shfl_sync(FG_FULL, v.x, t[u]),
                                                              __shfl_sync(FG_FULL, v.y, t[u]),
                                                              __shfl_sync(FG_FULL, v.z, t[u]), 0.f);
                                for (uint32_t k = lane; k < cnt[u]; k += 32u) {
                                    const uint32_t s = sm.hit[u][k];
                                    const float4 a = sm.a[s], b = sm.b[s];
                                    const float dx = fmaf(-a.x, scale, tx[u]), dy = fmaf(-a.y, scale, ty[u]),
                                                dz = fmaf(-a.z, scale, tz[u]);
                                    const float r2 = fmaf(dx, dx, fmaf(dy, dy, __fmul_rn(dz, dz)));
                                    fg_pair(f[u][0], f[u][1], f[u][2], dx, dy, dz, r2, h, kspiky, kv, rho_t, P_t, vt,
                                            a.w, b.w, b);
                                }
                            }
                            __syncwarp();
                            /* two targets' sums: one exchange leaves each half
                             * of the warp one target, a tree adds it up */
                            const bool hi = lane & 16u;
                            float r[3];
#pragma unroll
                            for (int c = 0; c < 3; c++) {
                                r[c] = __fadd_rn(hi ? f[1][c] : f[0][c],
                                                 __shfl_xor_sync(FG_FULL, hi ? f[0][c] : f[1][c], 16));
#pragma unroll
                                for (int o = 8; o; o >>= 1) r[c] = __fadd_rn(r[c], __shfl_xor_sync(FG_FULL, r[c], o));
                            }
#pragma unroll
                            for (int u = 0; u < 2; u++) {
                                const float x = __shfl_sync(FG_FULL, r[0], 16 * u);
                                const float y = __shfl_sync(FG_FULL, r[1], 16 * u);
                                const float z = __shfl_sync(FG_FULL, r[2], 16 * u);
                                if ((int)lane == t[u] && (u == 0 || two)) {
                                    fx = __fadd_rn(fx, x);
                                    fy = __fadd_rn(fy, y);
                                    fz = __fadd_rn(fz, z);
                                }
                            }
                        }
                    });
            }
            if (active && (sig.odd || walk)) {
                const float3 f = walk_terms_aside(S, i, kv, spos, svel, dp, start, end);
                fx = f.x; fy = f.y; fz = f.z;
            }
            __syncwarp();
            const uint32_t oi = valid ? __ldg(ids + i) : 0u;
            float3 sta, dyn;
            force_contacts(S, active, p, v, oi, R, sta, dyn);
            if (valid) force_finish(S, p, v, fx, fy, fz, mass, sta, dyn, oi, vel_out, pos_out);
        }
    }
}

/* The dispersed ranges of the launchers' force pass, a thread a target, as
 * k_density_dispersed: 1,048,576 random targets 0.8 h apart 610 us staged -> 527,
 * 1.2 h 749 -> 366, 3 h 799 -> 307; 262,144, 1.7 h 241 -> 75; 0.5 h, where no
 * range is dispersed, 584 -> 589.  Seven CTAs an SM: with six, 262,144 take 98. */
#define FG_WALK_FORCE_CTAS 7
__global__ void __launch_bounds__(FG_CHUNK, FG_WALK_FORCE_CTAS) k_forces_dispersed(
    uint32_t n_all, const __grid_constant__ FgScene scene, uint32_t most, const float4 *__restrict__ spos,
    const float4 *__restrict__ svel, const float2 *__restrict__ dp, const uint32_t *__restrict__ start,
    const uint32_t *__restrict__ end, const uint32_t *__restrict__ ids, float4 *__restrict__ vel_out,
    float4 *__restrict__ pos_out, const __grid_constant__ RigidArgs R, float mass, float visc)
{
    const FgScene *S = &scene;
    const StageGrid G(S);
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t i0 = blockIdx.x * FG_CHUNK + (threadIdx.x & ~31u);
    float4 ahead = __ldg(spos + min(i0 + lane, n_all - 1u));
    for (; i0 < n_all; i0 += gridDim.x * FG_CHUNK) {
        const uint32_t i = i0 + lane;
        const float4 p = ahead;
        ahead = __ldg(spos + min(i + gridDim.x * FG_CHUNK, n_all - 1u));
        if (!fg_stage_dispersed(fg_stage_cell(p, G), G, 32u, most)) continue;
        const bool valid = i < n_all, active = valid && p.w > 0.0f;
        const float4 v = valid ? __ldg(svel + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        float fx = 0.f, fy = 0.f, fz = 0.f;
        if (active) walk_terms(S, i, p, v, S->kvisc * visc, spos, svel, dp, start, end, fx, fy, fz);
        __syncwarp();
        const uint32_t oi = valid ? __ldg(ids + i) : 0u;
        float3 sta, dyn;
        force_contacts(S, active, p, v, oi, R, sta, dyn);
        if (valid) force_finish(S, p, v, fx, fy, fz, mass, sta, dyn, oi, vel_out, pos_out);
        __syncwarp();
    }
}

void launch_forces(const Launch &L, const float4 *spos, const float4 *svel, const float2 *dp, const uint32_t *start,
                   const uint32_t *end, const uint32_t *ids, ForceOut out, const RigidGrid *rigid,
                   const RigidGrid *statics, float mass_o, float visc_o, int use_o, const NbrList *list,
                   TargetOrder ord)
{
    if (!L.nwork) return;
    RigidArgs R;
    memset(&R, 0, sizeof(R));
    if (rigid) { R.dyn = *rigid; R.use_dyn = 1; }
    if (statics) { R.sta = *statics; R.use_sta = 1; }
    if (!list && use_o) {
        const uint32_t range = stage_range(L.nwork), warps = (L.n + range - 1u) / range;
        const uint32_t ctas = grid_for((warps + FG_FORCE_THREADS / 32u - 1u) / (FG_FORCE_THREADS / 32u), 128);
        uint32_t most;
        int dispersed = dispersed_ranges(L, range, most);
        const SideLaunch side(L, dispersed);
        if (side.use)
            k_forces_dispersed<<<grid_for(L.nwork, FG_WALK_FORCE_CTAS), FG_CHUNK, 0, L.side.stream>>>(
                L.n, *L.single, most, spos, svel, dp, start, end, ids, out.vel, out.pos, R, mass_o, visc_o);
        k_forces_search<<<ctas, FG_FORCE_THREADS, 0, L.stream>>>(L.n, *L.single, range, most, dispersed, spos, svel,
                                                                dp, start, end, ids, out.vel, out.pos, R, mass_o,
                                                                visc_o);
        return;
    }
    const uint32_t B = L.block ? L.block : FG_CHUNK;
    const uint32_t ipc = FG_ITEMS_PER_CTA(B);
    const int per_sm = (int)(((L.ctas_per_sm ? L.ctas_per_sm : 64u) * FG_CHUNK) / B);
    const uint32_t g = grid_for((L.nwork + ipc - 1u) / ipc, per_sm > 0 ? per_sm : 1);
#define FG_FORCES(BL)                                                                                              \
    if (list)                                                                                                      \
        k_forces<BL><<<g, BL, 0, L.stream>>>(L.work, L.nwork, L.n, L.table, *L.single, spos, svel, start, end, ids, \
                                             out.vel, out.pos, R, *list, ord);                                     \
    else                                                                                                           \
        k_forces_walk<BL><<<g, BL, 0, L.stream>>>(L.work, L.nwork, L.n, L.table, *L.single, spos, svel, dp, start, \
                                                  end, ids, out.vel, out.pos, R, ord)
    if (B == 64u) {
        FG_FORCES(64);
    } else if (B == 256u) {
        FG_FORCES(256);
    } else {
        FG_FORCES(128);
    }
#undef FG_FORCES
}

/* The fluid side of the fluid/rigid contact ahead of the force pass, by
 * particle id from the step's unsorted positions and velocities (the sorted
 * copies hold the same bits), so it runs right after the rigid-sphere grid
 * beside the fluid hash and sort.  The particles inside the bodies' AABB and
 * in a cell marked near a sphere (a shell around the bodies' surfaces) search
 * the rigid grid, a warp each: the pass is bound by the latency of those
 * searches, and a lane's own chain of 25 bucket rows and about 55 spheres,
 * diverging from its neighbours', takes as long as dozens of searches by
 * warp.  The CTA's eight warps share the searches of its 128 particles, which
 * ids along a surface may all need.  4M particles, eight bodies whose AABB is
 * the whole scene: 1007 -> 151 us by itself (a lane each inside the AABB ->
 * here; a lane each in marked cells only: 399; a warp per eight particles:
 * 235), some 230 beside the density pass.  The force pass adds the stored sum
 * where it would add the walked one: the same bits.
 * The launchers' pass goes over sorted particles and stores by id; within the
 * force search, whose shared memory leaves the bucket tables no L1, the same
 * searches took twice the time and more (262,144 particles: 4,096 spheres all
 * among them 652 -> 376 us for contact and forces; 32,768 and a half-width of
 * 4, half as many particles, 2584 -> 987; four bodies' surfaces, the whole
 * two-way pass, 488 -> 439). */
#define FG_CONTACT_THREADS 256u
/* Searches of a work item beyond which its particles walk by thread instead:
 * the 27 buckets of a half-width of 1 leave most of a searching warp idle, and
 * those of 3 and more are searched round by round.  Walking takes as long
 * however many lanes of a CTA need it, and an SM its 128 threads an item: such a
 * CTA takes two items, and walks or searches both (an item of each kind took as
 * long as the two forms one after the other, 556 us).  A step of 131,072
 * particles with spheres among 0.6, 0.8 and all of the width, searched -> by this
 * rule: half-width 1, 169, 200, 231 -> 164, 162, 173 us; 3, 287, 455, 612 -> 287,
 * 450, 454; 5, 836, 1548, 2196 -> 835, 1380, 1342.  (Half-width 2: 257 us walked
 * and 245 searched with 1,024 spheres, 437 and 353 with 32,768.)  Its registers
 * cost the other half-widths 3%, so they have a kernel without it; the choice
 * of the output's index (IDS) made while it runs cost 3% too. */
__host__ __device__ __forceinline__ uint32_t contact_searches(const int rel[3])
{
    const uint32_t total = (2u * rel[0] + 1u) * (2u * rel[1] + 1u) * (2u * rel[2] + 1u);
    return total <= 27u ? 44u : total <= 216u ? FG_CHUNK : 72u;
}
template <bool WALKS, bool IDS>
__global__ void __launch_bounds__(FG_CONTACT_THREADS) k_fluid_contact(const FgWork *__restrict__ work, uint32_t nwork,
                                                           uint32_t n_single, const FgScene *__restrict__ table,
                                                           const __grid_constant__ FgScene single,
                                                           const float4 *__restrict__ pos,
                                                           const float4 *__restrict__ vel,
                                                           const __grid_constant__ RigidGrid G,
                                                           const uint32_t *__restrict__ ids,
                                                           float4 *__restrict__ out)
{
    constexpr uint32_t ITEMS = WALKS ? FG_CONTACT_THREADS / FG_CHUNK : 1u; /* at a time */
    __shared__ uint32_t s_id[ITEMS][FG_CHUNK], s_n[ITEMS];
    const uint32_t lane = threadIdx.x & 31u;
    const bool dynamic = G.body_vel != nullptr;
    for (uint32_t w0 = ITEMS * blockIdx.x; w0 < nwork; w0 += ITEMS * gridDim.x) {
        const uint32_t items = min(ITEMS, nwork - w0), h = threadIdx.x / FG_CHUNK, t = threadIdx.x % FG_CHUNK;
        const FgWork it = fg_work(work, w0 + min(h, items - 1u), n_single);
        const FgScene *S = fg_scene(table, &single, it.scene);
        uint32_t some = 0u, bodies = S->flags & FG_SCENE_HAS_RB; /* some: searches beyond which all are walked */
        for (uint32_t q = 0; WALKS && q < items; q++) {
            const FgScene *Q = fg_scene(table, &single, fg_work(work, w0 + q, n_single).scene);
            bodies |= Q->flags & FG_SCENE_HAS_RB;
            some += contact_searches(Q->f2r_rel);
        }
        if (!bodies) continue; /* uniform over the CTA */
        if (threadIdx.x < ITEMS) s_n[threadIdx.x] = 0u;
        __syncthreads();
        if (h < items) {
            const uint32_t id = it.first + t;
            bool near = false;
            if (t < it.count && (S->flags & FG_SCENE_HAS_RB)) {
                const float4 p = __ldg(pos + id);
                near = p.w > 0.0f && !fg_contact_outside(S, it.scene, p, G) && fg_contact_marked(S, it.scene, p, G);
            }
            const uint32_t m = __ballot_sync(0xffffffffu, near);
            uint32_t base = 0u;
            if (lane == 0u && m) base = atomicAdd(&s_n[h], (uint32_t)__popc(m));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (near) s_id[h][base + __popc(m & ((1u << lane) - 1u))] = id;
        }
        __syncthreads();
        if (WALKS && s_n[0] + s_n[ITEMS - 1u] > some) {
            if (h < items && t < s_n[h]) {
                const uint32_t id = s_id[h][t];
                const float3 c = fg_fluid_rigid_contact(S, it.scene, __ldg(pos + id), __ldg(vel + id), G, dynamic);
                out[IDS ? __ldg(ids + id) : id] = make_float4(c.x, c.y, c.z, 0.0f);
            }
            __syncthreads();
            continue;
        }
        for (uint32_t q = 0; q < items; q++) {
            const FgScene *Q = WALKS ? fg_scene(table, &single, fg_work(work, w0 + q, n_single).scene) : S;
            const ContactShape C(Q);
            for (uint32_t k = threadIdx.x >> 5; k < s_n[q]; k += FG_CONTACT_THREADS / 32u) {
                const uint32_t id = s_id[q][k];
                const float3 c = fg_contact_warp(Q, C, __ldg(pos + id), __ldg(vel + id), G, dynamic);
                if (lane == 0u) out[IDS ? __ldg(ids + id) : id] = make_float4(c.x, c.y, c.z, 0.0f);
            }
        }
        __syncthreads();
    }
}

void launch_fluid_contact(const Launch &L, const float4 *pos, const float4 *vel, const RigidGrid &G, float4 *out,
                          bool may_walk, const uint32_t *ids)
{
    if (!L.nwork) return;
    /* an SM's worth of CTAs: a CTA per item queues ahead of the grid kernels
     * beside this one (64 worlds after 400 steps 896 us a step, here 883; 4M
     * particles 2163, here 2135) */
    const uint32_t g = grid_for(may_walk ? (L.nwork + 1u) / 2u : L.nwork, 8);
    auto *k = ids ? (may_walk ? k_fluid_contact<true, true> : k_fluid_contact<false, true>)
                  : (may_walk ? k_fluid_contact<true, false> : k_fluid_contact<false, false>);
    k<<<g, FG_CONTACT_THREADS, 0, L.stream>>>(L.work, L.nwork, L.n, L.table, *L.single, pos, vel, G, ids, out);
}

/* Many spheres favour the search, which takes them a lane each: 65,536
 * particles and a half-width of 8, a step with half as many spheres 4156 us
 * searched and 6842 walked, with a sixteenth 6372 and 4406; 131,072 and a
 * quarter 7381 and 6298. */
bool contact_may_walk(const int rel[3], uint32_t spheres, uint32_t particles)
{
    const uint32_t searches = contact_searches(rel);
    return searches < 64u || (searches < FG_CHUNK && spheres <= particles / 4u);
}

/* SPHIntegrateK (K_FluidSim.cu:418-438): pos += vel*(dt/scale) for active
 * particles, all four components, each operation rounded separately. */
__global__ void __launch_bounds__(FG_CHUNK) k_integrate(const FgWork *__restrict__ work, uint32_t nwork,
                                                       uint32_t n_single, const FgScene *__restrict__ table,
                                                       const __grid_constant__ FgScene single,
                                                       float4 *__restrict__ pos, const float4 *__restrict__ vel)
{
    for (uint32_t w = blockIdx.x; w < nwork; w += gridDim.x) {
        FgWork it = fg_work(work, w, n_single);
        if (threadIdx.x >= it.count) continue;
        const FgScene *S = fg_scene(table, &single, it.scene);
        const uint32_t i = it.first + threadIdx.x;
        float4 p = pos[i];
        if (p.w > 0.0f) {
            const float4 v = __ldg(vel + i);
            const float c = S->dt_over_scale;
            p.x = __fadd_rn(p.x, __fmul_rn(v.x, c));
            p.y = __fadd_rn(p.y, __fmul_rn(v.y, c));
            p.z = __fadd_rn(p.z, __fmul_rn(v.z, c));
            p.w = __fadd_rn(p.w, __fmul_rn(v.w, c));
            pos[i] = p;
        }
    }
}

void launch_integrate(const Launch &L, float4 *pos, const float4 *vel)
{
    if (!L.nwork) return;
    k_integrate<<<grid_for(L.nwork, 16), FG_CHUNK, 0, L.stream>>>(L.work, L.nwork, L.n, L.table, *L.single, pos,
                                                                  vel);
}

} // namespace fg
