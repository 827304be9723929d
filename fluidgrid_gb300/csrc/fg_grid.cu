/* Hash-grid build on GB300: particle hash, stable key/index radix sort, cell
 * start/end ranges with the sorted gather of position and velocity.
 *
 * Follows the reference's grid build (GPU_Kernels/K_HashGrid.cu:26-197 and the
 * thrust/CUDPP key-value sorts, K_FluidSim.cu:685-691,
 * RigidBodySimulator.cpp:195-196) with identical results: keys bit-exact,
 * ascending key order with ties in particle-index order, same start/end
 * entries.  All kernels stream coalesced 16-byte loads; the sort is a
 * reduce-then-scan LSD radix sort whose CTAs never wait on one another. */
#include <cuda_runtime.h>
#include <cooperative_groups.h>
#include <stdint.h>
#include <algorithm>
#include <atomic>
#include "fg_device.cuh"
#include "fg_kernels.h"

namespace fg {

int sm_count()
{
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
            sms = 152;
    }
    return sms;
}

uint32_t grid_for(uint32_t nwork, int ctas_per_sm)
{
    uint32_t cap = (uint32_t)sm_count() * (uint32_t)ctas_per_sm;
    return std::max(1u, std::min(nwork, cap));
}

/* ------------------------------------------------------------- hashing */

/* cnt[key] += 1 for every valid lane of the (converged) warp; the count that
 * the lane finds there, its own place in the bucket: one L2 atomic per run of
 * equal keys in neighbouring lanes (a match_any finds the same runs in as many
 * rounds as there are keys; 1M particles of a lattice: 15 -> 10.5 us). */
__device__ __forceinline__ uint32_t bs_count_in(uint32_t key, bool valid, uint32_t *__restrict__ cnt)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t prev = __shfl_up_sync(0xffffffffu, key, 1);
    const uint32_t act = __ballot_sync(0xffffffffu, valid); /* a prefix of the lanes */
    const uint32_t heads = __ballot_sync(0xffffffffu, valid && (lane == 0u || key != prev));
    const uint32_t upto = heads & (0xffffffffu >> (31u - lane)), later = heads & ~(0xffffffffu >> (31u - lane));
    const uint32_t head = upto ? 31u - (uint32_t)__clz((int)upto) : lane;
    uint32_t o = 0u;
    if (valid && head == lane) {
        const uint32_t next = later ? (uint32_t)__ffs((int)later) - 1u : (uint32_t)__popc(act);
        o = atomicAdd(cnt + key, next - lane);
    }
    return __shfl_sync(0xffffffffu, o, (int)head) + lane - head;
}

/* CalcHashKeyK (K_HashGrid.cu:26-38): key = bucket_base + HashKeyD(pos),
 * id = particle index.  With cnt, also the counting sort's first pass (as
 * k_bs_count): cnt[key] += 1 by L2 atomics, one per run of equal keys in a
 * warp, and off[i] = the count found there. */
__global__ void __launch_bounds__(FG_CHUNK) k_hash(const FgWork *__restrict__ work, uint32_t nwork, uint32_t n_single,
                                                  const FgScene *__restrict__ table,
                                                  const __grid_constant__ FgScene single,
                                                  const float4 *__restrict__ pos, uint32_t *__restrict__ keys,
                                                  uint32_t *__restrict__ ids, uint32_t *__restrict__ cnt,
                                                  uint32_t *__restrict__ off)
{
    for (uint32_t w = blockIdx.x; w < nwork; w += gridDim.x) {
        FgWork it = fg_work(work, w, n_single);
        const FgScene *S = fg_scene(table, &single, it.scene);
        const bool valid = threadIdx.x < it.count;
        const uint32_t i = it.first + threadIdx.x;
        uint32_t k = 0;
        if (valid) {
            float4 p = __ldg(pos + i);
            k = S->bucket_base + fg_hash(p.x, p.y, p.z, S->cell, S->nb, S->nb_mask);
            keys[i] = k;
            if (ids) ids[i] = i;
        }
        if (cnt) { /* uniform: every lane of the warp gets here */
            const uint32_t o = bs_count_in(k, valid, cnt);
            if (valid) off[i] = o;
        }
    }
}

void launch_hash(const Launch &L, const float4 *pos, uint32_t *keys, uint32_t *ids, uint32_t *cnt, uint32_t *off)
{
    if (!L.nwork) return;
    k_hash<<<grid_for(L.nwork, 64), FG_CHUNK, 0, L.stream>>>(L.work, L.nwork, L.n, L.table, *L.single, pos, keys,
                                                             ids, cnt, off);
}

/* CalcHashKeyWithOffsetK (K_HashGrid.cu:43-63): world = conj(q)*p*q + cm of
 * the sphere's body (w = body index), key of the world position in the
 * rigid grid.  Optionally grows the per-scene AABB of sphere centres (six
 * ordered ints: min xyz, max xyz) and marks the cells near each sphere. */
__global__ void __launch_bounds__(FG_CHUNK) k_hash_offset(const FgWork *__restrict__ work, uint32_t nwork,
                                                         uint32_t n_single, const FgScene *__restrict__ table,
                                                         const __grid_constant__ FgScene single,
                                                         const float4 *__restrict__ local,
                                                         const float4 *__restrict__ cm,
                                                         const float4 *__restrict__ q, float4 *__restrict__ world,
                                                         uint32_t *__restrict__ keys, uint32_t *__restrict__ ids,
                                                         int *__restrict__ aabb, uint32_t *__restrict__ near,
                                                         uint32_t near_mask)
{
    for (uint32_t w = blockIdx.x; w < nwork; w += gridDim.x) {
        FgWork it = fg_work(work, w, n_single);
        const FgScene *S = fg_scene(table, &single, it.scene);
        bool ok = threadIdx.x < it.count;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
        if (ok) {
            uint32_t i = it.first + threadIdx.x;
            float4 p = __ldg(local + i);
            int b = (int)p.w;
            float4 t = fg_qtransform_rn(p, __ldg(q + b));
            float4 o = __ldg(cm + b);
            a.x = __fadd_rn(t.x, o.x);
            a.y = __fadd_rn(t.y, o.y);
            a.z = __fadd_rn(t.z, o.z);
            a.w = p.w;
            world[i] = a;
            keys[i] = S->rb_bucket_base + fg_hash(a.x, a.y, a.z, S->rb_cell, S->rb_nb, S->rb_nb_mask);
            if (ids) ids[i] = i;
            if (near) {
                int cx, cy, cz;
                const float mind = S->fluid_radius + S->rb_radius + S->fluid_eps;
                fg_near_cell(a.x, a.y, a.z, fg_near_inv(mind), cx, cy, cz);
                fg_near_mark(cx, cy, cz, it.scene, near, near_mask);
            }
        }
        if (aabb) {
            /* warp-reduce then one atomic per warp per bound */
            float mn[3] = {ok ? a.x : 3.0e38f, ok ? a.y : 3.0e38f, ok ? a.z : 3.0e38f};
            float mx[3] = {ok ? a.x : -3.0e38f, ok ? a.y : -3.0e38f, ok ? a.z : -3.0e38f};
#pragma unroll
            for (int d = 0; d < 3; d++)
#pragma unroll
                for (int o = 16; o; o >>= 1) {
                    mn[d] = fminf(mn[d], __shfl_xor_sync(0xffffffffu, mn[d], o));
                    mx[d] = fmaxf(mx[d], __shfl_xor_sync(0xffffffffu, mx[d], o));
                }
            if ((threadIdx.x & 31) == 0 && (threadIdx.x >> 5) * 32 < it.count) {
                int *bx = aabb + 6 * it.scene;
#pragma unroll
                for (int d = 0; d < 3; d++) {
                    atomicMin(bx + d, fg_float_ord(mn[d]));
                    atomicMax(bx + 3 + d, fg_float_ord(mx[d]));
                }
            }
        }
    }
}

void launch_hash_with_offset(const Launch &L, const float4 *local, const float4 *cm, const float4 *q, float4 *world,
                             uint32_t *keys, uint32_t *ids, int *aabb, uint32_t *near, uint32_t near_mask)
{
    if (!L.nwork) return;
    k_hash_offset<<<grid_for(L.nwork, 16), FG_CHUNK, 0, L.stream>>>(L.work, L.nwork, L.n, L.table, *L.single, local,
                                                                    cm, q, world, keys, ids, aabb, near, near_mask);
}

/* ----------------------------------------------------------- radix sort
 * LSD radix sort, up to 8 bits per pass, tiles of RS_TILE keys:
 *   upsweep   per-tile digit counts          hist[d * T + t]
 *   scan      per digit, exclusive over tiles  (one CTA per digit) + totals
 *   downsweep stable in-tile ranking (a ballot a bit), shared-memory
 *             staging in digit order, coalesced scatter.
 * Ranks within a tile follow particle order (warp w holds keys
 * [w*512, w*512+512) of the tile, item k of lane l is key w*512 + 32k + l and
 * items are ranked k-major, lane-minor), so each pass is stable. */

#define RS_THREADS 256
#define RS_ITEMS 8
#define RS_TILE (RS_THREADS * RS_ITEMS)
static_assert(RS_TILE == FG_RS_TILE, "scratch sizes elsewhere assume FG_RS_TILE keys per tile");
#define RS_RADIX 256
#define RS_WARPS (RS_THREADS / 32)

size_t radix_hist_words(uint32_t n)
{
    size_t tiles = ((size_t)n + RS_TILE - 1) / RS_TILE;
    return (size_t)RS_RADIX * std::max<size_t>(tiles, 1) + RS_RADIX;
}

int radix_passes(uint32_t bits, uint32_t digit_bits)
{
    if (digit_bits < 1) digit_bits = 1;
    if (digit_bits > 8) digit_bits = 8;
    return (int)((bits + digit_bits - 1) / digit_bits);
}

/* The lanes of the warp whose digit (of `bits` bits) is the same: a ballot a
 * bit.  match_any takes a round for each distinct value of the warp: with it
 * the downsweep of 700,000 random pairs took 11.4 us, with the ballots 9.2; but
 * of keys in runs, as those of a fluid are, a sort of 4,000,000 (21 bits) took
 * 187 us with match_any, 173 with the ballots, and takes 156 choosing by the
 * runs of a warp's first keys (a lattice's keys 198, 174, 169; random ones 228,
 * 178, 180; 700,000 of these, chosen key by key, 83 instead of 82). */
__device__ __forceinline__ uint32_t rs_peers(uint32_t d, uint32_t bits)
{
    uint32_t peers = 0xffffffffu;
#pragma unroll
    for (uint32_t b = 0; b < 8u; b++)
        if (b < bits) {
            const bool one = d >> b & 1u;
            const uint32_t m = __ballot_sync(0xffffffffu, one);
            peers &= one ? m : ~m;
        }
    return peers;
}

/* keep_k, keep_v (optional): copies of the pass's input */
__global__ void __launch_bounds__(RS_THREADS) k_rs_upsweep(const uint32_t *__restrict__ keys, uint32_t n,
                                                          uint32_t shift, uint32_t mask, uint32_t *__restrict__ hist,
                                                          uint32_t T, const uint32_t *__restrict__ vals,
                                                          uint32_t *__restrict__ keep_k,
                                                          uint32_t *__restrict__ keep_v)
{
    __shared__ uint32_t cnt[RS_RADIX];
    cnt[threadIdx.x] = 0;
    __syncthreads();
    size_t base = (size_t)blockIdx.x * RS_TILE;
#pragma unroll
    for (int k = 0; k < RS_ITEMS; k++) {
        size_t i = base + (size_t)k * RS_THREADS + threadIdx.x;
        if (i < n) {
            const uint32_t key = __ldg(keys + i);
            atomicAdd(&cnt[(key >> shift) & mask], 1u);
            if (keep_k) {
                keep_k[i] = key;
                keep_v[i] = vals ? __ldg(vals + i) : (uint32_t)i;
            }
        }
    }
    __syncthreads();
    hist[(size_t)threadIdx.x * T + blockIdx.x] = cnt[threadIdx.x];
}

/* block-wide exclusive scan of one value per thread (RS_THREADS threads) */
__device__ __forceinline__ uint32_t rs_block_excl(uint32_t v, uint32_t *s_warp, uint32_t &total)
{
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) s_warp[wid] = x;
    __syncthreads();
    if (wid == 0) {
        uint32_t t = lane < RS_WARPS ? s_warp[lane] : 0;
        uint32_t u = t;
#pragma unroll
        for (int o = 1; o < RS_WARPS; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, u, o);
            if (lane >= (uint32_t)o) u += y;
        }
        if (lane < RS_WARPS) s_warp[lane] = u - t;
        if (lane == RS_WARPS - 1) s_warp[RS_WARPS] = u;
    }
    __syncthreads();
    uint32_t r = x - v + s_warp[wid];
    total = s_warp[RS_WARPS];
    __syncthreads();
    return r;
}

/* One CTA per digit: exclusive scan of hist[d*T .. d*T+T) in place. */
__global__ void __launch_bounds__(RS_THREADS) k_rs_scan(uint32_t *__restrict__ hist, uint32_t T,
                                                       uint32_t *__restrict__ totals)
{
    __shared__ uint32_t s_warp[RS_WARPS + 1];
    uint32_t *h = hist + (size_t)blockIdx.x * T;
    uint32_t carry = 0;
    for (uint32_t base = 0; base < T; base += RS_THREADS) {
        uint32_t i = base + threadIdx.x;
        uint32_t v = i < T ? h[i] : 0;
        uint32_t tot;
        uint32_t e = rs_block_excl(v, s_warp, tot);
        if (i < T) h[i] = e + carry;
        carry += tot;
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

__global__ void __launch_bounds__(RS_THREADS) k_rs_downsweep(const uint32_t *__restrict__ kin,
                                                            const uint32_t *__restrict__ vin,
                                                            uint32_t *__restrict__ kout, uint32_t *__restrict__ vout,
                                                            uint32_t n, uint32_t shift, uint32_t mask,
                                                            const uint32_t *__restrict__ hist,
                                                            const uint32_t *__restrict__ totals, uint32_t T)
{
    __shared__ uint32_t s_keys[RS_TILE];
    __shared__ uint32_t s_vals[RS_TILE];
    __shared__ uint32_t s_whist[RS_WARPS][RS_RADIX];
    __shared__ uint32_t s_goff[RS_RADIX];
    __shared__ uint32_t s_tstart[RS_RADIX];
    __shared__ uint32_t s_warp[RS_WARPS + 1];

    const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const size_t base = (size_t)blockIdx.x * RS_TILE;

    /* global offset of each digit for this tile */
    {
        uint32_t tot;
        uint32_t gb = rs_block_excl(totals[tid], s_warp, tot);
        s_goff[tid] = gb + hist[(size_t)tid * T + blockIdx.x];
    }
#pragma unroll
    for (int w = 0; w < RS_WARPS; w++) s_whist[w][tid] = 0;
    __syncthreads();

    uint32_t key[RS_ITEMS], val[RS_ITEMS], rank[RS_ITEMS];
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t bits = (uint32_t)__popc(mask);
#pragma unroll
    for (int k = 0; k < RS_ITEMS; k++) {
        const size_t i = base + (size_t)wid * (32 * RS_ITEMS) + (size_t)k * 32 + lane;
        key[k] = i < n ? __ldg(kin + i) : 0xffffffffu;
        val[k] = i < n ? (vin ? __ldg(vin + i) : (uint32_t)i) : 0u;
    }
    /* up to nine runs of equal digits in the warp's first 32: match_any, a round a digit */
    const uint32_t d0 = (key[0] >> shift) & mask;
    const bool few = (uint32_t)__popc(__ballot_sync(0xffffffffu, d0 != __shfl_up_sync(0xffffffffu, d0, 1))) < 9u;
    auto rank_all = [&](auto &&peers_of) {
#pragma unroll
        for (int k = 0; k < RS_ITEMS; k++) {
            const bool valid = base + (size_t)wid * (32 * RS_ITEMS) + (size_t)k * 32 + lane < n;
            const uint32_t d = (key[k] >> shift) & mask;
            const uint32_t peers = peers_of(d) & __ballot_sync(0xffffffffu, valid);
            const uint32_t leader = valid ? (uint32_t)__ffs((int)peers) - 1u : lane;
            uint32_t b = 0;
            if (valid && lane == leader) {
                b = s_whist[wid][d];
                s_whist[wid][d] = b + __popc(peers);
            }
            b = __shfl_sync(0xffffffffu, b, (int)leader);
            rank[k] = b + __popc(peers & lt);
            __syncwarp();
        }
    };
    if (few) rank_all([](uint32_t d) { return __match_any_sync(0xffffffffu, d); });
    else rank_all([bits](uint32_t d) { return rs_peers(d, bits); });
    __syncthreads();
    /* per digit: exclusive over warps, tile count */
    uint32_t run = 0;
#pragma unroll
    for (int w = 0; w < RS_WARPS; w++) {
        uint32_t c = s_whist[w][tid];
        s_whist[w][tid] = run;
        run += c;
    }
    {
        uint32_t tot;
        uint32_t ts = rs_block_excl(run, s_warp, tot);
        s_tstart[tid] = ts;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < RS_ITEMS; k++) {
        size_t i = base + (size_t)wid * (32 * RS_ITEMS) + (size_t)k * 32 + lane;
        if (i < n) {
            uint32_t d = (key[k] >> shift) & mask;
            uint32_t p = s_tstart[d] + s_whist[wid][d] + rank[k];
            s_keys[p] = key[k];
            s_vals[p] = val[k];
        }
    }
    __syncthreads();
    uint32_t tile_n = (n - base) < (size_t)RS_TILE ? (uint32_t)(n - base) : (uint32_t)RS_TILE;
    for (uint32_t i = tid; i < tile_n; i += RS_THREADS) {
        uint32_t kk = s_keys[i];
        uint32_t d = (kk >> shift) & mask;
        uint32_t g = s_goff[d] + (i - s_tstart[d]);
        kout[g] = kk;
        vout[g] = s_vals[i];
    }
}

__global__ void k_iota_copy(const uint32_t *__restrict__ kin, const uint32_t *__restrict__ vin,
                            uint32_t *__restrict__ kout, uint32_t *__restrict__ vout, uint32_t n)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        kout[i] = kin[i];
        vout[i] = vin ? vin[i] : i;
    }
}

/* ---- up to 65,536 pairs: the whole sort in one launch ----
 * One cluster of up to sixteen CTAs keeps the pairs on chip: ITEMS a thread in
 * registers, ranked in the CTA as k_rs_downsweep does; the CTAs read one
 * another's digit totals, order their tile by digit in shared memory and write
 * its runs into one another's, two cluster barriers a pass, 8 bits a pass.  A
 * digit that all keys share is skipped (a 32-bit sort of small keys).  The
 * three kernels a pass above are, at these sizes, launches and latency.
 * Measured in a captured graph, three kernels a pass before (with a
 * match_any a key) -> one launch, 17 bits: 39.9 -> 10.9 us at 4,096 pairs,
 * 40.6 -> 13.5 at 16,384, 42.4 -> 18.0 at 32,768, 42.7 -> 25.8 at 65,536; 32
 * bits, no digit shared: 52 -> 14.1, 17.8, 24.3, 56 -> 35.2.  The time is the
 * ranking and the staging of four pairs a thread on sixteen SMs by then (of
 * eight on eight, the portable cluster: 32.4 and 44.6).  Scattering each pair
 * straight into the other CTA's memory, a word at a time, took 43.3 us at
 * 65,536 pairs of 17 bits on eight: 32 destinations a warp. */
#define CS_THREADS 1024
#define CS_CTAS 16u

struct TileRank {
    uint16_t whist[CS_THREADS / 32][RS_RADIX];
    uint32_t part[4][RS_RADIX];
};

/* One digit of a CTA's tile (item k of lane l of warp w is pair
 * (w * ITEMS + k) * 32 + l): rank[] is each pair's place among its warp's of
 * the digit, R.whist[w][d] how many the warps before w hold; returns, in the
 * last 256 threads, the tile's count of digit threadIdx.x & 255.  A warp with
 * `idle` holds no pairs. */
template <int ITEMS>
__device__ __forceinline__ uint32_t rs_tile_rank(TileRank &R, const uint32_t (&key)[ITEMS], uint32_t (&rank)[ITEMS],
                                                 uint32_t shift, uint32_t db, bool idle)
{
    const uint32_t tid = threadIdx.x, wid = tid >> 5, lt = (1u << (tid & 31u)) - 1u, mask = (1u << db) - 1u;
    for (uint32_t w = tid; w < sizeof(R.whist) / 4u; w += CS_THREADS) ((uint32_t *)R.whist)[w] = 0u;
    __syncthreads();
    if (!idle) {
#pragma unroll
        for (int k = 0; k < ITEMS; k++) {
            const uint32_t d = key[k] >> shift & mask, peers = rs_peers(d, db);
            const uint32_t b = R.whist[wid][d];
            __syncwarp();
            if ((peers & lt) == 0u) R.whist[wid][d] = (uint16_t)(b + __popc(peers));
            rank[k] = b + __popc(peers & lt);
            __syncwarp();
        }
    }
    __syncthreads();
    /* per digit: exclusive over the warps, eight of them a thread */
    const uint32_t d = tid & 255u, q = tid >> 8;
    uint32_t run = 0u, c[8];
#pragma unroll
    for (int w = 0; w < 8; w++) {
        c[w] = R.whist[8u * q + w][d];
        run += c[w];
    }
    R.part[q][d] = run;
    __syncthreads();
    uint32_t before = 0u;
    for (uint32_t r = 0; r < q; r++) before += R.part[r][d];
#pragma unroll
    for (int w = 0; w < 8; w++) {
        R.whist[8u * q + w][d] = (uint16_t)before;
        before += c[w];
    }
    return before;
}

template <int ITEMS>
struct ClusterSort {
    uint2 stage[CS_THREADS * ITEMS]; /* the tile's pairs by digit */
    uint2 pair[CS_THREADS * ITEMS];  /* the cluster's, from any CTA */
    TileRank tile;
    uint32_t tot[2][RS_RADIX]; /* of alternate passes: the cluster may still read the one before */
    uint32_t goff[RS_RADIX], loff[RS_RADIX]; /* a digit's first place in the cluster and in the stage */
    uint32_t wsum[2 * RS_RADIX / 32];
    uint32_t same[2];
};

template <int ITEMS>
__global__ void __launch_bounds__(CS_THREADS, 1) k_sort_cluster(const uint32_t *kin, const uint32_t *vin,
                                                               uint32_t *kout, uint32_t *vout, uint32_t n,
                                                               uint32_t bits) /* kout may be kin, vout vin */
{
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) unsigned char smem[];
    ClusterSort<ITEMS> &S = *reinterpret_cast<ClusterSort<ITEMS> *>(smem);
    cg::cluster_group cl = cg::this_cluster();
    constexpr uint32_t TILE = CS_THREADS * ITEMS;
    const uint32_t me = cl.block_rank(), ctas = cl.num_blocks(), all = ctas * TILE;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, wid = tid >> 5;
    const uint32_t mine = wid * 32u * ITEMS + lane; /* item k: mine + 32 k of the tile */
    uint32_t key[ITEMS], val[ITEMS], rank[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; k++) {
        /* past the end: the largest key, after all equal ones */
        const uint32_t i = me * TILE + mine + 32u * k;
        key[k] = i < n ? kin[i] : 0xffffffffu;
        val[k] = i < n ? (vin ? vin[i] : i) : 0u;
    }
    uint32_t turn = 0u;
    for (uint32_t shift = 0u; shift < bits; shift += 8u, turn ^= 1u) {
        const uint32_t db = min(8u, bits - shift), mask = (1u << db) - 1u;
        const uint32_t count = rs_tile_rank<ITEMS>(S.tile, key, rank, shift, db, false);
        const uint32_t d = tid & 255u;
        if (tid >= CS_THREADS - RS_RADIX) S.tot[turn][d] = count;
        cl.sync();
        /* each digit's first place: of all its pairs and of the tile's among
         * them (threads 0 to 255), and in the staged tile (the next 256) */
        uint32_t ahead = 0u, total = 0u;
        if (tid < RS_RADIX) {
            for (uint32_t r = 0; r < ctas; r++) {
                const uint32_t t = *cl.map_shared_rank(&S.tot[turn][d], (int)r);
                total += t;
                if (r < me) ahead += t;
            }
            if (tid == 0u) S.same[turn] = 0u;
        } else if (tid < 2 * RS_RADIX) {
            total = S.tot[turn][d];
        }
        uint32_t incl = total;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += y;
        }
        if (tid < 2 * RS_RADIX && lane == 31u) S.wsum[wid] = incl;
        __syncthreads();
        if (tid < 2 * RS_RADIX) {
            uint32_t base = incl - total;
            for (uint32_t w = wid & ~(RS_RADIX / 32u - 1u); w < wid; w++) base += S.wsum[w];
            (tid < RS_RADIX ? S.goff : S.loff)[d] = base + ahead;
            /* all n keys in one digit: those past the end stay behind them */
            if (tid < RS_RADIX && total - (d == mask ? all - n : 0u) == n) S.same[turn] = 1u;
        }
        __syncthreads();
        if (S.same[turn]) continue; /* the same decision in every CTA */
#pragma unroll
        for (int k = 0; k < ITEMS; k++) {
            const uint32_t dk = key[k] >> shift & mask;
            S.stage[S.loff[dk] + S.tile.whist[wid][dk] + rank[k]] = make_uint2(key[k], val[k]);
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < ITEMS; k++) {
            const uint32_t i = tid + (uint32_t)k * CS_THREADS;
            const uint2 kv = S.stage[i];
            const uint32_t dk = kv.x >> shift & mask, g = S.goff[dk] + (i - S.loff[dk]);
            *cl.map_shared_rank(&S.pair[g % TILE], (int)(g / TILE)) = kv;
        }
        cl.sync();
#pragma unroll
        for (int k = 0; k < ITEMS; k++) {
            const uint2 kv = S.pair[mine + 32u * k];
            key[k] = kv.x;
            val[k] = kv.y;
        }
    }
    /* every CTA has its input in registers since the first barrier (in place) */
#pragma unroll
    for (int k = 0; k < ITEMS; k++) {
        const uint32_t i = me * TILE + mine + 32u * k;
        if (i < n) {
            kout[i] = key[k];
            vout[i] = val[k];
        }
    }
    cl.sync(); /* no CTA leaves while another may read its totals */
}

template <int ITEMS>
static cudaError_t cluster_config(cudaLaunchConfig_t &cfg, cudaLaunchAttribute &at, uint32_t ctas, cudaStream_t st)
{
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(CS_THREADS);
    cfg.dynamicSmemBytes = sizeof(ClusterSort<ITEMS>);
    cfg.stream = st;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = ctas;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaError_t e = cudaFuncSetAttribute(k_sort_cluster<ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)cfg.dynamicSmemBytes);
    if (e != cudaSuccess || ctas <= 8u) return e;
    return cudaFuncSetAttribute(k_sort_cluster<ITEMS>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
}

/* CTAs of the largest cluster that the current device places: sixteen, or the
 * portable eight where no part of it has sixteen SMs together (a partition).
 * Asked once a device; two threads that ask at once get the same answer. */
uint32_t cluster_ctas()
{
    constexpr int kDevices = 32;
    static std::atomic<uint32_t> known[kDevices];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) return 8u;
    uint32_t ctas = known[dev].load(std::memory_order_relaxed);
    if (!ctas) {
        const bool clean = cudaPeekAtLastError() == cudaSuccess;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at[1];
        int active = 0;
        if (cluster_config<4>(cfg, at[0], CS_CTAS, 0) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&active, k_sort_cluster<4>, &cfg) != cudaSuccess)
            active = 0;
        if (!active && clean) cudaGetLastError(); /* the query's own error */
        ctas = active > 0 ? CS_CTAS : 8u;
        known[dev].store(ctas, std::memory_order_relaxed);
    }
    return ctas;
}

template <int ITEMS>
static cudaError_t cluster_sort(const uint32_t *kin, const uint32_t *vin, uint32_t *kout, uint32_t *vout, uint32_t n,
                                uint32_t bits, cudaStream_t st)
{
    uint32_t ctas = 1u;
    while (ctas * CS_THREADS * ITEMS < n) ctas <<= 1;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    const cudaError_t e = cluster_config<ITEMS>(cfg, at[0], ctas, st);
    if (e != cudaSuccess) return e;
    return cudaLaunchKernelEx(&cfg, k_sort_cluster<ITEMS>, kin, vin, kout, vout, n, bits);
}

/* As many CTAs as give each thread one pair, up to `most`, then more pairs. */
cudaError_t one_launch_sort(const uint32_t *kin, const uint32_t *vin, uint32_t *kout, uint32_t *vout, uint32_t n,
                            uint32_t bits, uint32_t most, cudaStream_t st)
{
    const uint32_t per = most * CS_THREADS;
    if (n <= per) return cluster_sort<1>(kin, vin, kout, vout, n, bits, st);
    if (n <= 2u * per) return cluster_sort<2>(kin, vin, kout, vout, n, bits, st);
    if (n <= 4u * per) return cluster_sort<4>(kin, vin, kout, vout, n, bits, st);
    return cluster_sort<8>(kin, vin, kout, vout, n, bits, st);
}

/* Pairs that one launch sorts.  The three kernels a pass, over the whole chip,
 * take 34.6 us for one pair more (17 bits; 32 bits: 44.2), where the cluster
 * takes 25.8 (35.2, and less with each digit it skips); with eight pairs a
 * thread it meets them at 98,304 pairs (34.6 and 34.6; 24 bits: 37.0 and 35.2). */
#define CS_MAX (CS_CTAS * CS_THREADS * 4u)

bool radix_one_launch(uint32_t n) { return n <= CS_MAX; }

uint32_t radix_launches(uint32_t n, uint32_t bits, uint32_t digit_bits)
{
    return radix_one_launch(n) ? 1u : 3u * (uint32_t)radix_passes(bits, digit_bits);
}

cudaError_t radix_sort(const uint32_t *keys_in, const uint32_t *vals_in, uint32_t *keys_out, uint32_t *vals_out,
                       uint32_t n, uint32_t bits, uint32_t digit_bits, const RadixScratch &s, cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    if (digit_bits < 1) digit_bits = 1;
    if (digit_bits > 8) digit_bits = 8;
    const int P = radix_passes(bits, digit_bits);
    if (P == 0) {
        if (keys_in != keys_out || vals_in != vals_out || !vals_in)
            k_iota_copy<<<grid_for((n + 255) / 256, 8), 256, 0, st>>>(keys_in, vals_in, keys_out, vals_out, n);
        return cudaSuccess;
    }
    if (radix_one_launch(n)) return one_launch_sort(keys_in, vals_in, keys_out, vals_out, n, bits, cluster_ctas(), st);
    const uint32_t T = (n + RS_TILE - 1) / RS_TILE;
    uint32_t *totals = s.hist + (size_t)RS_RADIX * T;
    /* the last pass lands in *_out: an odd number of passes starts towards it,
     * from the input or, in place, from a copy that the first upsweep leaves
     * in the scratch */
    const bool copy = P % 2 == 1 && keys_in == keys_out;
    const uint32_t *kin = keys_in;
    const uint32_t *vin = vals_in;
    bool to_out = P % 2 == 1;
    for (int p = 0; p < P; p++) {
        uint32_t shift = (uint32_t)p * digit_bits;
        uint32_t b = std::min(digit_bits, bits - shift);
        uint32_t mask = (1u << b) - 1u;
        uint32_t *ko = to_out ? keys_out : s.keys_alt;
        uint32_t *vo = to_out ? vals_out : s.vals_alt;
        const bool keep = copy && p == 0;
        k_rs_upsweep<<<T, RS_THREADS, 0, st>>>(kin, n, shift, mask, s.hist, T, vin, keep ? s.keys_alt : nullptr,
                                               keep ? s.vals_alt : nullptr);
        if (keep) {
            kin = s.keys_alt;
            vin = s.vals_alt;
        }
        k_rs_scan<<<RS_RADIX, RS_THREADS, 0, st>>>(s.hist, T, totals);
        k_rs_downsweep<<<T, RS_THREADS, 0, st>>>(kin, vin, ko, vo, n, shift, mask, s.hist, totals, T);
        kin = ko;
        vin = vo;
        to_out = !to_out;
    }
    return cudaSuccess;
}

/* ------------------------------------------- counting sort by bucket
 * Sort variant 2.  The keys are bucket indices below B (the world's total
 * buckets), so the sort counts instead of ranking digits:
 *   end[] zeroed, then k_bs_count (or k_hash, when the step hashes right
 *           before) adds every particle to end[key] (L2 atomics, one per run
 *           of equal keys in a warp) and keeps the count it found there as
 *           the particle's offset in its bucket;
 *   k_bs_tile_sums: the sum of each tile of BS_TILE counts;
 *   k_bs_offsets: per tile, the preceding tiles' sums plus the exclusive
 *           prefix inside the tile give P; start[k] = P[k] for an occupied
 *           bucket, FG_EMPTY for an empty one; end[k] = P[k] + count;
 *   k_bs_scatter: slot = start[key] + offset: keys_out[slot] = key,
 *           tmp[slot] = particle index (in arrival order inside a bucket);
 *   k_bs_rank: the stable order inside each bucket: particle e's rank is
 *           the number of smaller particle indices in its bucket (a bucket
 *           of L particles costs L loads per particle, as the density walk
 *           over that bucket does), vals_out[start + rank] = e;
 *           k_bs_rank_reorder also does the ranges pass's gathers there.
 * The result is the stable sort: (key, particle index) ascending, and the
 * cell ranges come with it. */
#define BS_THREADS 256
#define BS_ITEMS 8
#define BS_TILE (BS_THREADS * BS_ITEMS)
static_assert(BS_THREADS == RS_THREADS, "the tile scans use rs_block_excl");
#define BS_RANKS 2u /* particles that a thread of k_bs_rank_reorder has in flight */

__global__ void __launch_bounds__(256) k_bs_count(const uint32_t *__restrict__ keys, uint32_t n,
                                                 uint32_t *__restrict__ cnt, uint32_t *__restrict__ off)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t stride = gridDim.x * blockDim.x;
    /* warp-uniform loop: a warp's 32 indices are consecutive */
    for (uint32_t b0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); b0 < n; b0 += stride) {
        const uint32_t i = b0 + lane;
        const bool valid = i < n;
        const uint32_t o = bs_count_in(valid ? __ldg(keys + i) : 0u, valid, cnt);
        if (valid) off[i] = o;
    }
}

/* one CTA per tile: the sum of its BS_TILE counts (coalesced reads) */
__global__ void __launch_bounds__(BS_THREADS) k_bs_tile_sums(const uint32_t *__restrict__ cnt, uint32_t nb,
                                                            uint32_t *__restrict__ tsum)
{
    __shared__ uint32_t s_warp[RS_WARPS + 1];
    const size_t base = (size_t)blockIdx.x * BS_TILE;
    uint32_t v = 0;
#pragma unroll
    for (int k = 0; k < BS_ITEMS; k++) {
        const size_t i = base + (size_t)k * BS_THREADS + threadIdx.x;
        if (i < nb) v += __ldg(cnt + i);
    }
    uint32_t tot;
    rs_block_excl(v, s_warp, tot);
    if (threadIdx.x == 0) tsum[blockIdx.x] = tot;
}

/* one CTA per tile: the tile's base (the preceding tiles' sums), then the
 * exclusive prefix of its counts in order, staged through shared memory so
 * that every global read and write is coalesced */
__global__ void __launch_bounds__(BS_THREADS) k_bs_offsets(uint32_t *__restrict__ cnt_end, uint32_t nb,
                                                          const uint32_t *__restrict__ tsum,
                                                          uint32_t *__restrict__ start)
{
    __shared__ uint32_t s_c[BS_TILE];
    __shared__ uint32_t s_warp[RS_WARPS + 1];
    const size_t base = (size_t)blockIdx.x * BS_TILE;
    /* the tile's base: the sum of all earlier tiles */
    uint32_t pre = 0;
    for (uint32_t t = threadIdx.x; t < blockIdx.x; t += BS_THREADS) pre += __ldg(tsum + t);
    uint32_t tbase;
    rs_block_excl(pre, s_warp, tbase);
#pragma unroll
    for (int k = 0; k < BS_ITEMS; k++) {
        const size_t i = base + (size_t)k * BS_THREADS + threadIdx.x;
        s_c[k * BS_THREADS + threadIdx.x] = i < nb ? cnt_end[i] : 0u;
    }
    __syncthreads();
    /* thread t scans items t*BS_ITEMS .. +BS_ITEMS of the tile */
    uint32_t c[BS_ITEMS], v = 0;
#pragma unroll
    for (int k = 0; k < BS_ITEMS; k++) {
        c[k] = s_c[threadIdx.x * BS_ITEMS + k];
        v += c[k];
    }
    uint32_t tot;
    uint32_t p = rs_block_excl(v, s_warp, tot) + tbase;
#pragma unroll
    for (int k = 0; k < BS_ITEMS; k++) {
        s_c[threadIdx.x * BS_ITEMS + k] = p; /* the bucket's first index */
        p += c[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BS_ITEMS; k++) {
        const size_t i = base + (size_t)k * BS_THREADS + threadIdx.x;
        if (i < nb) {
            const uint32_t first = s_c[k * BS_THREADS + threadIdx.x];
            const uint32_t count = cnt_end[i];
            start[i] = count ? first : FG_EMPTY;
            cnt_end[i] = first + count;
        }
    }
}

__global__ void __launch_bounds__(256) k_bs_scatter(const uint32_t *__restrict__ keys,
                                                   const uint32_t *__restrict__ off, uint32_t n,
                                                   const uint32_t *__restrict__ start,
                                                   uint32_t *__restrict__ keys_out, uint32_t *__restrict__ tmp)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t k = __ldg(keys + i);
        const uint32_t slot = __ldg(start + k) + __ldg(off + i);
        keys_out[slot] = k;
        tmp[slot] = i;
    }
}

__global__ void __launch_bounds__(256) k_bs_rank(const uint32_t *__restrict__ keys_out,
                                                const uint32_t *__restrict__ tmp, uint32_t n,
                                                const uint32_t *__restrict__ start, const uint32_t *__restrict__ end,
                                                uint32_t *__restrict__ vals_out)
{
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
        const uint32_t k = __ldg(keys_out + s);
        const uint32_t st = __ldg(start + k), en = __ldg(end + k);
        const uint32_t e = __ldg(tmp + s);
        uint32_t r = 0;
        for (uint32_t f = st; f < en; f++) r += __ldg(tmp + f) < e ? 1u : 0u;
        vals_out[st + r] = e;
    }
}

/* k_bs_rank and the ranges pass's reorder in one: the particle's sorted
 * index p = start + rank gets its id, position and velocity, inv[id] = p,
 * and a rank-0 particle appends its bucket's first index to runs (in no
 * particular order, as the ranges pass does).  Bound by the gathers' sectors
 * and by a chain of four loads a particle: two particles a thread at a time
 * take 123 us where one took 133 (4M; four: 118 there, no better at 1M). */
__global__ void __launch_bounds__(256) k_bs_rank_reorder(const uint32_t *__restrict__ keys_out,
                                                        const uint32_t *__restrict__ tmp, uint32_t n,
                                                        const uint32_t *__restrict__ start,
                                                        const uint32_t *__restrict__ end,
                                                        uint32_t *__restrict__ vals_out, BucketReorder R)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t b0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); b0 < n; b0 += BS_RANKS * stride) {
        uint32_t st[BS_RANKS], en[BS_RANKS], e[BS_RANKS], r[BS_RANKS];
#pragma unroll
        for (uint32_t u = 0; u < BS_RANKS; u++) {
            const uint32_t s = b0 + u * stride + lane;
            st[u] = s < n ? __ldg(keys_out + s) : 0u;
            e[u] = s < n ? __ldg(tmp + s) : 0u;
        }
#pragma unroll
        for (uint32_t u = 0; u < BS_RANKS; u++) {
            const uint32_t k = st[u];
            st[u] = en[u] = r[u] = 0u;
            if (b0 + u * stride + lane < n) {
                st[u] = __ldg(start + k);
                en[u] = __ldg(end + k);
            }
        }
#pragma unroll
        for (uint32_t u = 0; u < BS_RANKS; u++)
            for (uint32_t f = st[u]; f < en[u]; f++) r[u] += __ldg(tmp + f) < e[u] ? 1u : 0u;
        float4 x[BS_RANKS], v[BS_RANKS];
#pragma unroll
        for (uint32_t u = 0; u < BS_RANKS; u++)
            if (b0 + u * stride + lane < n) {
                x[u] = __ldg(R.pos + e[u]);
                if (R.vel) v[u] = __ldg(R.vel + e[u]);
            }
#pragma unroll
        for (uint32_t u = 0; u < BS_RANKS; u++) {
            if (b0 + u * stride + lane < n) {
                const uint32_t p = st[u] + r[u];
                vals_out[p] = e[u];
                R.spos[p] = x[u];
                if (R.vel) R.svel[p] = v[u];
                if (R.inv) R.inv[e[u]] = p;
            }
        }
        if (R.runs) {
#pragma unroll
            for (uint32_t u = 0; u < BS_RANKS; u++) {
                const bool head = b0 + u * stride + lane < n && r[u] == 0u;
                const uint32_t m = __ballot_sync(0xffffffffu, head);
                uint32_t base = 0;
                if (lane == 0 && m) base = atomicAdd(R.nruns, (uint32_t)__popc(m));
                base = __shfl_sync(0xffffffffu, base, 0);
                if (head) R.runs[base + __popc(m & ((1u << lane) - 1u))] = st[u];
            }
        }
    }
}

bool bucket_sort(const uint32_t *keys_in, uint32_t *keys_out, uint32_t *vals_out, uint32_t n, uint32_t nbuckets,
                 uint32_t *start, uint32_t *end, const RadixScratch &s, uint32_t scratch_words, cudaStream_t st,
                 const BucketReorder *reorder, bool counted)
{
    const uint32_t T = (nbuckets + BS_TILE - 1) / BS_TILE;
    if (!nbuckets || (size_t)T > scratch_words) return false; /* the tile sums would not fit */
    const uint32_t g = grid_for((n + 255) / 256, 8);
    if (!counted) {
        cudaMemsetAsync(end, 0, sizeof(uint32_t) * (size_t)nbuckets, st);
        if (n) k_bs_count<<<g, 256, 0, st>>>(keys_in, n, end, s.keys_alt);
    }
    k_bs_tile_sums<<<T, BS_THREADS, 0, st>>>(end, nbuckets, s.hist);
    k_bs_offsets<<<T, BS_THREADS, 0, st>>>(end, nbuckets, s.hist, start);
    if (n) {
        k_bs_scatter<<<g, 256, 0, st>>>(keys_in, s.keys_alt, n, start, keys_out, s.vals_alt);
        if (reorder)
            k_bs_rank_reorder<<<g, 256, 0, st>>>(keys_out, s.vals_alt, n, start, end, vals_out, *reorder);
        else
            k_bs_rank<<<g, 256, 0, st>>>(keys_out, s.vals_alt, n, start, end, vals_out);
    }
    return true;
}

/* ---------------------------------------------------------- onesweep
 * Stable LSD radix sort with one kernel per digit pass, after one histogram
 * kernel for all passes (decoupled look-back):
 *   k_os_hist  global digit counts of every pass (one read of the keys)
 *   k_os_scan  exclusive digit bases of every pass
 *   k_os_pass  per tile of RS_TILE keys, taken in launch order through a
 *              counter: rank the keys in the tile exactly as k_rs_downsweep
 *              does, publish the tile's per-digit counts, add up the
 *              preceding tiles' counts by looking back until a tile whose
 *              inclusive prefix is known, publish this tile's inclusive
 *              prefix, scatter.
 * A tile waits only on tiles taken before it, which publish their counts
 * before they wait themselves, so every wait ends; each wait is bounded all
 * the same, and one that gives up sets FG_DEV_SORT_TIMEOUT and goes on. */
#define OS_MAX_PASSES 6
#define OS_AGG 0x40000000u
#define OS_INC 0x80000000u
#define OS_CNT 0x3fffffffu
#define OS_SPIN_LIMIT (1u << 22)
#define OS_WINDOW 8

static uint32_t os_tiles(uint32_t n) { return std::max<uint32_t>((n + RS_TILE - 1) / RS_TILE, 1u); }

size_t onesweep_words(uint32_t n)
{
    /* status words [pass][tile][digit], digit counts/bases [pass][digit], tile counters */
    return (size_t)OS_MAX_PASSES * RS_RADIX * os_tiles(n) + (size_t)OS_MAX_PASSES * RS_RADIX + 32;
}

__global__ void __launch_bounds__(RS_THREADS) k_os_hist(const uint32_t *__restrict__ keys, uint32_t n,
                                                       uint32_t bits, uint32_t db, uint32_t passes,
                                                       uint32_t *__restrict__ counts)
{
    __shared__ uint32_t h[OS_MAX_PASSES][RS_RADIX];
#pragma unroll
    for (int p = 0; p < OS_MAX_PASSES; p++) h[p][threadIdx.x] = 0;
    __syncthreads();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t k = __ldg(keys + i);
        for (uint32_t p = 0; p < passes; p++) {
            const uint32_t shift = p * db, b = min(db, bits - shift);
            atomicAdd(&h[p][(k >> shift) & ((1u << b) - 1u)], 1u);
        }
    }
    __syncthreads();
    for (uint32_t p = 0; p < passes; p++) {
        const uint32_t v = h[p][threadIdx.x];
        if (v) atomicAdd(&counts[p * RS_RADIX + threadIdx.x], v);
    }
}

/* one CTA per pass: counts -> exclusive digit bases, in place */
__global__ void __launch_bounds__(RS_THREADS) k_os_scan(uint32_t *__restrict__ counts)
{
    __shared__ uint32_t s_warp[RS_WARPS + 1];
    uint32_t *c = counts + blockIdx.x * RS_RADIX;
    uint32_t tot;
    const uint32_t e = rs_block_excl(c[threadIdx.x], s_warp, tot);
    c[threadIdx.x] = e;
}

__global__ void __launch_bounds__(RS_THREADS) k_os_pass(const uint32_t *__restrict__ kin,
                                                       const uint32_t *__restrict__ vin,
                                                       uint32_t *__restrict__ kout, uint32_t *__restrict__ vout,
                                                       uint32_t n, uint32_t shift, uint32_t mask,
                                                       uint32_t *__restrict__ status,
                                                       const uint32_t *__restrict__ bases,
                                                       uint32_t *__restrict__ tile_ctr, uint32_t *__restrict__ err,
                                                       uint32_t spin_limit)
{
    __shared__ uint32_t s_keys[RS_TILE];
    __shared__ uint32_t s_vals[RS_TILE];
    __shared__ uint32_t s_whist[RS_WARPS][RS_RADIX];
    __shared__ uint32_t s_goff[RS_RADIX];
    __shared__ uint32_t s_tstart[RS_RADIX];
    __shared__ uint32_t s_warp[RS_WARPS + 1];
    __shared__ uint32_t s_tile;

    const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (tid == 0) s_tile = atomicAdd(tile_ctr, 1u);
#pragma unroll
    for (int w = 0; w < RS_WARPS; w++) s_whist[w][tid] = 0;
    __syncthreads();
    const uint32_t tile = s_tile;
    const size_t base = (size_t)tile * RS_TILE;

    uint32_t key[RS_ITEMS], val[RS_ITEMS], rank[RS_ITEMS];
    const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
    for (int k = 0; k < RS_ITEMS; k++) {
        const size_t i = base + (size_t)wid * (32 * RS_ITEMS) + (size_t)k * 32 + lane;
        key[k] = i < n ? __ldg(kin + i) : 0xffffffffu;
        val[k] = i < n ? (vin ? __ldg(vin + i) : (uint32_t)i) : 0u;
    }
#pragma unroll
    for (int k = 0; k < RS_ITEMS; k++) {
        const bool valid = base + (size_t)wid * (32 * RS_ITEMS) + (size_t)k * 32 + lane < n;
        const uint32_t d = (key[k] >> shift) & mask;
        /* not a ballot a bit, as k_rs_downsweep: this pass is bound by issue
         * beside its look-back (1M particles of a lattice, three passes: 65 us
         * so, 51.5 with match_any; random ones 66 and 60) */
        const uint32_t peers = __match_any_sync(0xffffffffu, valid ? d : 0xffffffffu);
        const uint32_t leader = valid ? (uint32_t)__ffs((int)peers) - 1u : lane;
        uint32_t b = 0;
        if (valid && lane == leader) {
            b = s_whist[wid][d];
            s_whist[wid][d] = b + __popc(peers);
        }
        b = __shfl_sync(0xffffffffu, b, (int)leader);
        rank[k] = b + __popc(peers & lt);
        __syncwarp();
    }
    __syncthreads();
    /* per digit: exclusive over warps, tile count */
    uint32_t run = 0;
#pragma unroll
    for (int w = 0; w < RS_WARPS; w++) {
        uint32_t c = s_whist[w][tid];
        s_whist[w][tid] = run;
        run += c;
    }
    /* publish this tile's count of digit tid, then look back */
    uint32_t *mine = status + (size_t)tile * RS_RADIX + tid;
    uint32_t excl = 0;
    if (tile == 0) {
        atomicExch(mine, OS_INC | run);
    } else {
        atomicExch(mine, OS_AGG | run);
        /* look back OS_WINDOW tiles per round trip: add aggregates from the
         * nearest tile outwards until an inclusive prefix; a tile that has
         * not published yet ends the round, which resumes there */
        int k = (int)tile - 1;
        uint32_t spins = 0;
        bool found = false;
        while (!found) {
            uint32_t v[OS_WINDOW];
#pragma unroll
            for (int q = 0; q < OS_WINDOW; q++)
                v[q] = (k - q >= 0) ? *(volatile const uint32_t *)(status + (size_t)(k - q) * RS_RADIX + tid)
                                    : OS_INC; /* before tile 0: an empty inclusive prefix */
            int used = 0;
            bool stalled = false;
#pragma unroll
            for (int q = 0; q < OS_WINDOW; q++) {
                if (found || stalled) continue;
                if (v[q] & OS_INC) {
                    excl += v[q] & OS_CNT;
                    found = true;
                } else if (v[q] & OS_AGG) {
                    excl += v[q] & OS_CNT;
                    used++;
                } else {
                    stalled = true;
                }
            }
            k -= used;
            if (stalled && ++spins > spin_limit) {
                atomicOr(err, FG_DEV_SORT_TIMEOUT);
                break;
            }
        }
        atomicExch(mine, OS_INC | (excl + run));
    }
    s_goff[tid] = __ldg(bases + tid) + excl;
    {
        uint32_t tot;
        s_tstart[tid] = rs_block_excl(run, s_warp, tot);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < RS_ITEMS; k++) {
        size_t i = base + (size_t)wid * (32 * RS_ITEMS) + (size_t)k * 32 + lane;
        if (i < n) {
            uint32_t d = (key[k] >> shift) & mask;
            uint32_t p = s_tstart[d] + s_whist[wid][d] + rank[k];
            s_keys[p] = key[k];
            s_vals[p] = val[k];
        }
    }
    __syncthreads();
    const uint32_t tile_n = (n - base) < (size_t)RS_TILE ? (uint32_t)(n - base) : (uint32_t)RS_TILE;
    for (uint32_t i = tid; i < tile_n; i += RS_THREADS) {
        uint32_t kk = s_keys[i];
        uint32_t d = (kk >> shift) & mask;
        uint32_t g = s_goff[d] + (i - s_tstart[d]);
        if (g < n) { /* only a wait that gave up leaves g unchecked */
            kout[g] = kk;
            vout[g] = s_vals[i];
        }
    }
}

bool onesweep_sort(const uint32_t *keys_in, uint32_t *keys_out, uint32_t *vals_out, uint32_t n, uint32_t bits,
                   uint32_t digit_bits, const RadixScratch &s, uint32_t *os, uint32_t *err, cudaStream_t st)
{
    if (digit_bits < 1) digit_bits = 1;
    if (digit_bits > 8) digit_bits = 8;
    const int P = radix_passes(bits, digit_bits);
    if (P < 1 || P > OS_MAX_PASSES || n == 0 || keys_in == keys_out) return false;
    const uint32_t T = os_tiles(n);
    uint32_t *status = os;                                        /* [P][T][256] */
    uint32_t *counts = os + (size_t)OS_MAX_PASSES * RS_RADIX * T; /* [P][256] */
    uint32_t *ctr = counts + (size_t)OS_MAX_PASSES * RS_RADIX;    /* [P] */
    cudaMemsetAsync(status, 0, 4 * ((size_t)P * RS_RADIX * T), st);
    cudaMemsetAsync(counts, 0, 4 * ((size_t)OS_MAX_PASSES * RS_RADIX + 32), st);
    k_os_hist<<<grid_for((n + RS_THREADS - 1) / RS_THREADS, 4), RS_THREADS, 0, st>>>(keys_in, n, bits, digit_bits,
                                                                                     (uint32_t)P, counts);
    k_os_scan<<<P, RS_THREADS, 0, st>>>(counts);
    const uint32_t *kin = keys_in;
    const uint32_t *vin = nullptr;
    bool to_out = (P % 2 == 1);
    for (int p = 0; p < P; p++) {
        const uint32_t shift = (uint32_t)p * digit_bits;
        const uint32_t b = std::min(digit_bits, bits - shift);
        const uint32_t mask = (1u << b) - 1u;
        uint32_t *ko = to_out ? keys_out : s.keys_alt;
        uint32_t *vo = to_out ? vals_out : s.vals_alt;
        k_os_pass<<<T, RS_THREADS, 0, st>>>(kin, vin, ko, vo, n, shift, mask, status + (size_t)p * RS_RADIX * T,
                                            counts + (size_t)p * RS_RADIX, ctr + p, err, OS_SPIN_LIMIT);
        kin = ko;
        vin = vo;
        to_out = !to_out;
    }
    return true;
}

/* Self-test of the look-back's bounded wait: one CTA takes tile 1 of a
 * two-tile sort whose tile 0 never publishes, waits spin_limit rounds, sets
 * FG_DEV_SORT_TIMEOUT and returns; every access stays inside the buffers
 * (the scatter skips the positions a wait that gave up leaves unchecked). */
int bounded_wait_selftest(uint32_t spin_limit, uint32_t *flags)
{
    const uint32_t n = 2 * RS_TILE;
    uint32_t *buf = nullptr;
    const size_t words = 3 * (size_t)n + 2 * RS_RADIX + RS_RADIX + 2;
    if (cudaMalloc(&buf, 4 * words) != cudaSuccess) return -1;
    uint32_t *keys = buf, *kout = buf + n, *vout = buf + 2 * n;
    uint32_t *status = buf + 3 * (size_t)n, *bases = status + 2 * RS_RADIX, *ctr = bases + RS_RADIX, *err = ctr + 1;
    cudaMemset(buf, 0, 4 * words);
    const uint32_t one = 1; /* the only CTA takes tile 1 */
    cudaMemcpy(ctr, &one, 4, cudaMemcpyHostToDevice);
    k_os_pass<<<1, RS_THREADS>>>(keys, nullptr, kout, vout, n, 0, 0xffu, status, bases, ctr, err, spin_limit);
    cudaError_t e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpy(flags, err, 4, cudaMemcpyDeviceToHost);
    cudaFree(buf);
    return e == cudaSuccess ? 0 : -1;
}

/* ------------------------------------------------------ ranges + reorder
 * FindCellOffsetOrderinPosVelK / FindCellOffsetOrderingPosK
 * (K_HashGrid.cu:70-197): start[key] at the first index of each key run,
 * end[previous key] = that index, end[last key] = n; sorted gather of
 * position (and velocity). */
__global__ void __launch_bounds__(256) k_cell_ranges(const uint32_t *__restrict__ keys,
                                                    const uint32_t *__restrict__ ids,
                                                    const float4 *__restrict__ pos, const float4 *__restrict__ vel,
                                                    uint32_t *__restrict__ start, uint32_t *__restrict__ end,
                                                    float4 *__restrict__ spos, float4 *__restrict__ svel, uint32_t n,
                                                    uint32_t *__restrict__ inv, uint32_t *__restrict__ runs,
                                                    uint32_t *__restrict__ nruns)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t k = __ldg(keys + i);
        uint32_t prev = i > 0 ? __ldg(keys + i - 1) : k;
        const bool head = (i == 0 || k != prev);
        if (head) {
            start[k] = i;
            if (i > 0) end[prev] = i;
        }
        if (runs) {
            /* append run heads, one atomic per warp */
            const uint32_t act = __activemask();
            const uint32_t m = __ballot_sync(act, head);
            const int lane = threadIdx.x & 31;
            const int leader = __ffs(act) - 1;
            uint32_t base = 0;
            if (lane == leader && m) base = atomicAdd(nruns, (uint32_t)__popc(m));
            base = __shfl_sync(act, base, leader);
            if (head) runs[base + __popc(m & ((1u << lane) - 1u))] = i;
        }
        if (i == n - 1) end[k] = n;
        uint32_t id = __ldg(ids + i);
        spos[i] = __ldg(pos + id);
        if (vel) svel[i] = __ldg(vel + id);
        if (inv) inv[id] = i; /* particle -> sorted index */
    }
}

void launch_cell_ranges(const uint32_t *keys, const uint32_t *ids, const float4 *pos, const float4 *vel,
                        uint32_t *start, uint32_t *end, float4 *spos, float4 *svel, uint32_t n, cudaStream_t st,
                        uint32_t *inv, uint32_t *runs, uint32_t *nruns)
{
    if (!n) return;
    k_cell_ranges<<<grid_for((n + 255) / 256, 32), 256, 0, st>>>(keys, ids, pos, vel, start, end, spos, svel, n,
                                                                inv, runs, nruns);
}

/* ------------------------------------------------ spatial target order
 * The force kernels process their targets in a spatially coherent order so
 * that a CTA's particles share listed neighbours and their loads hit L1 (the
 * hashed bucket order scatters a CTA over random cells); the density pass
 * stages by cell, in bucket order.  The key is the scene id above a Morton
 * code of the particle's cell, counted from that of the scene's volume_min and
 * clamped to 2^bits cells per axis; a particle outside that range only loses
 * locality, never correctness. */
__device__ __forceinline__ uint32_t fg_spread3(uint32_t v)
{
    v &= 0x3ffu;
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

__global__ void __launch_bounds__(FG_CHUNK) k_morton_keys(const FgWork *__restrict__ work, uint32_t nwork,
                                                         uint32_t n_single, const FgScene *__restrict__ table,
                                                         const __grid_constant__ FgScene single,
                                                         const float4 *__restrict__ pos, uint32_t *__restrict__ keys,
                                                         uint32_t bits, uint32_t scene_shift)
{
    const int lim = (1 << bits) - 1;
    for (uint32_t w = blockIdx.x; w < nwork; w += gridDim.x) {
        FgWork it = fg_work(work, w, n_single);
        if (threadIdx.x >= it.count) continue;
        const FgScene *S = fg_scene(table, &single, it.scene);
        const uint32_t t = it.first + threadIdx.x;
        const float4 p = __ldg(pos + t);
        int c[3];
        const float q[3] = {p.x, p.y, p.z};
#pragma unroll
        for (int a = 0; a < 3; a++) {
            /* the hash grid's own cell index (relative to the scene's lower
             * corner): a Morton cell is exactly one hashed cell, so a run of
             * targets shares its 27 buckets as in bucket order */
            const int v = fg_axis_index(q[a], S->cell[a]) - fg_axis_index(S->vmin[a], S->cell[a]) + 2;
            c[a] = v < 0 ? 0 : (v > lim ? lim : v);
        }
        const uint32_t m = (fg_spread3((uint32_t)c[0]) | (fg_spread3((uint32_t)c[1]) << 1) |
                            (fg_spread3((uint32_t)c[2]) << 2));
        keys[t] = (scene_shift < 32 ? (it.scene << scene_shift) : 0u) | m;
    }
}

void launch_morton_keys(const Launch &L, const float4 *pos, uint32_t *keys, uint32_t bits, uint32_t scene_shift)
{
    if (!L.nwork) return;
    k_morton_keys<<<grid_for(L.nwork, 16), FG_CHUNK, 0, L.stream>>>(L.work, L.nwork, L.n, L.table, *L.single, pos,
                                                                    keys, bits, scene_shift);
}

/* ------------------------------------------ rigid-sphere grid per scene
 * The sort + start/end of FindCellOffsetOrderingPosK (K_HashGrid.cu:140-197)
 * for the rigid-sphere grid, in one CTA per scene when every scene has at
 * most FG_RB_SCENE_MAX spheres: a stable radix sort of the scene's (key,
 * index) pairs in shared memory, four a thread, 8 bits a pass, so keys, ids
 * and ranges equal the general path's bit for bit.  A scene's spheres and rigid
 * buckets are its own ranges of the global arrays, and the global stable order
 * is the scenes' orders one after another (keys carry the scene's rigid bucket
 * base, which the sort leaves out: two or three passes).  Bound by the
 * latency of one CTA's barriers; a bitonic network of 64-bit words in its
 * place took 78 rounds of them for 4,096 spheres, 55 us, longer than the fluid
 * sort it runs beside (1M particles with one such body: 541 -> 519 us a step). */
#define RB_ITEMS 4
static_assert(FG_RB_SCENE_MAX <= CS_THREADS * RB_ITEMS, "a scene's spheres are one CTA's tile");

__global__ void __launch_bounds__(CS_THREADS) k_rb_sort_ranges(const FgScene *__restrict__ table,
                                                              const __grid_constant__ FgScene single,
                                                              const uint32_t *__restrict__ keys_u,
                                                              const float4 *__restrict__ world,
                                                              uint32_t *__restrict__ keys, uint32_t *__restrict__ ids,
                                                              float4 *__restrict__ spos, uint32_t *__restrict__ rstart,
                                                              uint32_t *__restrict__ rend)
{
    __shared__ TileRank R;
    __shared__ uint32_t s_key[CS_THREADS * RB_ITEMS];
    __shared__ uint16_t s_val[CS_THREADS * RB_ITEMS];
    __shared__ uint32_t s_off[RS_RADIX], s_wsum[RS_RADIX / 32];
    const FgScene *S = table ? table + blockIdx.x : &single;
    const uint32_t n = S->nsph, base = S->sph_base, bucket0 = S->rb_bucket_base, nb = S->rb_nb;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, wid = tid >> 5;
    if (!(S->flags & FG_SCENE_HAS_RB)) return; /* the scene has no rigid buckets */
    const uint32_t mine = wid * 32u * RB_ITEMS + lane;
    uint32_t key[RB_ITEMS], val[RB_ITEMS], rank[RB_ITEMS];
#pragma unroll
    for (int k = 0; k < RB_ITEMS; k++) {
        val[k] = mine + 32u * k;
        key[k] = val[k] < n ? __ldg(keys_u + base + val[k]) - bucket0 : 0xffffffffu; /* the largest, and last */
    }
    for (uint32_t b = tid; b < nb; b += CS_THREADS) rstart[bucket0 + b] = FG_EMPTY;
    if (!n) return;
    const bool idle = wid * 32u * RB_ITEMS >= n;
    const uint32_t bits = nb > 1u ? 32u - (uint32_t)__clz((int)(nb - 1u)) : 1u;
    for (uint32_t shift = 0u; shift < bits; shift += 8u) {
        const uint32_t db = min(8u, bits - shift), mask = (1u << db) - 1u;
        const uint32_t count = rs_tile_rank<RB_ITEMS>(R, key, rank, shift, db, idle);
        uint32_t incl = count;
        if (tid >= CS_THREADS - RS_RADIX) {
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= (uint32_t)o) incl += y;
            }
            if (lane == 31u) s_wsum[wid & 7u] = incl;
        }
        __syncthreads();
        if (tid >= CS_THREADS - RS_RADIX) {
            uint32_t first = incl - count;
            for (uint32_t w = 0; w < (wid & 7u); w++) first += s_wsum[w];
            s_off[tid & 255u] = first;
        }
        __syncthreads();
        if (!idle) {
#pragma unroll
            for (int k = 0; k < RB_ITEMS; k++) {
                const uint32_t d = key[k] >> shift & mask, to = s_off[d] + R.whist[wid][d] + rank[k];
                s_key[to] = key[k];
                s_val[to] = (uint16_t)val[k];
            }
        }
        __syncthreads();
        if (!idle) {
#pragma unroll
            for (int k = 0; k < RB_ITEMS; k++) {
                key[k] = s_key[mine + 32u * k];
                val[k] = s_val[mine + 32u * k];
            }
        }
    }
    for (uint32_t i = tid; i < n; i += CS_THREADS) {
        const uint32_t k = bucket0 + s_key[i], id = base + s_val[i];
        keys[base + i] = k;
        ids[base + i] = id;
        spos[base + i] = __ldg(world + id);
        const uint32_t prev = i ? bucket0 + s_key[i - 1] : k;
        if (i == 0 || k != prev) {
            rstart[k] = base + i;
            if (i) rend[prev] = base + i;
        }
        if (i == n - 1) rend[k] = base + n;
    }
}

void launch_rb_sort_ranges(const FgScene *table, const FgScene *single, uint32_t nscenes, const uint32_t *keys_u,
                           const float4 *world, uint32_t *keys, uint32_t *ids, float4 *spos, uint32_t *rstart,
                           uint32_t *rend, cudaStream_t s)
{
    if (!nscenes) return;
    k_rb_sort_ranges<<<nscenes, CS_THREADS, 0, s>>>(table, *single, keys_u, world, keys, ids, spos, rstart, rend);
}

__global__ void k_fill(uint32_t *buf, size_t words, uint32_t v)
{
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < words; i += (size_t)gridDim.x * blockDim.x)
        buf[i] = v;
}

void launch_fill(uint32_t *buf, size_t words, uint32_t v, cudaStream_t s)
{
    if (!words) return;
    k_fill<<<grid_for((uint32_t)std::min<size_t>((words + 255) / 256, 1u << 30), 8), 256, 0, s>>>(buf, words, v);
}

} // namespace fg
