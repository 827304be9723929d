/* Neighbour candidates of a warp's 32 consecutive sorted targets, staged in
 * shared memory.
 *
 * Particles of one cell share their 27 candidate buckets, and in sorted order
 * they stand together, so a warp's targets fall into a few groups.  Per group
 * the warp looks the 27 buckets up once (a lane each), lays their particles
 * end to end in visit order (z outer, x inner, ascending inside a bucket), and
 * keeps those within h of the box around the group's targets: 40-60% of them
 * (eight particles of a cell span about 0.55 h, not h).  Then every target, a
 * lane each, runs over its group's staged candidates: one flat loop with the
 * lanes of a group in step (a broadcast load each), where a walk by thread
 * has 27 short bucket loops over twice the candidates.
 *
 * The box test drops no in-range candidate, bit for bit: lo <= p <= hi per
 * axis (scaled target coordinates), every operation of the squared distance
 * is monotonic under rounding, and the box distance is evaluated by the same
 * operations on |dx|, |dy|, |dz| that are no larger. */
#ifndef FG_STAGE_CUH
#define FG_STAGE_CUH

#include "fg_device.cuh"

namespace fg {

#define FG_FULL 0xffffffffu

/* The scene's grid, in registers (a barrier has the compiler read memory
 * again, and the scene table is memory). */
struct StageGrid {
    float cell[3], scale, h2;
    uint32_t nb, mask, base;
    __device__ __forceinline__ explicit StageGrid(const FgScene *S)
        : scale(S->scale), h2(S->h2), nb(S->nb), mask(S->nb_mask), base(S->bucket_base)
    {
        cell[0] = S->cell[0];
        cell[1] = S->cell[1];
        cell[2] = S->cell[2];
    }
};

/* A target's cell and how its neighbour cells' indices differ from it (two
 * bits for each of the six; one in all but a few per cent, where p + 5000 and
 * p - cell + 5000 round apart).  Equal signatures mean the same 27 buckets. */
struct StageSig {
    int ix, iy, iz;
    uint32_t d;
    bool odd; /* a difference outside 0..3: the walk by thread handles it */
};

__device__ __forceinline__ StageSig fg_stage_sig(float4 p, const StageGrid &G)
{
    StageSig s;
    const float q[3] = {p.x, p.y, p.z};
    int c[3];
    s.d = 0u;
    s.odd = false;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        c[a] = fg_axis_index(q[a], G.cell[a]);
        const uint32_t m = (uint32_t)c[a] - (uint32_t)fg_axis_index_off(q[a], G.cell[a], -1);
        const uint32_t n = (uint32_t)fg_axis_index_off(q[a], G.cell[a], 1) - (uint32_t)c[a];
        s.odd |= (m | n) > 3u;
        s.d |= (m << (4 * a)) | (n << (4 * a + 2));
    }
    s.ix = c[0];
    s.iy = c[1];
    s.iz = c[2];
    return s;
}

/* The lane of the first target with the same signature, for each lane of
 * `todo` (whole warp, converged). */
__device__ __forceinline__ void fg_stage_groups(const StageSig &s, uint32_t todo, uint32_t &lead, uint32_t &leads)
{
    const uint32_t lane = threadIdx.x & 31u;
    leads = 0u;
    lead = 32u;
    while (todo) {
        const int l = __ffs(todo) - 1;
        const int ix = __shfl_sync(FG_FULL, s.ix, l), iy = __shfl_sync(FG_FULL, s.iy, l),
                  iz = __shfl_sync(FG_FULL, s.iz, l);
        const uint32_t d = __shfl_sync(FG_FULL, s.d, l);
        const bool same = (todo >> lane & 1u) && s.ix == ix && s.iy == iy && s.iz == iz && s.d == d;
        if (same) lead = (uint32_t)l;
        todo &= ~__ballot_sync(FG_FULL, same);
        leads |= 1u << l;
    }
}

/* minimum / maximum over the warp, NaN ignored */
__device__ __forceinline__ float fg_redux_min(float v)
{
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float fg_redux_max(float v)
{
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

#define FG_STAGE_WINDOW 256u /* candidate positions expanded at a time */
#define FG_STAGE_FLIGHT 4u   /* chunks of 32 candidates whose loads are in flight together */

struct StageCell {
    int x, y, z;
    bool active;
};
__device__ __forceinline__ StageCell fg_stage_cell(float4 p, const StageGrid &G)
{
    StageCell c = {fg_axis_index(p.x, G.cell[0]), fg_axis_index(p.y, G.cell[1]), fg_axis_index(p.z, G.cell[2]),
                   p.w > 0.0f};
    return c;
}

/* Buckets of a range of len targets, a lane each (past the scene's end its last
 * one's); cells of a shorter one where a bucket takes a modulo.  Buckets, not
 * cells: where many cells share a bucket, the candidates are many too. */
__device__ __forceinline__ uint32_t fg_stage_buckets(const StageCell &c, const StageGrid &G, uint32_t len)
{
    uint32_t b = (uint32_t)c.x * FG_PX ^ (uint32_t)c.y * FG_PY ^ (uint32_t)c.z * FG_PZ;
    if (G.mask) b &= G.mask;
    else if (len == 32u) b %= G.nb;
    const uint32_t lane = threadIdx.x & 31u, before = __shfl_up_sync(FG_FULL, b, 1);
    return (uint32_t)__popc(__ballot_sync(FG_FULL, lane < len && (lane == 0u || b != before)));
}

/* Whether its active targets are more than `most` and its buckets too: a
 * function of the range alone, so that two kernels that share the ranges agree
 * on it. */
__device__ __forceinline__ bool fg_stage_dispersed(const StageCell &c, const StageGrid &G, uint32_t len, uint32_t most)
{
    const uint32_t lane = threadIdx.x & 31u;
    return most < 32u && fg_stage_buckets(c, G, len) > most &&
           (uint32_t)__popc(__ballot_sync(FG_FULL, lane < len && c.active)) > most;
}

/* The targets [first, stop) of the warp whose nominal range is [b, b + len) of
 * a scene's [lo, hi), len <= 32: a cell that straddles two ranges goes to the
 * first one's warp as a whole, unless it fills a range.  (A cut cell would be
 * staged twice, and cells are two to four to a warp.)  Returns whether the
 * range is dispersed; with `apart` such ranges, which are not staged, stay as
 * they are. */
__device__ __forceinline__ bool fg_stage_range(uint32_t b, uint32_t len, uint32_t lo, uint32_t hi, uint32_t most,
                                               bool apart, const StageGrid &G, const float4 *__restrict__ spos,
                                               uint32_t &first, uint32_t &stop)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t own = min(len, hi - b);
    auto cell = [&](uint32_t i) { return fg_stage_cell(__ldg(spos + min(i, hi - 1u)), G); };
    auto pick = [&](const StageCell &c, uint32_t l) {
        StageCell r = {__shfl_sync(FG_FULL, c.x, (int)l), __shfl_sync(FG_FULL, c.y, (int)l),
                       __shfl_sync(FG_FULL, c.z, (int)l), true};
        return r;
    };
    auto same = [](const StageCell &a, const StageCell &c) { return a.x == c.x && a.y == c.y && a.z == c.z; };
    /* how many targets of a range begin by continuing the cell of the target before it */
    auto leading = [&](const StageCell &before, const StageCell &mine, uint32_t n) {
        return (uint32_t)__ffs((int)~(__ballot_sync(FG_FULL, lane < n && same(before, mine)))) - 1u; /* all 32: wraps */
    };
    const StageCell mine = cell(b + lane);
    first = b;
    stop = b + own;
    const bool dispersed = fg_stage_dispersed(mine, G, len, most);
    if (dispersed && apart) return true;
    if (b > lo) {
        const StageCell e = cell(b - len + lane);
        const StageCell before = pick(e, len - 1u), head = pick(e, 0u);
        const uint32_t m = leading(before, mine, own);
        if (m < len && !same(before, head) && !(apart && fg_stage_dispersed(e, G, len, most))) first += m;
    }
    if (b + len < hi) {
        const StageCell last = pick(mine, len - 1u), head = pick(mine, 0u), after = cell(b + len + lane);
        const uint32_t m = leading(last, after, min(len, hi - b - len));
        if (m < len && !same(last, head) && !(apart && fg_stage_dispersed(after, G, len, most))) stop += m;
    }
    return dispersed;
}

/* Of 32 targets, those before the last cell if the target after them, at
 * `after`, is in that cell too (all 32 if it is the only one). */
__device__ __forceinline__ uint32_t fg_stage_trim(const StageSig &s, float4 after, const StageGrid &G)
{
    const bool other = s.ix != fg_axis_index(after.x, G.cell[0]) || s.iy != fg_axis_index(after.y, G.cell[1]) ||
                       s.iz != fg_axis_index(after.z, G.cell[2]);
    const uint32_t m = __ballot_sync(FG_FULL, other);
    return m ? 32u - (uint32_t)__clz((int)m) : 32u;
}

/* Stages the candidates of up to GROUPS groups round after round (CAP slots) and calls
 * run(first, end, used) once a round, the whole warp: this lane's candidates
 * are slots [first, end) of [0, used), in visit order and a multiple of eight
 * of them, filled up with x = +inf, which is out of every range.  keep(slot, j, c) stores
 * candidate j at c.  Every round gets on: its first group's share of the slots
 * holds a chunk. */
template <uint32_t CAP, uint32_t GROUPS, class Keep, class Run>
__device__ __forceinline__ void fg_stage_rounds(const StageSig &sig, uint32_t lead, uint32_t leads, float px, float py,
                                                float pz, const StageGrid &G, const float4 *__restrict__ spos,
                                                const uint32_t *__restrict__ start, const uint32_t *__restrict__ end,
                                                uint32_t *idx /* FG_STAGE_WINDOW, shared */, Keep &&keep, Run &&run)
{
    static_assert(CAP % 8u == 0u && ((CAP / GROUPS) & ~7u) >= 32u, "a round in which no chunk fits would never end");
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t lt = (1u << lane) - 1u;
    const float scale = G.scale, h2 = G.h2;
    const uint32_t bx = lane % 3u, by = (lane / 3u) % 3u, bz = lane / 9u;
    const float inf = __int_as_float(0x7f800000);
    uint32_t next = 0u; /* leaders: the group's next candidate position */
    /* lane b < 27: bucket b's range, of the group that lane l leads */
    uint32_t a_next = FG_EMPTY, e_next = 0u;
    auto lookup = [&](int l) {
        const int ix = __shfl_sync(FG_FULL, sig.ix, l), iy = __shfl_sync(FG_FULL, sig.iy, l),
                  iz = __shfl_sync(FG_FULL, sig.iz, l);
        const uint32_t d = __shfl_sync(FG_FULL, sig.d, l);
        if (lane < 27u) {
            auto off = [&](uint32_t k, uint32_t sh) {
                return k == 0u ? 0u - ((d >> sh) & 3u) : (k == 2u ? (d >> (sh + 2u)) & 3u : 0u);
            };
            const uint32_t b = G.base + fg_bucket(((uint32_t)ix + off(bx, 0u)) * FG_PX,
                                                          ((uint32_t)iy + off(by, 4u)) * FG_PY,
                                                          ((uint32_t)iz + off(bz, 8u)) * FG_PZ, G.nb, G.mask);
            a_next = __ldg(start + b);
            e_next = __ldg(end + b);
        }
    };
    if (leads) lookup(__ffs((int)leads) - 1);
    while (leads) {
        uint32_t used = 0u, first = 0u, stop = 0u;
        for (uint32_t left = leads; left; left &= left - 1u) {
            const int l = __ffs((int)left) - 1;
            /* an even share of what is free; what a group leaves, the next get */
            const uint32_t quota = used + (((CAP - used) / (uint32_t)__popc(left)) & ~7u);
            const bool mine = lead == (uint32_t)l;
            uint32_t q0 = __shfl_sync(FG_FULL, next, l);
            /* lane b < 27: bucket b's first particle and count */
            uint32_t st = 0u, cnt = 0u;
            if (a_next != FG_EMPTY && e_next > a_next) {
                st = a_next;
                cnt = e_next - a_next;
            }
            /* the next group's on their way meanwhile (a full round's last
             * group may be the next round's first) */
            if (left & (left - 1u)) lookup(__ffs((int)(left & (left - 1u))) - 1);
            /* the targets' box */
            const float lx = fg_redux_min(mine ? px : inf), hx = fg_redux_max(mine ? px : -inf);
            const float ly = fg_redux_min(mine ? py : inf), hy = fg_redux_max(mine ? py : -inf);
            const float lz = fg_redux_min(mine ? pz : inf), hz = fg_redux_max(mine ? pz : -inf);
            /* bucket b's first position in the sequence */
            uint32_t incl = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(FG_FULL, incl, o);
                if (lane >= (uint32_t)o) incl += y;
            }
            const uint32_t total = __shfl_sync(FG_FULL, incl, 31);
            const uint32_t pre = incl - cnt;
            if (mine) first = used;
            bool room = true;
            while (room && q0 < total) {
                /* the indices of positions q0 .. q0 + FG_STAGE_WINDOW */
                const uint32_t w0 = q0, w1 = min(total, q0 + FG_STAGE_WINDOW);
                __syncwarp();
                for (uint32_t k = max(pre, w0), e = min(incl, w1); k < e; k++) idx[k - w0] = st + (k - pre);
                __syncwarp();
                /* four chunks of candidates in flight */
                while (room && q0 < w1) {
                    uint32_t j[FG_STAGE_FLIGHT];
                    float4 c[FG_STAGE_FLIGHT];
#pragma unroll
                    for (uint32_t u = 0; u < FG_STAGE_FLIGHT; u++) {
                        const uint32_t q = q0 + 32u * u + lane;
                        j[u] = q < w1 ? idx[q - w0] : 0u;
                        c[u] = q < w1 ? __ldg(spos + j[u]) : make_float4(inf, 0.f, 0.f, 0.f);
                    }
#pragma unroll
                    for (uint32_t u = 0; u < FG_STAGE_FLIGHT; u++) {
                        if (room && q0 < w1) {
                            /* distance to the box, by the operations of the pair distance */
                            const float ex = fmaxf(fmaxf(fmaf(-c[u].x, scale, lx), -fmaf(-c[u].x, scale, hx)), 0.f);
                            const float ey = fmaxf(fmaxf(fmaf(-c[u].y, scale, ly), -fmaf(-c[u].y, scale, hy)), 0.f);
                            const float ez = fmaxf(fmaxf(fmaf(-c[u].z, scale, lz), -fmaf(-c[u].z, scale, hz)), 0.f);
                            const float r2 = fmaf(ex, ex, fmaf(ey, ey, __fmul_rn(ez, ez)));
                            const bool in = !(r2 > h2) && q0 + lane < w1;
                            const uint32_t m = __ballot_sync(FG_FULL, in), n = (uint32_t)__popc(m);
                            if (used + n > quota) {
                                room = false; /* the next round's */
                            } else {
                                if (in) keep(used + (uint32_t)__popc(m & lt), j[u], c[u]);
                                used += n;
                                q0 += 32u;
                            }
                        }
                    }
                }
            }
            const uint32_t fill = (0u - used) & 7u;
            if (lane < fill) keep(used + lane, 0u, make_float4(inf, 0.f, 0.f, 0.f));
            used += fill;
            if (mine) stop = used;
            if (lane == (uint32_t)l) next = q0;
            if (q0 >= total) leads &= ~(1u << l);
        }
        if (leads) lookup(__ffs((int)leads) - 1);
        __syncwarp();
        run(first, stop, used);
        __syncwarp();
    }
}

} // namespace fg

#endif
