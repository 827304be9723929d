/* Rigid-body side of the two-way fluid/rigid coupling on GB300.
 *
 *   k_rb_from_fluid   CalculateRBForcesFromFluidsK (K_RigidBodySim.cu:66-99)
 *   k_rb_from_rb      CalculateRigidBodyForcesFromRBK (K_RigidBodySim.cu:18-61)
 *   k_body_update     applyForces' per-body sum (RigidBodySimulator.cpp:522-566:
 *                     sort by body, segmented scan, AddForceTorqueK) as one
 *                     deterministic FP64 block reduction per body, followed by
 *                     IntegrateRBK (K_RigidBodySim.cu:160-262) in FP64
 *   k_integrate_rb_f32  IntegrateRBK with the reference's FP32 arithmetic
 *   k_copy_rb_data / k_reorder_ft / k_segsum / k_add_ft
 *                     the reference's reduction data flow for the drop-in
 *                     launchers (K_RigidBodySim.cu:102-155 + CUDPP scan). */
#include <cuda_runtime.h>
#include <cooperative_groups.h>
#include <stdint.h>
#include <string.h>
#include "fg_device.cuh"
#include "fg_kernels.h"

namespace fg {

/* Contact sum of one rigid sphere against the fluid grid, then force and
 * torque written at the sphere's unsorted index (body-contiguous).  One warp
 * per sphere, so a few thousand spheres still fill the GPU: the lanes take
 * the (2r+1)^3 fluid buckets in turn and a fixed shuffle tree adds their
 * partial sums (deterministic; the FP32 terms are the reference's, their
 * summation order differs).  CTA = RBF_WARPS warps; CTA c takes spheres
 * RBF_WARPS (c % 32) + warp of work item c / 32. */
#define RBF_WARPS 4
__global__ void __launch_bounds__(RBF_WARPS * 32) k_rb_from_fluid(const FgWork *__restrict__ work, uint32_t nwork,
                                                                 uint32_t n_single, const FgScene *__restrict__ table,
                                                                 const __grid_constant__ FgScene single,
                                                                 const float4 *__restrict__ rb_spos,
                                                                 const uint32_t *__restrict__ rb_ids,
                                                                 const float4 *__restrict__ body_vel,
                                                                 const float4 *__restrict__ body_cm,
                                                                 const float4 *__restrict__ fl_spos,
                                                                 const float4 *__restrict__ fl_svel,
                                                                 const uint32_t *__restrict__ fl_start,
                                                                 const uint32_t *__restrict__ fl_end,
                                                                 float4 *__restrict__ force,
                                                                 float4 *__restrict__ torque, int add)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t w = blockIdx.x >> 5;
    if (w >= nwork) return;
    const FgWork it = fg_work(work, w, n_single);
    const uint32_t k = ((blockIdx.x & 31u) * RBF_WARPS) + (uint32_t)wid;
    if (k >= it.count) return; /* warp-uniform */
    const FgScene *S = fg_scene(table, &single, it.scene);
    const uint32_t i = it.first + k;
    const float4 p = rb_spos[i];
    const int b = (int)p.w;
    const float4 vb = __ldg(body_vel + b);
    const float3 P = make_float3(p.x, p.y, p.z), V = make_float3(vb.x, vb.y, vb.z);
    const float mind = S->rb_radius + S->fluid_radius + S->rb_eps;
    float3 acc = make_float3(0.f, 0.f, 0.f);
    const int rx = S->r2f_rel[0], ry = S->r2f_rel[1], rz = S->r2f_rel[2];
    const int nx = 2 * rx + 1, ny = 2 * ry + 1, nz = 2 * rz + 1;
    for (int q = lane; q < nx * ny * nz; q += 32) {
        const int z = q / (nx * ny) - rz, y = (q / nx) % ny - ry, x = q % nx - rx;
        const uint32_t bk = S->bucket_base + fg_bucket(fg_axis_hash_rel(p.x, S->cell[0], x, FG_PX),
                                                       fg_axis_hash_rel(p.y, S->cell[1], y, FG_PY),
                                                       fg_axis_hash_rel(p.z, S->cell[2], z, FG_PZ), S->nb, S->nb_mask);
        const uint32_t st = __ldg(fl_start + bk);
        if (st == FG_EMPTY) continue;
        const uint32_t en = __ldg(fl_end + bk);
        for (uint32_t j = st; j < en; j++)
            fg_contact(acc, P, V, __ldg(fl_spos + j), __ldg(fl_svel + j), mind, S->ck, S->ckd);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
        acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
        acc.z += __shfl_xor_sync(0xffffffffu, acc.z, o);
    }
    if (lane) return;
    const float4 cm = __ldg(body_cm + b);
    const float lw = (float)(b - (int)S->body_base); /* the reference stores the body index in w */
    const float dx = p.x - cm.x, dy = p.y - cm.y, dz = p.z - cm.z;
    float4 f = make_float4(acc.x, acc.y, acc.z, lw);
    float4 t = make_float4(dy * acc.z - dz * acc.y, dz * acc.x - dx * acc.z, dx * acc.y - dy * acc.x, lw);
    const uint32_t oi = rb_ids ? __ldg(rb_ids + i) : i;
    if (add) {
        const float4 f0 = force[oi], t0 = torque[oi];
        f.x += f0.x; f.y += f0.y; f.z += f0.z;
        t.x += t0.x; t.y += t0.y; t.z += t0.z;
    }
    force[oi] = f;
    torque[oi] = t;
}

void launch_rb_from_fluid(const Launch &L, const float4 *rb_spos, const uint32_t *rb_ids, const float4 *body_vel,
                          const float4 *body_cm, const float4 *fl_spos, const float4 *fl_svel,
                          const uint32_t *fl_start, const uint32_t *fl_end, float4 *force, float4 *torque, int add)
{
    if (!L.nwork) return;
    /* a work item holds up to FG_CHUNK spheres: FG_CHUNK / RBF_WARPS CTAs */
    k_rb_from_fluid<<<L.nwork * (FG_CHUNK / RBF_WARPS), RBF_WARPS * 32, 0, L.stream>>>(
        L.work, L.nwork, L.n, L.table, *L.single, rb_spos, rb_ids, body_vel, body_cm, fl_spos, fl_svel, fl_start,
        fl_end, force, torque, add);
}

/* Sphere/sphere contact between different bodies of one scene (same rigid
 * grid, half-width 1, spheres of the own body skipped) and, optionally,
 * against a static sphere grid (no velocity, no grouping). */
struct StaticArg {
    RigidGrid g;
    int use;
};

__global__ void __launch_bounds__(FG_CHUNK) k_rb_from_rb(const FgWork *__restrict__ work, uint32_t nwork,
                                                        uint32_t n_single, const FgScene *__restrict__ table,
                                                        const __grid_constant__ FgScene single,
                                                        const float4 *__restrict__ rb_spos,
                                                        const uint32_t *__restrict__ rb_ids,
                                                        const float4 *__restrict__ body_vel,
                                                        const float4 *__restrict__ body_cm,
                                                        const uint32_t *__restrict__ rb_start,
                                                        const uint32_t *__restrict__ rb_end,
                                                        float4 *__restrict__ force, float4 *__restrict__ torque,
                                                        const __grid_constant__ StaticArg sta, int add)
{
    for (uint32_t w = blockIdx.x; w < nwork; w += gridDim.x) {
        FgWork it = fg_work(work, w, n_single);
        if (threadIdx.x >= it.count) continue;
        const FgScene *S = fg_scene(table, &single, it.scene);
        const uint32_t i = it.first + threadIdx.x;
        const float4 p = rb_spos[i];
        const int b = (int)p.w;
        const float4 vb = __ldg(body_vel + b);
        const float4 cm = __ldg(body_cm + b);
        const float3 P = make_float3(p.x, p.y, p.z), V = make_float3(vb.x, vb.y, vb.z);
        const float mind = S->rb_radius + S->rb_radius + S->rbrb_eps;
        float3 acc = make_float3(0.f, 0.f, 0.f);
        for (int z = -1; z <= 1; z++) {
            const uint32_t hz = fg_axis_hash_rel(p.z, S->rb_cell[2], z, FG_PZ);
            for (int y = -1; y <= 1; y++) {
                const uint32_t hy = fg_axis_hash_rel(p.y, S->rb_cell[1], y, FG_PY);
                for (int x = -1; x <= 1; x++) {
                    const uint32_t hx = fg_axis_hash_rel(p.x, S->rb_cell[0], x, FG_PX);
                    const uint32_t bk = S->rb_bucket_base + fg_bucket(hx, hy, hz, S->rb_nb, S->rb_nb_mask);
                    const uint32_t st = __ldg(rb_start + bk);
                    if (st == FG_EMPTY) continue;
                    const uint32_t en = __ldg(rb_end + bk);
                    for (uint32_t j = st; j < en; j++) {
                        const float4 q = __ldg(rb_spos + j);
                        if ((int)q.w == b) continue;
                        fg_contact(acc, P, V, q, __ldg(body_vel + (int)q.w), mind, S->rbrb_k, S->rbrb_kd);
                    }
                }
            }
        }
        if (sta.use) {
            for (int z = -1; z <= 1; z++) {
                const uint32_t hz = fg_axis_hash_rel(p.z, S->rb_cell[2], z, FG_PZ);
                for (int y = -1; y <= 1; y++) {
                    const uint32_t hy = fg_axis_hash_rel(p.y, S->rb_cell[1], y, FG_PY);
                    for (int x = -1; x <= 1; x++) {
                        const uint32_t hx = fg_axis_hash_rel(p.x, S->rb_cell[0], x, FG_PX);
                        const uint32_t bk = fg_bucket(hx, hy, hz, sta.g.nb, sta.g.mask);
                        const uint32_t st = __ldg(sta.g.start + bk);
                        if (st == FG_EMPTY) continue;
                        const uint32_t en = __ldg(sta.g.end + bk);
                        for (uint32_t j = st; j < en; j++)
                            fg_contact(acc, P, V, __ldg(sta.g.spos + j), make_float4(0.f, 0.f, 0.f, 0.f), mind,
                                       S->rbrb_k, S->rbrb_kd);
                    }
                }
            }
        }
        const float dx = p.x - cm.x, dy = p.y - cm.y, dz = p.z - cm.z;
        const uint32_t oi = rb_ids ? __ldg(rb_ids + i) : i;
        const float tx = dy * acc.z - dz * acc.y, ty = dz * acc.x - dx * acc.z, tz = dx * acc.y - dy * acc.x;
        if (add) {
            float4 f = force[oi], t = torque[oi];
            f.x += acc.x; f.y += acc.y; f.z += acc.z;
            t.x += tx; t.y += ty; t.z += tz;
            force[oi] = f;
            torque[oi] = t;
        } else {
            const float lw = (float)(b - (int)S->body_base);
            force[oi] = make_float4(acc.x, acc.y, acc.z, lw);
            torque[oi] = make_float4(tx, ty, tz, lw);
        }
    }
}

void launch_rb_from_rb(const Launch &L, const float4 *rb_spos, const uint32_t *rb_ids, const float4 *body_vel,
                       const float4 *body_cm, const uint32_t *rb_start, const uint32_t *rb_end, float4 *force,
                       float4 *torque, const RigidGrid *statics, int add)
{
    if (!L.nwork) return;
    StaticArg sa;
    memset(&sa, 0, sizeof(sa));
    if (statics) { sa.g = *statics; sa.use = 1; }
    k_rb_from_rb<<<grid_for(L.nwork, 16), FG_CHUNK, 0, L.stream>>>(L.work, L.nwork, L.n, L.table, *L.single, rb_spos,
                                                                   rb_ids, body_vel, body_cm, rb_start, rb_end, force,
                                                                   torque, sa, add);
}

/* ---------------------------------------------------------- FP64 bodies */

#define BODY_THREADS 256

/* Sums of the eight components over the warp: lane l gets component l >> 2.
 * Halves the components a lane carries at each exchange: the sums of a
 * butterfly over all eight, bit for bit, for nine FP64 additions instead of
 * forty (the FP64 pipe takes a warp's addition in many cycles): 10 -> 4.3 us
 * for 32 bodies of 512 spheres. */
__device__ __forceinline__ double body_sum8(double (&a)[8])
{
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
    for (int o = 16, n = 4; o >= 4; o >>= 1, n >>= 1) {
        const bool upper = lane & (uint32_t)o;
#pragma unroll
        for (int q = 0; q < n; q++) {
            const double keep = upper ? a[n + q] : a[q], give = upper ? a[q] : a[n + q];
            a[q] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    a[0] += __shfl_xor_sync(0xffffffffu, a[0], 2);
    a[0] += __shfl_xor_sync(0xffffffffu, a[0], 1);
    return a[0];
}

/* One CTA's sums of force and torque (component threadIdx.x of eight, in the
 * first eight threads) over spheres first + [lo, hi): threads stride them, then
 * a warp tree and the warps in order (deterministic). */
__device__ __forceinline__ double body_sum_cta(uint32_t first, uint32_t lo, uint32_t hi,
                                               const float4 *__restrict__ force, const float4 *__restrict__ torque,
                                               double (*s_red)[8])
{
    double a[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (uint32_t k = lo + threadIdx.x; k < hi; k += BODY_THREADS) {
        const float4 f = __ldg(force + first + k), t = __ldg(torque + first + k);
        a[0] += f.x; a[1] += f.y; a[2] += f.z; a[3] += f.w;
        a[4] += t.x; a[5] += t.y; a[6] += t.z; a[7] += t.w;
    }
    const double sum = body_sum8(a);
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    if ((lane & 3u) == 0u) s_red[wid][lane >> 2] = sum;
    __syncthreads();
    double v = 0.0;
    if (threadIdx.x < 8)
        for (int wv = 0; wv < BODY_THREADS / 32; wv++) v += s_red[wv][threadIdx.x];
    return v;
}

/* FP64 partial force/torque sums of one body's spheres: chunk blockIdx.x of
 * FG_BODY_CHUNKS, body blockIdx.y. */
__global__ void __launch_bounds__(BODY_THREADS) k_body_partial(const uint32_t *__restrict__ body_first,
                                                              const uint32_t *__restrict__ body_count,
                                                              const float4 *__restrict__ force,
                                                              const float4 *__restrict__ torque,
                                                              double *__restrict__ partial)
{
    __shared__ double s_red[BODY_THREADS / 32][8];
    const uint32_t b = blockIdx.y, c = blockIdx.x;
    const uint32_t cnt = body_count[b];
    const uint32_t per = (cnt + FG_BODY_CHUNKS - 1) / FG_BODY_CHUNKS;
    const double v = body_sum_cta(body_first[b], min(cnt, c * per), min(cnt, (c + 1) * per), force, torque, s_red);
    if (threadIdx.x < 8) partial[((size_t)b * FG_BODY_CHUNKS + c) * 8 + threadIdx.x] = v;
}

/* What the lanes of a body's warp read of one another, by component x, y, z, w
 * or matrix element (row-major). */
struct BodyWarp {
    double F[4], L[4], q[4], om[4], R[9], Tm[9], G[9];
};

/* Component c of the quaternion product a * b, c = 3 the scalar part. */
__device__ __forceinline__ double body_qprod(const double *a, const double *b, uint32_t c)
{
    if (c == 3u) {
        const double dotv = a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
        return a[3] * b[3] - dotv;
    }
    const uint32_t d = c == 2u ? 0u : c + 1u, e = c == 0u ? 2u : c - 1u;
    return (a[3] * b[c]) + (b[3] * a[c]) + (a[d] * b[e] - a[e] * b[d]);
}

/* IntegrateRBK in double for one body by one warp: lane c < 4 has component c
 * of the sums F and T and of the vectors, lane e < 9 element e of the
 * matrices.  A body is a chain of some 60 FP64 operations, two square roots
 * and two divides that way, 11 us; one thread went through some 500, 22 us. */
__device__ __forceinline__ void body_integrate(const FgScene *S, uint32_t b, double F, double T, const BodyState &st,
                                               BodyWarp &W)
{
    const uint32_t lane = threadIdx.x & 31u, c = lane & 3u, e = min(lane, 8u), r = e / 3u, k = e % 3u;
    const double vl = S->rb_vlimit, dt = S->rb_dt;
    if (lane < 4u) {
        W.F[c] = F;
        W.q[c] = ((const double *)(st.q + b))[c];
    }
    __syncwarp();
    const double spd = sqrt(W.F[0] * W.F[0] + W.F[1] * W.F[1] + W.F[2] * W.F[2] + W.F[3] * W.F[3]);
    if (spd > vl) F *= vl / spd;
    const double acc = ((F + (double)S->rb_gravity[c]) / st.mass[b]) * dt;
    double v = ((const double *)(st.v + b))[c], x = ((const double *)(st.x + b))[c];
    v += acc * dt;
    if (c < 3u) x += v * dt;
    double L = ((const double *)(st.L + b))[c];
    L = (L + T * dt) * (double)0.9f;
    /* AngularVelocityD: R * Iinv * R^T * L.  R's diagonal: (1 - 2 a a) - 2 b b
     * of the other two components; else (2 q_r q_k) +- 2 w q_o of the third */
    {
        const bool diag = r == k, plus = !diag && (k == r + 1u || (r == 2u && k == 0u));
        const double a1 = W.q[diag ? (r == 0u ? 1u : 0u) : r], a2 = W.q[diag ? (r == 0u ? 1u : 0u) : k];
        const double b1 = diag ? W.q[r == 2u ? 1u : 2u] : W.q[3], b2 = W.q[diag ? (r == 2u ? 1u : 2u) : 3u - r - k];
        const double u = diag ? 1.0 - 2.0 * a1 * a2 : 2.0 * a1 * a2;
        if (lane < 9u) W.R[e] = plus ? u + 2.0 * b1 * b2 : u - 2.0 * b1 * b2;
        if (lane < 4u) W.L[c] = L;
    }
    __syncwarp();
    const double *I = st.inv_inertia + 9 * b;
    if (lane < 9u) W.Tm[e] = W.R[3u * r] * I[k] + W.R[3u * r + 1u] * I[3u + k] + W.R[3u * r + 2u] * I[6u + k];
    __syncwarp();
    if (lane < 9u)
        W.G[e] = W.Tm[3u * r] * W.R[3u * k] + W.Tm[3u * r + 1u] * W.R[3u * k + 1u] +
                 W.Tm[3u * r + 2u] * W.R[3u * k + 2u];
    __syncwarp();
    if (lane < 4u)
        W.om[c] = c < 3u ? W.G[3u * c] * W.L[0] + W.G[3u * c + 1u] * W.L[1] + W.G[3u * c + 2u] * W.L[2] : 0.0;
    __syncwarp();
    const double om = body_qprod(W.om, W.q, c) * (double)0.5f;
    __syncwarp();
    if (lane < 4u) W.om[c] = om * dt * (double)0.1f;
    __syncwarp();
    double q = W.q[c] + body_qprod(W.om, W.q, c);
    __syncwarp();
    if (lane < 4u) W.q[c] = q;
    __syncwarp();
    q /= sqrt(W.q[3] * W.q[3] + W.q[0] * W.q[0] + W.q[1] * W.q[1] + W.q[2] * W.q[2]);
    const double rest = (double)-0.7f;
    if (c == 1u) {
        if (x < (double)S->rb_vmin[1]) { x = S->rb_vmin[1]; v *= rest; }
    } else if (c != 3u) {
        if (x <= (double)S->rb_vmin[c]) { x = S->rb_vmin[c]; v *= rest; }
        else if (x >= (double)S->rb_vmax[c]) { x = S->rb_vmax[c]; v *= rest; }
    }
    if (lane < 4u) {
        ((double *)(st.x + b))[c] = x;
        ((double *)(st.v + b))[c] = v;
        ((double *)(st.L + b))[c] = L;
        ((double *)(st.q + b))[c] = q;
        ((float *)(st.x_f + b))[c] = (float)x;
        ((float *)(st.v_f + b))[c] = (float)v;
        ((float *)(st.q_f + b))[c] = (float)q;
    }
    __syncwarp();
}

/* A CTA per body: its sum, or its partial sums in order, then the first warp
 * integrates it. */
__global__ void __launch_bounds__(BODY_THREADS) k_body_update(const FgScene *__restrict__ table,
                                                             const __grid_constant__ FgScene single,
                                                             const uint32_t *__restrict__ body_scene,
                                                             const uint32_t *__restrict__ body_first,
                                                             const uint32_t *__restrict__ body_count,
                                                             uint32_t nbodies, const float4 *__restrict__ force,
                                                             const float4 *__restrict__ torque, BodyState st,
                                                             int integrate)
{
    __shared__ double s_red[BODY_THREADS / 32][8];
    __shared__ BodyWarp W;
    for (uint32_t b = blockIdx.x; b < nbodies; b += gridDim.x) {
        double v = 0.0;
        if (st.partial) {
            if (threadIdx.x < 8) {
                const double *pp = st.partial + (size_t)b * FG_BODY_CHUNKS * 8 + threadIdx.x;
#pragma unroll
                for (int ch = 0; ch < FG_BODY_CHUNKS; ch++) v += pp[ch * 8];
            }
        } else {
            v = body_sum_cta(body_first[b], 0u, body_count[b], force, torque, s_red);
        }
        if (threadIdx.x < 32) {
            FgD4 *const sum = threadIdx.x < 4 ? st.force_sum : st.torque_sum;
            if (threadIdx.x < 8) ((double *)(sum + b))[threadIdx.x & 3] = v;
            const double T = __shfl_sync(0xffffffffu, v, (threadIdx.x & 3) + 4);
            const double F = __shfl_sync(0xffffffffu, v, threadIdx.x & 3);
            /* mass 0: a static body (the reference's "static" rigid-body
             * file type), never integrated */
            if (integrate && st.mass[b] != 0.0)
                body_integrate(table ? table + body_scene[b] : &single, b, F, T, st, W);
        }
        __syncthreads();
    }
}

void launch_body_update(const FgScene *table, const FgScene *single, const uint32_t *body_scene,
                        const uint32_t *body_first, const uint32_t *body_count, uint32_t nbodies,
                        const float4 *force, const float4 *torque, BodyState st, int integrate, cudaStream_t s)
{
    if (!nbodies) return;
    if (st.partial && nbodies <= 65535u)
        k_body_partial<<<dim3(FG_BODY_CHUNKS, nbodies), BODY_THREADS, 0, s>>>(body_first, body_count, force, torque,
                                                                            st.partial);
    else
        st.partial = nullptr;
    const int per_sm = st.partial ? 16 : 4, threads = st.partial ? 32 : BODY_THREADS;
    k_body_update<<<grid_for(nbodies, per_sm), threads, 0, s>>>(table, *single, body_scene, body_first, body_count,
                                                                nbodies, force, torque, st, integrate);
}

/* ---------------------------------------------- FP32 IntegrateRBK (exact) */
__device__ __forceinline__ float4 f4add(float4 a, float4 b)
{
    return make_float4(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z), __fadd_rn(a.w, b.w));
}
__device__ __forceinline__ float4 f4muls(float4 a, float s)
{
    return make_float4(__fmul_rn(a.x, s), __fmul_rn(a.y, s), __fmul_rn(a.z, s), __fmul_rn(a.w, s));
}

__global__ void k_integrate_rb_f32(float4 *__restrict__ X, const float *__restrict__ mass, float4 *__restrict__ V,
                                   const float4 *__restrict__ Fin, uint32_t nrb, float dt, float4 ext, float3 vmin,
                                   float3 vmax, float4 *__restrict__ Lm, const float4 *__restrict__ Tq,
                                   float4 *__restrict__ Q, const float4 *__restrict__ inv, float vlimit)
{
    uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= nrb) return;
    float4 F = Fin[idx];
    float spd = __fsqrt_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(F.x, F.x), __fmul_rn(F.y, F.y)),
                                               __fmul_rn(F.z, F.z)),
                                     __fmul_rn(F.w, F.w)));
    if (spd > vlimit) F = f4muls(F, __fdiv_rn(vlimit, spd));
    float4 pos = X[idx];
    float m = mass[idx];
    float4 fe = f4add(F, ext);
    float4 acc = make_float4(__fmul_rn(__fdiv_rn(fe.x, m), dt), __fmul_rn(__fdiv_rn(fe.y, m), dt),
                             __fmul_rn(__fdiv_rn(fe.z, m), dt), __fmul_rn(__fdiv_rn(fe.w, m), dt));
    float4 vel = f4add(V[idx], f4muls(acc, dt));
    pos.x = __fadd_rn(pos.x, __fmul_rn(vel.x, dt));
    pos.y = __fadd_rn(pos.y, __fmul_rn(vel.y, dt));
    pos.z = __fadd_rn(pos.z, __fmul_rn(vel.z, dt));
    float4 L = f4add(Lm[idx], f4muls(Tq[idx], dt));
    L = f4muls(L, 0.9f);
    Lm[idx] = L;
    /* AngularVelocityD */
    float4 q = Q[idx];
    float R[3][3];
    R[0][0] = __fsub_rn(__fsub_rn(1.0f, __fmul_rn(__fmul_rn(2.0f, q.y), q.y)), __fmul_rn(__fmul_rn(2.0f, q.z), q.z));
    R[0][1] = __fadd_rn(__fmul_rn(__fmul_rn(2.0f, q.x), q.y), __fmul_rn(__fmul_rn(2.0f, q.w), q.z));
    R[0][2] = __fsub_rn(__fmul_rn(__fmul_rn(2.0f, q.x), q.z), __fmul_rn(__fmul_rn(2.0f, q.w), q.y));
    R[1][0] = __fsub_rn(__fmul_rn(__fmul_rn(2.0f, q.x), q.y), __fmul_rn(__fmul_rn(2.0f, q.w), q.z));
    R[1][1] = __fsub_rn(__fsub_rn(1.0f, __fmul_rn(__fmul_rn(2.0f, q.x), q.x)), __fmul_rn(__fmul_rn(2.0f, q.z), q.z));
    R[1][2] = __fadd_rn(__fmul_rn(__fmul_rn(2.0f, q.y), q.z), __fmul_rn(__fmul_rn(2.0f, q.w), q.x));
    R[2][0] = __fadd_rn(__fmul_rn(__fmul_rn(2.0f, q.x), q.z), __fmul_rn(__fmul_rn(2.0f, q.w), q.y));
    R[2][1] = __fsub_rn(__fmul_rn(__fmul_rn(2.0f, q.y), q.z), __fmul_rn(__fmul_rn(2.0f, q.w), q.x));
    R[2][2] = __fsub_rn(__fsub_rn(1.0f, __fmul_rn(__fmul_rn(2.0f, q.x), q.x)), __fmul_rn(__fmul_rn(2.0f, q.y), q.y));
    float I[3][3];
    for (int r = 0; r < 3; r++) {
        float4 row = inv[idx * 3 + r];
        I[r][0] = row.x; I[r][1] = row.y; I[r][2] = row.z;
    }
    float Tm[3][3], G[3][3];
    for (int r = 0; r < 3; r++)
        for (int c = 0; c < 3; c++)
            Tm[r][c] = __fadd_rn(__fadd_rn(__fmul_rn(R[r][0], I[0][c]), __fmul_rn(R[r][1], I[1][c])),
                                 __fmul_rn(R[r][2], I[2][c]));
    for (int r = 0; r < 3; r++)
        for (int c = 0; c < 3; c++)
            G[r][c] = __fadd_rn(__fadd_rn(__fmul_rn(Tm[r][0], R[c][0]), __fmul_rn(Tm[r][1], R[c][1])),
                                __fmul_rn(Tm[r][2], R[c][2]));
    float4 om;
    om.x = __fadd_rn(__fadd_rn(__fmul_rn(G[0][0], L.x), __fmul_rn(G[0][1], L.y)), __fmul_rn(G[0][2], L.z));
    om.y = __fadd_rn(__fadd_rn(__fmul_rn(G[1][0], L.x), __fmul_rn(G[1][1], L.y)), __fmul_rn(G[1][2], L.z));
    om.z = __fadd_rn(__fadd_rn(__fmul_rn(G[2][0], L.x), __fmul_rn(G[2][1], L.y)), __fmul_rn(G[2][2], L.z));
    om.w = 0.0f;
    om = f4muls(fg_qprod_rn(om, q), 0.5f);
    float4 dq = fg_qprod_rn(f4muls(f4muls(om, dt), 0.1f), q);
    q = f4add(q, dq);
    float nrm = __fsqrt_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(q.w, q.w), __fmul_rn(q.x, q.x)),
                                               __fmul_rn(q.y, q.y)),
                                     __fmul_rn(q.z, q.z)));
    q = make_float4(__fdiv_rn(q.x, nrm), __fdiv_rn(q.y, nrm), __fdiv_rn(q.z, nrm), __fdiv_rn(q.w, nrm));
    Q[idx] = q;
    if (pos.y < vmin.y) { pos.y = vmin.y; vel.y = __fmul_rn(vel.y, -0.7f); }
    if (pos.x <= vmin.x) { pos.x = vmin.x; vel.x = __fmul_rn(vel.x, -0.7f); }
    else if (pos.x >= vmax.x) { pos.x = vmax.x; vel.x = __fmul_rn(vel.x, -0.7f); }
    if (pos.z <= vmin.z) { pos.z = vmin.z; vel.z = __fmul_rn(vel.z, -0.7f); }
    else if (pos.z >= vmax.z) { pos.z = vmax.z; vel.z = __fmul_rn(vel.z, -0.7f); }
    X[idx] = pos;
    V[idx] = vel;
}

void launch_integrate_rb_f32(float4 *x, const float *mass, float4 *v, const float4 *f, uint32_t nrb, float dt,
                             float4 ext, float3 vmin, float3 vmax, float4 *L, const float4 *t, const float4 *inertia,
                             float4 *q, const float4 *inv, float vlimit, cudaStream_t s)
{
    (void)inertia;
    if (!nrb) return;
    k_integrate_rb_f32<<<(nrb + 127) / 128, 128, 0, s>>>(x, mass, v, f, nrb, dt, ext, vmin, vmax, L, t, q, inv,
                                                         vlimit);
}

/* ------------------------------- reference reduction data flow (drop-in) */

__global__ void k_copy_rb_data(uint32_t *key, uint32_t *idx, const float4 *force, uint32_t n)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        key[i] = (uint32_t)force[i].w;
        idx[i] = i;
    }
}

void launch_copy_rb_data_to_particle(uint32_t *key, uint32_t *idx, const float4 *force, uint32_t n, cudaStream_t s)
{
    if (!n) return;
    k_copy_rb_data<<<grid_for((n + 255) / 256, 8), 256, 0, s>>>(key, idx, force, n);
}

__global__ void k_reorder_ft(float4 *fo, float4 *to, const float4 *fi, const float4 *ti, const uint32_t *order,
                             uint32_t n)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t o = order[i];
        fo[i] = fi[o];
        to[i] = ti[o];
    }
}

void launch_reorder_force_torque(float4 *fo, float4 *to, const float4 *fi, const float4 *ti, const uint32_t *order,
                                 uint32_t n, cudaStream_t s)
{
    if (!n) return;
    k_reorder_ft<<<grid_for((n + 255) / 256, 8), 256, 0, s>>>(fo, to, fi, ti, order, n);
}

/* Inclusive forward segmented sum of float4 (segment heads flagged with a
 * non-zero flag) in 1,024-element chunks, a CTA of a cluster of up to eight
 * each: the chunks' own scans run side by side, and every CTA adds the totals
 * of the chunks before its own in order, so the sums are those of one CTA that
 * carries its total from chunk to chunk.  Bound by latency: one CTA took 11.2
 * us for 8,192 elements, eight 3.6. */
template <bool CLUSTER>
__global__ void __launch_bounds__(1024) k_segsum(const float4 *in, const uint32_t *__restrict__ flags, float4 *out,
                                                uint32_t n) /* out may be in */
{
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    __shared__ float4 s_v[32];
    __shared__ uint32_t s_f[32];
    __shared__ float4 s_tot[2]; /* the chunk's sum since its last flag, of alternate rounds */
    __shared__ uint32_t s_any[2];
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t me = CLUSTER ? cl.block_rank() : 0u, ctas = CLUSTER ? cl.num_blocks() : 1u;
    float4 carry = make_float4(0.f, 0.f, 0.f, 0.f); /* of all chunks before the round (warp 0) */
    uint32_t turn = 0u;
    for (uint32_t base = 0; base < n; base += ctas * 1024u, turn ^= 1u) {
        const uint32_t i = base + me * 1024u + threadIdx.x;
        float4 v = i < n ? in[i] : make_float4(0.f, 0.f, 0.f, 0.f);
        uint32_t f = i < n ? (flags[i] ? 1u : 0u) : 0u;
        /* warp segmented inclusive scan */
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            float4 u = make_float4(__shfl_up_sync(0xffffffffu, v.x, o), __shfl_up_sync(0xffffffffu, v.y, o),
                                   __shfl_up_sync(0xffffffffu, v.z, o), __shfl_up_sync(0xffffffffu, v.w, o));
            uint32_t g = __shfl_up_sync(0xffffffffu, f, o);
            if (lane >= (uint32_t)o && !f) {
                v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
            }
            if (lane >= (uint32_t)o) f |= g;
        }
        if (lane == 31) { s_v[wid] = v; s_f[wid] = f; }
        __syncthreads();
        /* warp `lane`'s exclusive prefix inside the chunk */
        float4 pv = make_float4(0.f, 0.f, 0.f, 0.f);
        uint32_t pf = 0u;
        if (wid == 0) {
            float4 wv = s_v[lane];
            uint32_t wf = s_f[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                float4 u = make_float4(__shfl_up_sync(0xffffffffu, wv.x, o), __shfl_up_sync(0xffffffffu, wv.y, o),
                                       __shfl_up_sync(0xffffffffu, wv.z, o), __shfl_up_sync(0xffffffffu, wv.w, o));
                uint32_t g = __shfl_up_sync(0xffffffffu, wf, o);
                if (lane >= (uint32_t)o && !wf) {
                    wv.x += u.x; wv.y += u.y; wv.z += u.z; wv.w += u.w;
                }
                if (lane >= (uint32_t)o) wf |= g;
            }
            pv = make_float4(__shfl_up_sync(0xffffffffu, wv.x, 1), __shfl_up_sync(0xffffffffu, wv.y, 1),
                             __shfl_up_sync(0xffffffffu, wv.z, 1), __shfl_up_sync(0xffffffffu, wv.w, 1));
            pf = __shfl_up_sync(0xffffffffu, wf, 1);
            if (lane == 31) { s_tot[turn] = wv; s_any[turn] = wf; }
        }
        if (CLUSTER) cl.sync();
        else __syncwarp(); /* the first warp reads what it wrote */
        if (wid == 0) {
            /* the chunks before mine, then the round's, in order */
            float4 c = carry, next = carry;
            for (uint32_t r = 0; r < ctas; r++) {
                if (r == me) c = next;
                float4 t = *cl.map_shared_rank(&s_tot[turn], (int)r);
                if (!*cl.map_shared_rank(&s_any[turn], (int)r)) {
                    t.x += next.x; t.y += next.y; t.z += next.z; t.w += next.w;
                }
                next = t;
            }
            carry = next;
            if (lane == 0) pv = c;
            else if (!pf) { pv.x += c.x; pv.y += c.y; pv.z += c.z; pv.w += c.w; }
            s_v[lane] = pv;
        }
        __syncthreads();
        if (i < n) {
            if (!f) {
                float4 p = s_v[wid];
                v.x += p.x; v.y += p.y; v.z += p.z; v.w += p.w;
            }
            out[i] = v;
        }
        __syncthreads();
    }
    if (CLUSTER) cl.sync(); /* no CTA leaves while another may read its sum */
}

void launch_segmented_sum(const float4 *in, const uint32_t *flags, float4 *out, uint32_t n, cudaStream_t s)
{
    if (!n) return;
    uint32_t ctas = 1u;
    while (ctas < 8u && ctas * 1024u < n) ctas <<= 1;
    if (ctas == 1u) { /* 1,000 elements: 6.6 us as a cluster of one, 5.4 so */
        k_segsum<false><<<1, 1024, 0, s>>>(in, flags, out, n);
        return;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(1024);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ctas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k_segsum<true>, in, flags, out, n);
}

__global__ void k_add_ft(const float4 *sum_f, const float4 *sum_t, const float4 *ordered_f, float4 *out_f,
                         float4 *out_t, const int *offsets, uint32_t nrb)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nrb) return;
    int o = offsets[i];
    int b = (int)ordered_f[o].w;
    float4 f = sum_f[o], t = sum_t[o];
    float4 a = out_f[b], c = out_t[b];
    out_f[b] = make_float4(a.x + f.x, a.y + f.y, a.z + f.z, a.w + f.w);
    out_t[b] = make_float4(c.x + t.x, c.y + t.y, c.z + t.z, c.w + t.w);
}

void launch_add_force_torque(const float4 *sum_f, const float4 *sum_t, const float4 *ordered_f, float4 *out_f,
                             float4 *out_t, const int *offsets, uint32_t nrb, cudaStream_t s)
{
    if (!nrb) return;
    k_add_ft<<<(nrb + 127) / 128, 128, 0, s>>>(sum_f, sum_t, ordered_f, out_f, out_t, offsets, nrb);
}

} // namespace fg
