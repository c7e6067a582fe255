/*
 * sph_pcisph.cu -- PCISPH passes (kernels/pcisph.cl) over the materialised neighbour lists.
 *
 *   k_pci_init_density  fill p = 0 (pcisphsimluation.cpp:118) + compute_initial_density
 *                       (pcisph.cl:33-102)
 *   k_pci_init_forces   fill F_p = 0 (pcisphsimluation.cpp:126) + compute_initial_forces
 *                       (pcisph.cl:134-222): viscosity + Akinci surface tension
 *   k_pci_loop          the whole predict-correct loop of pcisphsimluation.cpp:129-148 in ONE
 *                       persistent cooperative kernel: predict_pos (pcisph.cl:302-344),
 *                       update_pressure (:349-418) with a fused block max of the density
 *                       error (replacing clmax, clreduce.h:54-62, and its blocking read per
 *                       iteration), compute_pressure_force (:420-504).  The stop test runs on
 *                       the device after a grid barrier, so no host round trip per iteration.
 *                       Optionally the final predict_vel_n_pos (:240-284) is fused after it.
 *   k_pci_integrate     predict_vel_n_pos (pcisph.cl:240-284)
 * The grid barrier spins on a generation counter with a bounded poll count (2^24 polls of at
 * least 64 ns); on timeout the kernel sets SPH_FLAG_TIMEOUT and every CTA returns (the launch
 * is cooperative, so all CTAs are co-resident and the wait ends in practice).  The test of
 * that path injects a stall from the host (sph_inject_fault) instead of faulting anything.
 */
#include "sph_kernels.cuh"

namespace sph {

namespace {
__device__ __forceinline__ float block_max(float v) {
    __shared__ float s_w[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) s_w[w] = v;
    __syncthreads();
    if (w == 0) {
        v = lane < (int)(blockDim.x >> 5) ? s_w[lane] : 0.f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    }
    return v;
}

/* container clamp of both PCISPH integrators */
__device__ __forceinline__ void pci_advance(const Const& c, float4 p, float4 v, float4 fo, float4 fp, float& px,
                                            float& py, float& pz, float& vx, float& vy, float& vz, float& cx,
                                            float& cy, float& cz, float& d, float& vn) {
    const float md = c.mass_def, dt = c.dt, vm = c.vmax;
    const float ax = (fp.x + fo.x) / md, ay = c.g + (fp.y + fo.y) / md, az = (fp.z + fo.z) / md;
    vx = v.x + clampf(ax * dt, -vm, vm);
    vy = v.y + clampf(ay * dt, -vm, vm);
    vz = v.z + clampf(az * dt, -vm, vm);
    px = p.x + vx * dt;
    py = p.y + vy * dt;
    pz = p.z + vz * dt;
    vn = len3(vx, vy, vz);
    cx = clampf(px, (-c.lim_x) / 2.0f, c.lim_x / 2.0f);
    cy = clampf(py, (-c.lim_y) / 2.0f, 10.0f);
    cz = clampf(pz, (-c.lim_z) / 2.0f, c.lim_z / 2.0f);
    d = len3(cx - px, cy - py, cz - pz);
}

/* with the particle's (sorted) position p and pressure force fp */
__device__ __forceinline__ void pci_predict_one(const Const& c, const Bufs& b, int i, float4 p, float4 fp) {
    float px, py, pz, vx, vy, vz, cx, cy, cz, d, vn;
    pci_advance(c, p, __ldg(&b.vel_s[i]), __ldg(&b.f_other[i]), fp, px, py, pz, vx, vy, vz, cx, cy, cz, d, vn);
    if (d > 0.f && vn > 0.f) { px = cx; py = cy; pz = cz; }
    b.pos_pred[i] = make_float4(px, py, pz, 1.f);
}
__device__ __forceinline__ void pci_predict_one(const Const& c, const Bufs& b, int i) {
    pci_predict_one(c, b, i, __ldg(&b.pos_s[i]), b.f_press[i]);
}

__device__ __forceinline__ void pci_integrate_one(const Const& c, const Bufs& b, int i, float4 p, float4 fp) {
    float px, py, pz, vx, vy, vz, cx, cy, cz, d, vn;
    pci_advance(c, p, __ldg(&b.vel_s[i]), __ldg(&b.f_other[i]), fp, px, py, pz, vx, vy, vz, cx, cy, cz, d, vn);
    if (d > 0.f && vn > 0.f) {
        float sx = signf(cx - px), sy = signf(cy - py), sz = signf(cz - pz);
        const float sl = len3(sx, sy, sz);
        sx /= sl; sy /= sl; sz /= sl;
        const float rest = d / (c.dt * vn);
        const float k = (1.0f + rest) * (vx * sx + vy * sy + vz * sz);
        vx -= k * sx; vy -= k * sy; vz -= k * sz;
        px = cx; py = cy; pz = cz;
    }
    b.pos[i] = make_float4(px, py, pz, 1.f);
    b.vel[i] = make_float4(vx, vy, vz, 0.f);
    b.ids[i] = b.ids_s[i];
    const bool bad = !(isfinite(px) && isfinite(py) && isfinite(pz) && isfinite(vx) && isfinite(vy) && isfinite(vz));
    if (bad) atomicOr(b.flags, kFlagNan);
}
__device__ __forceinline__ void pci_integrate_one(const Const& c, const Bufs& b, int i) {
    pci_integrate_one(c, b, i, __ldg(&b.pos_s[i]), b.f_press[i]);
}

/* update_pressure for one particle: predicted density from the fixed lists at x*.  The
 * list is walked SPH_PCI_WALK_DEPTH entries deep, with the next ones' indices loaded during their
 * visits (the sum keeps list order).  x* is written by this kernel, so it is read with plain loads.
 * The updated pressure's p / rho^2 (the initial density, as compute_pressure_force uses it)
 * goes to pci_pc, beside the position, for the force phase: the same IEEE quotient the force
 * phase would form per pair, formed once per particle. */
/* The loop's list walks (walk_list) are bound by the latency of their dependent loads.  Four
 * deep, measured on GB300: the 4M PCISPH step 6.35 ms against 7.20 ms two deep (the 358k step
 * 0.620 against 0.618 ms); three deep 6.58 ms. */
#ifndef SPH_PCI_WALK_DEPTH
#define SPH_PCI_WALK_DEPTH 4
#endif
/* A boundary particle's position and Psi. */
struct BndRec {
    float4 p;
    float phi;
};
__device__ __forceinline__ BndRec load_bnd(const Bufs& b, int j) { return {__ldg(&b.bpos_s[j]), __ldg(&b.bphi_s[j])}; }
/* the boundary walks: four entries deep with one lane, the update's three with several.  A near-wall
 * particle's twenty-odd entries, walked one after the other behind its fluid pairs, were the
 * tail of every phase: 103,823 particles 28.8 -> 23.0 us an iteration. */
constexpr int kBndDepth = 4, kBndSplit = 3;
/* W > 1: W lanes of a particle (small scenes, PHYSICS): each forms the terms of entries w, w +
 * W, ..., and all add them in list order, so the sum is that of one thread.  w >= W: a lane
 * without a particle, which only takes part in the exchange. */
template <bool COMPAT, int W = 1>
__device__ __forceinline__ float pci_update_one(const Const& c, const Bufs& b, int i, int w = 0, bool full = true) {
    const float4 pi = b.pos_pred[i];
    const float H = c.h_def, HH = H * H;
    const size_t n = (size_t)c.n;
    float pd = 0.f, pdb = 0.f;
    const int len = __ldg(&b.nlen[i]);
    const int* __restrict__ e = b.nlist + i;
    /* every product and sum rounded on its own, in the kernel's order (r^2 as dot(r, r),
     * pown(h^2 - r^2, 3), the sum in list order): the result does not depend on how the
     * compiler would contract them */
    auto visit = [&](float4 pj) {
        const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
        const float r2 = r2_exact(dx, dy, dz);
        /* the range test as a select: a rejected pair adds +0 */
        if (COMPAT && c.monaghan) {
            pd += w_monaghan(r2, H, H);   /* W_DEFAULT(r^2, h), Monaghan kernels (pcisph.cl:396) */
        } else {
            const float t = (COMPAT || r2 < HH) ? HH - r2 : 0.f;
            pd = __fadd_rn(pd, __fmul_rn(__fmul_rn(t, t), t));
        }
    };
    const int blen = __ldg(&b.sblen[i]);
    if constexpr (W > 1) {
        auto cube = [&](float4 pj) {
            const float r2 = r2_exact(pi.x - pj.x, pi.y - pj.y, pi.z - pj.z);
            const float t = r2 < HH ? HH - r2 : 0.f;
            return __fmul_rn(__fmul_rn(t, t), t);
        };
        const int most = __reduce_max_sync(0xffffffffu, w < W ? len : 0);
        for (int k0 = 0; k0 < most; k0 += 4 * W) {
            float term[4];
            int j[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int k = k0 + u * W + w;
                j[u] = w < W && k < len ? __ldg(e + k * n) : -1;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) term[u] = j[u] >= 0 ? cube(b.pos_pred[j[u]]) : 0.f;
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int v = 0; v < W; ++v) pd = __fadd_rn(pd, __shfl_sync(0xffffffffu, term[u], v, W));
        }
        const int bmost = __reduce_max_sync(0xffffffffu, w < W ? blen : 0);
        for (int k0 = 0; k0 < bmost; k0 += kBndSplit * W) {
            float term[kBndSplit];
            int j[kBndSplit];
#pragma unroll
            for (int u = 0; u < kBndSplit; ++u) {
                const int k = k0 + u * W + w;
                j[u] = w < W && k < blen ? __ldg(&b.sblist[k * n + i]) : -1;
            }
#pragma unroll
            for (int u = 0; u < kBndSplit; ++u) {
                term[u] = 0.f;
                if (j[u] >= 0) {
                    const BndRec r = load_bnd(b, j[u]);
                    term[u] = __fmul_rn(cube(r.p), r.phi);
                }
            }
#pragma unroll
            for (int u = 0; u < kBndSplit; ++u)
#pragma unroll
                for (int v = 0; v < W; ++v) pdb = __fadd_rn(pdb, __shfl_sync(0xffffffffu, term[u], v, W));
        }
        if (w != 0) return 0.f;
    } else {
        walk_list<SPH_PCI_WALK_DEPTH>(e, n, len, i, [&](int j) { return b.pos_pred[j]; }, visit);
    }
    pd *= c.default_eval * c.mass_def;
    walk_list<kBndDepth>(b.sblist + i, n, W > 1 ? 0 : blen, 0, [&](int j) { return load_bnd(b, j); },
                                 [&](const BndRec& q) {
        const float r2 = r2_exact(pi.x - q.p.x, pi.y - q.p.y, pi.z - q.p.z);
        if (COMPAT && c.monaghan) {
            pdb += w_monaghan(r2, H, H) * q.phi;
        } else if (COMPAT || r2 < HH) {
            const float t = HH - r2;
            pdb = __fadd_rn(pdb, __fmul_rn(__fmul_rn(__fmul_rn(t, t), t), q.phi));
        }
    });
    pdb *= c.default_eval;
    const float e0 = pd + pdb - c.rho0_def;
    const float dv = (0.f < e0) ? e0 : 0.f;
    b.dens_var[i] = dv;
    const float p = __fadd_rn(b.pressure[i], __fmul_rn(dv, c.delta));
    b.pressure[i] = p;
    const float di = __ldg(&b.density[i]);
    const float q = p / (di * di);
    if (!full) {   /* the record has the position already */
        b.pci_pc[i].w = q;
        return dv;
    }
    const float4 ps = __ldg(&b.pos_s[i]);
    b.pci_pc[i] = make_float4(ps.x, ps.y, ps.z, q);   /* one record per neighbour for the force phase */
    return dv;
}

/* compute_pressure_force for one particle (initial density, updated pressure):
 * (p_i / rho_i^2 + p_j / rho_j^2) per pair; the particle's and each neighbour's position and
 * quotient come as one record from pci_pc (written by the update phase of this kernel, so
 * plain loads).  Gives done(record, force) to the particle's (first) lane. */
/* W > 1: W lanes of a particle, their sums in list order (w >= W as in pci_update_one; s_fac as
 * in ordered_walk, three a thread). */
template <bool MON = false, int W = 1, class F>
__device__ __forceinline__ void pci_pressure_force_one(const Const& c, const Bufs& b, int i, int w, float2* s_fac, F&& done) {
    const float4 pi = b.pci_pc[i];
    const float H = c.h_def;
    const size_t n = (size_t)c.n;
    const float C = pi.w;
    float fx = 0.f, fy = 0.f, fz = 0.f, gx = 0.f, gy = 0.f, gz = 0.f;
    const int len = __ldg(&b.nlen[i]);
    const int* __restrict__ e = b.nlist + i;
    auto visit = [&](float4 pj, float cj) {
        const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
        const float r2 = dx * dx + dy * dy + dz * dz;
        if constexpr (MON) {   /* GRAD_W_PRESSURE(r, l, h) with the Monaghan kernels (pcisph.cl:482) */
            const float l = sqrtf(r2);
            if (l >= 1e-5f) {
                float gx, gy, gz;
                grad_w_monaghan(dx, dy, dz, l, H, H, gx, gy, gz);
                const float q = C + cj;
                fx += q * gx;
                fy += q * gy;
                fz += q * gz;
            }
            return;
        }
        const float il0 = rsqrtf(r2), l0 = r2 * il0;
        /* the distance guard as selects: a rejected pair (the particle itself) adds zeros */
        const bool ok = l0 >= 1e-5f;
        const float il = ok ? il0 : 0.f, l = ok ? l0 : H;
        const float q = C + cj;
        const float t = (H - l) * (H - l);
        fx += q * ((dx * il) * t);
        fy += q * ((dy * il) * t);
        fz += q * ((dz * il) * t);
    };
    if constexpr (W > 1) {
        float total[3];
        ordered_walk<W>(i, c.n, b.nlist, w < W ? len : 0, i, s_fac, total, [&](int j) { return b.pci_pc[j]; },
                        [&](float4 pj, bool in, float2 (&f)[3]) {
            /* past the end: zeros, also for a particle that is not a number, whose list is empty */
            const float dx = in ? pi.x - pj.x : 0.f, dy = in ? pi.y - pj.y : 0.f, dz = in ? pi.z - pj.z : 0.f;
            const float r2 = dx * dx + dy * dy + dz * dz;
            const float il0 = rsqrtf(r2), l0 = r2 * il0;
            const bool ok = l0 >= 1e-5f;
            const float il = ok ? il0 : 0.f, l = ok ? l0 : H;
            const float q = in ? C + pj.w : 0.f;
            const float t = (H - l) * (H - l);
            f[0] = make_float2(q, (dx * il) * t);
            f[1] = make_float2(q, (dy * il) * t);
            f[2] = make_float2(q, (dz * il) * t);
        });
        fx = total[0];
        fy = total[1];
        fz = total[2];
    } else {
        walk_list<SPH_PCI_WALK_DEPTH>(e, n, len, i, [&](int j) { return b.pci_pc[j]; },
                                      [&](const float4& v) { visit(v, v.w); });
    }
    const float sf = (-(c.mass_def * c.mass_def)) * c.spiky_grad;
    fx *= sf; fy *= sf; fz *= sf;
    const int blen = __ldg(&b.sblen[i]);
    auto wall = [&](const BndRec& r) {
        const float dx = pi.x - r.p.x, dy = pi.y - r.p.y, dz = pi.z - r.p.z;
        const float l = sqrtf(dx * dx + dy * dy + dz * dz);
        const float q = r.phi * (2.0f * C);
        if constexpr (MON) {
            float wx, wy, wz;
            grad_w_monaghan(dx, dy, dz, l, H, H, wx, wy, wz);
            gx += q * wx;
            gy += q * wy;
            gz += q * wz;
            return;
        }
        const float il = 1.0f / l, t = (H - l) * (H - l);
        gx += q * ((dx * il) * t);
        gy += q * ((dy * il) * t);
        gz += q * ((dz * il) * t);
    };
    if constexpr (W > 1) {
        float total[3];
        ordered_walk<W>(i, c.n, b.sblist, w < W ? blen : 0, 0, s_fac, total, [&](int j) { return load_bnd(b, j); },
                        [&](const BndRec& r, bool in, float2 (&f)[3]) {
            const float dx = pi.x - r.p.x, dy = pi.y - r.p.y, dz = pi.z - r.p.z;
            const float l = sqrtf(dx * dx + dy * dy + dz * dz);
            const float q = r.phi * (2.0f * C);
            const float il = 1.0f / l, t = (H - l) * (H - l);
            f[0] = in ? make_float2(q, (dx * il) * t) : make_float2(0.f, 0.f);
            f[1] = in ? make_float2(q, (dy * il) * t) : make_float2(0.f, 0.f);
            f[2] = in ? make_float2(q, (dz * il) * t) : make_float2(0.f, 0.f);
        });
        gx = total[0];
        gy = total[1];
        gz = total[2];
    } else {
        walk_list<kBndDepth>(b.sblist + i, n, blen, 0, [&](int j) { return load_bnd(b, j); }, wall);
    }
    const float sb = (-c.mass_def) * c.spiky_grad;
    if (w == 0) done(pi, make_float4(fx + gx * sb, fy + gy * sb, fz + gz * sb, 0.f));
}
}  // namespace

template <bool COMPAT>
__global__ void __launch_bounds__(256) k_pci_init_density(Const c, Bufs b) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    b.pressure[i] = 0.f;
    const float4 pi = __ldg(&b.pos_s[i]);
    const float H = c.h_def, HH = H * H;
    float di = 0.f, bdi = 0.f;
    list_neighbors<2, true>(i, c.n, b.nlist, __ldg(&b.nlen[i]), b.pos_s, pi.x, pi.y, pi.z,
                   [&](int, float4, float dx, float dy, float dz) {
                       const float r2 = dx * dx + dy * dy + dz * dz;
                       if (COMPAT && c.monaghan) {   /* W_DEFAULT(r^2, h), Monaghan (pcisph.cl:81) */
                           di += w_monaghan(r2, H, H);
                       } else {
                           const float t = HH - r2;
                           di += (t * t) * t;
                       }
                   });
    list_neighbors(i, c.n, b.sblist, __ldg(&b.sblen[i]), b.bpos_s, pi.x, pi.y, pi.z,
                   [&](int j, float4, float dx, float dy, float dz) {
                       const float r2 = dx * dx + dy * dy + dz * dz;
                       if (COMPAT && c.monaghan) {
                           bdi += w_monaghan(r2, H, H) * __ldg(&b.bphi_s[j]);
                       } else {
                           const float t = HH - r2;
                           bdi += ((t * t) * t) * __ldg(&b.bphi_s[j]);
                       }
                   });
    const float d = c.default_eval * ((di * c.mass_def) + bdi);
    b.density[i] = d;
    b.aux[i] = make_float4(0.f, 1.0f / d, d, 0.f);
}

/* PACK (surface tension on, the normal pass wrote nrec): each neighbour's velocity, normal
 * and 1/rho come from nrec as two adjacent float4 (one 32-byte sector) instead of three
 * loads, and the pair terms use the forms of the WCSPH force pass: 1/r from rsqrtf,
 * (h - r) / rho_j as (h - r) * (1/rho_j), and 2 rho0 / (rho_i + rho_j) as
 * 2 rho0 R_j / (rho_i R_j + 1) with a fast division (FP32 results within a few ulp of the
 * IEEE forms).  Without PACK the pair terms are the kernel text's IEEE divisions. */
/* MON: LAPL_W_VISCOSITY(r, h) with the Monaghan kernels (pcisph.cl:208) instead of h - r. */
/* the walk two deep with the next entries loaded during the visits and a predicated last
 * batch: 4M 0.587 -> 0.557 ms, 358k 0.074 -> 0.066 ms against four deep without them */
#ifndef SPH_PCI_INIT_U
#define SPH_PCI_INIT_U 2
#endif
#ifndef SPH_PCI_INIT_PIPE
#define SPH_PCI_INIT_PIPE 1
#endif
/* W > 1 (small scenes, PACK): W lanes a particle, their sums in list order (ordered_walk). */
template <bool PACK, bool MON = false, int W = 1>
__global__ void __launch_bounds__(256) k_pci_init_forces(Const c, Bufs b) {
    chain_next();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (W == 1 && t >= c.n) return;
    const int w = W > 1 ? (t / W < c.n ? t & (W - 1) : W) : 0;
    const int i = W > 1 ? min(t / W, c.n - 1) : t;
    if (w == 0) b.f_press[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 pi = __ldg(&b.pos_s[i]), vi = __ldg(&b.vel_s[i]), ni = __ldg(&b.normal[i]);
    const float di = __ldg(&b.density[i]);
    const float H = c.h_def;
    const float two_rho0 = 2.0f * c.rho0_def;
    float vx = 0.f, vy = 0.f, vz = 0.f, ux = 0.f, uy = 0.f, uz = 0.f, ox = 0.f, oy = 0.f, oz = 0.f;
    auto pair = [&](int j, float4, float dx, float dy, float dz) {
                       float4 vj, nj;
                       float rn, inv, w, K;
                       const float r2 = dx * dx + dy * dy + dz * dz;
                       if constexpr (PACK) {
                           load_pair(&b.nrec[2 * (size_t)j], vj, nj);
                           const float Rj = nj.w;
                           inv = r2 > 0.f ? rsqrtf(r2) : 0.f;
                           rn = r2 * inv;
                           if constexpr (MON) rn = sqrtf(r2);
                           w = (MON ? lapl_w_monaghan(rn, H, H) : H - rn) * Rj;
                           K = __fdividef(two_rho0 * Rj, di * Rj + 1.0f);
                       } else {
                           vj = __ldg(&b.vel_s[j]);
                           nj = __ldg(&b.normal[j]);
                           const float dj = __ldg(&b.density[j]);
                           rn = sqrtf(r2);
                           w = (MON ? lapl_w_monaghan(rn, H, H) : H - rn) / dj;
                           K = st_corr(c.rho0_def, di, dj);
                           inv = rn > 0.f ? 1.0f / rn : 0.f;
                       }
                       vx += (vj.x - vi.x) * w;
                       vy += (vj.y - vi.y) * w;
                       vz += (vj.z - vi.z) * w;
                       ux += (ni.x - nj.x) * K;
                       uy += (ni.y - nj.y) * K;
                       uz += (ni.z - nj.z) * K;
                       const float sk = st_kernel_sel(rn, H, c.st_term);
                       ox += ((dx * inv) * sk) * K;
                       oy += ((dy * inv) * sk) * K;
                       oz += ((dz * inv) * sk) * K;
                   };
    if constexpr (W > 1) {
        struct Rec {
            float4 p, v, n;
        };
        __shared__ float2 s_fac[256 * 9];
        float total[9];
        ordered_walk<W>(i, c.n, b.nlist, w < W ? __ldg(&b.nlen[i]) : 0, i, s_fac, total, [&](int j) {
            Rec r;
            r.p = __ldg(&b.pos_s[j]);
            load_pair(&b.nrec[2 * (size_t)j], r.v, r.n);
            return r;
        }, [&](const Rec& q, bool in, float2 (&f)[9]) {
            const float dx = __fsub_rn(pi.x, q.p.x), dy = __fsub_rn(pi.y, q.p.y), dz = __fsub_rn(pi.z, q.p.z);
            const float r2 = dx * dx + dy * dy + dz * dz;
            const float Rj = q.n.w;
            const float inv = r2 > 0.f ? rsqrtf(r2) : 0.f;
            const float rn = r2 * inv;
            const float w = in ? (H - rn) * Rj : 0.f;
            const float K = in ? __fdividef(two_rho0 * Rj, di * Rj + 1.0f) : 0.f;
            const float sk = st_kernel_sel(rn, H, c.st_term);
            f[0] = make_float2(q.v.x - vi.x, w);
            f[1] = make_float2(q.v.y - vi.y, w);
            f[2] = make_float2(q.v.z - vi.z, w);
            f[3] = make_float2(ni.x - q.n.x, K);
            f[4] = make_float2(ni.y - q.n.y, K);
            f[5] = make_float2(ni.z - q.n.z, K);
            f[6] = make_float2((dx * inv) * sk, K);
            f[7] = make_float2((dy * inv) * sk, K);
            f[8] = make_float2((dz * inv) * sk, K);
        });
        if (w != 0) return;
        vx = total[0], vy = total[1], vz = total[2];
        ux = total[3], uy = total[4], uz = total[5];
        ox = total[6], oy = total[7], oz = total[8];
    } else {
        list_neighbors<SPH_PCI_INIT_U, SPH_PCI_INIT_PIPE, SPH_PCI_INIT_PIPE>(i, c.n, b.nlist, __ldg(&b.nlen[i]),
                                                                           b.pos_s, pi.x, pi.y, pi.z, pair);
    }
    const float md = c.mass_def;
    const float vsc = (c.mu * (md * md)) * (c.visc_lapl / di);
    const float csc = md * c.st_main;
    const float tsc = (-c.sigma) * md;
    float fx = vx * vsc + tsc * (ux + ox * csc), fy = vy * vsc + tsc * (uy + oy * csc),
          fz = vz * vsc + tsc * (uz + oz * csc);
    b.f_other[i] = make_float4(fx, fy, fz, 0.f);
}

/* The loop's own block size and blocks per SM, whatever the context's; bound by the L1 data
 * pipe once enough walks are in flight, by their latency before.  Scenes of more than three
 * rounds of 5 blocks/SM (583,680 particles) take 6 blocks/SM (40 registers, some spills).
 * Measured on GB300, us a step, 5 and 6 blocks: 357,911 particles 545 / 560; 512,000 769 / 793;
 * 592,704 972 / 945; 778,688 1268 / 1220; 4,194,304 5678 / 5503.  An iteration at 4M takes 7 and
 * 8 blocks/SM 10 to 30 % longer, 128 threads x 12 7 %; 512 threads x 3 gain 1 % there and lose
 * 7 % at 358k. */
constexpr int kLoopThreads = 256, kLoopBlocks = 5, kLoopDense = 6;
constexpr long long kLoopDenseFrom = 3LL * kLoopBlocks * kLoopThreads;   /* particles per SM */
/* W lanes a particle in small scenes (ordered_lanes): with one, a loop of 9,177 particles ran on
 * 36 SMs; measured on GB300, its three iterations 79 -> 47 us. */
/* An iteration's prediction is the epilogue of the force pass before it (as a pass of its own it
 * read and wrote 80 bytes a particle): 4M 538 -> 511 us an iteration, and 503 with the records'
 * positions written in the first iteration only. */
template <bool COMPAT, bool FUSE_INTEGRATE, int W = 1, int BLOCKS = kLoopBlocks>
__global__ void __launch_bounds__(kLoopThreads, BLOCKS) k_pci_loop(Const c, Bufs b, int min_iter, int max_iter) {
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int stride = gridDim.x * blockDim.x;
    const int n = c.n;
    /* the walks: W threads a particle, whole warps */
    const int walks = W > 1 ? (n * W + 31) & ~31 : n;
    auto lane_of = [&](int t) { return W > 1 ? (t / W < n ? t & (W - 1) : W) : 0; };
    auto particle = [&](int t) { return W > 1 ? min(t / W, n - 1) : t; };
    __shared__ float2 s_fac[W > 1 ? 3 * kLoopThreads : 1];
    int it = 1;
    if (max_iter >= 1)
        for (int t = tid; t < walks; t += stride)
            if (lane_of(t) == 0) pci_predict_one(c, b, particle(t));
    for (; it <= max_iter; ++it) {
        if (!grid_barrier(b.barrier, b.flags, (unsigned)c.barrier_extra)) return;
        float lmax = 0.f;
        for (int t = tid; t < walks; t += stride)
            lmax = fmaxf(lmax, pci_update_one<COMPAT, W>(c, b, particle(t), lane_of(t), it == 1));
        lmax = block_max(lmax);
        if (threadIdx.x == 0) atomicMax(reinterpret_cast<unsigned*>(&b.pci_maxerr[it - 1]), __float_as_uint(lmax));
        if (!grid_barrier(b.barrier, b.flags, (unsigned)c.barrier_extra)) return;
        const float mx = *reinterpret_cast<volatile float*>(&b.pci_maxerr[it - 1]);
        bool stop = false;
        if (it >= min_iter) {
            const float crit = COMPAT ? (mx - c.rho0) / c.rho0 : mx / c.rho0;
            stop = crit < c.pci_eta;
        }
        /* the force goes straight into the next prediction, or the step's integration */
        const bool last = stop || it == max_iter;
        auto apply = [&](int i, float4 p, float4 f) {
            if (!last) {
                pci_predict_one(c, b, i, p, f);
            } else {
                b.f_press[i] = f;
                if (FUSE_INTEGRATE) pci_integrate_one(c, b, i, p, f);
            }
        };
        if (COMPAT && c.monaghan) {
            for (int i = tid; i < n; i += stride)
                pci_pressure_force_one<true>(c, b, i, 0, nullptr, [&](float4 p, float4 f) { apply(i, p, f); });
        } else {
            for (int t = tid; t < walks; t += stride) {
                const int i = particle(t);
                pci_pressure_force_one<false, W>(c, b, i, lane_of(t), s_fac, [&](float4 p, float4 f) { apply(i, p, f); });
            }
        }
        if (stop) break;
    }
    if (tid == 0) {
        b.pci_iters[0] = it > max_iter ? max_iter : it;
        if (it > max_iter && !COMPAT) atomicOr(b.flags, kFlagNonconverged);
    }
    if (FUSE_INTEGRATE && max_iter < 1) {
        for (int t = tid; t < walks; t += stride)
            if (lane_of(t) == 0) pci_integrate_one(c, b, particle(t));
    }
}

__global__ void __launch_bounds__(256) k_pci_integrate(Const c, Bufs b) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    pci_integrate_one(c, b, i);
}

/* The loop's three passes as separate launches, for stage-by-stage parity on fields set
 * from outside: the same per-particle functions as k_pci_loop. */
__global__ void __launch_bounds__(256) k_pci_predict(Const c, Bufs b) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < c.n) pci_predict_one(c, b, i);
}

template <bool COMPAT>
__global__ void __launch_bounds__(256) k_pci_update_pressure(Const c, Bufs b) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < c.n) pci_update_one<COMPAT>(c, b, i);
}

/* p / rho^2 of every particle from the pressure and density fields as they stand (the
 * update pass forms it as a by-product in the loop). */
__global__ void __launch_bounds__(256) k_pci_quotient(Const c, Bufs b) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    const float di = b.density[i];
    const float q = b.pressure[i] / (di * di);
    const float4 ps = __ldg(&b.pos_s[i]);
    b.pci_pc[i] = make_float4(ps.x, ps.y, ps.z, q);
}

__global__ void __launch_bounds__(256) k_pci_pressure_force(Const c, Bufs b) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    auto store = [&](float4, float4 f) { b.f_press[i] = f; };
    if (c.monaghan) pci_pressure_force_one<true>(c, b, i, 0, nullptr, store);
    else pci_pressure_force_one(c, b, i, 0, nullptr, store);
}

static inline int nblk(int n, int bs) { return (n + bs - 1) / bs; }

void launch_pci_predict(cudaStream_t s, const Const& c, const Bufs& b, int bs) {
    if (c.n <= 0) return;
    k_pci_predict<<<nblk(c.n, bs), bs, 0, s>>>(c, b);
}
void launch_pci_update_pressure(cudaStream_t s, const Const& c, const Bufs& b, int bs) {
    if (c.n <= 0) return;
    if (c.compat) k_pci_update_pressure<true><<<nblk(c.n, bs), bs, 0, s>>>(c, b);
    else k_pci_update_pressure<false><<<nblk(c.n, bs), bs, 0, s>>>(c, b);
}
void launch_pci_pressure_force(cudaStream_t s, const Const& c, const Bufs& b, int bs) {
    if (c.n <= 0) return;
    k_pci_quotient<<<nblk(c.n, bs), bs, 0, s>>>(c, b);
    k_pci_pressure_force<<<nblk(c.n, bs), bs, 0, s>>>(c, b);
}

void launch_pci_init_density(cudaStream_t s, const Const& c, const Bufs& b, int bs) {
    if (c.n <= 0) return;
    if (c.compat) k_pci_init_density<true><<<nblk(c.n, bs), bs, 0, s>>>(c, b);
    else k_pci_init_density<false><<<nblk(c.n, bs), bs, 0, s>>>(c, b);
}
void launch_pci_init_forces(cudaStream_t s, const Const& c, const Bufs& b, int bs, int num_sms, bool pack) {
    if (c.n <= 0) return;
    if (pack && !c.compat) {
        switch (ordered_lanes(c.n, num_sms)) {
        case 8: launch_chained(s, k_pci_init_forces<true, false, 8>, nblk(8 * c.n, 256), 256, 0, c, b); return;
        case 4: launch_chained(s, k_pci_init_forces<true, false, 4>, nblk(4 * c.n, 256), 256, 0, c, b); return;
        }
    }
    if (c.monaghan) {
        if (pack) k_pci_init_forces<true, true><<<nblk(c.n, bs), bs, 0, s>>>(c, b);
        else k_pci_init_forces<false, true><<<nblk(c.n, bs), bs, 0, s>>>(c, b);
        return;
    }
    if (pack) launch_chained(s, k_pci_init_forces<true>, nblk(c.n, bs), bs, 0, c, b);
    else k_pci_init_forces<false><<<nblk(c.n, bs), bs, 0, s>>>(c, b);
}

static void* loop_fn(bool compat, bool fuse, int w, bool dense) {
    if (compat) return fuse ? (void*)k_pci_loop<true, true> : (void*)k_pci_loop<true, false>;
    if (dense)
        return fuse ? (void*)k_pci_loop<false, true, 1, kLoopDense> : (void*)k_pci_loop<false, false, 1, kLoopDense>;
    if (w == 8) return fuse ? (void*)k_pci_loop<false, true, 8> : (void*)k_pci_loop<false, false, 8>;
    if (w == 4) return fuse ? (void*)k_pci_loop<false, true, 4> : (void*)k_pci_loop<false, false, 4>;
    return fuse ? (void*)k_pci_loop<false, true> : (void*)k_pci_loop<false, false>;
}

LoopBlocks pci_loop_blocks(int num_sms) {
    int most[2] = {kLoopBlocks, kLoopDense};
    for (int dense = 0; dense < 2; ++dense)
        for (int w : {1, 4, 8})
            for (int k = 0; k < 4; ++k) {
                int v = 0;
                void* f = loop_fn((k & 1) != 0, (k & 2) != 0, w, dense != 0);
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, f, kLoopThreads, 0);
                if (v < most[dense]) most[dense] = v;
            }
    return {num_sms * (most[0] < 1 ? 1 : most[0]), num_sms * (most[1] < 1 ? 1 : most[1])};
}

cudaError_t launch_pci_loop(cudaStream_t s, const Const& c, const Bufs& b, int min_iter, int max_iter,
                            const LoopBlocks& fit, int num_sms, bool fuse) {
    if (c.n <= 0) return cudaSuccess;
    const int w = c.compat ? 1 : ordered_lanes(c.n, num_sms);
    const bool dense = !c.compat && c.n > kLoopDenseFrom * num_sms;
    /* the fewest blocks that need no more rounds over the particles, so that no round is nearly
     * empty: 216,000 particles (1.1 rounds of 760 blocks) 54 -> 37 us an iteration */
    const int need = nblk(c.n * w, kLoopThreads), rounds = nblk(need, dense ? fit.dense : fit.plain);
    const int blocks = nblk(need, rounds);
    Const cc = c;
    Bufs bb = b;
    int mi = min_iter, ma = max_iter;
    void* args[] = {&cc, &bb, &mi, &ma};
    return cudaLaunchCooperativeKernel(loop_fn(c.compat != 0, fuse, w, dense), dim3(blocks), dim3(kLoopThreads), args, 0,
                                       s);
}

void launch_pci_integrate(cudaStream_t s, const Const& c, const Bufs& b, int bs) {
    if (c.n <= 0) return;
    k_pci_integrate<<<nblk(c.n, bs), bs, 0, s>>>(c, b);
}

}  // namespace sph
