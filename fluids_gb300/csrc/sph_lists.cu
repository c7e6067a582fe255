/*
 * sph_lists.cu -- neighbour lists and density of the fused step for small scenes: several
 * lanes per particle, on the clamped (PHYSICS) grid.
 *
 *   k_lists_split  compute_neigh_list (kernels/grid.cl:145-182, fluid and boundary) with
 *                  compute_density_pressure (kernels/wcsph.cl:32-79) or, with PCI,
 *                  compute_initial_density (kernels/pcisph.cl:33-102) over the kept pairs:
 *                  the lists, list order, cap and density bits of k_lists_density.
 *
 * k_lists_density walks a particle's 27 cells (about 200 candidates) in one thread.  With
 * fewer particles than the GPU holds threads that walk's latency is the kernel's time,
 * whatever the size.  Here kSplitLanes lanes share a particle: they test as many candidates at a
 * time, in the list's order, and a ballot gives each hit its place.  The density terms go to shared memory
 * by entry, and one lane adds them in list order, so the sum has the order and rounding of
 * the one-thread walk.
 */
#include "sph_kernels.cuh"

namespace sph {

namespace {
constexpr int kSplitThreads = 256;
constexpr int kPer = kSplitThreads / kSplitLanes;
constexpr unsigned kAll = 0xffffffffu;

}  // namespace

/* REMAP (the adjoint's tape, particles in id order): the list of sorted particle i is row
 * remap[i] with entries remap[j], and its density, pressure and aux go to remap[i]. */
template <bool BATCH, bool REMAP, bool PCI>
__global__ void __launch_bounds__(kSplitThreads)
    k_lists_split(Const c0, const float4* __restrict__ spos, const int2* __restrict__ tab,
                  const float4* __restrict__ bpos_s, const int2* __restrict__ btab, const float* __restrict__ bphi_s,
                  int* __restrict__ nlist, int* __restrict__ nlen, int* __restrict__ sblist, int* __restrict__ sblen,
                  float* __restrict__ dens, float* __restrict__ pres, float4* __restrict__ aux,
                  const SceneDev* __restrict__ scenes, const int32_t* __restrict__ scene_of,
                  const int32_t* __restrict__ remap, unsigned* __restrict__ flags, const uint8_t* __restrict__ bnear,
                  float4* __restrict__ prho, const float4* __restrict__ vel, float4* __restrict__ rec) {
    extern __shared__ float2 s_term[];   /* per particle: cap entries, padded to an odd number */
    __shared__ int2 s_rng[kPer][27];
    chain_next();
    const int g = threadIdx.x & (kSplitLanes - 1), slot = threadIdx.x / kSplitLanes;
    const int i = blockIdx.x * kPer + slot;
    const bool live = i < c0.n;
    Const c = c0;
    const long long base = scene_setup_t<BATCH>(c, scenes, scene_of, live ? i : 0);
    const float4 p = __ldg(&spos[live ? i : 0]);
    int cx, cy, cz;
    cell_of(c, p.x, p.y, p.z, cx, cy, cz);
    bool near_b = false;
    if (!REMAP && c.nb > 0)
        near_b = live && (bnear == nullptr || __ldg(&bnear[base + cell_lin(c, cx, cy, cz)]) != 0);
    const int row = REMAP ? __ldg(&remap[live ? i : 0]) : i;
    const unsigned n4 = 4u * (unsigned)c.n;
    const float hd = PCI ? c.h_def : c.h;
    float2* const term = s_term + slot * (c.cap | 1);
    const int k = split_scan(c.nx, c.ny, c.nz, cx, cy, cz, live, c.h2_list, c.cap, tab + base, spos, p, g,
                                s_rng[slot], [&](int e, int j, float r2) {
        *list_slot(reinterpret_cast<char*>(nlist + row), e, n4) = REMAP ? __ldg(&remap[j]) : j;
        const float t = __fmaf_rn(hd, hd, -r2);
        term[e] = make_float2(__fmul_rn(t, t), t);
    });
    float di = 0.f, bdi = 0.f;
    int kb = 0;
    if (live && g == 0) {
#pragma unroll 4
        for (int e = 0; e < k; ++e) di = __fmaf_rn(term[e].x, term[e].y, di);
    }
    if (!REMAP && __any_sync(kAll, near_b)) {
        kb = split_scan(c.nx, c.ny, c.nz, cx, cy, cz, near_b, c.h2_list, c.cap, btab + base, bpos_s, p, g,
                           s_rng[slot], [&](int e, int j, float r2) {
            *list_slot(reinterpret_cast<char*>(sblist + i), e, n4) = j;
            const float t = __fmaf_rn(hd, hd, -r2);
            term[e] = make_float2(__fmul_rn(__fmul_rn(t, t), t), __ldg(&bphi_s[j]));
        });
        if (g == 0) {
#pragma unroll 4
            for (int e = 0; e < kb; ++e) bdi = __fmaf_rn(term[e].x, term[e].y, bdi);
        }
    }
    if (!live || g != 0) return;
    nlen[row] = k;
    if (REMAP && k >= c.cap) atomicOr(flags, kFlagOverflow);
    if (!REMAP) sblen[i] = kb;
    float d, pr = 0.f;
    if (PCI) {
        d = c.default_eval * __fmaf_rn(di, c.mass_def, bdi);
    } else {
        d = __fmaf_rn(c.poly6_eval, bdi, __fmul_rn(di, c.poly6_eval * c.mass));
        const float pv = c.kgas * (pown7(d / c.rho0) - 1.0f);
        pr = (0.f < pv) ? pv : 0.f;
    }
    dens[row] = d;
    if (prho) prho[row] = make_float4(p.x, p.y, p.z, d);
    pres[row] = pr;
    const float4 ax = PCI ? make_float4(0.f, 1.0f / d, d, 0.f) : make_aux(d, pr);
    aux[row] = ax;
    if (REMAP) store_rec(rec, row, p, __ldg(&vel[row]), ax);
}

/* The pass takes scenes of up to two waves of lanes (77,824 particles on 152 SMs): measured on
 * GB300, this kernel against k_lists_density (with the launch gap): 2,197 particles 14 against
 * 42 us, 9,261 16 / 47, 32,768 30 / 48, 64,000 43 / 49, 125,000 75 / 60.  4 lanes: 21, 23, 31,
 * 43, 71; 16 lanes: 14, 16, 34, 51, 93.  Longer lists than kMaxCap would not fit the shared
 * terms. */
constexpr int kMaxCap = 128;

template <bool BATCH, bool REMAP, bool PCI>
static void split_launch(cudaStream_t s, const Const& c, const Bufs& b, const int32_t* remap) {
    /* the adjoint's steps are not captured, and early launches save more there */
    const int grid = (c.n + kPer - 1) / kPer;
    launch_early(REMAP || grid <= kEarlyBlocks, s, k_lists_split<BATCH, REMAP, PCI>, grid, kSplitThreads,
                   sizeof(float2) * kPer * (size_t)(c.cap | 1), c, b.pos_s, b.tab, b.bpos_s, b.btab, b.bphi_s, b.nlist,
                   b.nlen, b.sblist, b.sblen, b.density, b.pressure, b.aux, b.scenes, b.scene_of, remap, b.flags,
                   b.bnear, b.prho, b.vel_s, b.nrec);
}

bool launch_lists_split(cudaStream_t s, const Const& c, const Bufs& b, bool pci, const int32_t* remap, int num_sms) {
    if (c.compat || c.wrap || c.cap > kMaxCap || c.n > 2 * 2048LL * num_sms / kSplitLanes) return false;
    if (remap) split_launch<false, true, false>(s, c, b, remap);
    else if (pci) split_launch<false, false, true>(s, c, b, nullptr);
    else if (c.batched) split_launch<true, false, false>(s, c, b, nullptr);
    else split_launch<false, false, false>(s, c, b, nullptr);
    return true;
}

}  // namespace sph
