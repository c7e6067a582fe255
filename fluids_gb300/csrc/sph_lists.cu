/*
 * sph_lists.cu -- neighbour lists and density of the fused step for small scenes: several
 * lanes or two threads per particle, on the clamped (PHYSICS) grid.
 *
 *   k_lists_split  compute_neigh_list (kernels/grid.cl:145-182, fluid and boundary) with
 *                  compute_density_pressure (kernels/wcsph.cl:32-79) or, with PCI,
 *                  compute_initial_density (kernels/pcisph.cl:33-102) over the kept pairs:
 *                  the lists, list order, cap and density bits of k_lists_density.
 *
 * k_lists_density walks a particle's 27 cells (about 200 candidates) in one thread.  With
 * fewer particles than the GPU holds threads that walk's latency is the kernel's time,
 * whatever the size.  Here kSplitLanes lanes share a particle: they test as many candidates at
 * a time, in the list's order, and a ballot gives each hit its place.  The density terms go to
 * shared memory by entry, and one lane adds them in list order, so the sum has the order and
 * rounding of the one-thread walk.
 *   k_lists_pair   the same with one thread a particle for the fluid and one for the boundary
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

/* The list pass of scenes with walls that are too large for the lanes above and leave the GPU
 * room for two threads a particle: half of a block's warps scan the fluid's cells as
 * k_lists_density does, the other half the boundary's of the same particles.  k_lists_density
 * takes as long as its longest warp, one that scans both: at 79,507 particles a warp took 57,000
 * cycles in the mean, the kernel 105,000.  Every sum and list is k_lists_density's. */
constexpr int kPairBlock = 256, kPairOf = kPairBlock / 2;
template <bool BATCH, bool PCI>
__global__ void __launch_bounds__(kPairBlock, 6)
    k_lists_pair(Const c0, const float4* __restrict__ spos, const int2* __restrict__ tab,
                 const float4* __restrict__ bpos_s, const int2* __restrict__ btab, const float* __restrict__ bphi_s,
                 int* __restrict__ nlist, int* __restrict__ nlen, int* __restrict__ sblist, int* __restrict__ sblen,
                 float* __restrict__ dens, float* __restrict__ pres, float4* __restrict__ aux,
                 const SceneDev* __restrict__ scenes, const int32_t* __restrict__ scene_of,
                 const uint8_t* __restrict__ bnear, float4* __restrict__ prho) {
    __shared__ float s_bdi[kPairOf];
    chain_next();
    const int slot = threadIdx.x & (kPairOf - 1), i = blockIdx.x * kPairOf + slot;
    const bool walls = threadIdx.x >= kPairOf, live = i < c0.n;
    const SceneDev* const sd = BATCH ? scenes + __ldg(&scene_of[live ? i : 0]) : scenes;
    Const c = c0;
    if (BATCH) apply_scene_grid(c, *sd);
    const long long base = BATCH ? sd->cell_base : 0;
    const float4 p = __ldg(&spos[live ? i : 0]);
    const float hh = PCI ? c.h_def * c.h_def : c.h * c.h;
    const unsigned n4 = 4u * (unsigned)c.n;
    int cx, cy, cz;
    cell_of(c, p.x, p.y, p.z, cx, cy, cz);
    float di = 0.f;
    if (walls) {
        int k = 0;
        if (live && (bnear == nullptr || __ldg(&bnear[base + cell_lin(c, cx, cy, cz)]) != 0)) {
            char* const row = reinterpret_cast<char*>(sblist + i);
            k = build_scan(c, p.x, p.y, p.z, cx, cy, cz, btab + base, bpos_s, sd->noff,
                           [&](bool hit, int j, float r2, int e) {
                if (hit) *list_slot(row, e, n4) = j;
                float w = 0.f;
                if (hit) w = __ldg(&bphi_s[j]);
                const float t = hit ? hh - r2 : 0.f;
                di += ((t * t) * t) * w;
            });
        }
        if (live) sblen[i] = k;
        s_bdi[slot] = di;
    } else if (live) {
        char* const row = reinterpret_cast<char*>(nlist + i);
        nlen[i] = build_scan(c, p.x, p.y, p.z, cx, cy, cz, tab + base, spos, sd->noff,
                             [&](bool hit, int j, float r2, int e) {
            if (hit) *list_slot(row, e, n4) = j;
            const float t = hit ? hh - r2 : 0.f;
            di += (t * t) * t;
        });
    }
    __syncthreads();
    if (walls || !live) return;
    const float bdi = s_bdi[slot];
    float d, pr = 0.f;
    if (PCI) {
        d = c.default_eval * ((di * c.mass_def) + bdi);
    } else {
        di *= c.poly6_eval * c.mass;
        d = di + c.poly6_eval * bdi;
        const float pv = (BATCH ? sd->kgas : c.kgas) * (pown7(d / c.rho0) - 1.0f);
        pr = (0.f < pv) ? pv : 0.f;
    }
    dens[i] = d;
    if (prho) prho[i] = make_float4(p.x, p.y, p.z, d);
    pres[i] = pr;
    aux[i] = PCI ? make_float4(0.f, 1.0f / d, d, 0.f) : make_aux(d, pr);
}

/* The lanes take scenes of up to 400 particles an SM (60,800), or 512 (77,824, two waves of lanes)
 * where there are no walls to scan or the adjoint's tape is written; two threads a particle, up
 * to 768 an SM (116,736, one wave of 6 blocks).  Measured on GB300 (us with the launch gap):
 * particles        2,197  9,261 32,768 54,872 64,000 79,507 103,823 157,464
 * 8 lanes             14     16     30     40     43
 * two threads                       40     42     42     43      46      73
 * k_lists_density     42     47     52     53     49     51      56      63
 * (4 lanes: 21, 23, 31, 43; 16 lanes: 14, 16, 34, 51.)  Longer lists than kMaxCap would not fit
 * the lanes' shared terms. */
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
    if (c.compat || c.wrap) return false;
    const bool two = !remap && c.nb > 0;
    if (c.cap > kMaxCap || c.n > (two ? 400LL : 512LL) * num_sms) {
        if (!two || c.n > 768LL * num_sms) return false;
        auto run = [&](auto kernel) {
            launch_chained(s, kernel, (c.n + kPairOf - 1) / kPairOf, kPairBlock, 0, c, b.pos_s, b.tab, b.bpos_s, b.btab,
                           b.bphi_s, b.nlist, b.nlen, b.sblist, b.sblen, b.density, b.pressure, b.aux, b.scenes,
                           b.scene_of, b.bnear, b.prho);
        };
        if (pci) run(k_lists_pair<false, true>);
        else if (c.batched) run(k_lists_pair<true, false>);
        else run(k_lists_pair<false, false>);
        return true;
    }
    if (remap) split_launch<false, true, false>(s, c, b, remap);
    else if (pci) split_launch<false, false, true>(s, c, b, nullptr);
    else if (c.batched) split_launch<true, false, false>(s, c, b, nullptr);
    else split_launch<false, false, false>(s, c, b, nullptr);
    return true;
}

}  // namespace sph
