/*
 * sph_kernels.cuh -- host-side launchers of the SPH kernels (one per reference launch point).
 */
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>

#include "sph_device.cuh"

namespace sph {

/* Device buffers of one context, passed to the launchers. */
struct Bufs {
    /* fluid */
    float4 *pos, *vel, *vhalf;             /* state between steps */
    float4 *pos_s, *vel_s, *vhalf_s;       /* this step's sorted copies */
    float4 *normal, *accel, *pos_pred, *f_other, *f_press;
    float *density, *pressure, *dens_var;
    float4* pci_pc;                        /* PCISPH loop: (x, y, z, p / rho^2), the force phase's record */
    float4* aux;                           /* per particle (p/rho^2, 1/rho, rho, p) */
    float4* nrec;                          /* 2 per particle: (v, p/rho^2), (normal, 1/rho) for the force pass */
    float4* prho;                          /* per particle (x, y, z, rho), written by the list + density pass of
                                              the step for the normal pass (one load per neighbour) */
    uint32_t *keys, *keys_alt;
    int32_t *mask, *mask_alt;
    uint32_t* keys_sorted;                 /* where the sort left the keys */
    int32_t* mask_sorted;
    int32_t *ids, *ids_s;
    int2* tab;                             /* fluid cell table */
    int32_t* cell_prev;                    /* cell id of each sorted particle (sparse clear) */
    int32_t* noff;                         /* 27 linear neighbour-cell offsets (single-scene grid) */
    int32_t *nlist, *nlen, *sblist, *sblen;
    void* sort_ws;
    void* inc_ws;                          /* the incremental sort's workspace (holds the last result) */
    /* boundary */
    float4 *braw, *bpos, *bvel, *bpos_s;
    float *bphi, *bphi_s;
    int32_t *bbody, *bbody_s;
    uint32_t *bkeys, *bkeys_alt;
    int32_t *bmask, *bmask_alt;
    uint32_t* bkeys_sorted;
    int32_t* bmask_sorted;
    int2* btab;
    int32_t* bcell_prev;
    uint8_t* bnear;                        /* per cell: 1 when a boundary particle is binned within one cell */
    void* bsort_ws;
    /* per-body data (device) */
    float* body_xf;                        /* 20 floats per body: rot3x4, lin4, ang4 */
    int32_t* body_range;                   /* origin, count, can_move, has_mass per body */
    float4 *body_force, *body_torque;
    int32_t* bmass;                        /* the boundary particles of bodies with mass */
    float4* bft;                           /* 2 per boundary particle: its fluid force and torque */
    float* body_dyn;                       /* 8 floats per body: dynamic, mass, inv inertia xyz, radius */
    /* batched contexts: scene table and the scene of each fluid particle (ranges never move) */
    const SceneDev* scenes;
    const int32_t* scene_of;
    const SceneTile* tiles;                /* batched: per-scene tiles of 32 particles (Const::ntiles) */
    unsigned* tile_next;                   /* batched: the tile counter (Const::tile_next), zero between launches */
    /* status */
    unsigned* flags;
    int32_t* pci_iters;
    float* pci_maxerr;
    unsigned* barrier;
    double* stats;
};

/* Launches a kernel that begins with chain_next(), with early: so that its blocks may be set up
 * while the kernel before it on the stream still runs (programmatic dependent launch; in a
 * captured step an edge of that kind).  Saves about a microsecond per launch of a chain of
 * short kernels. */
template <class... P, class... A>
inline void launch_early(bool early, cudaStream_t s, void (*kernel)(P...), int grid, int block, size_t smem,
                         A&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = early ? 1 : 0;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
/* The step's launches: early only for grids of at most one block per SM (152 on GB300).  Blocks set up beside
 * a running kernel go where it leaves room, not evenly over the SMs: measured on GB300, a step
 * of 103,823 particles 105 us without, 132 with early launches of its 406-block grids, of
 * 421,875 255 and 291; of 2,197 particles 40.9 and 39.0, of 9,261 42.6 and (this rule) 41.0. */
constexpr int kEarlyBlocks = 152;
template <class... P, class... A>
inline void launch_chained(cudaStream_t s, void (*kernel)(P...), int grid, int block, size_t smem, A&&... args) {
    launch_early(grid <= kEarlyBlocks, s, kernel, grid, block, smem, std::forward<A>(args)...);
}

/* sph_sort.cu */
int sort_passes(int key_bits);
size_t sort_workspace_bytes(int n, int key_bits);
struct SortBufs {
    const uint32_t* kin;
    const int32_t* vin;   /* null: the identity */
    uint32_t* k[4];       /* pass p's output (not its input) */
    int32_t* v[4];
};
void sort_launches(cudaStream_t s, const SortBufs& b, int n, int passes, uint32_t* hist, unsigned* flags,
                   const unsigned* gate, int hblocks, int sblocks);
void sort_pairs_passes(cudaStream_t s, const SortBufs& b, int n, const unsigned* gate, int key_bits, void* ws,
                       unsigned* flags, int num_sms);
void sort_pairs(cudaStream_t s, uint32_t* k0, int32_t* v0, uint32_t* k1, int32_t* v1, int n, int key_bits,
                void* ws, unsigned* flags, int num_sms, uint32_t** kres, int32_t** vres);
/* The stable sort of keys[0, n) (values: the indices) into kout / vout, computed as an update
 * of the previous call's result kept in inc_ws (bytes: sort_inc_workspace_bytes(n), zeroed
 * once before the first call; sort_ws: sort_workspace_bytes(n, key_bits)).  Same result as
 * sort_pairs over (keys, identity) for every input.  side / fork / join (all or none): a
 * second stream and two events on which the gated full sort runs beside the merge. */
size_t sort_inc_workspace_bytes(int n);
/* The step runs the incremental sort's first pass in its hash kernel and its last one in its
 * gather kernel (in_step). */
constexpr int kIncItems = 8;
constexpr int kIncTile = 256 * kIncItems;
struct IncFlags {
    const unsigned* valid;
    const uint32_t* prev;
    uint32_t* bits;
    uint32_t* tcnt;
    unsigned* over;
    int2* list;
    uint32_t* lcount;
};
IncFlags sort_inc_flags_args(void* inc_ws, int n);
struct IncKeep {
    const unsigned* opened;   /* 1: the full sort ran, so the previous keys are to be kept */
    unsigned *over, *valid;
    uint32_t *prev, *first, *sub;
    __device__ __forceinline__ void keep(int j, uint32_t key) const {
        if (over == nullptr) return;   /* keys of another sort */
        if (j == 0) {
            *over = 0u;
            *valid = 1u;
        }
        if (*opened != 0u) {
            prev[j] = key;
            if ((j & 31) == 0) sub[j >> 5] = key;
            if ((j & (kIncTile - 1)) == 0) first[j / kIncTile] = key;
        }
    }
};
IncKeep sort_inc_keep_args(void* inc_ws, int n);
void sort_pairs_incremental(cudaStream_t s, const uint32_t* keys, int n, int key_bits, uint32_t* kout,
                            int32_t* vout, void* inc_ws, void* sort_ws, unsigned* flags, int num_sms,
                            cudaStream_t side = nullptr, cudaEvent_t fork = nullptr, cudaEvent_t join = nullptr,
                            bool in_step = false);

/* sph_grid.cu */
/* scenes: the context's scene table (never null); scene_of: scene of each particle, or
 * null for a single-scene context. */
void launch_hashes(cudaStream_t s, const Const& c, const float4* pos, int n, uint32_t* keys, int32_t* mask,
                   int2* tab, const int32_t* cell_prev, unsigned* flags, int bs, const SceneDev* scenes,
                   const int32_t* scene_of);
void launch_hashes_flags(cudaStream_t s, const Const& c, const float4* pos, int n, uint32_t* keys, int2* tab,
                         const int32_t* cell_prev, unsigned* flags, const SceneDev* scenes, const int32_t* scene_of,
                         const IncFlags& inc);
void launch_gather_ranges(cudaStream_t s, const Const& c, int n, const int32_t* perm, const float4* a, float4* as,
                          const float4* b, float4* bs_, const float4* c3, float4* cs, const int32_t* ids,
                          int32_t* ids_s, const uint32_t* keys, int2* tab, int32_t* cell_out, unsigned* flags, int bs,
                          const SceneDev* scenes, const int32_t* scene_of, const IncKeep& inc);
void launch_gather(cudaStream_t s, int n, const int32_t* perm, const float4* a, float4* as, const float4* b,
                   float4* bs_, const float4* c3, float4* cs, const int32_t* ids, int32_t* ids_s, int bs);
void launch_gather_boundary(cudaStream_t s, int n, const int32_t* perm, const float4* pos, float4* pos_s,
                            const int32_t* body, int32_t* body_s, const float* phi, float* phi_s, int bs);
void launch_cell_ranges(cudaStream_t s, const Const& c, const float4* spos, const uint32_t* keys, int n,
                        int2* tab, int32_t* cell_out, unsigned* flags, int bs, const SceneDev* scenes,
                        const int32_t* scene_of);
void launch_neigh_lists(cudaStream_t s, const Const& c, const float4* spos, const int2* tab, const float4* bpos_s,
                        const int2* btab, int* nlist, int* nlen, int* sblist, int* sblen, int bs,
                        const SceneDev* scenes, const int32_t* scene_of, const uint8_t* bnear,
                        const int32_t* noff = nullptr);

/* sph_wcsph.cu */
void launch_wc_density(cudaStream_t s, const Const& c, const Bufs& b, bool lists, int bs);
/* pack: also write nrec (the force pass then reads 2 adjacent float4 per neighbour instead of
 * velocity, aux and normal); only the fused step uses it */
/* prho: the step's list + density pass wrote b.prho, which the walk then reads for both the
 * neighbour's position and its density.  ordered: several lanes' sums in list order */
void launch_normals(cudaStream_t s, const Const& c, const Bufs& b, bool lists, int bs, int num_sms, bool pack = false,
                    bool prho = false, bool ordered = false);
void launch_wc_forces(cudaStream_t s, const Const& c, const Bufs& b, bool lists, bool fuse_integrate,
                      bool write_acc, int bs, int num_sms, bool pack = false);
void launch_wc_integrate(cudaStream_t s, const Const& c, const Bufs& b, int bs);
void launch_aux(cudaStream_t s, const Const& c, const Bufs& b, int bs);
/* PHYSICS PCISPH: the neighbour lists and compute_initial_density in one pass */
void launch_lists_density_pci(cudaStream_t s, const Const& c, const Bufs& b, int bs, int num_sms);
void launch_lists_density(cudaStream_t s, const Const& c, const Bufs& b, int bs, int num_sms);
/* the list builder writing rows, entries and densities in id order (remap = sorted -> id) */
void launch_lists_density_remap(cudaStream_t s, const Const& c, const Bufs& b, const int32_t* remap, int bs,
                                int num_sms);

/* sph_lists.cu: the same passes for small scenes, several lanes per particle; false (nothing
 * launched) for contexts they do not take */
bool launch_lists_split(cudaStream_t s, const Const& c, const Bufs& b, bool pci, const int32_t* remap, int num_sms);

/* sph_pcisph.cu */
void launch_pci_init_density(cudaStream_t s, const Const& c, const Bufs& b, int bs);
void launch_pci_init_forces(cudaStream_t s, const Const& c, const Bufs& b, int bs, int num_sms, bool pack = false);
/* CTAs of the loop's kernels that run at once: of the plain and of the denser variant */
struct LoopBlocks {
    int plain, dense;
};
LoopBlocks pci_loop_blocks(int num_sms);
cudaError_t launch_pci_loop(cudaStream_t s, const Const& c, const Bufs& b, int min_iter, int max_iter,
                            const LoopBlocks& fit, int num_sms, bool fuse_integrate);
void launch_pci_integrate(cudaStream_t s, const Const& c, const Bufs& b, int bs);
void launch_pci_predict(cudaStream_t s, const Const& c, const Bufs& b, int bs);
void launch_pci_update_pressure(cudaStream_t s, const Const& c, const Bufs& b, int bs);
void launch_pci_pressure_force(cudaStream_t s, const Const& c, const Bufs& b, int bs);

/* sph_boundary.cu */
void launch_bnd_transform(cudaStream_t s, const Bufs& b, int nbodies, int nb, bool compat, bool only_movable,
                          int bs);
void launch_bnd_phi(cudaStream_t s, const Const& c, const Bufs& b, float phi_coeff, int bs);
/* marks bnear (zero before) for the 27 cells around every sorted boundary particle */
void launch_bnd_near(cudaStream_t s, const Const& c, const Bufs& b, int nb, int bs);
/* the fluid's force and torque on every body with mass (nmass particles of such bodies, listed
 * in b.bmass); dynamic: then advances every dynamic body by one step under them and gravity */
void launch_bnd_forces(cudaStream_t s, const Const& c, const Bufs& b, int nbodies, int nmass, bool dynamic, int bs,
                       int num_sms);
void launch_stats(cudaStream_t s, const Const& c, const Bufs& b);
void launch_scene_stats(cudaStream_t s, const Const& c, const Bufs& b, double* out, int nscenes);

}  // namespace sph
