// Host entry points of the line-move kernels (esm_linemove_impl.cuh).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "esm_common.cuh"

namespace esm {
template <class real>
size_t linemove_scratch_reals(const DevModel<real> &M);  // per warp
template <class real>
size_t linemove_smem_per_warp(const DevModel<real> &M);  // bytes of one move descriptor
// the moves walked by blocks (k_move_blocks) on `blocks` blocks (0: none, k_move walks every move) with
// smem bytes of shared memory: the separable moves of at least min_units units (0: none) with `region`
// bytes (0: none) and tmp_warp bytes of tmp a warp, and the other moves with walk_region bytes (0: none)
struct SepLaunch {
    int min_units, blocks, smem, region, tmp_warp, walk_region;
    char *tmp;
    int *redo;  // [tasks of a class] FP32: those of a move that the block walk leaves to k_move
};
// the whole class pass in one k_move_wave launch (on = 1), every move one task per lane: done
// holds the moves completed per work item (max_items), err is set when a bounded wait runs out
struct WaveLaunch {
    int on;
    unsigned int *done;
    int *err;
    size_t max_items;
};
template <class real>
int sep_region_bytes(const DevModel<real> &M);
template <class real>
int sep_tmp_bytes(const DevModel<real> &M);
template <class real>
int walk_region_bytes(const DevModel<real> &M);
template <class real>
int move_blocks(const DevModel<real> &M, int nsm, int smem, int max_warps);
// one colour class: the list and the descriptors of its moves into descs ((natoms + nextra) descriptors),
// then per move one k_move launch and one k_move_blocks launch (the kernel that does not take the move
// returns at once); the sweep index is read on the device from *sweep (graph-capturable)
template <class real>
cudaError_t launch_class_pass(const DevModel<real> &M, const int *steps, int nsteps, const uint32_t *sweep, int cls,
                              int limit, real *scratch, int wpb, int max_warps, unsigned long long *stats,
                              char *descs, unsigned int *counters, const SepLaunch &sep, const WaveLaunch &wave,
                              cudaStream_t s);
// resident k_move warps per SM with blocks of wpb (1, 2 or 4) warps
template <class real>
int linemove_blocks_per_sm(const DevModel<real> &M, int wpb);

// ---- a batch of models whose class passes run together: per pass one descriptor launch for all
// models and one k_move_batch launch per move index, each over the tasks of every model that has
// that move (the models sorted by decreasing move count, so those are a prefix of the models)
template <class real>
struct BatchModel {
    DevModel<real> M;           // the model (move log off)
    const int *steps[3];        // the step lists of its colour classes
    int nsteps[3];
    int nmoves;                 // moves of one of its class passes (natoms + nextra)
    char *descs;                // its descriptor buffer: nmoves descriptors of stride bytes
    size_t stride;
    unsigned long long *stats;  // its move counts, laid out as a context's
    int sep_on, walk_region;    // as in its own passes: separable moves from this many units (0: none); walk_run's bytes
};
struct BatchLaunch {
    int nm;                  // models
    int maxpass;             // colour classes per sweep, the most of any model (2, or 3 with an odd T)
    int maxmoves;            // moves per class pass of the first model (the most)
    int npass, nmove;        // the passes and the moves per pass launched (maxpass, maxmoves: all)
    const int *nact;         // host [maxmoves]: the models that have move mi (a prefix)
    int wpb, warps;          // k_move_batch: warps per block (1 or 2) and warps launched
    size_t prep_smem;        // the largest descriptor stride
    void *scratch;           // global walk slabs for the models whose buffers exceed the local arrays
    size_t scratch_per_warp; // reals of one warp's slab (0: no model needs one)
    int *pass_cls;           // device [maxpass * nm]: the class model b runs in pass p (-1: none)
    unsigned int *off;       // device [maxpass * (nm + 1)]: the item prefix over the models of pass p
    unsigned int *choff;     // device [maxpass * (nm + 1)]: the chunk prefix (k_move_blocks_batch)
    unsigned int *counters;  // device [3 * maxpass * maxmoves]: the item, chunk and redo counters of the launches
    unsigned long long *redo;  // device [tasks of a pass] FP32: chunk (high word) and task left to k_move_batch
    int bblocks, region, tmp_warp;  // k_move_blocks_batch: blocks (0: not used), shared memory, sort buffer
    char *tmp;
};
// the passes of one sweep of every model of the batch (the sweep index read from *sweep on the
// device, graph-capturable); the caching rebuild at the sweep start is the caller's
template <class real>
cudaError_t launch_batch_passes(const BatchModel<real> *bm, const BatchLaunch &bl, const uint32_t *sweep,
                                cudaStream_t s);
// resident k_move_batch warps per SM with blocks of wpb (1 or 2) warps; sets the kernels' limits
template <class real>
int batch_warps_per_sm(int wpb);
template <class real>
int batch_blocks_per_sm(int region);

// ---- storage multiscale sweep (esm_plateau.cuh)
#define ESM_PLAT_MAXU 32  // units of one plateau move (a cell-class aggregate)
#define ESM_PLAT_MAXK 8   // dispatchable units at one node taking part in the compensation
// the moves of one class pass, drawn on the host
struct PlatMoves {
    int L, o, cls, li, nb;      // length, offset, block parity, length index, blocks of the class
    int nu[8];                  // units per move
    int j[8][ESM_PLAT_MAXU];    // storage unit indices (into stor)
};
// maxd: the most dispatchable units at a node
// reals of the storage kernels' global scratch (*least: with which they still run, a task at a time)
template <class real>
size_t plateau_scratch_reals(const DevModel<real> &M, int maxd, size_t *least);
template <class real>
cudaError_t launch_plateau(const DevModel<real> &M, int maxd, const PlatMoves &mv, uint32_t sweep, real *scratch,
                           size_t reals, unsigned long long *stats, cudaStream_t s);
// ---- long-range storage sweep: per unit [stor index, moves, (L, a) per move], at most 5 moves
#define ESM_SL_STRIDE 12
template <class real>
cudaError_t launch_storage_long(const DevModel<real> &M, int maxd, const int *plan, int nunits, uint32_t sweep,
                                real *scratch, size_t reals, unsigned long long *stats, cudaStream_t s);
}  // namespace esm
