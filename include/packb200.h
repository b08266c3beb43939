/*
 * packb200.h -- C ABI of the B200 (sm_100a) packing hot path.
 *
 * Every entry point returns an int status: PK_OK (0) on success, a negative
 * PK_E* code otherwise, with a message readable through pk_last_error().
 * Nothing here traps or aborts.  Pointers are device pointers unless a name
 * says "host".  `stream` is a cudaStream_t passed as void* (NULL = legacy
 * default stream).  All launches are asynchronous on that stream.
 *
 * Layouts (reference core/pack_cuda.py:1040-1064, 1186-1207):
 *   xyt   float32 C-contiguous (E, n, 3) = [x, y, theta(rad)] per tree
 *   h     float32 (E, 3) = [square side, x offset, y offset]
 *   cost  float32 (E,)      grad float32 (E, n, 3)   grad_h float32 (E, 3)
 * Ragged batches pack the trees of instance e at rows offsets[e] ..
 * offsets[e+1]-1 of a (sum n, 3) array; offsets is int32 (E+1,).
 *
 * Outputs are caller-allocated and fully overwritten (no zeroing needed).
 */
#ifndef PACKB200_H
#define PACKB200_H

#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

#define PK_OK 0
#define PK_EINVAL -1      /* bad argument (shape, size, null pointer) */
#define PK_ECUDA -2       /* CUDA runtime error */
#define PK_ENOTINIT -3    /* pk_init not called on this device */
#define PK_ERANGE -4      /* size beyond a documented maximum */

#define PK_NUM_PIECES 4
#define PK_MAX_TREE_VERTS 16
#define PK_MAX_TREES 1024     /* trees per instance in the cost / relax kernels */
#define PK_MAX_LAP_N 256      /* Hungarian matrix side (reference: 200) */

/* Tree geometry: convex pieces (any orientation; the library makes them
 * CCW as shapely.orient does, pack_cuda.py:824-826) and the outline used by
 * the boundary cost.  Replaces kaggle_support.py:241-354 +
 * pack_cuda.py:787-849 (_build_convex_piece_arrays). */
typedef struct PkGeometry {
    double piece_xy[PK_NUM_PIECES][4][2];
    int piece_nv[PK_NUM_PIECES];          /* 3 or 4 */
    double tree_xy[PK_MAX_TREE_VERTS][2];
    int n_tree_verts;                     /* <= 16 */
    double max_radius;                    /* max |vertex| of the outline */
    double area;                          /* outline area (informational) */
    /* Legality tree (pk_validate_fp64): the Kaggle metric's unexpanded tree
     * (pack_metric.py:27-79) in the same pose frame, i.e. offset by the
     * search tree's centroid (pack_io.py:150-158).  has_legal = 0: the search
     * geometry above is used for legality too. */
    int has_legal;
    double legal_piece_xy[PK_NUM_PIECES][4][2];
    double legal_tree_xy[PK_MAX_TREE_VERTS][2];
} PkGeometry;

/* Fills *out with the reference Christmas tree (kaggle_support.py:241-324)
 * for a given TREE_EXPANSION (kaggle_support.py:98 uses 20*(1.000001-1)),
 * recentred on its centroid. */
int pk_default_geometry(double tree_expansion, PkGeometry* out);

/* Uploads the geometry to the current device; geom NULL = default tree.
 * Must be called once per device before any compute call.  Replaces the
 * lazy _ensure_initialized of pack_cuda.py:852-1032 (no runtime nvcc). */
int pk_init(const PkGeometry* geom);

/* Message of the last failing call on this host thread. */
const char* pk_last_error(void);

/* ---- cost and gradient (pack_cuda.py, pack_cuda_lut.py) --------------- */

#define PK_PAIR_NONE 0
#define PK_PAIR_AREA 1        /* overlap area,  CollisionCostOverlappingArea */
#define PK_PAIR_SEP 2         /* sum of sep^2,  CollisionCostSeparation */
#define PK_PAIR_LUT 3         /* LUT lookup,    pack_cuda_lut */

/* LUT grid (pack_cuda_lut.py:30-86, constants :653-695).  vals is a device
 * float32 (nx, ny, nt) C-order table over X (x >= one negative sample,
 * mirrored), Y and theta. */
typedef struct PkLut {
    const float* vals;
    int nx, ny, nt;
    float x_min, x_max, y_min, y_max, t_min, t_max;
    int quadratic;        /* apply max(0, v)^2 per pair */
} PkLut;

/* One fused pass per instance: total = w_area*h0^2 + w_boundary*boundary +
 * w_pair*pairs, as CostCompound sums its terms (pack_cost.py:245-277).
 * fixed_h zeroes grad_h (Cost.compute_cost, pack_cost.py:178-195). */
typedef struct PkCostSpec {
    int pair_mode;        /* PK_PAIR_* */
    float w_pair;
    float w_boundary;     /* 0 disables the boundary term (h may be NULL) */
    float w_area;         /* AreaCost of a square: h0^2 (kaggle_support.py:803-816) */
    int fixed_h;
    PkLut lut;            /* used when pair_mode == PK_PAIR_LUT */
    int symmetry;         /* 0 or 1: xyt holds every tree; 2 / 4: xyt holds the genotype of a
                             180 / 90 degree symmetric packing (SolutionCollectionSquareSymmetric180
                             / 90, kaggle_support.py:1272-1393 / 1039-1195): the cost is that of the
                             2 n / 4 n image trees and the gradient is the genotype's */
} PkCostSpec;

/* Compound cost over a uniform (offsets == NULL, all n_uniform trees) or
 * ragged batch.  grad / grad_h may be NULL.  Deterministic: an instance's
 * result does not depend on the rest of the batch.  No scratch memory.
 * Replaces CostCompound.compute_cost over pack_cuda.overlap_multi_ensemble
 * (pack_cuda.py:1040), boundary_distance_multi_ensemble (:1186) and
 * pack_cuda_lut.overlap_multi_ensemble (pack_cuda_lut.py:783). */
int pk_cost(const float* xyt, const int* offsets, int E, int n_uniform, const float* h,
            const PkCostSpec* spec, float* cost, float* grad, float* grad_h, void* stream);

/* pk_cost on a part of a launch order: the count instances order[0 ..
 * count-1] (order is required) of a batch of E, n_max bounding their
 * sizes, threads per CTA (0: the default for n_max; else a multiple of 32 in
 * [32, 256] with 8 * threads >= n_max - 1).  Instances keep their indices in
 * every array, so calls with disjoint parts of one largest-first order --
 * size classes of a ragged batch, on different streams -- fill the same
 * outputs side by side.  Results equal pk_cost's bit for bit. */
int pk_cost_ordered(const float* xyt, const int* offsets, const int* order, int count, int E, int n_max,
                    const float* h, const PkCostSpec* spec, int threads, float* cost, float* grad, float* grad_h,
                    void* stream);

/* pk_cost_ordered for every size class of a largest-first order: class k is
 * order[start .. start + count - 1] (the classes cover it once), none with more
 * than n_max trees, on CTAs of `threads` (0: the library's choice), on
 * stream side[k], forked from and joined to `stream` (a single class runs on
 * `stream` itself).  A batch that the GPU takes in a few waves of the largest
 * class's CTAs goes in one launch on `stream` instead, with the library's choice
 * of threads; the classes' bounds hold all the same (a packing beyond its
 * class's n_max costs NaN), and a class with bad threads or n_max is refused.
 * The same results either way. */
typedef struct PkSizeClass { int start, count, n_max, threads; } PkSizeClass;
int pk_cost_classes(const float* xyt, const int* offsets, const int* order, const PkSizeClass* classes, int n_classes,
                    int E, int n_max, const float* h, const PkCostSpec* spec, float* cost, float* grad, float* grad_h,
                    void* stream, void* const* side);

/* pack_cuda.overlap_multi_ensemble(xyt, xyt, use_separation, out_cost,
 * out_grads) (pack_cuda.py:1040-1183), non-periodic form. */
int pk_overlap(const float* xyt, int E, int n, int use_separation, float* cost, float* grad,
               void* stream);

/* Periodic form of pk_overlap (overlap_multi_ensemble with crystal_axes,
 * pack_cuda.py:1040-1183; kernel :254-464 with ENABLE_CRYSTAL_AXES): every
 * tree against every tree's images under cx A + cy B, |cx|, |cy| <=
 * n_periodic, crystal_axes (E, 4) = [ax, ay, bx, by] float32.  Images of a
 * tree itself count half (all of it with only_self, which keeps only those)
 * and add no gradient, as in the reference.  grad nullable. */
int pk_overlap_crystal(const float* xyt, int E, int n, int use_separation, const float* crystal_axes, int only_self,
                       int n_periodic, float* cost, float* grad, void* stream);

/* pack_cuda.boundary_distance_multi_ensemble (pack_cuda.py:1186-1295). */
int pk_boundary(const float* xyt, const float* h, int E, int n, float* cost, float* grad,
                float* grad_h, void* stream);

/* pack_cuda_lut.overlap_multi_ensemble (pack_cuda_lut.py:783-862); ragged
 * batches allowed through offsets. */
int pk_overlap_lut(const float* xyt, const int* offsets, int E, int n_uniform, const PkLut* lut,
                   float* cost, float* grad, void* stream);


/* Fills vals (nx, ny, nt) with the analytic pair cost (PK_PAIR_AREA or
 * PK_PAIR_SEP) of a tree at the origin against one at (X[ix], Y[iy], T[it])
 * -- the LUT that CollisionCost._ensure_lut_initialized builds through
 * LookupTable.build_from_function (pack_cost.py:322-377,
 * pack_cuda_lut.py:90-169), evaluated on the GPU.  X, Y, T are device
 * float32 vectors. */
int pk_lut_build(const float* X, int nx, const float* Y, int ny, const float* T, int nt, int pair_mode,
                 float* vals, void* stream);

/* Fills vals (nx, ny, nt) with the exact signed separation of a tree at the
 * origin and one at (X[ix], Y[iy]) rotated by T[it]: + the distance to the
 * boundary of their Minkowski difference (the union of the 16 convex piece
 * differences) when the trees overlap, - that distance when they do not --
 * pack_minkowski.separation_distance (pack_minkowski.py:210-266), the
 * function CollisionCostExactSeparation tabulates through
 * LookupTable.build_from_function (pack_cost.py:1144-1215), evaluated in FP64
 * on the GPU.  Each slice uses the rotation angle the reference's float32
 * theta gives through np.degrees and shapely's rotate.  X, Y, T are device
 * float32 vectors; synchronises the stream. */
int pk_lut_build_exact_sep(const float* X, int nx, const float* Y, int ny, const float* T, int nt,
                           float* vals, void* stream);

/* ---- batched linear assignment (lap_batch.py) ------------------------- */

/* Hungarian on B float32 N x N matrices (solve_lap_batch with the default
 * LAPConfig, lap_batch.py:457-534; kernel :62-165, totals :173-196).
 * Assignments and totals are bit-identical to the reference's sequential
 * kernel.  row_match int32 (B, N); total float32 (B,); status int32 (B,)
 * nullable: 1 where a problem had no finite augmenting slack (rows -1,
 * total NaN).  N <= 256.  No scratch memory. */
int pk_lap_solve(const float* C, int B, int N, int* row_match, float* total, int* status, void* stream);

/* Diversity between two sets of packings (compute_genetic_diversity_matrix,
 * kaggle_support.py:2014-2129): for every (pop, ref) pair the minimum over
 * the 8 symmetry transforms (transform != 0; else identity only) of the
 * optimal assignment cost with entries sqrt(dx^2 + dy^2 + wrap(dtheta)^2).
 * pop (Np, n, 3), ref (Nr, n, 3) float32; out (Np, Nr).  Cost rows are
 * generated inside the assignment kernel; no (8 Np Nr, n, n) tensor. */
int pk_diversity_matrix(const float* pop, const float* ref, int Np, int Nr, int n, int transform, float* out,
                        void* stream);

/* The same result with the caller's scratch: work is a 128-byte aligned device
 * array of at least pk_diversity_work_floats(Np, Nr, n, transform) floats
 * (asked with the launch's device current), in which every running warp keeps
 * the cost matrix of its problem (1.4 to 2 times faster).  Calls that may
 * overlap need a work array each. */
int pk_diversity_matrix_work(const float* pop, const float* ref, int Np, int Nr, int n, int transform, float* out,
                             float* work, size_t work_floats, void* stream);
size_t pk_diversity_work_floats(int Np, int Nr, int n, int transform);

/* The (transforms * Np * Nr, n, n) cost matrices of the same computation
 * in the reference's stacking order (kaggle_support.py:2118-2119). */
int pk_diversity_costs(const float* pop, const float* ref, int Np, int Nr, int n, int transform, float* out,
                       void* stream);

/* compute_diversity_shortcut_kernel (lap_batch.py:537-607, kernel :216-331). */
int pk_diversity_shortcut(const float* pop, const float* ref, int Np, int Nr, int n, float cos_a, float sin_a,
                          int mirror, float* out, void* stream);

/* ---- FP64 legality (pack_metric.py) ------------------------------------ */

/* Strict FP64 check of E packings of n trees: overlaps[e] = number of tree
 * pairs whose interiors intersect (pack_metric.score's "intersects and not
 * touches", :134-141: touching is legal), side[e] = side of the smallest
 * axis-aligned square holding every tree (max of the bounding box's width
 * and height, :144-147), both on the legality tree in double precision.
 * xyt is float32 (dtype_bytes 4) or float64 (8), (E, n, 3).  n <= 1024. */
int pk_validate_fp64(const void* xyt, int dtype_bytes, int E, int n, int* overlaps, double* side, void* stream);

/* ---- batched L-BFGS (lbfgs_torch_parallel.py) ------------------------- */

/* One phase of one iteration of lbfgs (lbfgs_torch_parallel.py:411-729,
 * line_search_fn=None) for M systems of N parameters, history m, while the
 * objective stays with the caller.  arrays[17] = device pointers, in order:
 * x, g, loss, d, prev_g, prev_loss, loss0 (M,N)/(M,) of the dtype;
 * S, Y (M, m, N); ro (M, m); H, t (M,); hlen, hstart, evals, active (M,)
 * int32; any_active (1,) int32.  dtype_bytes 4 (float32) or 8 (float64).
 *   phase 0 init:      p0 = tolerance_grad
 *   phase 1 direction: p0 = lr, p1 = max_step, i1 = has max_step, p2 = tolerance_change
 *   phase 2 step:      x += t d
 *   phase 3 update:    p0 = tolerance_grad, p1 = tolerance_change,
 *                      p2 = tolerance_rel_change, i1 = stop_on_cost_increase, i2 = max_eval */
int pk_lbfgs_phase(int phase, int dtype_bytes, void* const* arrays, int M, int N, int m, int n_iter, double p0,
                   double p1, double p2, double p3, int i1, int i2, void* stream);

/* Iteration n_iter (1, 2, ...) of the same loop without a line search, up to and
 * including its step, in two launches: phase 3 of the iteration before (phase 0
 * for n_iter = 1) with loss and gradient at the current x, phase 1, and x += t d
 * if any system is active.  The arrays of pk_lbfgs_phase, with any_active int32
 * (2,), zero before the first call; arrays[1] and arrays[2] (gradient, loss) may
 * be the objective's own output.  host_flag: pinned host memory that holds, once
 * the stream has been waited for, whether any system is active. */
typedef struct PkLbfgsParams {
    double lr, max_step, tol_grad, tol_change, tol_rel_change;
    int has_max_step, stop_on_cost_increase, max_eval;
} PkLbfgsParams;
int pk_lbfgs_iterate(int dtype_bytes, void* const* arrays, int M, int N, int m, int n_iter, const PkLbfgsParams* params,
                     int* host_flag, void* stream);

/* Batched strong-Wolfe line search of the drop-in lbfgs
 * (_strong_wolfe_batched, lbfgs_torch_parallel.py:70-407, with its defaults
 * c1 = 1e-4, c2 = 0.9, tolerance_change = 1e-9, max_ls = 25 as the main loop
 * calls it, :613-617).  A per-system state machine run in phases by the
 * host, which calls the objective between them on the rows the reference
 * evaluates:
 *   0 init (g . d, |d|max, first trial x + t d)      -> objective on rows with in_ls, is_main
 *   1 after an evaluation (g_new . d, count; flag_arg = 1 for the first one)
 *   2 bracketing pass (ls_iter)                       -> flag: any active -> objective on active rows
 *   3 zoom start (flag_arg = 1 when the bracketing ran out of evaluations)
 *   4 zoom pass before its evaluation (tol_change)   -> flag: any active -> objective on active rows
 *   5 zoom bracket update after the evaluation
 *   6 result: t, f_new, g_new of each searched system
 * arrays: x, d, g, f, gtd, t, x_new, g_new, f_new, gtd_new, g_prev, f_prev,
 * gtd_prev, t_prev, bg (M,2,N), bt, bf, bgtd (M,2), d_norm, t_new (dtype of
 * dtype_bytes), then int32: bsize, done, active, low, insuf, evals, in_ls,
 * flag (1).  Replaces the reference's module-private helper, split at its
 * objective evaluations. */
int pk_wolfe_phase(int phase, int dtype_bytes, void* const* arrays, int M, int N, int ls_iter, double c1, double c2,
                   double tol_change, int flag_arg, void* stream);

/* After a search (:621-624, :632): rows with in_ls take x += t d and the
 * search's loss and gradient; evals are adjusted so the history phase leaves
 * func_evals += ls_evals for them and += 0 for the rest. */
int pk_wolfe_apply(int dtype_bytes, void* x, void* g, void* loss, int* evals, const void* d, const void* t,
                   const void* f_new, const void* g_new, const int* in_ls, const int* ls_evals, int M, int N,
                   void* stream);

typedef struct PkRelaxParams {
    int max_iter;             /* n_iterations */
    int history;              /* history_size, 1..64 */
    float lr;
    float max_step;
    int has_max_step;
    float tol_grad;           /* pack_dynamics passes 0 (pack_dynamics.py:127-137) */
    float tol_change;         /* 0 there too */
    float tol_rel_change;
    int stop_on_cost_increase;
    int max_eval;             /* reference default max_iter * 5 / 4 */
    int final_eval;           /* 1: loss_out is the cost at the returned x */
    unsigned long long* counters;  /* device (6,) or NULL: enumerated pairs, near pairs,
                                      piece pairs, cost evaluations, iterations,
                                      history entries streamed -- accumulated */
    int threads;              /* threads per packing: 0 = library default for n_max, else
                                 a multiple of 32 in [32, 256] with 8 * threads >= n_max - 1
                                 (an autotuned choice); results do not depend on it */
    int persistent;           /* 1: one CTA per resident slot, each walking the launch
                                 order with the grid's stride; 0: one CTA per packing */
} PkRelaxParams;

/* Fused batched relaxation (OptimizerBFGS.run_simulation,
 * pack_dynamics.py:54-149, over lbfgs :411-729): one launch relaxes every
 * instance to max_iter with the compound cost of *spec, x = [xyt, h].
 * Uniform (offsets NULL, n_max trees each) or ragged (offsets, n_max >= every
 * size) batches; order (nullable) is a permutation of instances giving the
 * launch order (largest first balances ragged batches).  xyt_out may alias
 * xyt_in.  loss_out (E,) float32; iters_out (E,) int32 nullable.
 * work: pk_relax_workspace_floats() floats of device scratch for the
 * L-BFGS history.  An instance stops when it turns inactive, so its result
 * does not depend on the rest of the batch. */
int pk_relax(const float* xyt_in, const float* h_in, const int* offsets, const int* order, int E, int n_max,
             const PkCostSpec* spec, const PkRelaxParams* params, float* xyt_out, float* h_out, float* loss_out,
             int* iters_out, float* work, void* stream);

/* pk_relax on a part of the launch order: the count instances order[0 ..
 * count-1] (order is required), with n_max bounding only their sizes and
 * prm->threads sized for them; instances keep their indices 0 .. E-1 in
 * every array, so several calls with disjoint parts of one largest-first
 * order fill the same outputs and share one work buffer.  Launched on
 * different streams, the parts -- size classes of a ragged batch, each with
 * CTAs sized for its own trees -- run side by side.  Results equal
 * pk_relax's bit for bit. */
int pk_relax_ordered(const float* xyt_in, const float* h_in, const int* offsets, const int* order, int count, int E,
                     int n_max, const PkCostSpec* spec, const PkRelaxParams* prm, float* xyt_out, float* h_out,
                     float* loss_out, int* iters_out, float* work, void* stream);

/* ---- serving: resumable device-resident relaxation jobs ---------------- */

#define PK_JOB_NEW 0
#define PK_JOB_RUNNING 1
#define PK_JOB_DONE 2

/* One relaxation job of the serving loop.  Its state lives in a caller pool:
 * pool[x_off ..] = x (3n + 3: xyt then h), g (3n + 3), ro (history);
 * pool[h_off ..] = S, Y (2 * history * (3n + 3)).  The caller writes x and
 * sets status = PK_JOB_NEW; the library fills the rest. */
typedef struct PkJob {
    int n;
    int max_iter;
    long long x_off;
    long long h_off;
    int status;
    int it, evals, hlen, hstart;
    float H, loss, loss0;
} PkJob;

/* Advances every job listed (device int32 indices into jobs, largest n
 * first balances the launch) by up to chunk_iters L-BFGS iterations of the
 * compound cost *spec; params->history and the step / tolerance settings
 * apply to all jobs, each job's own max_iter to itself; the final loss is
 * evaluated at the returned x.  A job's result does not depend on which
 * jobs share its launches or on how its iterations are split into chunks.
 * The continuous-batching form of pack_dynamics.run_simulation_list
 * (pack_dynamics.py:152-236), which runs one blocking relaxation per tree
 * count. */
int pk_relax_jobs(PkJob* jobs, const int* list, int njobs, float* pool, int n_max, const PkCostSpec* spec,
                  const PkRelaxParams* params, int chunk_iters, void* stream);

/* Allocation-free form of pk_relax for a uniform batch (E packings of n
 * trees).  No counterpart in the reference: it exists for callers that must
 * not allocate device memory while they run -- code inside CUDA stream
 * capture, where cudaMalloc is not permitted; hosts whose allocator or memory
 * budget owns every device byte; and latency-bound loops, where cudaMalloc /
 * cudaFree may synchronise the device.  It allocates nothing: the L-BFGS
 * history lives in a 16 MiB array built into the library, which every GPU
 * that loads the library keeps until the process exits.  The caller still
 * provides inputs and outputs as for pk_relax.
 *   - Limit: 2 * history * E * (3 n + 3) <= 4194304 floats (e.g. E = 256,
 *     n = 200, history = 10); larger batches return PK_ERANGE with a message.
 *   - The first call on each device looks up the array's device address
 *     (cudaGetSymbolAddress) with that device current; make that first call
 *     before any stream capture.  Like every entry point it needs pk_init on
 *     the device first (PK_ENOTINIT otherwise, before any CUDA call).
 *   - The address is remembered per device until pk_init runs there again.
 *     After cudaDeviceReset (or any re-creation of the primary context) call
 *     pk_init again, as the geometry tables need anyway; the next call then
 *     fetches the address afresh -- again before any stream capture.
 *   - All calls share the one array and it keeps the previous call's
 *     contents.  Nothing in it needs clearing (every history slot is written
 *     before it is read), but two calls whose kernels overlap on the GPU --
 *     on different streams, or from different host threads -- race on it:
 *     serialise them. */
int pk_relax_noalloc(const float* xyt_in, const float* h_in, int E, int n, const PkCostSpec* spec,
                     const PkRelaxParams* params, float* xyt_out, float* h_out, float* loss_out, int* iters_out,
                     void* stream);

/* SolutionCollectionSquare.snap (kaggle_support.py:824-879): each packing's
 * trees re-centred on the bounding box of their (search-tree) vertices and h
 * = (min(side, h_in[0]), 0, 0), side = max(width, height); h_in nullable
 * (then h = (side, 0, 0)).  xyt_out may alias xyt_in. */
int pk_snap(const float* xyt_in, const float* h_in, int E, int n, float* xyt_out, float* h_out, void* stream);

/* ---- GA offspring moves (pack_move.py) -------------------------------- */

#define PK_MOVE_RANDOM_TREE 0     /* MoveRandomTree,   pack_move.py:161 */
#define PK_MOVE_JIGGLE_TREE 1     /* JiggleRandomTree, :191 */
#define PK_MOVE_JIGGLE_CLUSTER 2  /* JiggleCluster,    :227 */
#define PK_MOVE_TRANSLATE 3       /* Translate,        :301 */
#define PK_MOVE_TWIST 4           /* Twist,            :336 */
#define PK_MOVE_CROSSOVER 5       /* Crossover,        :406 */
#define PK_MOVE_CROSSOVER2 6      /* Crossover2,       :635 */
#define PK_MAX_MOVE_TYPES 16

#define PK_GENO_SQUARE 0          /* SolutionCollectionSquare */
#define PK_GENO_SYM90 1           /* SolutionCollectionSquareSymmetric90 */
#define PK_GENO_SYM180 2          /* SolutionCollectionSquareSymmetric180 */

#define PK_XDIST_STRIPE 0         /* Crossover2.distance_function */
#define PK_XDIST_SQUARE 1
#define PK_XDIST_SQUARE90 2
#define PK_XDIST_SQUARE180 3

/* One entry of a MoveSelector: the move class and its fields. */
typedef struct PkMove {
    int type;                          /* PK_MOVE_* */
    int respect_edge_spacer_filter;
    double max_xy_move, max_theta_move;        /* JiggleRandomTree, JiggleCluster */
    int min_n_trees, max_n_trees;              /* JiggleCluster; min_n_trees also for the crossovers */
    double max_n_trees_ratio;                  /* Crossover, Crossover2 */
    double min_radius, max_radius;             /* Twist */
    int simple_mate_location;                  /* Crossover */
    int distance_function;                     /* Crossover2: PK_XDIST_* */
    int decouple_mate_location;                /* Crossover2 */
    int use_edge_clearance_when_decoupled;     /* Crossover2 */
    int do_90_rotation;                        /* Crossover2 */
} PkMove;

/* The population's genotype class and its move-location filter
 * (kaggle_support.py:454-535): EdgeSpacerDummy (spacer 0) or
 * EdgeSpacerBasic (spacer 1). */
typedef struct PkGenotype {
    int kind;                 /* PK_GENO_* of the population: move centres, N_trees */
    int mate_kind;            /* PK_GENO_* of the mate collection: canonicalisation, N_trees */
    int filter;               /* filter_move_locations_with_edge_spacer */
    int spacer;
    double margin;            /* filter_move_locations_margin */
    double dist_x, dist_y, dist_corner;
} PkGenotype;

/* MoveSelector (pack_move.py:119-158): cum_prob holds the float32 cumulative
 * normalised weights; a draw u picks the first move with u <= cum_prob. */
typedef struct PkMoveSet {
    int n_moves;
    double cum_prob[PK_MAX_MOVE_TYPES];
    PkMove moves[PK_MAX_MOVE_TYPES];
    PkGenotype geno;
} PkMoveSet;

/* Move.do_move_vec of a MoveSelector (pack_move.py:31-55, 119-158) on the
 * rows inds_to_do (C,) of xyt (E, n, 3), in place, with mates
 * mate_xyt[inds_mate] (mate_xyt (M, n, 3), mate_h (M, 3)); h (E, 3).  One CTA
 * per row: the move is chosen and applied with random draws from
 * Philox4x32-10 keyed by seed and counted by (call, row position, draw), so a
 * call is reproducible and independent of the batch split.  chosen (C,)
 * int32 receives the move index (-1: none), status (device int, nullable)
 * is or-ed with 1 when a rejection sampler hit its limit, 2 for a request
 * the reference rejects by assertion (edge-spacer filter on a 90-degree
 * genotype, edge clearance above a quarter of the side) and 4 for a row or
 * mate index out of range (that row is left unchanged).  Rows must be
 * distinct and mate_xyt must not alias xyt; n <= 1024. */
int pk_moves(float* xyt, const float* h, int E, int n, const int* inds_to_do, int C, const float* mate_xyt,
             const float* mate_h, int M, const int* inds_mate, const PkMoveSet* set, uint64_t seed, uint64_t call,
             int* chosen, int* status, void* stream);

/* Philox4x32-10 draws of the move kernels (tests): out (count,) float64
 * uniforms of (seed, call, row position), draws first .. first+count-1. */
int pk_move_draws(uint64_t seed, uint64_t call, int row, int first, int count, double* out, void* stream);

/* Floats of work needed by pk_relax: sizes_host (E,) host int32 tree counts
 * for a ragged batch, or NULL and n_uniform for a uniform one. */
size_t pk_relax_workspace_floats(const int* sizes_host, int E, int n_uniform, int history);

/* FP32 FMA throughput probe: blocks x threads x iters x 16 flops, for the
 * roofline denominator of the SIMT-bound kernels. */
int pk_fma_probe(float* out, int blocks, int threads, int iters, void* stream);

/* Trilinear-lookup probe: blocks x threads x iters x 2 lookups, each the 8
 * corner loads of a random cell of the C-ordered (nx, ny, nt) float table, for
 * the roofline denominator of the LUT kernel (lookups per second). */
int pk_gather_probe(const float* table, int nx, int ny, int nt, float* out, int blocks, int threads, int iters,
                    unsigned seed, void* stream);

int pk_version(void);

#ifdef __cplusplus
}
#endif

#endif /* PACKB200_H */
