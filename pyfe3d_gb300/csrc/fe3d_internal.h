// Opaque objects behind the C ABI (device arrays owned by the library).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

// Free-row layout of one node in a pattern built from element connectivity:
// its free rows are consecutive, start at CSR position rs (-1 when the node
// has no free DOF) and all have L entries; fm holds the free-DOF bits.
struct __align__(16) fe3d_noderow {
    long long rs;
    int L;
    int fm;
};

struct fe3d_pattern {
    int64_t N = 0;          // DOFs of the full system
    int64_t nrows = 0;      // free DOFs (rows of the reduced system)
    int64_t nnz = 0;        // CSR entries of the reduced system
    int64_t nnz_in = 0;     // COO slots the pattern was built from
    int64_t nnz_valid = 0;  // COO slots with a free row and a free column
    int32_t *row_of_dof = nullptr;  // [N] reduced row of a DOF, -1 when fixed
    int64_t *dof_of_row = nullptr;  // [nrows] full DOF of a reduced row
    int32_t *perm = nullptr;        // [nnz_in] COO slots sorted by (row, col)
    int32_t *seg = nullptr;         // [nnz + 1] segment starts in perm
    int4 *runs = nullptr;           // [2 nruns] runs of entries summed alike (assembly.cu), or NULL
    int64_t nruns = 0;
    int32_t *colind = nullptr;      // [nnz]
    int64_t *rowptr = nullptr;      // [nrows + 1]
    // compressed columns for the solver's SpMV when every row spans fewer than
    // 65,536 columns: colind[k] = colbase[row] + col16[k] (else both NULL)
    int32_t *colbase = nullptr;     // [nrows]
    uint16_t *col16 = nullptr;      // [nnz]
    // node-block structure (patterns built from element connectivity only;
    // perm and seg are then NULL): the neighbours of node a are
    // nbr[nbrptr[a] .. nbrptr[a+1]) in ascending order, and the free columns
    // of neighbour nbr[k] start at offset nboff[k] within node a's rows
    int64_t nnodes = 0;
    int64_t *nbrptr = nullptr;      // [nnodes + 1]
    int32_t *nbr = nullptr;         // [npairs]
    int32_t *nboff = nullptr;       // [npairs]
    fe3d_noderow *noderow = nullptr;  // [nnodes]
    int max_row_len = 0;            // largest L over the nodes
};

// Element -> CSR scatter map of one element group (fused assembly).
struct fe3d_fmap_group {
    int64_t E = 0;
    int nn = 0;                     // nodes per element
    int32_t *node = nullptr;        // [E, nn] node indices
    int32_t *boff = nullptr;        // [E, nn, nn] offset of node j's columns in node i's rows
    uint32_t *first = nullptr;      // [E] bit i nn + j: this element assigns block (i, j)
    int32_t *order = nullptr;       // [E] elements sorted by colour
    int ncolors = 0;
    int64_t cstart[65] = {};        // colour c is order[cstart[c] .. cstart[c+1])
};

constexpr int kFmapMaxGroups = 8;

struct fe3d_fmap {
    const fe3d_pattern *pat = nullptr;
    int ngroups = 0;
    fe3d_fmap_group g[kFmapMaxGroups];
};

// Resident PCG (team_pcg.cu): the split of one or more systems over co-resident
// blocks, the slice layout of the non-zero values and the exchange words.
// Rows per block wanted while blocks are left, fewer FP64 instructions per block
// against a slower exchange: us per iteration with 8 / 16 / 32 / 64 rows, 486 rows
// 5.5 / 5.9 / 6.3 / 6.1, 2,166 rows 5.6 / 5.7 / 5.6 / 6.0, 9,126 rows 6.8 / 6.8 /
// 6.8 / 6.9.
constexpr int kTeamRows = 16;
constexpr int64_t kTeamIters = 4096;   // iterations of one resident launch at most (a quarter of a second)

// One system of a launch: limits in, iterations out.
struct TeamSys {
    double stop2;   // r.r at which to stop
    int maxiter;    // iterations of this launch at most
    int phase;      // convergence is looked at where phase + iterations is a multiple of chunk
    int iters;      // iterations run
    int pad;
};

// Rows [row0, row1) of system sys on so many blocks.
struct TeamPart {
    int64_t row0, row1, sys;
    int blocks;
};

struct fe3d_team {
    int blocks = 0;                    // blocks of a launch at most
    size_t smem_max = 0;
    int G = 0, L = 1;                  // blocks in use, lanes per row
    int nmax = 0;                      // largest row count of a block
    size_t smem = 0;                   // of the block that needs most, without matrix entries
    size_t smem_run = 0;               // of a launch
    int rows = 0;                      // where the matrix rows are kept (team_pcg.cu)
    int32_t *ints = nullptr;           // the per-block arrays below
    int32_t *rbeg = nullptr, *rend = nullptr, *slice0 = nullptr, *cmin = nullptr, *cmax = nullptr;
    int32_t *tfirst = nullptr, *tcount = nullptr, *tsys = nullptr;
    int64_t slices = 0;                // allocated in slen, soff
    int32_t *slen = nullptr;
    int64_t *soff = nullptr;
    double *sval = nullptr;
    uint16_t *scol = nullptr;
    int64_t cap = 0;                   // entries allocated in sval, scol
    unsigned long long *total = nullptr;
    ulonglong2 *z = nullptr, *slots = nullptr;
    double *dval = nullptr;            // [6][n] non-zeros of the rows of the block inverses
    uint32_t *dinf = nullptr;          // [n]
    TeamSys *sys = nullptr;
    int *done = nullptr;
    unsigned epoch = 1;
    // polls of one word before a block gives up: about a second, and about a
    // minute at the first exchange, where blocks may still wait for SMs that
    // another stream's kernel holds
    int poll = 1 << 21, poll_first = 1 << 27;
};

// Block-Jacobi PCG state (pcg.cu); the batched solver (bpcg.cu) reuses its
// node blocks, block inverses, work vectors and private stream.
struct fe3d_solver {
    const fe3d_pattern *pat = nullptr;
    int64_t n = 0, nnodes = 0;
    int bs = 6;  // DOFs per node
    int32_t *start = nullptr;
    int8_t *size = nullptr;
    double *Dinv = nullptr;
    float *Dinv32 = nullptr;
    const double *vals = nullptr;  // FP64 values (caller-owned, set by setup)
    int ready = 0;                 // setup has run (vals may be NULL when nnz == 0)
    float *vals32 = nullptr;
    double *r = nullptr;
    double *z = nullptr, *p = nullptr, *q = nullptr;
    float *z32 = nullptr, *p32 = nullptr, *q32 = nullptr;
    double *ppq = nullptr, *prz = nullptr, *prr = nullptr, *prf = nullptr;
    double *scal = nullptr;  // [0..1] rz double buffer, [2] rr, [3] alpha, [4] ff, [5..7] spare
    int *nonpos = nullptr;
    int nparts = 0;
    int spmv_grid = 0, node_grid = 0, vec_grid = 0;
    int have32 = 0;
    // private stream: iteration chunks are captured once as CUDA graphs
    // (the legacy default stream cannot be captured) and replayed
    cudaStream_t stream = nullptr;
    cudaEvent_t ev_in = nullptr, ev_out = nullptr;
    double *uin = nullptr, *fin = nullptr;  // stable operands of the graphs
    double *xhi = nullptr, *xlo = nullptr;  // double-double solution base
    double *sc = nullptr;  // [2n]: row scales sqrt(K_ii), then their inverses; FP32 data hold
                           // S^-1 K S^-1 and S Dinv S
    cudaGraphExec_t graph[3][2] = {};     // [precision][parity]
    int graph_chunk[3][2] = {};
    int graph_flex[3][2] = {};
    int graph_lanes[3][2] = {};
    int lanes[3] = {0, 0, 0};             // SpMV lanes per row [precision], tuned at setup
    float2 *vals2 = nullptr, *p2 = nullptr;  // split-FP32 (hi, lo) values and direction
    int have2 = 0;
    unsigned int *counter = nullptr;      // last-block-done counter of the reductions
    // FP64 solves: the non-zero values in slices of 32 rows (entry k of row i
    // at 32 (soff[i / 32] + k) + i % 32, rows padded with zeros to the slice's
    // longest), rebuilt from the caller's values by every solve; sell_on: the
    // current solve uses it
    int64_t *soff = nullptr;
    int32_t *slen = nullptr;
    double *sval = nullptr;
    uint16_t *scol = nullptr;             // offsets from the pattern's colbase
    int64_t sell_cap = 0;                 // entries allocated in sval / scol
    unsigned long long *sell_total = nullptr;
    int sell_on = 0;
    int sell_grid = 0;                    // blocks of the slice kernels (one wave of resident ones)
    // row-wise update: rows of each 32-node chunk, and each row's non-zeros of
    // the block inverses (rebuilt by every solve)
    int32_t *chunk_row = nullptr;         // [nchunks + 1]
    int64_t nchunks = 0;
    int upd_grid = 0;
    double *dval = nullptr;               // [6][n]
    uint32_t *dinf = nullptr;             // [n]
    int *xnz = nullptr;                   // [0] non-zero initial guess, [1] non-finite matrix value
    fe3d_team *team = nullptr;            // resident iterations (FP64, systems that fit)
    int team_tried = 0;
};

// Batched PCG state (bpcg.cu).
struct fe3d_bsolver {
    fe3d_solver *base = nullptr;  // node blocks, block inverses, work vectors, stream
    int64_t ninst = 0;
    int32_t *inst = nullptr;       // [nrows] instance of each reduced row
    int32_t *node_inst = nullptr;  // [nnodes]
    int *active = nullptr, *flag = nullptr;
    int *bad = nullptr;
    double *pq = nullptr, *rz = nullptr /* [2][ninst] */, *rr = nullptr, *ff = nullptr, *rt = nullptr;
    int lanes[2] = {0, 0};  // autotuned lanes per row [precision]
    int32_t *rowlist = nullptr, *nodelist = nullptr;  // rows / nodes of active instances
    int *lcount = nullptr;                            // [0] rows, [1] nodes in the lists
    int *blockcount = nullptr;                        // compaction scratch [2][kCompactGrid]
    cudaGraphExec_t graph[2][2] = {{nullptr, nullptr}, {nullptr, nullptr}};  // [precision][parity]
    int graph_chunk[2][2] = {{0, 0}, {0, 0}};
    // work split: row and node ranges per instance, the rows of the
    // instances whose rows are contiguous (0 otherwise), the size limit, and
    // the block-resident solver's list, results and stream
    int32_t *rlo = nullptr, *rhi = nullptr, *nlo = nullptr, *nhi = nullptr, *rcnt = nullptr, *ncnt = nullptr;
    std::vector<int64_t> contig_rows, first_row;
    fe3d_team *team = nullptr;     // resident teams, made by the first solve that can use them
    int team_tried = 0;
    std::vector<int32_t> reach;    // column reach of each instance
    int64_t split_rows = 0;
    int32_t *cta_list = nullptr;
    int *cta_status = nullptr;
    int64_t *cta_iters = nullptr;
    cudaStream_t cta_stream = nullptr;
    cudaEvent_t cta_start = nullptr, cta_done = nullptr;
};

namespace fe3d {
void team_free(fe3d_team *t);
fe3d_team *team_create(const fe3d_solver *s, int64_t nsys, cudaStream_t st);
size_t team_smem(int64_t rows, int64_t bw);
int team_split(fe3d_team *t, const fe3d_solver *s, const std::vector<TeamPart> &parts, cudaStream_t st);
// Counts into t->total the entries of all slices and of the block with most;
// team_build lays them out once the caller has read both; team_inverses takes
// the block inverses.
int team_plan(fe3d_team *t, const fe3d_solver *s, cudaStream_t st);
int team_build(fe3d_team *t, const fe3d_solver *s, const unsigned long long (&total)[2], cudaStream_t st);
int team_inverses(fe3d_team *t, const fe3d_solver *s, cudaStream_t st);
// Iterations of every system of the split from s->r, s->p, u and rz (per
// system), until its limits are met or the teams of enough blocks have
// finished; rr per system, sys updated (synchronises).  FE3D_ERR_LAUNCH where
// the launch is refused or a poll gave up: u is then an earlier iterate in some
// or all rows, and r, p and rz do not belong to it.
int team_run(fe3d_team *t, const fe3d_solver *s, double *u, double *rz, double *rr, std::vector<TeamSys> &sys,
             int chunk, int enough, cudaStream_t st);
}  // namespace fe3d
