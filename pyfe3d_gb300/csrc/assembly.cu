// COO -> CSR assembly with boundary-condition elimination.
//
// Replaces the caller-side `coo_matrix((v, (r, c))).tocsc()` followed by
// `K[bu, :][:, bu]` of the reference's tests
// (tests/test_quad4_static_point_load.py:80-99).
//
// Pattern (once per mesh): every COO slot whose row and column are free DOFs
// gets the key (row', col') in the reduced numbering; keys are radix-sorted
// together with the slot index, equal keys form a segment, and the segment
// heads give the CSR row pointer and column indices.  The pattern keeps the
// sorted slot permutation `perm` and the segment starts `seg`.
// Numeric assembly (every update): vals[s] = sum of Kv[perm[t]] over the
// segment t in [seg[s], seg[s+1]), summed in ascending slot order, so the
// result is deterministic.  The six (free) columns of a node in a row of the
// matrix come from six consecutive slots of every element that has both nodes,
// so the segments of neighbouring entries are the same slots shifted by one:
// the pattern describes such a run, which ends with the node, by one 32-byte
// record, and the numeric assembly reads 5 instead of 11 bytes of indices per entry
// and two slots per load.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include "common.cuh"
#include "fe3d_internal.h"

namespace fe3d {
namespace {

__global__ void free_flags_kernel(int64_t N, const uint8_t *fixed, int32_t *flag) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < N) flag[i] = fixed ? (fixed[i] ? 0 : 1) : 1;
}

__global__ void reduced_index_kernel(int64_t N, const int32_t *flag, const int32_t *scan,
                                     int32_t *row_of_dof, int64_t *dof_of_row) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= N) return;
    if (flag[i]) {
        row_of_dof[i] = scan[i];
        dof_of_row[scan[i]] = i;
    } else {
        row_of_dof[i] = -1;
    }
}

__global__ void coo_keys_kernel(int64_t nnz, const int64_t *Kr, const int64_t *Kc, int64_t N,
                                const int32_t *row_of_dof, int64_t nfree, uint64_t *keys,
                                int32_t *idx, int *err) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= nnz) return;
    const int64_t r = Kr[t], c = Kc[t];
    uint64_t key = ~0ull;
    if (r < 0 || c < 0 || r >= N || c >= N) {
        raise_error(err, kErrBounds);
    } else {
        const int32_t rr = row_of_dof[r], cc = row_of_dof[c];
        if (rr >= 0 && cc >= 0) key = (uint64_t)rr * (uint64_t)nfree + (uint64_t)cc;
    }
    keys[t] = key;
    idx[t] = (int32_t)t;
}

__global__ void head_flags_kernel(int64_t nnz, const uint64_t *keys, int32_t *head) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= nnz) return;
    const uint64_t k = keys[t];
    head[t] = (k != ~0ull && (t == 0 || keys[t - 1] != k)) ? 1 : 0;
}

__global__ void segments_kernel(int64_t nnz, const uint64_t *keys, const int32_t *head,
                                const int32_t *hscan, int64_t nfree, int32_t *seg,
                                int32_t *colind, int32_t *row_count) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= nnz) return;
    if (head[t]) {
        const int32_t s = hscan[t];
        const uint64_t k = keys[t];
        seg[s] = (int32_t)t;
        colind[s] = (int32_t)(k % (uint64_t)nfree);
        atomicAdd(row_count + (k / (uint64_t)nfree), 1);
    }
}

__global__ void seg_end_kernel(int64_t nnz_valid, int64_t nseg, int32_t *seg) {
    seg[nseg] = (int32_t)nnz_valid;
}

__global__ void count_valid_kernel(int64_t nnz, const uint64_t *keys, unsigned long long *cnt) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t < nnz && keys[t] != ~0ull) atomicAdd(cnt, 1ull);
}

// Per row: the first (smallest) column as the base and 16-bit offsets of the
// row's columns from it; too_wide is set when a row spans 65,536 columns or more.
__global__ void col16_kernel(int64_t n, const int64_t *rowptr, const int32_t *colind, int32_t *colbase,
                             uint16_t *col16, int *too_wide) {
    const int64_t row = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (row >= n) return;
    const int64_t k0 = rowptr[row], k1 = rowptr[row + 1];
    const int32_t base = k1 > k0 ? colind[k0] : 0;
    colbase[row] = base;
    if (k1 > k0 && (int64_t)colind[k1 - 1] - base > 65535) {
        atomicOr(too_wide, 1);
        return;
    }
    for (int64_t k = k0; k < k1; k++) col16[k] = (uint16_t)(colind[k] - base);
}

__global__ void rowptr_kernel(int64_t n, const int64_t *scan, int64_t *rowptr, int64_t total) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) rowptr[i] = scan[i];
    if (i == n) rowptr[n] = total;
}

__global__ void widen_kernel(int64_t n, const int32_t *a, int64_t *b) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) b[i] = a[i];
}

// ---- runs of entries ----------------------------------------------------
// A run is entries s, s + 1, .. of one row and one node's columns whose
// segments are as long and whose slots are each one further.  It ends with the
// node, whichever of the node's DOFs are free, so it has at most RUN_MAX entries,
// which is what the lanes of a run write.  Record: {first entry, length, slots
// per entry, first place in perm}, {its first four slots}.
constexpr int RUN_SLOTS = 4;
constexpr int RUN_MAX = 6, RUN_LANES = RUN_MAX / 2;

// flag[s] = 1 where entry s does not continue the run of entry s - 1 (rows:
// run_rows_kernel).
__global__ void run_flags_kernel(int64_t nnz, const int32_t *seg, const int32_t *perm, const int32_t *colind,
                                 const int64_t *dof_of_row, int32_t *flag) {
    const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (s >= nnz) return;
    bool head = s == 0;
    if (!head) {
        const int32_t b = seg[s], e = seg[s + 1], a = seg[s - 1];
        head = e - b != b - a || colind[s] != colind[s - 1] + 1 ||
               dof_of_row[colind[s]] / RUN_MAX != dof_of_row[colind[s - 1]] / RUN_MAX;
        for (int32_t t = 0; !head && t < e - b; t++) head = perm[b + t] != perm[a + t] + 1;
    }
    flag[s] = head;
}

__global__ void run_rows_kernel(int64_t nrows, const int64_t *rowptr, int64_t nnz, int32_t *flag) {
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r < nrows && rowptr[r] < nnz) flag[rowptr[r]] = 1;
}

__global__ void run_fill_kernel(int64_t nnz, const int32_t *flag, const int32_t *scan, const int32_t *seg,
                                const int32_t *perm, int4 *runs) {
    const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (s >= nnz || !flag[s]) return;
    const int32_t b = seg[s], k = seg[s + 1] - b;
    int32_t q[RUN_SLOTS];
    for (int t = 0; t < RUN_SLOTS; t++) q[t] = t < k ? perm[b + t] : 0;
    runs[2 * (int64_t)scan[s]] = make_int4((int)s, 0, k, b);
    runs[2 * (int64_t)scan[s] + 1] = make_int4(q[0], q[1], q[2], q[3]);
}

__global__ void run_lengths_kernel(int64_t nruns, int64_t nnz, int4 *runs) {
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r >= nruns) return;
    const int next = r + 1 < nruns ? runs[2 * (r + 1)].x : (int)nnz;
    runs[2 * r].y = next - runs[2 * r].x;
}

// Sorts every RUN_CHUNK runs by their slots per entry (4 and more, 3, 2, 1;
// stable).  An FP64 addition takes a sub-partition's pipe for 64 cycles
// whatever its active lanes, and with the runs of a row side by side (1 2 1 2 4
// 2 1 2 1 slots in a plate) every warp made the additions of the longest.
constexpr int RUN_CHUNK = 256;
__global__ void __launch_bounds__(RUN_CHUNK) run_sort_kernel(int64_t nruns, int4 *runs) {
    __shared__ int cnt[4][RUN_CHUNK / 32];
    const int64_t r = blockIdx.x * (int64_t)RUN_CHUNK + threadIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool in = r < nruns;
    int4 h = make_int4(0, 0, 0, 0), q = h;
    if (in) {
        h = runs[2 * r];
        q = runs[2 * r + 1];
    }
    const int k = h.z, cls = !in ? -1 : k >= 4 ? 0 : 4 - k;
    int below = 0;
    for (int c = 0; c < 4; c++) {
        const unsigned m = __ballot_sync(0xffffffffu, cls == c);
        if (lane == 0) cnt[c][warp] = __popc(m);
        if (cls == c) below = __popc(m & ((1u << lane) - 1u));
    }
    __syncthreads();
    if (!in) return;
    int at = below;
    for (int c = 0; c <= cls; c++)
        for (int w = 0; w < RUN_CHUNK / 32; w++)
            if (c < cls || w < warp) at += cnt[c][w];
    const int64_t o = blockIdx.x * (int64_t)RUN_CHUNK + at;
    runs[2 * o] = h;
    runs[2 * o + 1] = q;
}

__device__ __forceinline__ double2 run_load(const double *a, bool two, bool wide) {
    if (wide) return __ldg(reinterpret_cast<const double2 *>(a));
    return make_double2(__ldg(a), two ? __ldg(a + 1) : 0.);
}

// Numeric assembly over runs: three lanes a run, two entries a lane; 8 bytes
// per slot and per entry and 32 per run.  301x301-node plate (51.8 M slots, 29 M
// entries): 0.354 ms by entries, 0.234 ms with the runs unsorted (78 % of the
// FP64 pipe), 0.144 ms sorted (5.6 TB/s, 0.82 of the measured copy rate).
__global__ void __launch_bounds__(256) assemble_runs_kernel(int64_t nruns, const int4 *__restrict__ runs,
                                                            const int32_t *__restrict__ perm,
                                                            const double *__restrict__ Kv, double *__restrict__ vals,
                                                            int vec16) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, r = t / RUN_LANES;
    const int j = 2 * (int)(t - RUN_LANES * r);
    int4 h = make_int4(0, 0, 0, 0), q = h;
    if (r < nruns) {
        h = __ldg(runs + 2 * r);
        q = __ldg(runs + 2 * r + 1);
    }
    const int len = h.y, k = h.z;
    const bool in = j < len, two = j + 1 < len;
    // one path per warp, its loads in flight together
    const int most = __reduce_max_sync(0xffffffffu, in ? k : 0);
    const bool wide = two && vec16;
    double2 s = make_double2(0., 0.);
    if (most == 0) return;
    if (most == 1) {
        if (in) s = run_load(Kv + q.x + j, two, wide && !(q.x & 1));
    } else if (most == 2) {
        double2 v = s;
        if (in) s = run_load(Kv + q.x + j, two, wide && !(q.x & 1));
        if (in && k > 1) v = run_load(Kv + q.y + j, two, wide && !(q.y & 1));
        s.x += v.x;
        s.y += v.y;
    } else if (most <= RUN_SLOTS) {
        double2 v1 = s, v2 = s, v3 = s;
        if (in) s = run_load(Kv + q.x + j, two, wide && !(q.x & 1));
        if (in && k > 1) v1 = run_load(Kv + q.y + j, two, wide && !(q.y & 1));
        if (in && k > 2) v2 = run_load(Kv + q.z + j, two, wide && !(q.z & 1));
        if (in && k > 3) v3 = run_load(Kv + q.w + j, two, wide && !(q.w & 1));
        s.x = ((s.x + v1.x) + v2.x) + v3.x;
        s.y = ((s.y + v1.y) + v2.y) + v3.y;
    } else if (in) {
        for (int i = 0; i < k; i++) {
            s.x += __ldg(Kv + __ldg(perm + h.w + j * k + i));
            if (two) s.y += __ldg(Kv + __ldg(perm + h.w + (j + 1) * k + i));
        }
    }
    if (in) vals[h.x + j] = s.x;
    if (two) vals[h.x + j + 1] = s.y;
}

// Numeric assembly without runs: one thread per CSR entry (segment).
__global__ void __launch_bounds__(256) assemble_kernel(int64_t nseg, const int32_t *__restrict__ seg,
                                                       const int32_t *__restrict__ perm,
                                                       const double *__restrict__ Kv,
                                                       double *__restrict__ vals) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < nseg; s += stride) {
        const int32_t b = __ldg(seg + s), e = __ldg(seg + s + 1);
        double acc = 0.;
        for (int32_t t = b; t < e; t++) acc += __ldg(Kv + __ldg(perm + t));
        vals[s] = acc;
    }
}

template <typename T>
int dalloc(T **p, size_t n) {
    if (n == 0) n = 1;
    return cudaMalloc((void **)p, n * sizeof(T)) == cudaSuccess ? 0 : FE3D_ERR_NOMEM;
}

inline unsigned nblk(int64_t n, int bs = 256) { return (unsigned)((n + bs - 1) / bs > 0 ? (n + bs - 1) / bs : 1); }

}  // namespace
}  // namespace fe3d

using namespace fe3d;

extern "C" int fe3d_pattern_build(const int64_t *Kr, const int64_t *Kc, int64_t nnz_in, int64_t N,
                                  const uint8_t *fixed, fe3d_pattern **out, int *err, void *stream) {
    if (!out || nnz_in < 0 || N <= 0 || (nnz_in > 0 && (!Kr || !Kc))) return FE3D_ERR_ARG;
    if (nnz_in >= (int64_t)INT32_MAX || N >= (int64_t)INT32_MAX) return FE3D_ERR_ARG;
    *out = nullptr;
    cudaStream_t st = as_stream(stream);
    fe3d_pattern *p = new fe3d_pattern();
    p->N = N;
    p->nnz_in = nnz_in;
    int rc = 0;
    int32_t *flag = nullptr, *scan = nullptr, *idx = nullptr, *head = nullptr, *hscan = nullptr;
    int32_t *row_count = nullptr;
    int64_t *rc64 = nullptr, *rscan = nullptr;
    uint64_t *keys = nullptr, *keys_sorted = nullptr;
    void *tmp = nullptr;
    size_t tmp_bytes = 0, need = 0;
    unsigned long long *dcount = nullptr;
    int *wide = nullptr;
    int hwide = 0;
    unsigned long long hcount = 0;
    int32_t nfree32 = 0, nseg32 = 0, last_head = 0, last_hscan = 0;
    int32_t last_flag = 0, last_scan = 0;
#define TRY(x)                  \
    do {                        \
        rc = (x);               \
        if (rc) goto fail;      \
    } while (0)
#define TRYC(x)                                     \
    do {                                            \
        if ((x) != cudaSuccess) {                   \
            rc = FE3D_ERR_CUDA;                     \
            goto fail;                              \
        }                                           \
    } while (0)
    // reduced numbering of the free DOFs
    TRY(dalloc(&flag, N));
    TRY(dalloc(&scan, N));
    TRY(dalloc(&p->row_of_dof, N));
    free_flags_kernel<<<nblk(N), 256, 0, st>>>(N, fixed, flag);
    TRYC(cub::DeviceScan::ExclusiveSum(nullptr, need, flag, scan, (int)N, st));
    tmp_bytes = need;
    TRYC(cudaMalloc(&tmp, tmp_bytes));
    TRYC(cub::DeviceScan::ExclusiveSum(tmp, tmp_bytes, flag, scan, (int)N, st));
    TRYC(cudaMemcpyAsync(&last_flag, flag + N - 1, 4, cudaMemcpyDeviceToHost, st));
    TRYC(cudaMemcpyAsync(&last_scan, scan + N - 1, 4, cudaMemcpyDeviceToHost, st));
    TRYC(cudaStreamSynchronize(st));
    nfree32 = last_flag + last_scan;
    p->nrows = nfree32;
    TRY(dalloc(&p->dof_of_row, p->nrows));
    reduced_index_kernel<<<nblk(N), 256, 0, st>>>(N, flag, scan, p->row_of_dof, p->dof_of_row);
    // keys of the kept slots, sorted with their slot index
    TRY(dalloc(&keys, nnz_in));
    TRY(dalloc(&keys_sorted, nnz_in));
    TRY(dalloc(&idx, nnz_in));
    TRY(dalloc(&p->perm, nnz_in));
    if (nnz_in > 0) {
        coo_keys_kernel<<<nblk(nnz_in), 256, 0, st>>>(nnz_in, Kr, Kc, N, p->row_of_dof,
                                                      p->nrows > 0 ? p->nrows : 1, keys, idx, err);
        {
            int end_bit = 1;
            while (end_bit < 64 && ((1ull << end_bit) - 1) < (uint64_t)p->nrows * (uint64_t)p->nrows) end_bit++;
            // the drop marker ~0 must sort last: use all 64 bits when needed
            end_bit = 64;
            TRYC(cub::DeviceRadixSort::SortPairs(nullptr, need, keys, keys_sorted, idx, p->perm,
                                                 (int)nnz_in, 0, end_bit, st));
            if (need > tmp_bytes) {
                cudaFree(tmp);
                tmp_bytes = need;
                TRYC(cudaMalloc(&tmp, tmp_bytes));
            }
            TRYC(cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, keys, keys_sorted, idx, p->perm,
                                                 (int)nnz_in, 0, end_bit, st));
        }
        // segments
        TRY(dalloc(&head, nnz_in));
        TRY(dalloc(&hscan, nnz_in));
        head_flags_kernel<<<nblk(nnz_in), 256, 0, st>>>(nnz_in, keys_sorted, head);
        TRYC(cub::DeviceScan::ExclusiveSum(nullptr, need, head, hscan, (int)nnz_in, st));
        if (need > tmp_bytes) {
            cudaFree(tmp);
            tmp_bytes = need;
            TRYC(cudaMalloc(&tmp, tmp_bytes));
        }
        TRYC(cub::DeviceScan::ExclusiveSum(tmp, tmp_bytes, head, hscan, (int)nnz_in, st));
        TRYC(cudaMemcpyAsync(&last_head, head + nnz_in - 1, 4, cudaMemcpyDeviceToHost, st));
        TRYC(cudaMemcpyAsync(&last_hscan, hscan + nnz_in - 1, 4, cudaMemcpyDeviceToHost, st));
        TRY(dalloc(&dcount, 1));
        TRYC(cudaMemsetAsync(dcount, 0, sizeof(*dcount), st));
        count_valid_kernel<<<nblk(nnz_in), 256, 0, st>>>(nnz_in, keys_sorted, dcount);
        TRYC(cudaMemcpyAsync(&hcount, dcount, sizeof(hcount), cudaMemcpyDeviceToHost, st));
        TRYC(cudaStreamSynchronize(st));
        nseg32 = last_head + last_hscan;
    }
    p->nnz = nseg32;
    p->nnz_valid = (int64_t)hcount;
    TRY(dalloc(&p->seg, p->nnz + 1));
    TRY(dalloc(&p->colind, p->nnz));
    TRY(dalloc(&row_count, p->nrows + 1));
    TRY(dalloc(&p->rowptr, p->nrows + 1));
    TRYC(cudaMemsetAsync(row_count, 0, sizeof(int32_t) * (p->nrows + 1), st));
    if (nnz_in > 0) {
        segments_kernel<<<nblk(nnz_in), 256, 0, st>>>(nnz_in, keys_sorted, head, hscan, p->nrows > 0 ? p->nrows : 1,
                                                      p->seg, p->colind, row_count);
    }
    seg_end_kernel<<<1, 1, 0, st>>>(p->nnz_valid, p->nnz, p->seg);
    // row pointer = exclusive scan of the per-row counts (64-bit)
    TRY(dalloc(&rc64, p->nrows + 1));
    TRY(dalloc(&rscan, p->nrows + 1));
    widen_kernel<<<nblk(p->nrows + 1), 256, 0, st>>>(p->nrows + 1, row_count, rc64);
    TRYC(cub::DeviceScan::ExclusiveSum(nullptr, need, rc64, rscan, (int)(p->nrows + 1), st));
    if (need > tmp_bytes) {
        cudaFree(tmp);
        tmp_bytes = need;
        TRYC(cudaMalloc(&tmp, tmp_bytes));
    }
    TRYC(cub::DeviceScan::ExclusiveSum(tmp, tmp_bytes, rc64, rscan, (int)(p->nrows + 1), st));
    rowptr_kernel<<<nblk(p->nrows + 1), 256, 0, st>>>(p->nrows, rscan, p->rowptr, p->nnz);
    if (p->nnz > 0) {
        // runs of entries (head and hscan are free again)
        run_flags_kernel<<<nblk(p->nnz), 256, 0, st>>>(p->nnz, p->seg, p->perm, p->colind, p->dof_of_row, head);
        run_rows_kernel<<<nblk(p->nrows), 256, 0, st>>>(p->nrows, p->rowptr, p->nnz, head);
        TRYC(cub::DeviceScan::ExclusiveSum(nullptr, need, head, hscan, (int)p->nnz, st));
        if (need > tmp_bytes) {
            cudaFree(tmp);
            tmp = nullptr;
            tmp_bytes = need;
            TRYC(cudaMalloc(&tmp, tmp_bytes));
        }
        TRYC(cub::DeviceScan::ExclusiveSum(tmp, tmp_bytes, head, hscan, (int)p->nnz, st));
        TRYC(cudaMemcpyAsync(&last_head, head + p->nnz - 1, 4, cudaMemcpyDeviceToHost, st));
        TRYC(cudaMemcpyAsync(&last_hscan, hscan + p->nnz - 1, 4, cudaMemcpyDeviceToHost, st));
        TRYC(cudaStreamSynchronize(st));
        p->nruns = last_head + last_hscan;
        // shorter than two entries on average: the records would be the larger part
        if (2 * p->nruns <= p->nnz && dalloc(&p->runs, 2 * (size_t)p->nruns) == 0) {
            run_fill_kernel<<<nblk(p->nnz), 256, 0, st>>>(p->nnz, head, hscan, p->seg, p->perm, p->runs);
            run_lengths_kernel<<<nblk(p->nruns), 256, 0, st>>>(p->nruns, p->nnz, p->runs);
            run_sort_kernel<<<nblk(p->nruns, RUN_CHUNK), RUN_CHUNK, 0, st>>>(p->nruns, p->runs);
        } else {
            (void)cudaGetLastError();
            p->nruns = 0;
        }
    }
    if (p->nrows > 0 && p->nnz > 0) {
        // compressed columns for the SpMV (2 bytes per entry instead of 4)
        TRY(dalloc(&p->colbase, p->nrows));
        TRY(dalloc(&p->col16, p->nnz));
        TRY(dalloc(&wide, 1));
        TRYC(cudaMemsetAsync(wide, 0, sizeof(int), st));
        col16_kernel<<<nblk(p->nrows), 256, 0, st>>>(p->nrows, p->rowptr, p->colind, p->colbase, p->col16, wide);
        TRYC(cudaMemcpyAsync(&hwide, wide, sizeof(int), cudaMemcpyDeviceToHost, st));
    }
    TRYC(cudaStreamSynchronize(st));
    TRYC(cudaGetLastError());
    if (hwide) {
        cudaFree(p->colbase);
        cudaFree(p->col16);
        p->colbase = nullptr;
        p->col16 = nullptr;
    }
    cudaFree(wide);
    wide = nullptr;
    cudaFree(flag); cudaFree(scan); cudaFree(keys); cudaFree(keys_sorted); cudaFree(idx);
    cudaFree(head); cudaFree(hscan); cudaFree(row_count); cudaFree(rc64); cudaFree(rscan);
    cudaFree(tmp); cudaFree(dcount);
    *out = p;
    return FE3D_OK;
fail:
    cudaFree(flag); cudaFree(scan); cudaFree(keys); cudaFree(keys_sorted); cudaFree(idx);
    cudaFree(head); cudaFree(hscan); cudaFree(row_count); cudaFree(rc64); cudaFree(rscan);
    cudaFree(tmp); cudaFree(dcount); cudaFree(wide);
    fe3d_pattern_free(p);
    return rc;
#undef TRY
#undef TRYC
}

extern "C" int fe3d_pattern_free(fe3d_pattern *p) {
    if (!p) return FE3D_OK;
    cudaFree(p->row_of_dof);
    cudaFree(p->dof_of_row);
    cudaFree(p->perm);
    cudaFree(p->seg);
    cudaFree(p->runs);
    cudaFree(p->colind);
    cudaFree(p->rowptr);
    cudaFree(p->colbase);
    cudaFree(p->col16);
    cudaFree(p->nbrptr);
    cudaFree(p->nbr);
    cudaFree(p->nboff);
    cudaFree(p->noderow);
    delete p;
    return FE3D_OK;
}

extern "C" int fe3d_pattern_info(const fe3d_pattern *p, int64_t *nrows, int64_t *nnz,
                                 int64_t *nnz_in) {
    if (!p) return FE3D_ERR_ARG;
    if (nrows) *nrows = p->nrows;
    if (nnz) *nnz = p->nnz;
    if (nnz_in) *nnz_in = p->nnz_in;
    return FE3D_OK;
}

extern "C" int fe3d_pattern_arrays(const fe3d_pattern *p, const int64_t **rowptr,
                                   const int32_t **colind, const int64_t **dof_of_row,
                                   const int32_t **row_of_dof) {
    if (!p) return FE3D_ERR_ARG;
    if (rowptr) *rowptr = p->rowptr;
    if (colind) *colind = p->colind;
    if (dof_of_row) *dof_of_row = p->dof_of_row;
    if (row_of_dof) *row_of_dof = p->row_of_dof;
    return FE3D_OK;
}

extern "C" int fe3d_pattern_copy(const fe3d_pattern *p, int64_t *rowptr, int32_t *colind,
                                 int64_t *dof_of_row, void *stream) {
    if (!p) return FE3D_ERR_ARG;
    cudaStream_t st = as_stream(stream);
    if (rowptr)
        FE3D_CUDA(cudaMemcpyAsync(rowptr, p->rowptr, sizeof(int64_t) * (p->nrows + 1),
                                  cudaMemcpyDeviceToDevice, st));
    if (colind && p->nnz)
        FE3D_CUDA(cudaMemcpyAsync(colind, p->colind, sizeof(int32_t) * p->nnz, cudaMemcpyDeviceToDevice, st));
    if (dof_of_row && p->nrows)
        FE3D_CUDA(cudaMemcpyAsync(dof_of_row, p->dof_of_row, sizeof(int64_t) * p->nrows,
                                  cudaMemcpyDeviceToDevice, st));
    return FE3D_OK;
}

extern "C" int fe3d_assemble(const fe3d_pattern *p, const double *Kv, double *vals, void *stream) {
    if (!p || (p->nnz > 0 && (!Kv || !vals))) return FE3D_ERR_ARG;
    if (p->nnz > 0 && !p->perm) return FE3D_ERR_STATE;  // pattern built from elements: no COO slots
    if (p->nnz == 0) return FE3D_OK;
    if (p->nruns) {
        assemble_runs_kernel<<<nblk(RUN_LANES * p->nruns), 256, 0, as_stream(stream)>>>(p->nruns, p->runs, p->perm, Kv, vals,
                                                                               ((uintptr_t)Kv & 15u) == 0);
        FE3D_CHECK_LAUNCH();
        return FE3D_OK;
    }
    const int64_t blocks = (p->nnz + 255) / 256;
    const unsigned grid = (unsigned)(blocks < kSMs * 16 ? blocks : kSMs * 16);
    assemble_kernel<<<grid, 256, 0, as_stream(stream)>>>(p->nnz, p->seg, p->perm, Kv, vals);
    FE3D_CHECK_LAUNCH();
    return FE3D_OK;
}
