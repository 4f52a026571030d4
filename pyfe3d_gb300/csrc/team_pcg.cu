// Resident block-Jacobi PCG: many iterations of the FP64 recurrence of pcg.cu
// in one cooperative launch, for systems whose vectors fit the shared memory
// of the SMs.  Stands in for the same reference call as pcg.cu
// (tests/test_quad4_static_point_load.py:102).
//
// What bounds it: with three launches per iteration a plate of up to 60,000
// DOFs spends 20-30 us per iteration, of which its FP64 work is 0.3-5 us; the
// rest is launches, their tails and vectors going through L2.  Here each block
// owns the rows of a contiguous range of nodes and keeps their r, u and K p
// in shared memory, together with the search direction over the window of
// columns its rows reach; p = z + beta p is recomputed by every block for its
// own window, so z is the only vector that travels.
//
// Exchange: every value that crosses blocks (z, the partial sums of p.q, r.z
// and r.r) travels as two 8-byte words, each holding half of the double and
// the iteration's number.  A reader polls the words themselves: no fence, no
// counter, one trip through L2 per exchange, two exchanges per iteration.  A
// slot is written again only after every reader of its previous value has
// sent something that the writer waited for.  Sums over blocks are taken in a
// fixed order by each block, so all blocks hold the same scalars and the
// result does not depend on scheduling.  Every poll is bounded; a block that
// gives up raises a flag and returns.  The partial sums sit a 128-byte line
// apart: 152 blocks exchange a value in 3.1k cycles, 5.8k with four to a line.
//
// Matrix: the non-zero values in slices of 32 / L rows, L lanes per row (L
// grows as the rows per block shrink), anchored at the block's first row.  An
// FP64 instruction holds its sub-partition's pipe for 64 cycles whatever its
// active lanes, so reductions go through shared memory to one warp per
// sub-partition instead of shuffles in all warps, comparisons of doubles are
// left to one warp, and blocks of few rows keep them in registers.
//
// Measured on clamped perturbed plates, us per iteration, three launches /
// resident: 486 rows 20.8 / 5.9, 2,166 rows 20.8 / 6.2, 9,126 rows 22.2 / 8.2,
// 58,806 rows 25.5 / 11.6, 237,606 rows 43 / 25, 536,406 rows 69.5 / 60 (there
// the matrix no longer fits L2 and bounds both).
#include "common.cuh"
#include "fe3d_internal.h"

namespace fe3d {
namespace {

constexpr int TT = 512;               // threads per block
constexpr int TEAM_MAX = kSMs;        // blocks of one system
// Polls of one word before a block gives up: about a second, and about a
// minute at the first exchange, where blocks may still wait for SMs that
// another stream's kernel holds.
constexpr int POLL_MAX = 1 << 21, POLL_FIRST = 1 << 27;
constexpr int TZ = TT - 32;           // threads that fetch z; the last warp sums r.z meanwhile
constexpr int SLOT = 8;               // words (16 bytes) per slot: a 128-byte line each

__device__ __forceinline__ void ll_store(ulonglong2 *p, double v, unsigned ep) {
    const unsigned long long e = (unsigned long long)ep << 32;
    const unsigned long long a = e | (unsigned)__double2loint(v), b = e | (unsigned)__double2hiint(v);
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}

// Polls N words base[i0 + j step], i0 + j step < lim, into v (0 past the end),
// all loads of a round in flight together; false when one did not arrive.
template <int N>
__device__ __forceinline__ bool ll_poll(const ulonglong2 *base, int i0, int step, int lim, unsigned ep,
                                        double (&v)[N], int limit = POLL_MAX) {
#pragma unroll
    for (int j = 0; j < N; j++) v[j] = 0.;
    if (i0 >= lim) return true;
    bool all = false;
    for (int spin = 0; !all && spin < limit; spin++) {
        unsigned long long a[N], b[N];
#pragma unroll
        for (int j = 0; j < N; j++) {
            const ulonglong2 *p = base + (i0 + j * step < lim ? i0 + j * step : i0);
            asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a[j]), "=l"(b[j]) : "l"(p) : "memory");
        }
        all = true;
#pragma unroll
        for (int j = 0; j < N; j++) {
            all &= (unsigned)(a[j] >> 32) == ep && (unsigned)(b[j] >> 32) == ep;
            if (i0 + j * step < lim) v[j] = __hiloint2double((int)(unsigned)b[j], (int)(unsigned)a[j]);
        }
    }
    return all;
}

// Sum over the block of values held by its first nw warps (by the lanes that
// are multiples of lo in a group of more than four), valid in warp 0.  red:
// TT + 4 doubles; a block-wide barrier has to come before the next use.
__device__ __forceinline__ double team_block_sum(double v, int nw, int lo, double *red) {
    const int warp = threadIdx.x >> 5;
    if (nw > 4) {
        red[threadIdx.x] = v;
        __syncthreads();
        v = threadIdx.x < 128
                ? (red[threadIdx.x] + red[threadIdx.x + 128]) + (red[threadIdx.x + 256] + red[threadIdx.x + 384]) : 0.;
        nw = 4;
        lo = 1;
    }
    if (warp < nw) {
        for (int o = 16; o >= lo; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0) red[TT + warp] = v;
    }
    __syncthreads();
    v = 0.;
    if (warp == 0) {
        v = red[TT];
        for (int w = 1; w < nw; w++) v += red[TT + w];
    }
    return v;
}

constexpr int TEAM_WORDS = (TEAM_MAX + 31) / 32;

// One warp: the blocks' partial sums, then their sum in a fixed order (lane 0).
__device__ __forceinline__ bool team_poll(const ulonglong2 *slots, int G, unsigned ep, double (&v)[TEAM_WORDS],
                                          int limit = POLL_MAX) {
    return ll_poll(slots, SLOT * (int)(threadIdx.x & 31), SLOT * 32, SLOT * G, ep, v, limit);
}
__device__ __forceinline__ double team_add(const double (&v)[TEAM_WORDS], int G) {
    double s = v[0];
#pragma unroll
    for (int j = 1; j < TEAM_WORDS; j++)
        if (32 * j < G) s += v[j];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        if (o < G) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

struct TeamArgs {
    const int32_t *r0, *slice0, *cmin, *cmax;  // per block: first row, first slice, column window
    const int32_t *slen;
    const int64_t *soff;
    const double *sval;
    const uint16_t *scol;
    const int32_t *colbase;
    const int64_t *dof_of_row;
    const int32_t *start;
    int bs;
    const double *dval;      // [6][n] non-zeros of each row of the block inverse
    const uint32_t *dinf;    // [n] their number and, 3 bits each, their columns
    double *u, *r, *p;
    int64_t n;
    double *scal;        // [rz_index] rz in / out, [2] r.r out, [6] iterations run, [7] 1: a poll gave up
    int rz_index;
    ulonglong2 *z;       // [n]
    ulonglong2 *slots;   // [3][TEAM_MAX] slots: p.q, r.z, r.r
    unsigned epoch;      // of the launch's first iteration
    int maxiter;         // iterations of this launch at most
    int chunk, phase;    // convergence is looked at where phase + iterations is a multiple of chunk
    double stop2;        // r.r at which to stop
    int wmax, nmax;      // largest window and row count of a block
};

// Entries per lane that a block of at most TT / L rows keeps in registers.
constexpr int team_regs(int L) { return L == 1 ? 28 : L == 2 ? 16 : 8; }

template <int L, bool REG>
__global__ void __launch_bounds__(TT, 1) team_pcg_kernel(TeamArgs a) {
    extern __shared__ __align__(16) double sm[];
    __shared__ double red[TT + 4];
    __shared__ double bc[3];
    __shared__ int fail, fresh, dmax;  // a poll gave up; beta = 0; most non-zeros in a row of the block inverses
    const int tid = threadIdx.x, G = gridDim.x, bid = blockIdx.x;
    const int r0 = a.r0[bid], n = a.r0[bid + 1] - r0, c0 = a.cmin[bid], W = n > 0 ? a.cmax[bid] - c0 + 1 : 0;
    const int s0 = a.slice0[bid];
    double *pw = sm, *rs = pw + a.wmax, *us = rs + a.nmax, *qs = us + a.nmax;
    int *rfirst = reinterpret_cast<int *>(qs + a.nmax);  // first row of the row's node
    uint32_t *rinf = reinterpret_cast<uint32_t *>(rfirst + a.nmax);
    const int own = r0 - c0;  // window index of the block's first row
    ulonglong2 *slot_pq = a.slots, *slot_rz = slot_pq + SLOT * TEAM_MAX, *slot_rr = slot_rz + SLOT * TEAM_MAX;
    if (tid == 0) {
        fail = 0;
        dmax = 0;
    }
    __syncthreads();
    for (int c = tid; c < W; c += TT) pw[c] = a.p[c0 + c];
    for (int i = tid; i < n; i += TT) {
        rs[i] = a.r[r0 + i];
        us[i] = a.u[r0 + i];
        rfirst[i] = a.start[a.dof_of_row[r0 + i] / a.bs] - r0;
        rinf[i] = a.dinf[r0 + i];
        atomicMax(&dmax, (int)(rinf[i] & 7));
    }
    double rz = a.scal[a.rz_index], rr = 0., irz = 0.;
    const int rows32 = (n * L + 31) & ~31;
    // REG: the block's rows of the matrix and of the block inverses stay in registers
    constexpr int MK = REG ? team_regs(L) : 4;
    double dreg[6], vreg[MK];
    uint32_t creg[MK / 2], dinf = 0;
    int mylen = 0, dfirst = 0, cb = 0;
    if (REG) {
        dinf = tid < n ? a.dinf[r0 + tid] : 0;
        dfirst = tid < n ? a.start[a.dof_of_row[r0 + tid] / a.bs] - r0 : 0;
#pragma unroll
        for (int k = 0; k < 6; k++) dreg[k] = k < (int)(dinf & 7) ? a.dval[k * a.n + r0 + tid] : 0.;
        if (tid < rows32) {
            mylen = a.slen[s0 + (tid >> 5)];
            cb = tid / L < n ? a.colbase[r0 + tid / L] - c0 : 0;
        }
        const int64_t o = tid < rows32 ? a.soff[s0 + (tid >> 5)] * 32 + (tid & 31) : 0;
        uint32_t c = 0;
#pragma unroll
        for (int k = 0; k < MK; k++) {
            vreg[k] = k < mylen ? a.sval[o + 32 * k] : 0.;
            if (k < mylen) c = cb + a.scol[o + 32 * k];  // window index (the window has at most 28,000 columns)
            if (k & 1) creg[k / 2] |= c << 16;
            else creg[k / 2] = c;
        }
    }
    __syncthreads();
    int it = 0, left = a.chunk - a.phase;  // iterations to the next look at convergence
    bool stop = it >= a.maxiter;
    const bool few = dmax <= 3;
    const int nwq = max(1, min(rows32, TT) >> 5), nwz = max(1, (min(n, TT) + 31) >> 5);
    while (!stop) {
        const unsigned ep = a.epoch + (unsigned)it;
        // q = K p over the block's rows, and p.q
        double dot = 0.;
        for (int t = tid; t < rows32; t += REG ? (1 << 20) : TT) {
            const int i = t / L;
            double acc = 0.;
            if (REG) {
                // four entries at a time; those past the slice's end are zeros
#pragma unroll
                for (int k = 0; k < MK; k += 4)
                    if (k < mylen) {
                        const double x0 = pw[creg[k / 2] & 0xffff], x1 = pw[creg[k / 2] >> 16];
                        const double x2 = pw[creg[k / 2 + 1] & 0xffff], x3 = pw[creg[k / 2 + 1] >> 16];
                        acc += vreg[k] * x0;
                        acc += vreg[k + 1] * x1;
                        acc += vreg[k + 2] * x2;
                        acc += vreg[k + 3] * x3;
                    }
            } else {
                const int slice = s0 + (t >> 5);
                const int len = __ldg(a.slen + slice);
                const int64_t o = __ldg(a.soff + slice) * 32 + (t & 31);
                const double *sv = a.sval + o;
                const uint16_t *sc = a.scol + o;
                const double *xb = pw + (i < n ? __ldg(a.colbase + r0 + i) - c0 : 0);
#pragma unroll 9
                for (int k = 0; k < len; k++) acc += __ldg(sv + 32 * k) * xb[__ldg(sc + 32 * k)];
            }
#pragma unroll
            for (int o2 = L / 2; o2 > 0; o2 >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o2);
            if (i < n) {
                qs[i] = acc;
                if (L == 1 || (t & (L - 1)) == 0) dot += pw[own + i] * acc;
            }
        }
        dot = team_block_sum(dot, nwq, L, red);
        if (tid < 32) {
            if (tid == 0) ll_store(slot_pq + SLOT * bid, dot, ep);
            double v[TEAM_WORDS];
            if (!team_poll(slot_pq, G, ep, v, it == 0 ? POLL_FIRST : POLL_MAX)) fail = 1;
            const double pq = team_add(v, G);
            if (tid == 0) bc[0] = pq != 0. ? rz / pq : 0.;
        } else if (tid >= TZ) {
            irz = fabs(rz) > 1e-290 ? 1. / rz : 0.;  // for beta, while alpha is waited for
        }
        __syncthreads();
        const double alpha = bc[0];
        for (int i = tid; i < n; i += REG ? (1 << 20) : TT) rs[i] -= alpha * qs[i];
        __syncthreads();
        // z = Minv r, r.z (and r.r where convergence is looked at)
        it++;
        const bool look = --left == 0 || it >= a.maxiter;
        if (left == 0) left = a.chunk;
        double lrz = 0., lrr = 0.;
        for (int i = tid; i < n; i += REG ? (1 << 20) : TT) {
            const uint32_t inf = REG ? dinf : rinf[i];
            const double *rn = rs + (REG ? dfirst : rfirst[i]);
            double acc = 0.;
            if (REG) {
#pragma unroll
                for (int k = 0; k < 3; k++) acc += dreg[k] * rn[(inf >> (3 + 3 * k)) & 7];
                if (!few) {
#pragma unroll
                    for (int k = 3; k < 6; k++) acc += dreg[k] * rn[(inf >> (3 + 3 * k)) & 7];
                }
            } else {
                const int cnt = inf & 7;
                for (int k = 0; k < cnt; k++) acc += __ldg(a.dval + k * a.n + r0 + i) * rn[(inf >> (3 + 3 * k)) & 7];
            }
            ll_store(a.z + r0 + i, acc, ep);
            lrz += rs[i] * acc;
            if (look) lrr += rs[i] * rs[i];
        }
        lrz = team_block_sum(lrz, nwz, 1, red);
        if (tid == 0) ll_store(slot_rz + SLOT * bid, lrz, ep);
        if (look) {
            __syncthreads();
            lrr = team_block_sum(lrr, nwz, 1, red);
            if (tid == 0) ll_store(slot_rr + SLOT * bid, lrr, ep);
        }
        for (int i = tid; i < n; i += REG ? (1 << 20) : TT) us[i] += alpha * pw[own + i];
        // p = z + beta p over the window.  The words of z are asked for once
        // r.z has come from every block: polling them earlier would crowd the
        // lines that their owners are about to write
        double zv[4], vz[TEAM_WORDS], vr[TEAM_WORDS];
        if (tid >= TZ) {
            if (!team_poll(slot_rz, G, ep, vz)) fail = 1;
            if (look && !team_poll(slot_rr, G, ep, vr)) fail = 1;
        }
        __syncthreads();
        if (tid < TZ) {
            if (!ll_poll(a.z + c0, tid, TZ, W, ep, zv)) fail = 1;
        } else {
            const double rzn = team_add(vz, G), s = look ? team_add(vr, G) : 0.;
            if (tid == TZ) {
                const double be = rz == 0. ? 0. : irz != 0. ? rzn * irz : rzn / rz;
                bc[0] = be;
                fresh = be == 0.;
                bc[1] = rzn;
                bc[2] = s;
            }
        }
        __syncthreads();
        // (comparisons of doubles run on the FP64 pipe too: one warp makes them)
        const double beta = bc[0];
        const bool reset = fresh;
        rz = bc[1];
        if (look) rr = bc[2];
        if (tid < TZ && tid < W) {
            for (int c1 = tid;;) {
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int c = c1 + j * TZ;
                    if (c < W) pw[c] = reset ? zv[j] : zv[j] + beta * pw[c];
                }
                c1 += 4 * TZ;
                if (c1 >= W) break;
                if (!ll_poll(a.z + c0, c1, TZ, W, ep, zv)) fail = 1;
            }
        }
        __syncthreads();
        stop = fail || it >= a.maxiter || (look && !(rr > a.stop2 && rr <= 1.7e308));
    }
    for (int i = tid; i < n; i += TT) {
        a.u[r0 + i] = us[i];
        a.r[r0 + i] = rs[i];
        a.p[r0 + i] = pw[own + i];
    }
    if (fail && tid == 0) a.scal[7] = 1.;
    if (bid == 0 && tid == 0) {
        a.scal[a.rz_index] = rz;
        a.scal[2] = rr;
        a.scal[6] = (double)it;
    }
}

// Non-zeros of each row of the block inverses (a flat plate's blocks couple
// (u, v, rz) and (w, rx, ry) only).
__global__ void __launch_bounds__(256) team_blocks_kernel(int64_t n, const int64_t *dof_of_row, const int32_t *start,
                                                          const int8_t *size, int bs, const double *Dinv,
                                                          double *dval, uint32_t *dinf) {
    const int64_t row = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (row >= n) return;
    const int64_t node = dof_of_row[row] / bs;
    const int i = (int)(row - start[node]), b = size[node];
    int cnt = 0;
    uint32_t inf = 0;
    for (int k = 0; k < b; k++) {
        const double v = Dinv[36 * node + 6 * i + k];
        if (v != 0.) {
            dval[cnt * n + row] = v;
            cnt++;
            inf |= (uint32_t)k << (3 * cnt);
        }
    }
    dinf[row] = inf | (uint32_t)cnt;
}

// Block boundaries: rows split by stored entries, moved back to the first row
// of the node they fall in.
__global__ void team_split_kernel(int G, int64_t n, int64_t nnz, const int64_t *rowptr, const int64_t *dof_of_row,
                                  const int32_t *start, int bs, int32_t *r0) {
    const int b = threadIdx.x;
    if (b > G) return;
    if (b == 0 || b == G) {
        r0[b] = b == 0 ? 0 : (int32_t)n;
        return;
    }
    const int64_t want = nnz / G * b;
    int64_t lo = 0, hi = n;  // first row whose entries start at or after want
    while (lo < hi) {
        const int64_t m = (lo + hi) / 2;
        if (rowptr[m] < want) lo = m + 1;
        else hi = m;
    }
    r0[b] = lo < n ? start[dof_of_row[lo] / bs] : (int32_t)n;
}

// Column window of each block: its rows' columns and its own rows.
__global__ void __launch_bounds__(256) team_window_kernel(const int32_t *r0, const int64_t *rowptr,
                                                          const int32_t *colind, int32_t *cmin, int32_t *cmax) {
    __shared__ int lo, hi;
    const int a = r0[blockIdx.x], e = r0[blockIdx.x + 1];
    if (threadIdx.x == 0) {
        lo = a;
        hi = e - 1;
    }
    __syncthreads();
    int l = a, h = e - 1;
    for (int i = a + threadIdx.x; i < e; i += blockDim.x)
        if (rowptr[i + 1] > rowptr[i]) {
            l = min(l, colind[rowptr[i]]);
            h = max(h, colind[rowptr[i + 1] - 1]);
        }
    atomicMin(&lo, l);
    atomicMax(&hi, h);
    __syncthreads();
    if (threadIdx.x == 0) {
        cmin[blockIdx.x] = lo;
        cmax[blockIdx.x] = hi;
    }
}

// Lengths (entries per lane) and places of a block's slices.
__global__ void __launch_bounds__(256) team_count_kernel(const int32_t *r0, const int32_t *slice0, int L,
                                                         const int64_t *rowptr, const double *vals, int32_t *slen,
                                                         int64_t *soff, unsigned long long *total) {
    const int a = r0[blockIdx.x], e = r0[blockIdx.x + 1], s0 = slice0[blockIdx.x], s1 = slice0[blockIdx.x + 1];
    const int lane = threadIdx.x & 31, per = 32 / L;
    for (int s = s0 + (threadIdx.x >> 5); s < s1; s += blockDim.x >> 5) {
        int longest = 0;
        for (int j = 0; j < per; j++) {
            const int row = a + (s - s0) * per + j;
            if (row >= e) break;
            const int64_t kb = rowptr[row], ke = rowptr[row + 1];
            int cnt = 0;
            for (int64_t k = kb; k < ke; k += 32)
                cnt += __popc(__ballot_sync(0xffffffffu, k + lane < ke && vals[k + lane < ke ? k + lane : kb] != 0.));
            longest = max(longest, (cnt + L - 1) / L);
        }
        if (lane == 0) {
            slen[s] = longest;
            soff[s] = (int64_t)atomicAdd(total, (unsigned long long)longest);
            atomicMax(total + 1, (unsigned long long)longest);
        }
    }
}

// Entry k of a row goes to lane k % L of its L lanes; lanes that end early
// repeat the row's last column with the value 0.
__global__ void __launch_bounds__(256) team_fill_kernel(const int32_t *r0, const int32_t *slice0, int L,
                                                        const int64_t *rowptr, const uint16_t *col16,
                                                        const double *vals, const int32_t *slen,
                                                        const int64_t *soff, double *sval, uint16_t *scol) {
    const int a = r0[blockIdx.x], e = r0[blockIdx.x + 1], s0 = slice0[blockIdx.x], s1 = slice0[blockIdx.x + 1];
    const int lane = threadIdx.x & 31, per = 32 / L;
    for (int s = s0 + (threadIdx.x >> 5); s < s1; s += blockDim.x >> 5) {
        const int row = a + (s - s0) * per + lane / L, sub = lane % L, len = slen[s];
        double *sv = sval + soff[s] * 32 + lane;
        uint16_t *sc = scol + soff[s] * 32 + lane;
        int at = 0, nz = 0;
        uint16_t c = 0;
        if (row < e) {
            const int64_t ke = rowptr[row + 1];
            for (int64_t k = rowptr[row]; k < ke; k++) {
                const double v = vals[k];
                if (v != 0.) {
                    c = col16[k];
                    if (nz % L == sub) {
                        sv[32 * at] = v;
                        sc[32 * at] = c;
                        at++;
                    }
                    nz++;
                }
            }
        }
        for (; at < len; at++) {
            sv[32 * at] = 0.;
            sc[32 * at] = c;
        }
    }
}

typedef void (*TeamKernel)(TeamArgs);

TeamKernel team_kernel(int L, bool reg) {
    switch (L) {
        case 1: return reg ? team_pcg_kernel<1, true> : team_pcg_kernel<1, false>;
        case 2: return reg ? team_pcg_kernel<2, true> : team_pcg_kernel<2, false>;
        case 4: return reg ? team_pcg_kernel<4, true> : team_pcg_kernel<4, false>;
        default: return reg ? team_pcg_kernel<8, true> : team_pcg_kernel<8, false>;
    }
}

template <typename T>
bool get(T **p, size_t n) {
    return cudaMalloc((void **)p, (n ? n : 1) * sizeof(T)) == cudaSuccess;
}

}  // namespace

void team_free(fe3d_team *t) {
    if (!t) return;
    cudaFree(t->r0);
    cudaFree(t->slice0);
    cudaFree(t->cmin);
    cudaFree(t->cmax);
    cudaFree(t->slen);
    cudaFree(t->soff);
    cudaFree(t->sval);
    cudaFree(t->scol);
    cudaFree(t->total);
    cudaFree(t->z);
    cudaFree(t->dval);
    cudaFree(t->dinf);
    cudaFree(t->slots);
    delete t;
}

// Splits the solver's system over blocks; nullptr where it does not fit (or
// memory is short): the launch-per-kernel iteration is used then.
fe3d_team *team_create(const fe3d_solver *s, cudaStream_t st) {
    const fe3d_pattern *p = s->pat;
    if (s->n < 1 || s->n > kTeamMaxRows || !p->col16) return nullptr;
    int dev = 0, sms = 0, coop = 0, optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess || !coop)
        return nullptr;
    fe3d_team *t = new fe3d_team();
    const int64_t g = (s->n + kTeamRows - 1) / kTeamRows;
    t->G = (int)(g < 1 ? 1 : g > TEAM_MAX ? TEAM_MAX : g);
    if (t->G > sms) t->G = sms;
    const int G = t->G;
    int32_t h[3 * (TEAM_MAX + 1)];
    bool ok = get(&t->r0, G + 1) && get(&t->slice0, G + 1) && get(&t->cmin, G) && get(&t->cmax, G) &&
              get(&t->total, 2) && get(&t->z, s->n) && get(&t->slots, 3 * SLOT * TEAM_MAX) &&
              get(&t->dval, 6 * s->n) && get(&t->dinf, s->n);
    if (ok) {
        team_split_kernel<<<1, TEAM_MAX + 8, 0, st>>>(G, s->n, p->nnz, p->rowptr, p->dof_of_row, s->start, s->bs, t->r0);
        team_window_kernel<<<G, 256, 0, st>>>(t->r0, p->rowptr, p->colind, t->cmin, t->cmax);
        ok = cudaMemcpyAsync(h, t->r0, sizeof(int32_t) * (G + 1), cudaMemcpyDeviceToHost, st) == cudaSuccess &&
             cudaMemcpyAsync(h + G + 1, t->cmin, sizeof(int32_t) * G, cudaMemcpyDeviceToHost, st) == cudaSuccess &&
             cudaMemcpyAsync(h + 2 * G + 1, t->cmax, sizeof(int32_t) * G, cudaMemcpyDeviceToHost, st) == cudaSuccess &&
             cudaMemsetAsync(t->z, 0, sizeof(ulonglong2) * s->n, st) == cudaSuccess &&
             cudaMemsetAsync(t->slots, 0, sizeof(ulonglong2) * 3 * SLOT * TEAM_MAX, st) == cudaSuccess &&
             cudaStreamSynchronize(st) == cudaSuccess;
    }
    if (ok) {
        for (int b = 0; b < G; b++) {
            const int n = h[b + 1] - h[b], w = n > 0 ? h[2 * G + 1 + b] - h[G + 1 + b] + 1 : 0;
            if (n < 0) ok = false;
            if (n > t->nmax) t->nmax = n;
            if (w > t->wmax) t->wmax = w;
        }
        t->smem = sizeof(double) * ((size_t)t->wmax + 3 * (size_t)t->nmax) + 2 * sizeof(int) * (size_t)t->nmax;
        ok = ok && t->smem + 8192 <= (size_t)optin;
    }
    if (ok) {
        // lanes per row: the fewest FP64 instructions on one sub-partition's
        // warps for a row of 27 non-zeros (a node of a flat plate's inside)
        int best = 1 << 30;
        for (int L = 1; L <= 8; L *= 2) {
            int cost = 28 / L + 1, lg = L;
            while (lg > 1) {
                cost++;
                lg /= 2;
            }
            cost *= (t->nmax * L + 127) / 128;
            if (cost < best) {
                best = cost;
                t->L = L;
            }
        }
        const int per = 32 / t->L;
        int32_t first[TEAM_MAX + 1];
        first[0] = 0;
        for (int b = 0; b < G; b++) first[b + 1] = first[b] + (h[b + 1] - h[b] + per - 1) / per;
        ok = get(&t->slen, first[G]) && get(&t->soff, first[G]) &&
             cudaMemcpyAsync(t->slice0, first, sizeof(int32_t) * (G + 1), cudaMemcpyHostToDevice, st) == cudaSuccess &&
             cudaStreamSynchronize(st) == cudaSuccess;
        for (int reg = 0; ok && reg < 2; reg++) {
            int res = 0;
            ok = cudaFuncSetAttribute(team_kernel(t->L, reg), cudaFuncAttributeMaxDynamicSharedMemorySize, optin - 8192) ==
                     cudaSuccess &&
                 cudaOccupancyMaxActiveBlocksPerMultiprocessor(&res, team_kernel(t->L, reg), TT, t->smem) ==
                     cudaSuccess &&
                 res >= 1;
        }
    }
    if (!ok) {
        (void)cudaGetLastError();
        team_free(t);
        return nullptr;
    }
    return t;
}

int team_plan(fe3d_team *t, const fe3d_solver *s, cudaStream_t st) {
    FE3D_CUDA(cudaMemsetAsync(t->total, 0, 2 * sizeof(unsigned long long), st));
    team_count_kernel<<<t->G, 256, 0, st>>>(t->r0, t->slice0, t->L, s->pat->rowptr, s->vals, t->slen, t->soff,
                                            t->total);
    FE3D_CHECK_LAUNCH();
    return FE3D_OK;
}

int team_build(fe3d_team *t, const fe3d_solver *s, unsigned long long total, unsigned long long longest,
               cudaStream_t st) {
    t->reg = t->nmax * t->L <= TT && (int64_t)longest <= team_regs(t->L);
    const int64_t entries = 32 * (int64_t)total;
    if (entries > t->cap) {
        cudaFree(t->sval);
        cudaFree(t->scol);
        t->sval = nullptr;
        t->scol = nullptr;
        t->cap = 0;
        if (!get(&t->sval, entries) || !get(&t->scol, entries)) {
            (void)cudaGetLastError();
            return FE3D_ERR_NOMEM;
        }
        t->cap = entries;
    }
    team_fill_kernel<<<t->G, 256, 0, st>>>(t->r0, t->slice0, t->L, s->pat->rowptr, s->pat->col16, s->vals, t->slen,
                                           t->soff, t->sval, t->scol);
    team_blocks_kernel<<<(unsigned)((s->n + 255) / 256), 256, 0, st>>>(s->n, s->pat->dof_of_row, s->start, s->size,
                                                                       s->bs, s->Dinv, t->dval, t->dinf);
    FE3D_CHECK_LAUNCH();
    return FE3D_OK;
}

int team_run(fe3d_team *t, const fe3d_solver *s, double *u, int rz_index, int maxiter, int chunk, int phase,
             double stop2, cudaStream_t st) {
    if (t->epoch > 0xffffffffu - (unsigned)maxiter - 2u) {
        FE3D_CUDA(cudaMemsetAsync(t->z, 0, sizeof(ulonglong2) * s->n, st));
        FE3D_CUDA(cudaMemsetAsync(t->slots, 0, sizeof(ulonglong2) * 3 * SLOT * TEAM_MAX, st));
        t->epoch = 1;
    }
    TeamArgs a{t->r0, t->slice0, t->cmin, t->cmax, t->slen, t->soff, t->sval, t->scol, s->pat->colbase,
               s->pat->dof_of_row, s->start, s->bs, t->dval, t->dinf, u, s->r, s->p, s->n, s->scal, rz_index,
               t->z, t->slots, t->epoch, maxiter, chunk, phase, stop2, t->wmax, t->nmax};
    t->epoch += (unsigned)maxiter + 1u;
    FE3D_CUDA(cudaMemsetAsync(s->scal + 6, 0, 2 * sizeof(double), st));
    void *args[] = {&a};
    if (cudaLaunchCooperativeKernel((const void *)team_kernel(t->L, t->reg), dim3(t->G), dim3(TT), args, t->smem, st) !=
        cudaSuccess)
        return FE3D_ERR_LAUNCH;
    return FE3D_OK;
}

}  // namespace fe3d
