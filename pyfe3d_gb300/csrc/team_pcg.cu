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
// Several independent systems run in one launch, each on a team of its own
// blocks (bpcg.cu); teams do not wait for one another, and once the blocks of
// finished teams pass a share of the grid the others stop at their next look at
// the residual, so that the host can deal the blocks out anew.
//
// Exchange: every value that crosses blocks (z, the partial sums of p.q, r.z
// and r.r) travels as two 8-byte words, each holding half of the double and
// the iteration's number.  A reader polls the words themselves: no fence, no
// counter, one trip through L2 per exchange, two exchanges per iteration.  A
// slot is written again only after every reader of its previous value has
// sent something that the writer waited for.  Each block makes the same sum over
// blocks, so all hold the same scalars, and the result of a launch with one system
// does not depend on scheduling (with several, when a team stops for the blocks to
// be dealt out anew depends on when the others finish).  Every poll is bounded; a block that
// gives up raises a flag and returns.  The partial sums sit a 128-byte line
// apart: 152 blocks exchange a value in 3.1k cycles, 5.8k with four to a line.
//
// Matrix: the non-zero values in slices of 32 / L rows, L lanes per row (L
// grows as the rows per block shrink), anchored at the block's first row and
// copied to shared memory where they fit.  An FP64 instruction holds its
// sub-partition's pipe for 64 cycles whatever its active lanes, so sums over
// lanes and blocks are made with integer reductions (fixed_sum), comparisons of
// doubles with integer operations, and rare FP64 work stands behind branches
// and calls.
//
// Measured on clamped perturbed plates, us per iteration, three launches /
// resident, rows in registers and FP64 sums / now: 486 rows 20.8 / 5.9 / 5.8,
// 2,166 rows 20.8 / 6.7 / 5.7, 9,126 rows 22.2 / 8.2 / 6.6, 58,806 rows 25.5 /
// 11.6 / 9.8, 237,606 rows 43 / 25 / 22.6, 536,406 rows 69.5 / 60 / 45 (there the
// matrix no longer fits L2).  Other matrices, three launches / resident: laminated
// cylinder (54 non-zeros a row) 1,080 rows 20.1 / 6.2, 42,480 rows 28.3 / 12.8,
// 387,714 rows 91 / 66; laminated panel 616,324 rows 131 / 90; lattice of nodes with
// 3 DOFs 81,000 rows 25.3 / 15.3; plate with shuffled nodes 20,184 rows 25.6 / 13.9;
// chain with one node joined to 200 others (rows of 1,200 entries) 6,000 rows 44 / 46.  At 20,886 rows a block's 12,700 cycles are: product
// 3,300, sums over the block 2,800, waiting for p.q 1,800, for r.z and z 3,000, z 400,
// sums over blocks and division 1,900 -- of which the FP64 pipe needs 3,900.
#include <limits.h>

#include <vector>

#include "common.cuh"
#include "fe3d_internal.h"
#include "fixed_sum.h"
#include "quotient.cuh"

namespace fe3d {
namespace {

constexpr int TT = 512;               // threads per block
constexpr int TEAM_MAX = kSMs;        // blocks of one system
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
                                        double (&v)[N], int limit) {
#pragma unroll
    for (int j = 0; j < N; j++) v[j] = 0.;
    if (i0 >= lim) return true;
    bool all = false;
    for (int spin = 0; !all && spin < limit; spin++) {
        unsigned long long a[N], b[N];
#pragma unroll
        for (int j = 0; j < N; j++) {
            a[j] = b[j] = (unsigned long long)ep << 32;
            if (i0 + j * step < lim)
                asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
                             : "=l"(a[j]), "=l"(b[j]) : "l"(base + i0 + j * step) : "memory");
        }
        all = true;
#pragma unroll
        for (int j = 0; j < N; j++) {
            all &= (unsigned)(a[j] >> 32) == ep && (unsigned)(b[j] >> 32) == ep;
            v[j] = __hiloint2double((int)(unsigned)b[j], (int)(unsigned)a[j]);
        }
    }
    return all;
}

// Sum of N doubles a lane over the warp (all lanes get it), in fixed point
// relative to the largest (fixed_sum.h), the limbs added with the warp's integer
// reductions: free of the FP64 pipe, where a tree of five additions takes 450
// cycles and this 150.  Infinities, NaN and sums near the ends of the range are
// left to such a tree (plain_sum, a call, so that the compiler does not predicate
// its additions into the common path).
__device__ __noinline__ double plain_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __noinline__ double plain_add(double a, double b) { return a + b; }
template <int N>
__device__ __forceinline__ double fixed_sum_of(const double (&v)[N]) {
    unsigned top = 0;
#pragma unroll
    for (int j = 0; j < N; j++) top = max(top, (unsigned)__double2hiint(v[j]) & 0x7fffffffu);
    const int emax = (int)(__reduce_max_sync(0xffffffffu, top) >> 20);
    if (!fixed_range(emax)) {
        double s = v[0];
        for (int j = 1; j < N; j++) s = plain_add(s, v[j]);
        return plain_sum(s);
    }
    static_assert(32 * N <= FS_TERMS, "terms of a fixed-point sum");
    FixedLimbs f{0u, 0u, 0};
#pragma unroll
    for (int j = 0; j < N; j++) fixed_add(f, __double_as_longlong(v[j]), emax);
    f.lo = __reduce_add_sync(0xffffffffu, f.lo);
    f.mid = __reduce_add_sync(0xffffffffu, f.mid);
    f.hi = __reduce_add_sync(0xffffffffu, f.hi);
    return __longlong_as_double((long long)fixed_round(f, emax));
}

constexpr int TEAM_WORDS = (TEAM_MAX + 31) / 32;

// Calls, not inlined: the iteration's code runs once per iteration in one warp
// at a time, and the less of it there is the more stays in the instruction cache.
__device__ __noinline__ double fixed_sum(double v) {
    const double one[1] = {v};
    return fixed_sum_of(one);
}
__device__ __noinline__ double fixed_sum(double a, double b, double c, double d, double e) {
    const double five[5] = {a, b, c, d, e};
    return fixed_sum_of(five);
}
__device__ __forceinline__ double fixed_sum(const double (&v)[TEAM_WORDS]) {
    static_assert(TEAM_WORDS == 5, "words per lane");
    return fixed_sum(v[0], v[1], v[2], v[3], v[4]);
}

// Sum over the block of values held by its first nw warps, valid in warp 0.
// red: 16 doubles; a block-wide barrier has to come before the next use.
__device__ __forceinline__ double team_block_sum(double v, int nw, double *red) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp < nw) {
        v = fixed_sum(v);
        if (nw == 1) return v;
        if (lane == 0) red[warp] = v;
    }
    if (nw == 1) return 0.;
    __syncthreads();
    if (warp != 0) return 0.;
    if (nw > 4) return fixed_sum(lane < nw ? red[lane] : 0.);
    v = red[0];
#pragma unroll 1
    for (int w = 1; w < nw; w++) v += red[w];  // 64 cycles each, fixed_sum 320
    return v;
}

// One warp: the blocks' partial sums.
__device__ __forceinline__ bool team_poll(const ulonglong2 *slots, int G, unsigned ep, double (&v)[TEAM_WORDS],
                                          int limit) {
    return ll_poll(slots, SLOT * (int)(threadIdx.x & 31), SLOT * 32, SLOT * G, ep, v, limit);
}

struct TeamArgs {
    // per block: rows, first slice, column window, and its team: first block,
    // number of blocks and system
    const int32_t *rbeg, *rend, *slice0, *cmin, *cmax, *tfirst, *tcount, *tsys;
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
    double *rz, *rr;         // per system: r.z in and out, r.r out
    TeamSys *sys;            // per system: limits in, iterations run out
    ulonglong2 *z;           // [n]
    ulonglong2 *slots;       // [3][blocks] slots: p.q, r.z, r.r
    unsigned epoch;          // of the launch's first iteration
    int chunk;               // convergence is looked at every chunk iterations
    int *done;               // [0] blocks of finished teams, [1] a poll gave up
    int enough;              // finished blocks at which the other teams stop too
    int poll, poll_first;    // polls of a word before a block gives up, and at the first exchange
};

// Where a block's rows of the matrix are between two iterations, and how they
// are read: from shared memory where they fit; else from L1 and L2 in a plain
// loop (NEAR), or a chunk ahead of their use where all rows together exceed what
// L2 holds next to the vectors (FAR, above kFarEntries entries of 10 bytes).  us
// per iteration: 58,806 rows SHARED 10.2, NEAR 10.6, FAR 11.1; 84,966 rows 12.7,
// 13.6, 14.0; 133,206 rows (too many for SHARED) NEAR 14.8, FAR 16.6; 237,606
// rows 23.4, 25.9; 314,646 rows 31.2, 32.0; 536,406 rows 50, 47.
enum { SHARED, NEAR, FAR };
constexpr int64_t kFarEntries = 8400000;

template <int L, int ROWS>
__global__ void __launch_bounds__(TT, 1) team_pcg_kernel(TeamArgs a) {
    extern __shared__ __align__(16) double sm[];
    __shared__ double red[TT / 32];
    __shared__ double bc[4];
    // a poll gave up; beta = 0; others finished
    __shared__ int fail, fresh, yield;
    const int tid = threadIdx.x, G = a.tcount[blockIdx.x], t0 = a.tfirst[blockIdx.x], bid = blockIdx.x - t0;
    const int sys = a.tsys[blockIdx.x];
    const int r0 = a.rbeg[blockIdx.x], n = a.rend[blockIdx.x] - r0, c0 = a.cmin[blockIdx.x];
    const int W = n > 0 ? a.cmax[blockIdx.x] - c0 + 1 : 0, s0 = a.slice0[blockIdx.x];
    const TeamSys lim = a.sys[sys];
    double *pw = sm, *rs = pw + W, *us = rs + n, *qs = us + n;
    const int ns = (n * L + 31) >> 5;
    int64_t *sinf = reinterpret_cast<int64_t *>(qs + n);  // offset << 16 | length of the block's slices
    int *rfirst = reinterpret_cast<int *>(sinf + ns);     // first row of the row's node
    uint32_t *rinf = reinterpret_cast<uint32_t *>(rfirst + n);
    uint16_t *rbase = reinterpret_cast<uint16_t *>(rinf + n);  // window index of the row's column base
    const int own = r0 - c0;  // window index of the block's first row
    ulonglong2 *slot_pq = a.slots + SLOT * t0, *slot_rz = slot_pq + SLOT * gridDim.x,
               *slot_rr = slot_rz + SLOT * gridDim.x;
    if (tid == 0) fail = 0;
    __syncthreads();
    for (int c = tid; c < W; c += TT) pw[c] = a.p[c0 + c];
    for (int i = tid; i < n; i += TT) {
        rs[i] = a.r[r0 + i];
        us[i] = a.u[r0 + i];
        rfirst[i] = a.start[a.dof_of_row[r0 + i] / a.bs] - r0;
        rinf[i] = a.dinf[r0 + i];
        // (a row without entries has the base 0, which the window may not hold)
        rbase[i] = (uint16_t)max(a.colbase[r0 + i] - c0, 0);
    }
    for (int i = tid; i < ns; i += TT) sinf[i] = a.soff[s0 + i] << 16 | a.slen[s0 + i];
    double *mv = nullptr;      // SHARED: the block's slices, and their places in sinf
    uint16_t *mc = nullptr;
    if (ROWS == SHARED) {
        const size_t base = (reinterpret_cast<char *>(rbase + n) - reinterpret_cast<char *>(sm) + 7) & ~(size_t)7;
        mv = reinterpret_cast<double *>(reinterpret_cast<char *>(sm) + base);
        __syncthreads();
        int at = 0, tot = 0;
        for (int i = 0; i < ns; i++) tot += (int)(sinf[i] & 0xffff);
        mc = reinterpret_cast<uint16_t *>(mv + 32 * tot);
        for (int i = 0; i < ns; i++) {
            const int64_t si = sinf[i];
            const int len = (int)(si & 0xffff);
            if ((i & (TT / 32 - 1)) == tid >> 5)
                for (int e = 0; e < len; e++) {
                    const int64_t o = 32 * ((si >> 16) + e) + (tid & 31);
                    mv[32 * (at + e) + (tid & 31)] = a.sval[o];
                    mc[32 * (at + e) + (tid & 31)] = a.scol[o];
                }
            at += len;
        }
        __syncthreads();
        if (tid == 0) {
            at = 0;
            for (int i = 0; i < ns; i++) {
                const int len = (int)(sinf[i] & 0xffff);
                sinf[i] = (int64_t)at << 16 | len;
                at += len;
            }
        }
    }
    double rz = a.rz[sys], rr = 0., irz = 0.;
    __syncthreads();
    const int rows32 = (n * L + 31) & ~31;
    double dreg[3];
    // the first entries of the thread's first row of the block inverses
    const uint32_t dinf = tid < n ? rinf[tid] : 0;
#pragma unroll
    for (int k = 0; k < 3; k++) dreg[k] = k < (int)(dinf & 7) ? a.dval[k * a.n + r0 + tid] : 0.;
    __syncthreads();
    // FAR: CH entries a lane of the warp's slice from entry k on, loaded one
    // chunk ahead of their use (the first of an iteration at the end of the one
    // before), past the slice's end its last entry again
    constexpr int CH = 7;
    double cv[CH];
    uint16_t cc[CH];
    auto fetch = [&](int64_t si, int k, double(&v)[CH], uint16_t(&c)[CH]) {
        const int last = (int)(si & 0xffff) - 1;
        if (k > last) return;
        const double *sv = a.sval + 32 * (si >> 16) + (tid & 31);
        const uint16_t *sc = a.scol + 32 * (si >> 16) + (tid & 31);
#pragma unroll
        for (int j = 0; j < CH; j++) {
            const int e = 32 * min(k + j, last);
            v[j] = __ldg(sv + e);
            c[j] = __ldg(sc + e);
        }
    };
    for (int j = 0; j < CH; j++) cv[j] = 0., cc[j] = 0;
    if (ROWS == FAR && tid < rows32) fetch(sinf[tid >> 5], 0, cv, cc);
    int it = 0, left = a.chunk - lim.phase;  // iterations to the next look at convergence
    bool stop = it >= lim.maxiter;
    const int nwq = max(1, min(rows32, TT) >> 5), nwz = max(1, (min(n, TT) + 31) >> 5);
    while (!stop) {
        const unsigned ep = a.epoch + (unsigned)it;
        // q = K p over the block's rows, and p.q
        double dot = 0.;
        if (ROWS == SHARED) {
            for (int t = tid; t < rows32; t += TT) {
                const int i = t / L, len = (int)(sinf[t >> 5] & 0xffff), o = 32 * (int)(sinf[t >> 5] >> 16) + (t & 31);
                const double *xb = pw + (i < n ? rbase[i] : 0), *sv = mv + o;
                const uint16_t *sc = mc + o;
                double acc = 0.;
#pragma unroll 7
                for (int k = 0; k < len; k++) acc += sv[32 * k] * xb[sc[32 * k]];
#pragma unroll
                for (int o2 = L / 2; o2 > 0; o2 >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o2);
                if (i < n) {
                    qs[i] = acc;
                    if (L == 1 || (t & (L - 1)) == 0) dot += pw[own + i] * acc;
                }
            }
        }
        if (ROWS == NEAR) {
            for (int t = tid; t < rows32; t += TT) {
                const int i = t / L, len = (int)(sinf[t >> 5] & 0xffff);
                const int64_t o = 32 * (sinf[t >> 5] >> 16) + (t & 31);
                const double *xb = pw + (i < n ? rbase[i] : 0), *sv = a.sval + o;
                const uint16_t *sc = a.scol + o;
                double acc = 0.;
#pragma unroll 9
                for (int k = 0; k < len; k++) acc += __ldg(sv + 32 * k) * xb[__ldg(sc + 32 * k)];
#pragma unroll
                for (int o2 = L / 2; o2 > 0; o2 >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o2);
                if (i < n) {
                    qs[i] = acc;
                    if (L == 1 || (t & (L - 1)) == 0) dot += pw[own + i] * acc;
                }
            }
        }
        if (ROWS == FAR) {
            int t = tid, k = 0;
            int64_t si = t < rows32 ? sinf[t >> 5] : 0;
            double acc = 0.;
#pragma unroll 1
            while (t < rows32) {
                const int i = t / L, m = (int)(si & 0xffff) - k;
                const double *xb = pw + (i < n ? rbase[i] : 0);
                double nv[CH];
                uint16_t nc[CH];
                int64_t sn = si;
                const bool end = m <= CH;
                k += CH;
                if (end) {
                    t += TT;
                    k = 0;
                    if (t < rows32) sn = sinf[t >> 5];
                }
                if (t < rows32) fetch(sn, k, nv, nc);
                double x[CH];
#pragma unroll
                for (int j = 0; j < CH; j++) x[j] = m > 0 ? xb[cc[j]] : 0.;  // an empty slice has no columns
                // (a jump into the additions: predicated-off ones would take the FP64 pipe)
                switch (m < CH ? m : CH) {
                case 7: acc += cv[6] * x[6]; [[fallthrough]];
                case 6: acc += cv[5] * x[5]; [[fallthrough]];
                case 5: acc += cv[4] * x[4]; [[fallthrough]];
                case 4: acc += cv[3] * x[3]; [[fallthrough]];
                case 3: acc += cv[2] * x[2]; [[fallthrough]];
                case 2: acc += cv[1] * x[1]; [[fallthrough]];
                case 1: acc += cv[0] * x[0];
                }
                if (end) {
#pragma unroll
                    for (int o2 = L / 2; o2 > 0; o2 >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o2);
                    if (i < n) {
                        qs[i] = acc;
                        if (L == 1 || (tid & (L - 1)) == 0) dot += pw[own + i] * acc;
                    }
                    acc = 0.;
                }
#pragma unroll
                for (int j = 0; j < CH; j++) cv[j] = nv[j], cc[j] = nc[j];
                si = sn;
            }
        }
        dot = team_block_sum(dot, nwq, red);
        if (tid < 32) {
            // (the word leaves before the warp's other lanes start to poll, which
            // they otherwise may do first: 0.4 us per iteration)
            if (tid == 0) ll_store(slot_pq + SLOT * bid, dot, ep);
            __syncwarp();
            double v[TEAM_WORDS];
            if (!team_poll(slot_pq, G, ep, v, it == 0 ? a.poll_first : a.poll)) fail = 1;
            const double pq = fixed_sum(v);
            if (tid == 0) bc[0] = quotient(rz, pq);
        } else if (tid >= TZ) {
            irz = quotient_range(rz) ? 1. / rz : 0.;  // for beta
        }
        __syncthreads();
        // z = Minv r, r.z
        const double alpha = bc[0];
        double lrz = 0.;
        // (z from the new r, not as Minv r - alpha Minv q made while alpha is waited
        // for: 0.4 us less, but where r drops by orders of magnitude in one
        // iteration, as with one node or uncoupled ones, that z has no correct digit)
        for (int i = tid; i < n; i += TT) rs[i] -= alpha * qs[i];
        __syncthreads();
        // the first three entries of a row of the block inverses are asked for a row ahead
        double d[3] = {dreg[0], dreg[1], dreg[2]};
        uint32_t inf = dinf;
#pragma unroll 1
        for (int i = tid; i < n; i += TT) {
            const uint32_t ninf = i + TT < n ? rinf[i + TT] : 0;
            double nd[3];
#pragma unroll
            for (int k = 0; k < 3; k++)
                nd[k] = k < (int)(ninf & 7) ? __ldg(a.dval + k * a.n + r0 + i + TT) : 0.;
            const double *rn = rs + rfirst[i];
            double acc = 0.;
#pragma unroll
            for (int k = 0; k < 3; k++) acc += d[k] * rn[(inf >> (3 + 3 * k)) & 7];
#pragma unroll 1
            for (int k = 3; k < (int)(inf & 7); k++)
                acc += __ldg(a.dval + k * a.n + r0 + i) * rn[(inf >> (3 + 3 * k)) & 7];
            ll_store(a.z + r0 + i, acc, ep);
            lrz += rs[i] * acc;
#pragma unroll
            for (int k = 0; k < 3; k++) d[k] = nd[k];
            inf = ninf;
        }
        lrz = team_block_sum(lrz, nwz, red);
        if (tid == 0) ll_store(slot_rz + SLOT * bid, lrz, ep);
        __syncwarp();
        it++;
        const bool look = --left == 0 || it >= lim.maxiter;
        if (left == 0) left = a.chunk;
        if (look) {
            __syncthreads();
            double lrr = 0.;
            for (int i = tid; i < n; i += TT) lrr += rs[i] * rs[i];
            lrr = team_block_sum(lrr, nwz, red);
            if (tid == 0) {
                ll_store(slot_rr + SLOT * bid, lrr, ep);
                // the team's first block decides for all whether others have finished
                if (bid == 0) ll_store(slot_rr + 1, *(volatile int *)a.done >= a.enough ? 1. : 0., ep);
            }
        }
        for (int i = tid; i < n; i += TT) us[i] += alpha * pw[own + i];
        // p = z + beta p over the window
        constexpr int ZW = ROWS == FAR ? 4 : 6;  // words a thread asks for at a time
        double zv[ZW];
        if (tid < TZ) {
            if (!ll_poll(a.z + c0, tid, TZ, W, ep, zv, a.poll)) fail = 1;
        } else {
            double vz[TEAM_WORDS], vr[TEAM_WORDS], vy[1];
            if (!team_poll(slot_rz, G, ep, vz, a.poll)) fail = 1;
            if (look && !(team_poll(slot_rr, G, ep, vr, a.poll) && ll_poll(slot_rr + 1, 0, 1, 1, ep, vy, a.poll)))
                fail = 1;
            const double rzn = fixed_sum(vz);
            double s = 0.;
            if (look) s = fixed_sum(vr);
            if (tid == TZ) {
                const double be = bits_zero(irz) ? plain_quotient(rzn, rz) : quotient_by(rzn, rz, irz);
                bc[1] = be;
                fresh = bits_zero(be);
                bc[2] = rzn;
                bc[3] = s;
                if (look) yield = vy[0] != 0.;
            }
        }
        __syncthreads();
        // (comparisons of doubles run on the FP64 pipe too: one warp makes them)
        const double beta = bc[1];
        const bool reset = fresh;
        rz = bc[2];
        if (look) rr = bc[3];
        if (W <= TZ) {
            if (tid < W) pw[tid] = reset ? zv[0] : zv[0] + beta * pw[tid];
        } else if (W <= 2 * TZ) {
            // (a path of its own: predicated-off FP64 instructions take the pipe too)
            if (tid < TZ) pw[tid] = reset ? zv[0] : zv[0] + beta * pw[tid];
            if (tid + TZ < W && tid < TZ) pw[tid + TZ] = reset ? zv[1] : zv[1] + beta * pw[tid + TZ];
        } else if (tid < TZ) {
            for (int c1 = tid;;) {
#pragma unroll
                for (int j = 0; j < ZW; j++) {
                    const int c = c1 + j * TZ;
                    if (c1 - tid + j * TZ >= W) break;  // (for the whole block: a branch, not predicates)
                    if (c < W) pw[c] = reset ? zv[j] : zv[j] + beta * pw[c];
                }
                c1 += ZW * TZ;
                if (c1 >= W) break;
                if (!ll_poll(a.z + c0, c1, TZ, W, ep, zv, a.poll)) fail = 1;
            }
        }
        if (ROWS == FAR && tid < rows32) fetch(sinf[tid >> 5], 0, cv, cc);
        __syncthreads();
        stop = fail || it >= lim.maxiter || (look && (yield || !(rr > lim.stop2 && rr <= 1.7e308)));
    }
    if (fail) {
        // the rows keep the u of before the launch, from which the host restarts
        if (tid == 0) a.done[1] = 1;
        return;
    }
    for (int i = tid; i < n; i += TT) {
        a.u[r0 + i] = us[i];
        a.r[r0 + i] = rs[i];
        a.p[r0 + i] = pw[own + i];
    }
    if (bid == 0 && tid == 0) {
        a.rz[sys] = rz;
        a.rr[sys] = rr;
        a.sys[sys].iters = it;
        atomicAdd(a.done, G);
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

// First rows of the blocks: the wanted ones moved back to the first row of the
// node they fall in (a team's first block keeps the system's first row); a
// block ends where the next of its team begins.
__global__ void team_split_kernel(int B, const int32_t *want, const int32_t *tfirst, const int32_t *tcount,
                                  const int32_t *tend, const int64_t *dof_of_row, const int32_t *start, int bs,
                                  int32_t *rbeg, int32_t *rend) {
    const int b = threadIdx.x;
    auto at = [&](int i) { return i == tfirst[i] ? want[i] : start[dof_of_row[want[i]] / bs]; };
    if (b >= B) return;
    rbeg[b] = at(b);
    rend[b] = b + 1 < tfirst[b] + tcount[b] ? at(b + 1) : tend[b];
}

// Column window of each block: its rows' columns and its own rows.
__global__ void __launch_bounds__(256) team_window_kernel(const int32_t *rbeg, const int32_t *rend,
                                                          const int64_t *rowptr,
                                                          const int32_t *colind, int32_t *cmin, int32_t *cmax) {
    __shared__ int lo, hi;
    const int a = rbeg[blockIdx.x], e = rend[blockIdx.x];
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
__global__ void __launch_bounds__(256) team_count_kernel(const int32_t *rbeg, const int32_t *rend, const int32_t *slice0,
                                                         int L,
                                                         const int64_t *rowptr, const double *vals, int32_t *slen,
                                                         int64_t *soff, unsigned long long *total) {
    const int a = rbeg[blockIdx.x], e = rend[blockIdx.x], s0 = slice0[blockIdx.x], s1 = slice0[blockIdx.x + 1];
    const int lane = threadIdx.x & 31, per = 32 / L;
    __shared__ int all;
    if (threadIdx.x == 0) all = 0;
    __syncthreads();
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
            atomicAdd(&all, longest);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) atomicMax(total + 1, (unsigned long long)all);
}

// Entry k of a row goes to lane k % L of its L lanes; lanes that end early
// repeat the row's last column with the value 0.
__global__ void __launch_bounds__(256) team_fill_kernel(const int32_t *rbeg, const int32_t *rend, const int32_t *slice0,
                                                         int L,
                                                        const int64_t *rowptr, const uint16_t *col16,
                                                        const double *vals, const int32_t *slen,
                                                        const int64_t *soff, double *sval, uint16_t *scol) {
    const int a = rbeg[blockIdx.x], e = rend[blockIdx.x], s0 = slice0[blockIdx.x], s1 = slice0[blockIdx.x + 1];
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

template <int L>
TeamKernel team_kernel(int rows) {
    return rows == SHARED ? team_pcg_kernel<L, SHARED> : rows == NEAR ? team_pcg_kernel<L, NEAR>
                                                                      : team_pcg_kernel<L, FAR>;
}
TeamKernel team_kernel(int L, int rows) {
    return L == 1 ? team_kernel<1>(rows) : L == 2 ? team_kernel<2>(rows) : L == 4 ? team_kernel<4>(rows)
                                                                                 : team_kernel<8>(rows);
}

template <typename T>
bool get(T **p, size_t n) {
    return cudaMalloc((void **)p, (n ? n : 1) * sizeof(T)) == cudaSuccess;
}

}  // namespace

void team_free(fe3d_team *t) {
    if (!t) return;
    cudaFree(t->ints);
    cudaFree(t->slen);
    cudaFree(t->soff);
    cudaFree(t->sval);
    cudaFree(t->scol);
    cudaFree(t->total);
    cudaFree(t->z);
    cudaFree(t->slots);
    cudaFree(t->dval);
    cudaFree(t->dinf);
    cudaFree(t->sys);
    cudaFree(t->done);
    delete t;
}

// Memory for up to nsys systems of the solver's matrix; nullptr where the
// device or the pattern does not allow it or memory is short.
fe3d_team *team_create(const fe3d_solver *s, int64_t nsys, cudaStream_t st) {
    if (s->n < 1 || s->n > INT32_MAX || !s->pat->col16) return nullptr;
    int dev = 0, sms = 0, coop = 0, optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess || !coop)
        return nullptr;
    fe3d_team *t = new fe3d_team();
    t->blocks = sms < TEAM_MAX ? sms : TEAM_MAX;
    t->smem_max = (size_t)optin - 8192;
    const size_t slots = 3 * SLOT * TEAM_MAX;
    bool ok = get(&t->ints, 10 * (TEAM_MAX + 1)) && get(&t->total, 2) && get(&t->z, s->n) && get(&t->slots, slots) &&
              get(&t->dval, 6 * s->n) && get(&t->dinf, s->n) && get(&t->sys, nsys) && get(&t->done, 2) &&
              cudaMemsetAsync(t->z, 0, sizeof(ulonglong2) * s->n, st) == cudaSuccess &&
              cudaMemsetAsync(t->slots, 0, sizeof(ulonglong2) * slots, st) == cudaSuccess;
    for (int L = 1; ok && L <= 8; L *= 2)
        for (int rows = SHARED; ok && rows <= FAR; rows++) {
            int res = 0;
            ok = cudaFuncSetAttribute(team_kernel(L, rows), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)t->smem_max) == cudaSuccess &&
                 cudaOccupancyMaxActiveBlocksPerMultiprocessor(&res, team_kernel(L, rows), TT, t->smem_max) ==
                     cudaSuccess &&
                 res >= 1;
        }
    if (!ok) {
        (void)cudaGetLastError();
        team_free(t);
        return nullptr;
    }
    return t;
}

// Shared memory of a block of rows rows whose columns reach bw rows further on
// either side.
size_t team_smem(int64_t rows, int64_t bw) {
    return sizeof(double) * (size_t)(4 * rows + 2 * bw + rows / 4 + 1) + 10 * (size_t)rows;
}

// Deals the systems out: part i on parts[i].blocks blocks.  Returns 0, or
// FE3D_ERR_TOO_LARGE where a block's rows do not fit shared memory.
int team_split(fe3d_team *t, const fe3d_solver *s, const std::vector<TeamPart> &parts, cudaStream_t st) {
    constexpr int S = TEAM_MAX + 1;
    std::vector<int32_t> h(10 * S, 0);
    int32_t *want = &h[0], *tfirst = &h[S], *tcount = &h[2 * S], *tend = &h[3 * S], *tsys = &h[4 * S];
    int B = 0;
    for (const TeamPart &q : parts) {
        const int first = B;
        for (int j = 0; j < q.blocks; j++, B++) {
            if (B >= t->blocks) return FE3D_ERR_ARG;
            want[B] = (int32_t)(q.row0 + (q.row1 - q.row0) * j / q.blocks);
            tfirst[B] = first;
            tcount[B] = q.blocks;
            tend[B] = (int32_t)q.row1;
            tsys[B] = (int32_t)q.sys;
        }
    }
    t->G = B;
    int32_t *d = t->ints;
    t->tfirst = d + S;
    t->tcount = d + 2 * S;
    t->tsys = d + 4 * S;
    t->rbeg = d + 5 * S;
    t->rend = d + 6 * S;
    t->cmin = d + 7 * S;
    t->cmax = d + 8 * S;
    t->slice0 = d + 9 * S;
    FE3D_CUDA(cudaMemcpyAsync(d, h.data(), sizeof(int32_t) * 5 * S, cudaMemcpyHostToDevice, st));
    team_split_kernel<<<1, TEAM_MAX + 8, 0, st>>>(B, d, t->tfirst, t->tcount, d + 3 * S, s->pat->dof_of_row, s->start,
                                                  s->bs, t->rbeg, t->rend);
    team_window_kernel<<<B, 256, 0, st>>>(t->rbeg, t->rend, s->pat->rowptr, s->pat->colind, t->cmin, t->cmax);
    FE3D_CHECK_LAUNCH();
    FE3D_CUDA(cudaMemcpyAsync(&h[5 * S], t->rbeg, sizeof(int32_t) * 4 * S, cudaMemcpyDeviceToHost, st));
    FE3D_CUDA(cudaStreamSynchronize(st));
    t->nmax = 0;
    for (int b = 0; b < B; b++) {
        const int n = h[6 * S + b] - h[5 * S + b];
        if (n < 0) return FE3D_ERR_ARG;
        if (n > t->nmax) t->nmax = n;
    }
    // lanes per row: the fewest FP64 instructions on one sub-partition's warps
    // for a row of 27 non-zeros (a node of a flat plate's inside).  us per
    // iteration with 1 / 2 / 4 / 8 lanes, * the chosen ones: plate 2,166 rows 6.4 /
    // 5.9 / 5.7* / 5.7, 9,126 rows 7.0 / 6.5* / 6.5 / 6.9, 20,886 rows 7.2* / 7.3 /
    // 7.9 / 8.9, 237,606 rows 23* / 27 / 34 / 45; rows of 54: cylinder 1,080 rows 7.7 /
    // 6.7 / 6.2* / 6.1, 10,440 rows 8.9* / 8.0 / 7.9 / 8.7, 42,480 rows 11.8 / 12.9* /
    // 13.0 / 14.4, 387,714 rows 67* / 73 / 78 / 90, panel 21,964 rows 8.6 / 8.5* / 9.4 /
    // 10.0
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
    t->smem = 0;
    for (int b = 0; b < B; b++) {
        const size_t n = h[6 * S + b] - h[5 * S + b], w = n > 0 ? h[8 * S + b] - h[7 * S + b] + 1 : 0;
        const size_t need = sizeof(double) * (w + 3 * n + (n * t->L + 31) / 32) +
                            (2 * sizeof(int) + sizeof(uint16_t)) * n;
        if (need > t->smem) t->smem = need;
    }
    if (t->smem > t->smem_max) return FE3D_ERR_TOO_LARGE;
    const int per = 32 / t->L;
    int32_t *slice0 = &h[9 * S];
    slice0[0] = 0;
    for (int b = 0; b < B; b++) slice0[b + 1] = slice0[b] + (h[6 * S + b] - h[5 * S + b] + per - 1) / per;
    if (slice0[B] > t->slices) {
        cudaFree(t->slen);
        cudaFree(t->soff);
        t->slen = nullptr;
        t->soff = nullptr;
        t->slices = 0;
        if (!get(&t->slen, slice0[B]) || !get(&t->soff, slice0[B])) {
            (void)cudaGetLastError();
            return FE3D_ERR_NOMEM;
        }
        t->slices = slice0[B];
    }
    FE3D_CUDA(cudaMemcpyAsync(t->slice0, slice0, sizeof(int32_t) * (B + 1), cudaMemcpyHostToDevice, st));
    FE3D_CUDA(cudaStreamSynchronize(st));
    return FE3D_OK;
}

int team_plan(fe3d_team *t, const fe3d_solver *s, cudaStream_t st) {
    FE3D_CUDA(cudaMemsetAsync(t->total, 0, 2 * sizeof(unsigned long long), st));
    team_count_kernel<<<t->G, 256, 0, st>>>(t->rbeg, t->rend, t->slice0, t->L, s->pat->rowptr, s->vals, t->slen,
                                            t->soff, t->total);
    FE3D_CHECK_LAUNCH();
    return FE3D_OK;
}

int team_build(fe3d_team *t, const fe3d_solver *s, const unsigned long long (&total)[2], cudaStream_t st) {
    const size_t shared = ((t->smem + 7) & ~(size_t)7) + 32 * (sizeof(double) + sizeof(uint16_t)) * (size_t)total[1];
    const int64_t entries = 32 * (int64_t)total[0];
    t->rows = shared <= t->smem_max ? SHARED : entries <= kFarEntries ? NEAR : FAR;
    t->smem_run = t->rows == SHARED ? shared : t->smem;
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
    team_fill_kernel<<<t->G, 256, 0, st>>>(t->rbeg, t->rend, t->slice0, t->L, s->pat->rowptr, s->pat->col16, s->vals,
                                           t->slen, t->soff, t->sval, t->scol);
    FE3D_CHECK_LAUNCH();
    return FE3D_OK;
}

int team_inverses(fe3d_team *t, const fe3d_solver *s, cudaStream_t st) {
    team_blocks_kernel<<<(unsigned)((s->n + 255) / 256), 256, 0, st>>>(s->n, s->pat->dof_of_row, s->start, s->size,
                                                                       s->bs, s->Dinv, t->dval, t->dinf);
    FE3D_CHECK_LAUNCH();
    return FE3D_OK;
}

int team_run(fe3d_team *t, const fe3d_solver *s, double *u, double *rz, double *rr, std::vector<TeamSys> &sys,
             int chunk, int enough, cudaStream_t st) {
    int most = 0;
    for (const TeamSys &q : sys)
        if (q.maxiter > most) most = q.maxiter;
    if (t->epoch > 0xffffffffu - (unsigned)most - 2u) {
        FE3D_CUDA(cudaMemsetAsync(t->z, 0, sizeof(ulonglong2) * s->n, st));
        FE3D_CUDA(cudaMemsetAsync(t->slots, 0, sizeof(ulonglong2) * 3 * SLOT * TEAM_MAX, st));
        t->epoch = 1;
    }
    FE3D_CUDA(cudaMemcpyAsync(t->sys, sys.data(), sizeof(TeamSys) * sys.size(), cudaMemcpyHostToDevice, st));
    FE3D_CUDA(cudaMemsetAsync(t->done, 0, 2 * sizeof(int), st));
    TeamArgs a{t->rbeg, t->rend, t->slice0, t->cmin, t->cmax, t->tfirst, t->tcount, t->tsys, t->slen, t->soff,
               t->sval, t->scol, s->pat->colbase, s->pat->dof_of_row, s->start, s->bs, t->dval, t->dinf, u, s->r,
               s->p, s->n, rz, rr, t->sys, t->z, t->slots, t->epoch, chunk, t->done, enough, t->poll, t->poll_first};
    t->epoch += (unsigned)most + 1u;
    void *args[] = {&a};
    if (cudaLaunchCooperativeKernel((const void *)team_kernel(t->L, t->rows), dim3(t->G), dim3(TT), args,
                                    t->smem_run, st) != cudaSuccess) {
        (void)cudaGetLastError();
        return FE3D_ERR_LAUNCH;
    }
    int done[2] = {0, 0};
    FE3D_CUDA(cudaMemcpyAsync(sys.data(), t->sys, sizeof(TeamSys) * sys.size(), cudaMemcpyDeviceToHost, st));
    FE3D_CUDA(cudaMemcpyAsync(done, t->done, sizeof(done), cudaMemcpyDeviceToHost, st));
    FE3D_CUDA(cudaStreamSynchronize(st));
    return done[1] ? FE3D_ERR_LAUNCH : FE3D_OK;
}

}  // namespace fe3d
