// Resident kernels of the single-LP engine: a whole block of iterations, the evaluation of both points or the whole
// power iteration in ONE launch, for LPs whose phases are bound by latency rather than by throughput.
//
// What bounds a small or medium LP on the phase kernels (kernels.cuh) is not its bytes but the chain of dependent
// steps of each phase -- launch, metadata, matrix entries, gathers, row sums, fused step -- of which only the gathers
// depend on the phase before. Here the CTAs stay on their SMs, and between two phases there is a barrier instead of a
// kernel boundary: a CTA that has arrived at the barrier loads its next tile's matrix entries, row pointers and step
// operands into registers and shared memory while it waits, so behind the barrier only gathers, sums and the fused
// step are left.
//
//   team   -- 256 threads, one row block (tile) of the block list at a time, exactly as a CTA of k_rowblock takes
//             it on the default row split: the same products, the same summation order per row, hence the same iterates
//             bit for bit (blocks that a context tuned to kMidGroups or kSegmented are summed by the default rule here);
//   CTA    -- kTeams teams, one CTA per SM (its teams share the CTA's arrival at the barrier);
//   grid   -- a cooperative launch, so that every CTA is resident while others wait for it at the barrier, a counter
//             in global memory.
//
// The gathered vectors change from phase to phase, so they are read with plain (coherent) loads; the acquire side of
// the barrier drops stale L1 lines, and within a phase L1 serves the columns that the rows of an SM share.
#pragma once
#include "kernels.cuh"

namespace taral {

// Teams per CTA: 2 teams of 256 threads leave 128 registers a thread, which hold a tile in flight beside the step's
// FP64 operands and the interleaved sums of long rows; 3 or 4 teams spill them to local memory.
constexpr int kTeams = 2;
constexpr int kBarrierPolls = 1 << 22;  // bound of a barrier wait (seconds); the launch is cooperative, so it ends sooner

template <class T>
struct ResidentMat {
    const int *ptr, *idx;
    const T* val;
    const int4* blk;
    int nblk;
};

template <class T>
struct ResidentArgs {
    ResidentMat<T> A, AT;
    int m, n;
    T *x, *z, *Ax, *ATz;
    double *xs, *zs;
    const T *c, *l, *u, *rl, *ru, *Dr, *Dc, *xlast, *zlast;
    const double* par;
    double *tmp_m, *tmp_n, *part, *out;
    unsigned *bar, *other_bar, *ticket;  // grid barrier's counter (zero at launch) and the next launch's, zeroed here
    int* err;   // set when a wait gave up: the launch left its work half done
    int polls;  // after which a wait gives up
};

// ------------------------------------------------------------------------------------------ barriers
// arrive() publishes this CTA's writes; wait() returns when every CTA of the grid has arrived (false: gave up).
struct GridBarrier {
    unsigned *bar, target = 0;
    int* err;
    int polls;
    bool* ok;  // shared
    template <class T>
    __device__ GridBarrier(const ResidentArgs<T>& a, bool* shared_ok) : bar(a.bar), err(a.err), polls(a.polls), ok(shared_ok) {
        if (threadIdx.x == 0) {
            *ok = true;
            if (blockIdx.x == 0) *a.other_bar = 0;
        }
    }
    __device__ __forceinline__ void arrive() {
        target += gridDim.x;
        __syncthreads();
        if (threadIdx.x == 0)
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
    }
    __device__ __forceinline__ bool wait() {
        if (threadIdx.x == 0) {
            bool there = false;
            for (int i = 0; i < polls && !there; ++i) {
                unsigned v;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
                there = int(v - target) >= 0;
            }
            if (!there) *ok = false, atomicExch(err, 1);
        }
        __syncthreads();
        return *ok;
    }
};

struct Team {  // 256 consecutive threads of the CTA with a named barrier of their own
    int id, tid;
    __device__ Team() : id(int(threadIdx.x) / kThreads), tid(int(threadIdx.x) % kThreads) {}
    __device__ __forceinline__ void sync() const { asm volatile("bar.sync %0, 256;" ::"r"(id + 1) : "memory"); }
};

// ------------------------------------------------------------------------------------------ tiles
template <class T>
struct Tile {
    int4 meta;
    T v[kQuads][4];
    int c[kQuads][4];
};

// The matrix entries of the tile q.meta into registers: nothing here depends on the phase before. A row longer than a
// tile (alone in its block) is streamed by tile_sum instead.
template <class T, class P>
__device__ __forceinline__ void load_tile(const ResidentMat<T>& a, const Team& t, RowSmem<P>& sm, Tile<T>& q) {
    const int p0 = q.meta.z, p1 = q.meta.w;
    if (p1 - p0 > kTile) return;
    const int a0 = p0 & ~3;
#pragma unroll
    for (int i = 0; i < kQuads; ++i) {
        const int k = a0 + 4 * (t.tid + i * kThreads);
        if (k >= p0 && k + 4 <= p1) {
            Quad<T>::load(a.val + k, q.v[i]), load_idx4(a.idx + k, q.c[i]);
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const bool in = k + e >= p0 && k + e < p1;
                q.v[i][e] = in ? __ldg(a.val + k + e) : T(0);
                q.c[i][e] = in ? __ldg(a.idx + k + e) : -1;
            }
        }
    }
    if (t.tid == 0) sm.nlong = 0;
}

// The tile's row pointers, relative to its first entry, into shared memory.
template <class T>
__device__ __forceinline__ void load_rows(const ResidentMat<T>& a, int4 meta, const Team& t, int* rptr) {
    for (int r = t.tid; r <= (meta.y & 0xffff); r += kThreads) rptr[r] = __ldg(a.ptr + meta.x + r) - meta.z;
}

// The sum of row tid of the tile, in the order of block_sums (kernels.cuh): rows of at most kShort nonzeros (every
// row of a uniform block) in entry order by their own thread, longer ones by a warp (lanes strided, shuffle tree), a
// row longer than a tile by the whole team. `in(k)`: entry k of the gathered vector. Every thread of the team calls
// it; the result is meaningful where tid < rows.
template <class P, class T, class In>
__device__ __forceinline__ double tile_sum(const ResidentMat<T>& a, const Tile<T>& q, const Team& t, RowSmem<P>& sm,
                                           const int* rptr, In in) {
    const int tid = t.tid, lane = tid & 31, warp = tid >> 5;
    const int nrows = q.meta.y & 0xffff, p0 = q.meta.z, p1 = q.meta.w;
    if (p1 - p0 > kTile) {
        double s = 0;
        for (int k = (p0 & ~3) + 4 * tid; k < p1; k += 4 * kThreads) {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (k + e >= p0 && k + e < p1) s += double(__ldg(a.val + k + e)) * double(in(__ldg(a.idx + k + e)));
        }
        for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
        if (lane == 0) sm.rowsum[1 + warp] = s;
        t.sync();
        s = 0;
        for (int w = 0; w < kThreads / 32; ++w) s += sm.rowsum[1 + w];
        t.sync();
        return s;
    }
    const int a0 = p0 & ~3;
    {
        decltype(in(0)) g[kQuads][4];
#pragma unroll
        for (int i = 0; i < kQuads; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) g[i][e] = q.c[i][e] >= 0 ? in(q.c[i][e]) : decltype(in(0))(0);
#pragma unroll
        for (int i = 0; i < kQuads; ++i) {
            const int k = a0 + 4 * (tid + i * kThreads);
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (q.c[i][e] >= 0) sm.prod[pidx(k + e - p0)] = mul_rn(P(q.v[i][e]), P(g[i][e]));
        }
    }
    t.sync();
    const int thread_max = (q.meta.y & kUniformRows) ? kTile : kShort;
    const bool queue = (q.meta.y & kLongRows) && !(q.meta.y & kUniformRows);  // the same for the whole team
    double s = 0;
    bool queued = false;
    if (tid < nrows) {
        const int lo = rptr[tid], hi = rptr[tid + 1];
        if (hi - lo <= thread_max) {
            int k = lo;
            for (; k + 4 <= hi; k += 4) {
                P v[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] = sm.prod[pidx(k + e)];
#pragma unroll
                for (int e = 0; e < 4; ++e) s += double(v[e]);
            }
            for (; k < hi; ++k) s += double(sm.prod[pidx(k)]);
        } else {
            queued = true;
            sm.longrow[atomicAdd(&sm.nlong, 1)] = short(tid);
        }
    }
    if (!queue) return s;
    t.sync();
    // a warp takes four queued rows at a time: their loads and shuffle trees are independent, so their latencies overlap
    constexpr int kAtOnce = 4;
    const int nlong = sm.nlong;
    for (int i = warp * kAtOnce; i < nlong; i += kAtOnce * (kThreads / 32)) {
        double v[kAtOnce];
        int row[kAtOnce], k[kAtOnce], hi[kAtOnce], longest = 0;
#pragma unroll
        for (int j = 0; j < kAtOnce; ++j) {
            row[j] = i + j < nlong ? sm.longrow[i + j] : -1;
            k[j] = row[j] >= 0 ? rptr[row[j]] : 0, hi[j] = row[j] >= 0 ? rptr[row[j] + 1] : 0;
            longest = max(longest, hi[j] - k[j]);
            v[j] = 0;
        }
        for (int d = lane; d < longest; d += 64) {  // two strides of loads, then the adds in order (zeros change no sum)
            P e[kAtOnce][2];
#pragma unroll
            for (int j = 0; j < kAtOnce; ++j)
#pragma unroll
                for (int i = 0; i < 2; ++i) e[j][i] = k[j] + d + 32 * i < hi[j] ? sm.prod[pidx(k[j] + d + 32 * i)] : P(0);
#pragma unroll
            for (int j = 0; j < kAtOnce; ++j)
#pragma unroll
                for (int i = 0; i < 2; ++i) v[j] += double(e[j][i]);
        }
        for (int off = 16; off > 0; off >>= 1)
#pragma unroll
            for (int j = 0; j < kAtOnce; ++j) v[j] += __shfl_xor_sync(0xffffffffu, v[j], off);
#pragma unroll
        for (int j = 0; j < kAtOnce; ++j)
            if (lane == j && row[j] >= 0) sm.rowsum[row[j]] = v[j];
    }
    t.sync();
    return queued ? sm.rowsum[tid] : s;
}

// A team's first tile of one matrix, held for the whole launch: its metadata and its row pointers (in shared memory).
struct FirstTile {
    int4 meta;
    int* rptr;
};
template <class T>
__device__ __forceinline__ FirstTile first_tile(const ResidentMat<T>& a, const Team& t, int b, int* rptr) {
    FirstTile f{b < a.nblk ? __ldg(a.blk + b) : make_int4(0, 0, 0, 0), rptr};
    load_rows(a, f.meta, t, rptr);
    return f;
}

// One phase: every tile of the matrix with the fused step `epi`, gathering through `in`. Called after arrive(); the
// first tile's entries and operands are loaded before the wait.
template <class P, class T, class E, class In>
__device__ __forceinline__ bool phase(GridBarrier& barrier, const ResidentMat<T>& a, const FirstTile& f, const Team& t,
                                      RowSmem<P>& sm, const E& epi, In in) {
    const int first = t.id * int(gridDim.x) + int(blockIdx.x), teams = int(gridDim.x) * (int(blockDim.x) / kThreads);
    Tile<T> q;
    typename E::Ops ops{};
    if (first < a.nblk) {
        q.meta = f.meta;
        load_tile(a, t, sm, q);
        if (t.tid < (q.meta.y & 0xffff)) ops = epi.load(q.meta.x + t.tid, 0);
    }
    if (!barrier.wait()) return false;
    const int* rptr = f.rptr;
    for (int b = first; b < a.nblk; b += teams) {
        if (b != first) {
            t.sync();  // the last tile's row pointers have been read
            q.meta = __ldg(a.blk + b);
            load_tile(a, t, sm, q);
            load_rows(a, q.meta, t, sm.rptr);
            rptr = sm.rptr;
            if (t.tid < (q.meta.y & 0xffff)) ops = epi.load(q.meta.x + t.tid, 0);
            t.sync();
        }
        const double s = tile_sum<P>(a, q, t, sm, rptr, in);
        if (t.tid < (q.meta.y & 0xffff)) epi.apply(q.meta.x + t.tid, s, ops);
    }
    return true;
}

// The dual step of EpiRow (kernels.cuh) with the reciprocal of sigma taken once per launch.
template <class T>
struct ResidentRow {
    T *Ax, *z;
    double* zs;
    const T *rl, *ru;
    double sigma, inv_sigma;
    struct Ops { double z, ax, rl, ru, zs; };
    __device__ __forceinline__ Ops load(int r, int) const {
        return {double(z[r]), double(Ax[r]), double(rl[r]), double(ru[r]), zs[r]};
    }
    __device__ __forceinline__ void apply(int r, double s, const Ops& o) const {
        const T st = T(s), zn = T(dual_prox(o.z + sigma * (2.0 * double(st) - o.ax), o.rl, o.ru, sigma, inv_sigma));
        z[r] = zn, Ax[r] = st, zs[r] = o.zs + double(zn);
    }
};

// ------------------------------------------------------------------------------------------ kernels
// A block of `steps` iterations: the first primal step, then row and column phase per step (as the engine's launch
// of k_xupd and 2 steps phase kernels, bit for bit).
template <class T>
__global__ void __launch_bounds__(kThreads * kTeams, 1) k_resident_iterate(const ResidentArgs<T> a, int steps) {
    extern __shared__ __align__(16) unsigned char raw[];
    __shared__ bool ok;
    __shared__ int held[2][kTeams][kRowsMax + 1];
    const Team t;
    RowSmem<T>& sm = reinterpret_cast<RowSmem<T>*>(raw)[t.id];
    GridBarrier barrier(a, &ok);
    const int first = t.id * int(gridDim.x) + int(blockIdx.x), teams = int(gridDim.x) * (int(blockDim.x) / kThreads);
    const FirstTile fa = first_tile(a.A, t, first, held[0][t.id]), ft = first_tile(a.AT, t, first, held[1][t.id]);
    const double tau = a.par[0], sigma = a.par[1];
    for (int b = first; b < a.AT.nblk; b += teams) {  // the thread that owns a column in the column phases takes it
        const int4 meta = __ldg(a.AT.blk + b);
        if (t.tid < (meta.y & 0xffff)) {
            const int j = meta.x + t.tid;
            const T xn = T(clampv(double(a.x[j]) - tau * (double(a.c[j]) + double(a.ATz[j])), double(a.l[j]), double(a.u[j])));
            a.x[j] = xn, a.xs[j] += double(xn);
        }
    }
    const ResidentRow<T> row{a.Ax, a.z, a.zs, a.rl, a.ru, sigma, 1.0 / sigma};
    EpiCol<T> col{a.ATz, a.x, a.xs, a.c, a.l, a.u, a.par, 1};
    for (int s = 0; s < steps; ++s) {
        barrier.arrive();
        if (!phase<T>(barrier, a.A, fa, t, sm, row, [&](int k) { return a.x[k]; })) return;
        barrier.arrive();
        col.upd = s + 1 < steps ? 1 : 0;
        if (!phase<T>(barrier, a.AT, ft, t, sm, col, [&](int k) { return a.z[k]; })) return;
    }
}

constexpr int kResidentDone = 20;  // out[kResidentDone] = 1: this launch ran to its end, and no barrier ever gave up

// The sum of K values over a team: shuffle tree per warp, then the warps in order, as reduce_finish sums a CTA
// (kernels.cuh); thread k < K writes dst[k]. Ends with a team barrier.
template <int K>
__device__ __forceinline__ void team_sums(double (&v)[K], const Team& t, double* sh, double* dst) {
    const int lane = t.tid & 31, w = t.tid >> 5;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        double s = v[k];
        for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
        if (lane == 0) sh[k * (kThreads / 32) + w] = s;
    }
    t.sync();
    if (t.tid < K) {
        double s = 0;
        for (int i = 0; i < kThreads / 32; ++i) s += sh[t.tid * (kThreads / 32) + i];
        dst[t.tid] = s;
    }
    t.sync();
}

// The KKT scalars of the current point (out[0..9]) and of the average sums * f (out[10..19]): the average's products
// and the current point's partial sums, a barrier, the average's partial sums; the CTA that finishes last adds the
// partials. The partials are those of k_eval_row / k_eval_col at gr / gc CTAs -- a team takes their CTAs one after
// another -- and are added in the same order, so the scalars are the same bits. `out` may be pinned host memory.
constexpr int kEvalCtas = kRedCtas;
template <class T>
__global__ void __launch_bounds__(kThreads * kTeams, 1) k_resident_eval(const ResidentArgs<T> a, double f, int gr, int gc) {
    extern __shared__ __align__(16) unsigned char raw[];
    __shared__ bool ok, last;
    __shared__ double sh[kTeams][5 * (kThreads / 32)];
    const Team t;
    RowSmem<double>& sm = reinterpret_cast<RowSmem<double>*>(raw)[t.id];
    GridBarrier barrier(a, &ok);
    const int first = t.id * int(gridDim.x) + int(blockIdx.x), teams = int(gridDim.x) * (int(blockDim.x) / kThreads);
    auto products = [&](const ResidentMat<T>& mat, const double* in, double* to) {
        for (int b = first; b < mat.nblk; b += teams) {
            Tile<T> q;
            t.sync();
            q.meta = __ldg(mat.blk + b);
            load_tile(mat, t, sm, q);
            load_rows(mat, q.meta, t, sm.rptr);
            t.sync();
            const double s = tile_sum<double>(mat, q, t, sm, sm.rptr, [&](int k) { return in[k]; });
            if (t.tid < (q.meta.y & 0xffff)) to[q.meta.x + t.tid] = s;
        }
    };
    auto partials = [&](bool avg) {
        double* p = a.part + (avg ? 10 * kEvalCtas : 0);
        for (int job = first; job < gr + gc; job += teams) {
            double v[5] = {0, 0, 0, 0, 0};
            if (job < gr) {
                const int i = job * kThreads + t.tid, G = gr * kThreads;
                if (avg) eval_rows(v, i, G, a.m, f, (const double*)a.tmp_m, (const double*)a.zs, a.rl, a.ru, a.Dr, a.zlast);
                else eval_rows(v, i, G, a.m, 1.0, (const T*)a.Ax, (const T*)a.z, a.rl, a.ru, a.Dr, a.zlast);
                team_sums<5>(v, t, sh[t.id], p + 5 * job);
            } else {
                const int j = (job - gr) * kThreads + t.tid, G = gc * kThreads;
                if (avg) eval_cols(v, j, G, a.n, f, (const double*)a.xs, (const double*)a.tmp_n, a.c, a.l, a.u, a.Dc, a.xlast);
                else eval_cols(v, j, G, a.n, 1.0, (const T*)a.x, (const T*)a.ATz, a.c, a.l, a.u, a.Dc, a.xlast);
                team_sums<5>(v, t, sh[t.id], p + 5 * (kEvalCtas + job - gr));
            }
        }
    };
    products(a.A, a.xs, a.tmp_m);
    products(a.AT, a.zs, a.tmp_n);
    barrier.arrive();
    partials(false);
    if (!barrier.wait()) return;
    partials(true);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(a.ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    double* all = reinterpret_cast<double*>(raw);  // 4 x kEvalCtas x 5 partials, loaded at once, then added in order
    for (int i = threadIdx.x; i < 20 * kEvalCtas; i += blockDim.x) {
        const int cta = i / 5 % kEvalCtas;
        all[i] = cta < (i / (5 * kEvalCtas) & 1 ? gc : gr) ? __ldcg(a.part + i) : 0.0;
    }
    __syncthreads();
    if (threadIdx.x < 20) {
        const int q = threadIdx.x / 5, k = threadIdx.x % 5;  // q: current rows, current columns, average rows, columns
        double s = 0;
        for (int b = 0; b < (q & 1 ? gc : gr); ++b) s += all[(q * kEvalCtas + b) * 5 + k];
        a.out[threadIdx.x] = s;
    }
    if (threadIdx.x == 0) *a.ticket = 0, a.out[kResidentDone] = *a.err ? 0.0 : 1.0;
}

// The power iteration on A^T A from v (the steps of k_power_* and two products each, bit for bit): out[0] = the
// estimate, out[1] = the steps taken. The normalisation of v is applied where v is gathered.
template <class T>
__global__ void __launch_bounds__(kThreads * kTeams, 1) k_resident_power(const ResidentArgs<T> a, T* v, T* w, int iters, int gc) {
    extern __shared__ __align__(16) unsigned char raw[];
    __shared__ bool ok;
    __shared__ int held[2][kTeams][kRowsMax + 1];
    __shared__ double sh[kTeams][kThreads / 32], parts[kEvalCtas], total;
    const Team t;
    RowSmem<T>& sm = reinterpret_cast<RowSmem<T>*>(raw)[t.id];
    GridBarrier barrier(a, &ok);
    const int first = t.id * int(gridDim.x) + int(blockIdx.x), teams = int(gridDim.x) * (int(blockDim.x) / kThreads);
    const FirstTile fa = first_tile(a.A, t, first, held[0][t.id]), ft = first_tile(a.AT, t, first, held[1][t.id]);
    double est = 0, f = 0;
    int it = 0;
    while (it < iters) {
        barrier.arrive();
        const bool scale = it > 0;
        if (!phase<T>(barrier, a.A, fa, t, sm, EpiStore<T>{w}, [&](int k) { return scale ? T(double(v[k]) * f) : v[k]; })) return;
        barrier.arrive();
        if (!phase<T>(barrier, a.AT, ft, t, sm, EpiStore<T>{v}, [&](int k) { return w[k]; })) return;
        barrier.arrive();
        if (!barrier.wait()) return;
        for (int job = first; job < gc; job += teams) {
            double q[1] = {0};
            for (int j = job * kThreads + t.tid; j < a.n; j += gc * kThreads) q[0] += double(v[j]) * double(v[j]);
            team_sums<1>(q, t, sh[t.id], a.part + job);
        }
        barrier.arrive();
        if (!barrier.wait()) return;
        for (int i = threadIdx.x; i < gc; i += blockDim.x) parts[i] = __ldcg(a.part + i);
        __syncthreads();
        if (threadIdx.x == 0) {
            double s = 0;
            for (int b = 0; b < gc; ++b) s += parts[b];
            total = s;
        }
        __syncthreads();
        const double s = total, prev = est;
        ++it;
        if (s <= 0) {
            est = 0;
            break;
        }
        est = sqrt(sqrt(s)), f = 1 / sqrt(s);
        if (it > 10 && fabs(est - prev) <= 1e-7 * est) break;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) a.out[0] = est, a.out[1] = double(it), a.out[kResidentDone] = *a.err ? 0.0 : 1.0;
}

}  // namespace taral
