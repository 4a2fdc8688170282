// Iterations of small LPs inside one thread-block cluster per LP, everything on chip.
//
// An LP whose vectors and matrix slices fit the shared memory of 1 to 16 CTAs has no work that could fill the GPU: its
// time is the length of the dependent chain of a phase. Here that chain leaves the caches alone:
//   * every CTA of the cluster holds a full copy of the gathered vectors x and z, and a slice of the rows of A and of
//     A^T (indices as 16 bits, values, step operands) for the whole launch;
//   * a phase is: the sums of the slice's rows, the fused step, and the new entries of z (or x) stored into every CTA's
//     copy through distributed shared memory;
//   * the hardware cluster barrier (463 cycles with the remote stores, against 1,012 with stores to global memory that
//     it has to release) ends the phase; a single CTA needs only a CTA barrier.
// Products, summation order and steps are those of the phase kernels (kernels.cuh), so the iterates are the same bits.
#pragma once
#include <algorithm>
#include <vector>

#include "kernels.cuh"

namespace taral {

constexpr int kClusterThreads = 512;
constexpr int kClusterRows = 65535;  // most rows or columns: positions are 16 bits
constexpr int kClusterMax = 16;  // CTAs per cluster (the largest, non-portable size)

// One LP on the device. Row pointers hold offsets into idx / val. Rows are renumbered for the cluster: a CTA's slice is a
// contiguous range of the rows sorted by descending length (its rows of more than kShort nonzeros come first), and the
// position of a row counts through the slices in order. The copies of x and z are in positions, so that a warp's new
// entries are neighbours in them.
template <class T>
struct ClusterLp {
    const int *a_ptr, *a_idx, *t_ptr, *t_idx;
    const T *a_val, *t_val;
    int m, n;
    T *x, *z, *Ax, *ATz;
    double *xs, *zs;
    const T *c, *l, *u, *rl, *ru;
    const double* par;
    const T* v0;        // the power iteration's start
    const int* plan;    // the CTAs' headers (ClusterCta) and what they refer to, see cluster_plan
    const int* active;  // NULL, or the LP is left alone when *active == 0
};

// The slices of one CTA: its header of the plan. Offsets are ints into the plan, counts in rows and entries.
struct ClusterCta {
    int rows[2], nlong[2];   // positions of A and of A^T, and how many of them are long rows
    int first[2];            // the first position
    int order[2], base[2];   // the rows at the positions; the entry offset of every group of 32 short rows (and the end)
    int where[2];            // the position of every row of A and of every row of A^T
    int entries[2];          // entries stored: groups padded to their longest row, then the long rows
    __host__ __device__ int groups(int k) const { return (rows[k] - nlong[k] + 31) / 32; }
    __host__ __device__ int bases(int k) const { return groups(k) + (nlong[k] > 1 ? nlong[k] : 1); }
};

__host__ __device__ constexpr size_t align16(size_t b) { return (b + 15) & ~size_t(15); }

// Offsets of a CTA's arrays in shared memory. The arrays that other CTAs write (the copies of x and z, the power
// iteration's partial sums) come first, at the same offsets in every CTA.
struct ClusterLayout {
    size_t x, z, squares, val[2], state[2], idx[2], base[2], len[2], end;
};
template <class T>
__host__ __device__ inline ClusterLayout cluster_layout(int m, int n, const ClusterCta& h) {
    ClusterLayout o;
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t p = at;
        at = align16(at + bytes);
        return p;
    };
    o.x = take(size_t(n) * sizeof(T)), o.z = take(size_t(m) * sizeof(T)), o.squares = take(size_t(n / 32 + 1) * 8);
    for (int k = 0; k < 2; ++k) {
        const size_t rows = size_t(h.rows[k]);
        o.val[k] = take(size_t(h.entries[k]) * sizeof(T));
        o.state[k] = take(rows * (8 + 3 * sizeof(T)));  // the FP64 running sum, then three vectors of T
        o.idx[k] = take(size_t(h.entries[k]) * 2);
        o.base[k] = take(size_t(h.bases(k)) * 4), o.len[k] = take(rows * 2);
    }
    o.end = at;
    return o;
}

// Barrier of the LP's CTAs: remote stores before it are visible after it.
template <bool MANY>
__device__ __forceinline__ void lp_barrier() {
    if (MANY) asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
    else __syncthreads();
}

// dst (the address of an entry of a vector copy in this CTA) = v in every CTA of the cluster.
__device__ __forceinline__ void store_remote(unsigned addr, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void store_remote(unsigned addr, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
template <bool MANY, class T>
__device__ __forceinline__ void store_all(T* dst, T v, int ctas) {
    if (!MANY) {
        *dst = v;
        return;
    }
    const unsigned a = unsigned(__cvta_generic_to_shared(dst));
    for (int q = 0; q < ctas; ++q) {
        unsigned r;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(q));
        store_remote(r, v);
    }
}

// A CTA's slice of one matrix in shared memory: the row at the slice's position t has len[t] entries. Entry e of the
// short row at position nlong + i is at base[i / 32] + 32 e + i % 32: the lanes of a warp read neighbouring values, and every
// warp's rows have about one length. Long row t's entries are contiguous from base[groups + t].
template <class T>
struct Slice {
    const T* val;
    const unsigned short* idx;
    const int* base;
    const short* len;
    int rows, nlong, groups;
};

// done(t, s) for every position t of the slice with its row's sum s of val * in: rows of at most kShort nonzeros in
// entry order by a thread, longer ones by a warp (lanes strided, shuffle tree; lane 0 calls done). The products go
// straight from registers into the sum: staging them for a balanced product pass, as the large kernels do, costs a
// barrier and more instructions than is left of the rows' imbalance after the sort.
template <class T, class In, class Done>
__device__ __forceinline__ void slice_phase(const Slice<T>& a, In in, Done done) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int g = warp; g < a.groups; g += kClusterThreads / 32) {
        const int t = a.nlong + 32 * g + lane, at = a.base[g], width = (a.base[g + 1] - at) >> 5;
        const int len = t < a.rows ? a.len[t] : 0;
        const T* val = a.val + at + lane;
        const unsigned short* idx = a.idx + at + lane;
        // the next four entries are loaded while four products are formed and added; past the row's end zeros are
        // added, which changes no sum (a sum that starts at +0 is never -0)
        double s = 0;
        T v[4];
        int c[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = e < len ? val[32 * e] : T(0), c[e] = e < len ? idx[32 * e] : -1;
        for (int k = 4; k < width + 4; k += 4) {
            T p[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) p[e] = c[e] >= 0 ? mul_rn(v[e], in(c[e])) : T(0);
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = k + e < len ? val[32 * (k + e)] : T(0), c[e] = k + e < len ? idx[32 * (k + e)] : -1;
#pragma unroll
            for (int e = 0; e < 4; ++e) s += double(p[e]);
        }
        if (t < a.rows) done(t, s);
    }
    for (int t = warp; t < a.nlong; t += kClusterThreads / 32) {
        const int lo = a.base[a.groups + t], len = a.len[t];
        double s = 0;
        for (int k = lane; k < len; k += 128) {  // four strides of products, then the adds in order
            T p[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) p[e] = k + 32 * e < len ? mul_rn(a.val[lo + k + 32 * e], in(a.idx[lo + k + 32 * e])) : T(0);
#pragma unroll
            for (int e = 0; e < 4; ++e) s += double(p[e]);
        }
        for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        if (lane == 0) done(t, s);
    }
}

// This CTA's slice of matrix k (0: A, 1: A^T) from global into shared memory. No barrier.
template <class T>
__device__ __forceinline__ Slice<T> load_slice(const int* plan, const ClusterCta& h, int k, const ClusterLayout& o, unsigned char* raw,
                                               const int* ptr, const int* idx, const T* val) {
    T* sval = reinterpret_cast<T*>(raw + o.val[k]);
    auto* sidx = reinterpret_cast<unsigned short*>(raw + o.idx[k]);
    int* sbase = reinterpret_cast<int*>(raw + o.base[k]);
    short* slen = reinterpret_cast<short*>(raw + o.len[k]);
    const int rows = h.rows[k], nlong = h.nlong[k], groups = h.groups(k), tid = threadIdx.x;
    const int *order = plan + h.order[k], *base = plan + h.base[k], *where = plan + h.where[1 - k];
    for (int i = tid; i < h.bases(k); i += kClusterThreads) sbase[i] = base[i];
    for (int t = nlong + tid; t < rows; t += kClusterThreads) {
        const int r = order[t], p0 = ptr[r], len = ptr[r + 1] - p0, i = t - nlong, at = base[i / 32] + i % 32;
        slen[t] = short(len);
#pragma unroll 4
        for (int e = 0; e < len; ++e) sval[at + 32 * e] = __ldg(val + p0 + e), sidx[at + 32 * e] = (unsigned short)where[__ldg(idx + p0 + e)];
    }
    for (int t = tid >> 5; t < nlong; t += kClusterThreads / 32) {
        const int r = order[t], p0 = ptr[r], len = ptr[r + 1] - p0, at = base[groups + t];
        if ((tid & 31) == 0) slen[t] = short(len);
        for (int e = tid & 31; e < len; e += 32) sval[at + e] = __ldg(val + p0 + e), sidx[at + e] = (unsigned short)where[__ldg(idx + p0 + e)];
    }
    return {sval, sidx, sbase, slen, rows, nlong, groups};
}

// The vectors of a slice's positions in shared memory.
template <class T>
struct SliceState {
    double* sum;
    T *a, *b, *c;
    __device__ SliceState(unsigned char* at, int rows)
        : sum(reinterpret_cast<double*>(at)), a(reinterpret_cast<T*>(at + 8 * rows)), b(a + rows), c(b + rows) {}
};

// `steps` iterations of each LP lps[cluster]: the first primal step, then row and column phase per step.
template <class T, bool MANY>
__global__ void __launch_bounds__(kClusterThreads, 1) k_cluster_iterate(const ClusterLp<T>* __restrict__ lps, int ctas, int steps) {
    extern __shared__ __align__(16) unsigned char raw[];
    const ClusterLp<T> p = lps[blockIdx.x / ctas];
    if (p.active && !*p.active) return;  // the same for every CTA of the cluster
    const ClusterCta h = reinterpret_cast<const ClusterCta*>(p.plan)[blockIdx.x % ctas];
    const ClusterLayout o = cluster_layout<T>(p.m, p.n, h);
    const int tid = threadIdx.x;
    T *x = reinterpret_cast<T*>(raw + o.x), *z = reinterpret_cast<T*>(raw + o.z);
    const double tau = p.par[0], sigma = p.par[1], inv_sigma = 1.0 / sigma;
    const Slice<T> A = load_slice(p.plan, h, 0, o, raw, p.a_ptr, p.a_idx, p.a_val);
    const Slice<T> AT = load_slice(p.plan, h, 1, o, raw, p.t_ptr, p.t_idx, p.t_val);
    const SliceState<T> rs(raw + o.state[0], A.rows), cs(raw + o.state[1], AT.rows);  // {zs, ax, rl, ru}, {xs, c, l, u}
    const int *row = p.plan + h.order[0], *col = p.plan + h.order[1];
    T *zo = z + h.first[0], *xo = x + h.first[1];  // this CTA's own entries
    lp_barrier<MANY>();  // every CTA of the cluster runs before it is written to
    for (int t = tid; t < A.rows; t += kClusterThreads) {
        const int r = row[t];
        zo[t] = p.z[r], rs.a[t] = p.Ax[r], rs.b[t] = p.rl[r], rs.c[t] = p.ru[r], rs.sum[t] = p.zs[r];
    }
    for (int t = tid; t < AT.rows; t += kClusterThreads) {
        const int j = col[t];
        const T cj = p.c[j], lj = p.l[j], uj = p.u[j];
        const T xn = T(clampv(double(p.x[j]) - tau * (double(cj) + double(p.ATz[j])), double(lj), double(uj)));
        cs.a[t] = cj, cs.b[t] = lj, cs.c[t] = uj, cs.sum[t] = p.xs[j] + double(xn);
        store_all<MANY>(xo + t, xn, ctas);
    }
    lp_barrier<MANY>();
    for (int s = 0; s < steps; ++s) {
        slice_phase(A, [&](int k) { return x[k]; }, [&](int t, double sum) {
            const T st = T(sum);
            const double v = double(zo[t]) + sigma * (2.0 * double(st) - double(rs.a[t]));
            const T zn = T(dual_prox(v, double(rs.b[t]), double(rs.c[t]), sigma, inv_sigma));
            store_all<MANY>(zo + t, zn, ctas);
            rs.a[t] = st, rs.sum[t] += double(zn);
        });
        lp_barrier<MANY>();
        const bool last = s + 1 == steps;
        slice_phase(AT, [&](int k) { return z[k]; }, [&](int t, double sum) {
            const T st = T(sum);
            if (last) {
                p.ATz[col[t]] = st;
            } else {
                const T xn = T(clampv(double(xo[t]) - tau * (double(cs.a[t]) + double(st)), double(cs.b[t]), double(cs.c[t])));
                store_all<MANY>(xo + t, xn, ctas);
                cs.sum[t] += double(xn);
            }
        });
        lp_barrier<MANY>();
    }
    for (int t = tid; t < A.rows; t += kClusterThreads) {
        const int r = row[t];
        p.z[r] = zo[t], p.Ax[r] = rs.a[t], p.zs[r] = rs.sum[t];
    }
    for (int t = tid; t < AT.rows; t += kClusterThreads) {
        const int j = col[t];
        p.x[j] = xo[t], p.xs[j] = cs.sum[t];
    }
}

// The power iteration on A^T A of each LP from its v0 (column order): est = the estimate, taken = the steps, as the
// steps of k_power_* with two products each compute them. The squares are added in column order, each group of 32 by a
// shuffle tree, then 8 groups, then all of them: the CTAs and warps of k_power_sumsq. v stays unnormalised in the copies;
// the factor is applied where it is gathered.
template <class T, bool MANY>
__global__ void __launch_bounds__(kClusterThreads, 1) k_cluster_power(const ClusterLp<T>* __restrict__ lps, int ctas, int iters, double* out) {
    extern __shared__ __align__(16) unsigned char raw[];
    __shared__ double sums[kClusterRows / 256 + 1], total;
    const ClusterLp<T> p = lps[blockIdx.x / ctas];
    const int rank = int(blockIdx.x) % ctas;
    const ClusterCta h = reinterpret_cast<const ClusterCta*>(p.plan)[rank];
    const ClusterLayout o = cluster_layout<T>(p.m, p.n, h);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    T *v = reinterpret_cast<T*>(raw + o.x), *w = reinterpret_cast<T*>(raw + o.z);
    const Slice<T> A = load_slice(p.plan, h, 0, o, raw, p.a_ptr, p.a_idx, p.a_val);
    const Slice<T> AT = load_slice(p.plan, h, 1, o, raw, p.t_ptr, p.t_idx, p.t_val);
    const int* where = p.plan + h.where[1];
    // the sums of 32 squares, a copy per CTA
    double* squares = reinterpret_cast<double*>(raw + o.squares);
    const int groups = (p.n + 31) / 32, blocks = (p.n + 255) / 256;
    lp_barrier<MANY>();
    for (int j = tid; j < p.n; j += kClusterThreads) v[where[j]] = p.v0[j];  // every CTA fills its own copy
    __syncthreads();
    double est = 0, f = 0;
    int it = 0;
    while (it < iters) {
        const bool scale = it > 0;
        slice_phase(A, [&](int k) { return scale ? T(double(v[k]) * f) : v[k]; },
                    [&](int t, double sum) { store_all<MANY>(w + h.first[0] + t, T(sum), ctas); });
        lp_barrier<MANY>();
        slice_phase(AT, [&](int k) { return w[k]; }, [&](int t, double sum) { store_all<MANY>(v + h.first[1] + t, T(sum), ctas); });
        lp_barrier<MANY>();
        for (int g = rank * (kClusterThreads / 32) + warp; g < groups; g += ctas * (kClusterThreads / 32)) {
            const int j = 32 * g + lane;
            const double e = j < p.n ? double(v[__ldg(where + j)]) : 0.0;
            double s = 0.0 + e * e;
            for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
            if (lane == 0) store_all<MANY>(squares + g, s, ctas);
        }
        lp_barrier<MANY>();
        static_assert(kClusterRows / 256 + 1 <= kClusterThreads, "a thread per block");
        if (tid < blocks) {  // 8 groups make a block; then the blocks in order
            double s = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) s += 8 * tid + i < groups ? squares[8 * tid + i] : 0.0;
            sums[tid] = s;
        }
        __syncthreads();
        if (tid == 0) {
            double all = 0;
#pragma unroll 8
            for (int i = 0; i < blocks; ++i) all += sums[i];
            total = all;
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
    if (rank == 0 && tid == 0) out[2 * (blockIdx.x / ctas)] = est, out[2 * (blockIdx.x / ctas) + 1] = double(it);
    lp_barrier<MANY>();
}

// ------------------------------------------------------------------------------------------ host side
constexpr size_t kClusterSmem = 224 * 1024;  // dynamic shared memory a CTA may use (227 KB less the static arrays)

// The plan of an LP on `ctas` CTAs: the CTAs' headers, then their row orders and group bases. A and A^T are cut into
// contiguous ranges of about equal cost (nonzeros plus 4 per row, the weight of a row's step). Returns the largest
// CTA's shared memory; offsets in the headers count from the plan's start.
//
// *us: what an iteration takes. A phase lasts as long as the warp with the most work; in us, FP32 (FP64): 0.33 (0.40) a
// group of 32 short rows, 0.027 (0.014) a step of its longest row, 0.63 (0.64) a long row (a shuffle tree in FP64, and one
// lane's fused step), 0.12 (0.075) its stride of 128. Several CTAs add 0.56 of barriers and 0.037 (0.028) a KB of x and z,
// which every SM takes in. Within 20 % of the time measured on 70 LPs of 360 to 60,000 nonzeros.
template <class T>
size_t cluster_plan(const int* a_ptr, const int* t_ptr, int m, int n, int ctas, std::vector<int>& plan, double* us) {
    constexpr int kHeader = int(sizeof(ClusterCta) / sizeof(int));
    std::vector<ClusterCta> head(static_cast<size_t>(ctas));
    plan.assign(size_t(ctas) * kHeader, 0);
    constexpr bool fp32 = sizeof(T) == 4;
    constexpr double group = fp32 ? 0.33 : 0.40, step = fp32 ? 0.027 : 0.014, long_row = fp32 ? 0.63 : 0.64, stride = fp32 ? 0.12 : 0.075;
    *us = ctas > 1 ? 0.56 + (fp32 ? 0.037e-3 : 0.028e-3) * double(size_t(m + n) * sizeof(T)) : 0;
    for (int k = 0; k < 2; ++k) {
        const int *ptr = k ? t_ptr : a_ptr, rows = k ? n : m;
        const double all = double(ptr[rows] - ptr[0]) + 4.0 * rows;
        int end = 0;
        double phase = 0;
        for (int q = 0; q < ctas; ++q) {
            double warp[kClusterThreads / 32] = {0};
            const int begin = end;
            while (end < rows && (q + 1 == ctas || double(ptr[end] - ptr[0]) + 4.0 * end < all * (q + 1) / ctas)) ++end;
            ClusterCta& h = head[size_t(q)];
            h.rows[k] = end - begin, h.first[k] = begin, h.order[k] = int(plan.size());
            for (int r = begin; r < end; ++r) plan.push_back(r);
            auto len = [&](int r) { return ptr[r + 1] - ptr[r]; };
            const auto first = plan.end() - (end - begin);
            std::stable_sort(first, plan.end(), [&](int x, int y) { return len(x) > len(y); });
            int nlong = 0;
            while (nlong < h.rows[k] && len(first[nlong]) > kShort) ++nlong;
            h.nlong[k] = nlong;
            std::vector<int> base;
            int at = 0;
            for (int t = nlong; t < h.rows[k]; t += 32) {
                base.push_back(at), at += 32 * len(first[t]);
                warp[(t - nlong) / 32 % (kClusterThreads / 32)] += group + step * ((len(first[t]) + 3) / 4 * 4);
            }
            base.push_back(at);  // the last group's end, and the first long row
            for (int t = 0; t < nlong; ++t) {
                if (t) base.push_back(at);
                at += len(first[t]);
                warp[t % (kClusterThreads / 32)] += long_row + stride * ((len(first[t]) + 127) / 128);
            }
            phase = std::max(phase, *std::max_element(warp, warp + kClusterThreads / 32));
            h.entries[k] = at, h.base[k] = int(plan.size());
            plan.insert(plan.end(), base.begin(), base.end());
        }
        *us += phase;
    }
    for (int k = 0; k < 2; ++k) {
        const size_t at = plan.size();
        plan.resize(at + size_t(k ? n : m));
        for (ClusterCta& h : head) {
            h.where[k] = int(at);
            for (int t = 0; t < h.rows[k]; ++t) plan[at + size_t(plan[size_t(h.order[k] + t)])] = h.first[k] + t;
        }
    }
    size_t most = 0;
    for (int q = 0; q < ctas; ++q) {
        std::copy_n(reinterpret_cast<const int*>(&head[size_t(q)]), kHeader, plan.begin() + q * kHeader);
        most = std::max(most, cluster_layout<T>(m, n, head[size_t(q)]).end);
    }
    return most;
}

// CTAs for an LP, by its nonzeros: one up to 3,000 a CTA, at most 8. Measured (us an iteration, FP64, 1 / 4 / 8 / 16
// CTAs): 1,400 nonzeros 1.33 / 1.92 / 1.95 / 2.17, 2,804: 1.98 / 1.99 / 2.07 / 2.35, 8,000: 3.09 / 2.48 / 2.39 / 2.90,
// 17,500: - / - / 3.31 / 3.64. Beyond 8 the remote stores of x and z, whose bytes into each SM do not shrink (distributed
// shared memory takes about 22 bytes a cycle), outweigh the shorter slices. Larger only where the LP does not fit.
inline int cluster_size(int64_t nnz) {
    int c = 1;
    while (c < 8 && nnz > 3000 * int64_t(c)) c *= 2;
    return c;
}

// Clusters of `ctas` CTAs with `smem` bytes each that the device runs at the same time (on 148 SMs 14 or 15 of 8 CTAs, 30
// to 33 of 4).
template <class T>
cudaError_t clusters_at_once(int ctas, size_t smem, int* count) {
    const void* kernel = ctas > 1 ? reinterpret_cast<const void*>(&k_cluster_iterate<T, true>)
                                  : reinterpret_cast<const void*>(&k_cluster_iterate<T, false>);
    const cudaError_t e = allow_launches(kernel, kClusterSmem, ctas > 1);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(ctas)), cfg.blockDim = dim3(kClusterThreads), cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = unsigned(ctas), attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr, cfg.numAttrs = 1;
    return cudaOccupancyMaxActiveClusters(count, kernel, &cfg);
}

// One cluster of `ctas` CTAs per LP of lps[0 .. count). Returns the launch's status.
template <class T, class... P, class... Args>
cudaError_t launch_cluster(void (*many)(const ClusterLp<T>*, int, P...), void (*one)(const ClusterLp<T>*, int, P...),
                           const ClusterLp<T>* lps, int count, int ctas, size_t smem, cudaStream_t st, Args... args) {
    auto kernel = ctas > 1 ? many : one;
    const cudaError_t e = allow_launches(reinterpret_cast<const void*>(kernel), kClusterSmem, ctas > 1);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(count * ctas)), cfg.blockDim = dim3(kClusterThreads);
    cfg.dynamicSmemBytes = smem, cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = unsigned(ctas), attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr, cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, lps, ctas, static_cast<P>(args)...);
}

}  // namespace taral
