// Products with matrices whose rows share columns: panels of rows with the columns they use in shared memory.
//
// What bounds the row-block kernels (kernels.cuh) on such a matrix -- a multi-period model, where the rows of a period use
// the columns of that period -- is neither HBM (6-12 % busy) nor the arithmetic but L1: a warp's 32 gathered entries lie in
// about 28 cache lines, one tag lookup each, whether they hit or not. Shared memory serves 32 random words in 3-4 cycles.
//   panel  -- consecutive rows (kPanelRows at most) and the sorted list of the columns they use (kPanelCols at most). A
//             CTA copies those entries of the gathered vector to shared memory once and gathers there.
//   slices -- the panel's rows of at most kShort nonzeros, sorted by descending length, in groups of 32: a lane per row,
//             its entries in order, four at a time, stored so that a warp reads 32 x 16 (or 32) bytes of values and 32 x 8
//             bytes of 16-bit positions in the column list. Rows are filled up with zero values at a position that
//             holds zero.
//   long   -- longer rows, a warp each with its lanes strided; four sums at a time (4 / W rows of W instances) share one
//             shuffle tree whose first two levels split them between the lanes (6 exchanges instead of 20).
//   W      -- instances that share the matrix (batches): their entries of one column are neighbours in shared memory, one
//             gather serves all W, and the panel's matrix entries and column list are read once for them.
// Every row's products and summation order are those of the row blocks (block_sums), so the results are the same bits; the
// sums go through shared memory, so that the fused step reads and writes its vectors in row order.
#pragma once
#include <algorithm>
#include <cstdint>
#include <new>
#include <type_traits>
#include <vector>

#include "host.hpp"
#include "kernels.cuh"

namespace taral {

constexpr int kPanelRows = 1024, kPanelCols = 6144;
constexpr int kPanelThreads = 512;
struct Panel {
    int row0, rows;      // rows of the matrix
    int slice0, slices;  // slices of 32 short rows
    int long0, nlong;    // longer rows
    int col0, cols;      // the column list
};
// Device arrays of one matrix (or of several, one after another): entries of slice s at (slice[s].x + k) * 32 + lane, k <
// slice[s].y; order[32 s + lane]: the lane's row in its panel, 0xffff: none. Long row q = {first entry in lval / lplace,
// entries, row in its panel, -}.
template <class T>
struct alignas(16) Four {
    T v[4];
};
struct alignas(8) Places {
    unsigned short p[4];
};
template <class T>
struct PanelMat {
    const Panel* panels;
    const int2* slice;
    const unsigned short* order;
    const int* cols;
    const Four<T>* val;
    const Places* place;
    const int4* longrow;
    const T* lval;
    const unsigned short* lplace;
};
// A CTA's work in a batch: a panel and up to W instances; row shifts and gather offsets as for k_rowblock_batch. An unused
// slot has inst -1 and the shifts of slot 0.
template <int W>
struct alignas(16) PanelWork {
    Panel panel;
    int inst[W], row[W], gather[W];
};

// Fused steps on a row's sum, with the constants of its instance formed once per CTA (scale: two doubles per instance):
// load the row's operands, then apply.
template <class Y>
struct PanelStore {
    Y* y;
    struct Ops {};
    __device__ __forceinline__ double2 scale(int) const { return make_double2(0, 0); }
    __device__ __forceinline__ Ops load(int) const { return {}; }
    __device__ __forceinline__ void apply(int r, double s, double2, const Ops&) const { y[r] = Y(s); }
};
// The gathered vector times f, rounded as if it had been scaled in memory: a power step then needs no launch to scale it
// (refinery LP of 3.4M nonzeros FP64, a step: 2 products and 3 launches 39 us, 2 products and 1 launch 35).
template <class Y>
struct PanelScaled : PanelStore<Y> {
    static constexpr bool kScaled = true;
    const double* f;  // per instance
    __device__ __forceinline__ double2 scale(int inst) const { return make_double2(f[inst], 0); }
};
template <class E, class = void>
struct ScalesGather : std::false_type {};
template <class E>
struct ScalesGather<E, std::void_t<decltype(E::kScaled)>> : std::true_type {};
template <class T>
struct PanelRow {  // EpiRow, the division by sigma as in dual_prox
    T *Ax, *z;
    double* zs;
    const T *rl, *ru;
    const double* par;
    struct Ops { T z, ax, rl, ru; double zs; };
    __device__ __forceinline__ double2 scale(int inst) const { return make_double2(par[2 * inst + 1], 1.0 / par[2 * inst + 1]); }
    __device__ __forceinline__ Ops load(int r) const { return {z[r], Ax[r], rl[r], ru[r], zs[r]}; }
    __device__ __forceinline__ void apply(int r, double s, double2 k, const Ops& o) const {
        const T st = T(s);
        const T zn = T(dual_prox(double(o.z) + k.x * (2.0 * double(st) - double(o.ax)), double(o.rl), double(o.ru), k.x, k.y));
        Ax[r] = st, z[r] = zn, zs[r] = o.zs + double(zn);
    }
};
template <class T>
struct PanelCol {  // EpiCol
    T *ATz, *x;
    double* xs;
    const T *c, *l, *u;
    const double* par;
    int upd;
    struct Ops { T x, c, l, u; double xs; };
    __device__ __forceinline__ double2 scale(int inst) const { return make_double2(par[2 * inst], 0); }
    __device__ __forceinline__ Ops load(int r) const {
        if (!upd) return {T(0), T(0), T(0), T(0), 0.0};
        return {x[r], c[r], l[r], u[r], xs[r]};
    }
    __device__ __forceinline__ void apply(int r, double s, double2 k, const Ops& o) const {
        const T st = T(s);
        ATz[r] = st;
        if (upd) {
            const T xn = T(clampv(double(o.x) - k.x * (double(o.c) + double(st)), double(o.l), double(o.u)));
            x[r] = xn, xs[r] = o.xs + double(xn);
        }
    }
};

template <class X, int W>
constexpr size_t panel_smem(int cols, int rows, int nlong) {
    return (size_t(cols) + 1) * W * sizeof(X) + 16 + (size_t(rows) * W + 1) * sizeof(double) + size_t(nlong) * sizeof(int4);
}

// A lane's entries of R long rows q .. q + R - 1 (below end): STRIDES strides of 32 from entry k of each.
template <class T, int R, int STRIDES>
struct LongRows {
    T m[R][STRIDES];
    unsigned c[R][STRIDES / 2];  // places, two to a register
    __device__ __forceinline__ int place(int r, int e) const { return int(e & 1 ? c[r][e / 2] >> 16 : c[r][e / 2] & 0xffff); }
    __device__ __forceinline__ void load(const PanelMat<T>& a, const int4* heads, int q, int end, int none, int k) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int2 h = q + r < end ? *reinterpret_cast<const int2*>(heads + q + r) : make_int2(0, 0);
#pragma unroll
            for (int e = 0; e < STRIDES; ++e) {
                const bool in = k + 32 * e < h.y;
                m[r][e] = in ? __ldg(a.lval + h.x + k + 32 * e) : T(0);
                const unsigned p = in ? __ldg(a.lplace + h.x + k + 32 * e) : unsigned(none);  // the entry that holds zero
                c[r][e / 2] = e & 1 ? c[r][e / 2] | p << 16 : p;
            }
        }
    }
};

// One CTA per panel (work NULL: panel blockIdx.x, one instance) or per work item. A panel's latency is what a phase of a
// single LP takes, so every load that does not need the gathered entries is issued before the copy of those is waited for:
// the first long rows of each warp here, and in the loop the next ones before the current are summed. (More rows in
// flight per warp spill, and ranges prefetched into L2 compete with the loads: 10% slower each.) The lists and the first
// long rows are read while the phase before ends (launch_early; what that phase writes is then read past L1 or by plain
// loads): a refinery LP of 3.4M nonzeros takes 26.1 us an iteration in FP64 instead of 27.3, in FP32 18.0 instead of 19.8.
template <class T, class X, int W, class E>
__global__ void __launch_bounds__(kPanelThreads, 2) k_panel(const PanelMat<T> a, const X* __restrict__ xin,
                                                            const PanelWork<W>* __restrict__ work,
                                                            const int* __restrict__ active, E epi) {
    using P = typename ProdT<T, X>::type;
    constexpr int kWarps = kPanelThreads / 32, R = 4 / W, STRIDES = W == 4 ? 4 : 2;
    extern __shared__ __align__(16) unsigned char raw[];
    __shared__ double2 scale[W];
    launch_next();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const Panel p = work ? work[blockIdx.x].panel : a.panels[blockIdx.x];
    const int* list = a.cols + p.col0;
    constexpr int kAtOnce = 4;
    int c0[kAtOnce];  // the first columns this thread copies
#pragma unroll
    for (int i = 0; i < kAtOnce; ++i) c0[i] = tid + i * kPanelThreads < p.cols ? __ldg(list + tid + i * kPanelThreads) : -1;
    X* xs = reinterpret_cast<X*>(raw);
    double* sums = reinterpret_cast<double*>(raw + ((size_t(p.cols + 1) * W * sizeof(X) + 15) & ~size_t(15)));
    int4* heads = reinterpret_cast<int4*>(sums + (size_t(p.rows) * W + 1) / 2 * 2);
    for (int q = tid; q < p.nlong; q += kPanelThreads) heads[q] = __ldg(a.longrow + p.long0 + q);
    // a warp's long rows are consecutive
    const int per = ((p.nlong + kWarps - 1) / kWarps + R - 1) / R * R, lq0 = warp * per, lq1 = min(p.nlong, lq0 + per);
    LongRows<T, R, STRIDES> rows;
    __syncthreads();
    rows.load(a, heads, lq0, lq1, p.cols, lane);
    // everything before is the same in every launch; what follows is written by the launches before
    wait_previous();
    int gather[W];
    bool on[W];
    double factor[W];
    if (work) {
        int any = 0;
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const int i = work[blockIdx.x].inst[w];
            on[w] = i >= 0 && (!active || active[i]);
            gather[w] = work[blockIdx.x].gather[w], any |= on[w];
            if (tid == w) scale[w] = on[w] ? epi.scale(i) : make_double2(0, 0);
            if constexpr (ScalesGather<E>::value) factor[w] = on[w] ? epi.scale(i).x : 0;
        }
        if (!any) return;  // the same for the whole CTA
    } else {
        on[0] = true, gather[0] = 0;
        if (tid == 0) scale[0] = epi.scale(0);
        if constexpr (ScalesGather<E>::value) factor[0] = epi.scale(0).x;
    }
    auto entry = [&](X v, int w) {
        if constexpr (ScalesGather<E>::value) return X(double(v) * factor[w]);
        else return v;
    };
    {
        X g[kAtOnce][W];
#pragma unroll
        for (int i = 0; i < kAtOnce; ++i)
#pragma unroll
            for (int w = 0; w < W; ++w) g[i][w] = c0[i] >= 0 ? __ldcg(xin + gather[w] + c0[i]) : X(0);
#pragma unroll
        for (int i = 0; i < kAtOnce; ++i)
            if (c0[i] >= 0)
#pragma unroll
                for (int w = 0; w < W; ++w) xs[(tid + i * kPanelThreads) * W + w] = entry(g[i][w], w);
    }
#pragma unroll 4
    for (int i = tid + kAtOnce * kPanelThreads; i < p.cols; i += kPanelThreads) {
        const int c = __ldg(list + i);
#pragma unroll
        for (int w = 0; w < W; ++w) xs[i * W + w] = entry(__ldcg(xin + gather[w] + c), w);
    }
    if (tid < W) xs[p.cols * W + tid] = X(0);
    __syncthreads();
    // long rows: R at a time, four sums per lane
    for (int q0 = lq0; q0 < lq1; q0 += R) {
        const LongRows<T, R, STRIDES> now = rows;
        rows.load(a, heads, q0 + R, lq1, p.cols, lane);  // the next rows' entries, while these are summed
        double v[4] = {0, 0, 0, 0};
        auto add = [&](const LongRows<T, R, STRIDES>& x, int left) {  // left: entries of the longest row from here on
#pragma unroll
            for (int e = 0; e < STRIDES; ++e) {
                if (32 * e >= left) break;  // the same for the whole warp
#pragma unroll
                for (int r = 0; r < R; ++r)
#pragma unroll
                    for (int w = 0; w < W; ++w) v[r * W + w] += double(mul_rn(P(x.m[r][e]), P(xs[x.place(r, e) * W + w])));
            }
        };
        int longest = 0;
#pragma unroll
        for (int r = 0; r < R; ++r) longest = max(longest, q0 + r < lq1 ? heads[q0 + r].y : 0);
        add(now, longest);
        for (int k = 32 * STRIDES; k < longest; k += 32 * STRIDES) {
            LongRows<T, R, STRIDES> more;
            more.load(a, heads, q0, lq1, p.cols, k + lane);
            add(more, longest - k);
        }
        // each lane keeps two of the four sums, then one; a sum's tree is that of xor 16, 8, 4, 2, 1
        const bool hi = lane & 16, odd = lane & 8;
        double s0 = hi ? v[2] : v[0], s1 = hi ? v[3] : v[1];
        s0 += __shfl_xor_sync(0xffffffffu, hi ? v[0] : v[2], 16);
        s1 += __shfl_xor_sync(0xffffffffu, hi ? v[1] : v[3], 16);
        double s = odd ? s1 : s0;
        s += __shfl_xor_sync(0xffffffffu, odd ? s0 : s1, 8);
        for (int off = 4; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        const int which = lane >> 3, r = which / W, w = which % W;
        if ((lane & 7) == 0 && q0 + r < lq1) sums[w * p.rows + heads[q0 + r].z] = s;
    }
    // slices, the last warps first: the first ones have the most long rows
    for (int s = kWarps - 1 - warp; s < p.slices; s += kWarps) {
        const int2 sl = __ldg(a.slice + p.slice0 + s);
        const int local = a.order[32 * (p.slice0 + s) + lane];
        const Four<T>* val = a.val + size_t(sl.x) * 32 + lane;
        const Places* place = a.place + size_t(sl.x) * 32 + lane;
        double sum[W];
#pragma unroll
        for (int w = 0; w < W; ++w) sum[w] = 0;
        constexpr int G = W > 1 && sizeof(T) == 4 ? 4 : 2;  // groups of four entries in flight
        for (int k = 0; k < sl.y; k += G) {
            Four<T> v[G];
            Places c[G];
#pragma unroll
            for (int g = 0; g < G; ++g)
                if (k + g < sl.y) v[g] = val[32 * (k + g)], c[g] = place[32 * (k + g)];
#pragma unroll
            for (int g = 0; g < G; ++g)
                if (k + g < sl.y) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const X* from = xs + int(c[g].p[e]) * W;
#pragma unroll
                        for (int w = 0; w < W; ++w) sum[w] += double(mul_rn(P(v[g].v[e]), P(from[w])));
                    }
                }
        }
        if (local < p.rows) {
#pragma unroll
            for (int w = 0; w < W; ++w) sums[w * p.rows + local] = sum[w];
        }
    }
    __syncthreads();
    int shift[W];
#pragma unroll
    for (int w = 0; w < W; ++w) shift[w] = p.row0 + (work ? work[blockIdx.x].row[w] : 0);
    for (int t = tid; t < p.rows; t += kPanelThreads) {
        typename E::Ops ops[W];
#pragma unroll
        for (int w = 0; w < W; ++w) ops[w] = epi.load(shift[w] + t);  // of every slot: no branch between the loads
#pragma unroll
        for (int w = 0; w < W; ++w)
            if (on[w]) epi.apply(shift[w] + t, sums[w * p.rows + t], scale[w], ops[w]);
    }
}

// The slices' entries from the CSR matrix (a CTA per panel): values, and positions in the panel's column list found by
// bisection in shared memory.
template <class T>
__global__ void __launch_bounds__(kThreads) k_panel_fill(const Panel* __restrict__ panels, const int2* __restrict__ slice,
                                                         const unsigned short* __restrict__ order, const int* __restrict__ cols,
                                                         const int4* __restrict__ longrow, const int* __restrict__ ptr,
                                                         const int* __restrict__ idx, const T* __restrict__ val,
                                                         Four<T>* out, Places* place, T* lval, unsigned short* lplace) {
    __shared__ int list[kPanelCols];
    const Panel p = panels[blockIdx.x];
    for (int i = threadIdx.x; i < p.cols; i += kThreads) list[i] = cols[p.col0 + i];
    __syncthreads();
    auto find = [&](int want) {
        int lo = 0, hi = p.cols - 1;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (list[mid] < want) lo = mid + 1;
            else hi = mid;
        }
        return (unsigned short)lo;
    };
    const int lane = threadIdx.x & 31;
    for (int q = threadIdx.x >> 5; q < p.nlong; q += kThreads / 32) {
        const int4 row = longrow[p.long0 + q];
        const int b = ptr[p.row0 + row.z];
        for (int k = lane; k < row.y; k += 32) lval[row.x + k] = val[b + k], lplace[row.x + k] = find(idx[b + k]);
    }
    for (int s = threadIdx.x >> 5; s < p.slices; s += kThreads / 32) {
        const int2 sl = slice[p.slice0 + s];
        const int local = order[32 * (p.slice0 + s) + lane];
        const int b = local < p.rows ? ptr[p.row0 + local] : 0, len = local < p.rows ? ptr[p.row0 + local + 1] - b : 0;
        for (int k = 0; k < sl.y; ++k) {
            Four<T> v;
            Places c;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int at = 4 * k + e;
                if (at >= len) {
                    v.v[e] = T(0), c.p[e] = (unsigned short)p.cols;
                    continue;
                }
                v.v[e] = val[b + at], c.p[e] = find(idx[b + at]);
            }
            out[(size_t(sl.x) + k) * 32 + lane] = v, place[(size_t(sl.x) + k) * 32 + lane] = c;
        }
    }
}

// ------------------------------------------------------------------------------------------ host side
struct PanelSize {  // the largest panel's columns, rows and long rows
    int cols = 0, rows = 0, nlong = 0;
    void cover(const PanelSize& o) { cols = std::max(cols, o.cols), rows = std::max(rows, o.rows), nlong = std::max(nlong, o.nlong); }
};
struct PanelPlan {
    std::vector<Panel> panels;
    std::vector<int2> slice;
    std::vector<unsigned short> order;
    std::vector<int4> longrow;
    std::vector<int> cols;
    int groups = 0;             // entry groups of 32 lanes x 4
    int long_entries = 0;
    int64_t padded = 0;         // entries stored
    int64_t listed = 0;         // columns in the panels' lists
    PanelSize most;
    bool empty() const { return panels.empty(); }
    void append(const PanelPlan& p, int row_shift) {
        for (Panel h : p.panels) {
            h.row0 += row_shift, h.slice0 += int(slice.size()), h.long0 += int(longrow.size()), h.col0 += int(cols.size());
            panels.push_back(h);
        }
        for (int2 q : p.slice) slice.push_back(make_int2(q.x + groups, q.y));
        for (int4 q : p.longrow) longrow.push_back(make_int4(q.x + long_entries, q.y, q.z, 0));
        order.insert(order.end(), p.order.begin(), p.order.end());
        cols.insert(cols.end(), p.cols.begin(), p.cols.end());
        groups += p.groups, long_entries += p.long_entries, padded += p.padded, listed += p.listed;
        most.cover(p.most);
    }
};

// Marks of the columns that a panel has used, kept from panel to panel.
struct PanelMarks {
    std::vector<int> seen;
    int stamp = 0;
    explicit PanelMarks(int cols) : seen(size_t(cols), 0) {}
};
// Panels of about `target` nonzeros and at most max_cols columns for the rows [first, last); empty where a single row uses
// more columns than that. lists = false: their sizes only, without the column lists in order.
template <class I>
PanelPlan panels_of(const I* ptr, const int32_t* idx, int first, int last, int cols, int target, int max_cols, PanelMarks& marks,
                    bool lists = true) {
    PanelPlan plan;
    std::vector<int>& seen = marks.seen;
    std::vector<int> list;
    int &stamp = marks.stamp, low = 0, high = 0;
    auto unique = [&](int r0, int r1) {  // columns of the rows [r0, r1) into list, unsorted, all of them in [low, high]
        list.clear(), ++stamp, low = cols, high = -1;
        for (I k = ptr[r0]; k < ptr[r1]; ++k) {
            const int c = idx[k];
            if (seen[size_t(c)] != stamp) seen[size_t(c)] = stamp, list.push_back(c), low = std::min(low, c), high = std::max(high, c);
        }
    };
    auto len = [&](int r) { return int(ptr[r + 1] - ptr[r]); };
    std::vector<int> by, shorter, count(size_t(kShort) + 2);
    for (int r0 = first; r0 < last;) {
        int r1 = r0;
        while (r1 < last && r1 - r0 < kPanelRows && (r1 == r0 || ptr[r1 + 1] - ptr[r0] <= I(target))) ++r1;
        for (unique(r0, r1); int(list.size()) > max_cols; unique(r0, r1)) {  // too many columns: half the rows
            if (r1 - r0 == 1) return PanelPlan();
            r1 = r0 + (r1 - r0) / 2;
        }
        Panel p{};
        p.row0 = r0, p.rows = r1 - r0, p.slice0 = int(plan.slice.size()), p.col0 = int(plan.cols.size()), p.cols = int(list.size());
        p.long0 = int(plan.longrow.size());
        plan.listed += int64_t(list.size());
        if (!lists) {
        } else if (int64_t(high) - low < 16 * int64_t(list.size())) {  // in column order: the marks of the range
            for (int c = low; c <= high; ++c)
                if (seen[size_t(c)] == stamp) plan.cols.push_back(c);
        } else {
            std::sort(list.begin(), list.end());
            plan.cols.insert(plan.cols.end(), list.begin(), list.end());
        }
        // long rows in row order, the others by descending length (stable counting sort)
        shorter.clear(), std::fill(count.begin(), count.end(), 0);
        for (int r = r0; r < r1; ++r) {
            const int l = len(r);
            if (l > kShort) {
                plan.longrow.push_back(make_int4(plan.long_entries, l, r - r0, 0));
                plan.long_entries += l, plan.padded += l;
            } else {
                shorter.push_back(r), ++count[size_t(kShort - l) + 1];
            }
        }
        p.nlong = int(plan.longrow.size()) - p.long0;
        for (size_t l = 1; l < count.size(); ++l) count[l] += count[l - 1];
        by.resize(shorter.size());
        for (int r : shorter) by[size_t(count[size_t(kShort - len(r))]++)] = r;
        for (size_t t = 0; t < by.size(); t += 32) {
            const int width = (len(by[t]) + 3) / 4;
            plan.slice.push_back(make_int2(plan.groups, width));
            plan.groups += width, plan.padded += 128 * int64_t(width);
            for (size_t l = t; l < t + 32; ++l) plan.order.push_back(l < by.size() ? (unsigned short)(by[l] - r0) : 0xffff);
        }
        p.slices = int(plan.slice.size()) - p.slice0;
        plan.most.cover({p.cols, p.rows, p.nlong});
        plan.panels.push_back(p);
        r0 = r1;
    }
    return plan;
}

// Whether an LP's products are faster on panels than on row blocks, by the number of panels of A and of A^T (a lower bound
// refuses before they are planned). A panel kernel has 2 CTAs an SM: a second wave of panels costs what a first does (a
// tenth of one starts as the first panels end), and a panel of short rows is bound by its 1,024 rows, not by its nonzeros.
// Measured (us an iteration, row blocks / panels):
//   up to 2.2 an SM: refinery of 64 periods (304 panels) FP32 29.8 / 25.6, FP64 52.3 / 40.1; band of 8 (280,000 rows) 12.7 /
//              10.0 and 21.9 / 12.8; band of 20 (4.4M nonzeros) 20.4 / 14.8 and 42.3 / 26.0; blocks of 50 x 60 16.3 / 14.2,
//              33.5 / 17.4; random in blocks of 300 x 500 (5M, 320 panels) 30.8 / 25.1 and 54.4 / 43.7
//   more, FP32: refinery of 96 41.7 / 50.1, band of 20 (6M) 26.5 / 32.9, band of 100 (9M) 41.2 / 46.2, blocks of 150 x 200
//              (6M) 33.2 / 30.5, (9.9M) 49.0 / 58.7, band of 8 (1M rows) 37.7 / 58.6
//   more, FP64, full panels: refinery of 96 73.7 / 60.4, band of 100 (9M) 83.9 / 56.2, band of 20 (6M) 46.9 / 45.4; filled by
//              their rows: band of 10 (400,000 rows) 33.5 / 39.7, band of 7 (600,000) 35.6 / 38.1
//   rows of fewer than 8: band of 6 (350,000 rows) 10.8 / 17.7 and 13.8 / 24.5, band of 7 (304 panels) 10.8 / 14.9
constexpr int kFullPanel = 15000;  // of the largest target, 16,384
inline bool panels_suit(int64_t nnz, int64_t m, int64_t n, int64_t panels_a, int64_t panels_t, int sms, bool fp64) {
    const int64_t most = std::max(panels_a, panels_t);
    return nnz >= 8 * std::max(m, n) && (5 * most <= 11 * int64_t(sms) || (fp64 && nnz >= kFullPanel * most));
}
inline int64_t least_panels(int64_t nnz, int64_t rows, int target) {
    return std::max((nnz + target - 1) / target, (rows + kPanelRows - 1) / kPanelRows);
}

// Panels for the CSR rows on `threads` host threads (max_cols <= kPanelCols), or none where they do not pay: the column
// lists must hold at most a third as many columns as the panels hold nonzeros (a list and its entries of x cost about as
// much to read as they save otherwise), and padding at most 40 % of the nonzeros.
template <class I>
PanelPlan plan_of_panels(const I* ptr, const int32_t* idx, int rows, int cols, int target, int max_cols, int threads) {
    PanelPlan plan;
    if (rows == 0 || ptr[rows] == ptr[0]) return plan;
    for (int r = 0; r < rows; ++r)
        if (ptr[r + 1] - ptr[r] > I(kTile)) return plan;  // summed by a whole CTA in the row blocks
    const int64_t all = int64_t(ptr[rows] - ptr[0]);
    auto pays = [](const PanelPlan& p, int64_t nnz) { return nnz >= 3 * p.listed && 10 * p.padded <= 14 * nnz; };
    {  // a look at a few rows first: most matrices without shared columns are refused here
        PanelMarks marks(cols);
        PanelPlan look;
        int64_t nnz = 0;
        for (int q = 0; q < 4; ++q) {
            const int r0 = int(int64_t(rows) * q / 4);
            int r1 = r0;
            while (r1 < rows && ptr[r1] - ptr[r0] < I(target)) ++r1;
            const PanelPlan p = panels_of(ptr, idx, r0, r1, cols, target, max_cols, marks, false);
            if (p.empty()) return plan;
            look.append(p, 0), nnz += int64_t(ptr[r1] - ptr[r0]);
        }
        if (!pays(look, nnz)) return plan;
    }
    // parts planned on their own (each ends with a panel that is not full), the same on every host
    const int parts = int(std::max<int64_t>(1, std::min<int64_t>(16, all / (8 * int64_t(target)))));
    std::vector<PanelPlan> part(static_cast<size_t>(parts));
    split_ranges(parts, threads, [&](int, int64_t q0, int64_t q1) {
        try {
            PanelMarks marks(cols);
            for (int64_t q = q0; q < q1; ++q) {
                auto cut = [&](int64_t k) {
                    return k >= parts ? rows : int(std::lower_bound(ptr, ptr + rows, ptr[0] + I(all * k / parts)) - ptr);
                };
                part[size_t(q)] = panels_of(ptr, idx, cut(q), cut(q + 1), cols, target, max_cols, marks);
            }
        } catch (const std::bad_alloc&) {  // no exception leaves a thread
            for (int64_t q = q0; q < q1; ++q) part[size_t(q)] = PanelPlan();
        }
    });
    for (const PanelPlan& p : part) plan.append(p, 0);
    int covered = 0;
    for (const Panel& p : plan.panels) covered += p.rows;
    return covered == rows && pays(plan, all) ? plan : PanelPlan();
}
// The same; none either where the host has no memory for the plan.
template <class I>
PanelPlan build_panels(const I* ptr, const int32_t* idx, int rows, int cols, int target, int max_cols, int threads) {
    try {
        return plan_of_panels(ptr, idx, rows, cols, target, max_cols, threads);
    } catch (const std::bad_alloc&) {
        return PanelPlan();
    }
}

// The panel counterparts of the row blocks' fused steps.
template <class Y> PanelStore<Y> panel_step(const EpiStore<Y>& e) { return {e.y}; }
template <class T> PanelRow<T> panel_step(const EpiRow<T>& e) { return {e.Ax, e.z, e.zs, e.rl, e.ru, e.par}; }
template <class T> PanelCol<T> panel_step(const EpiCol<T>& e) { return {e.ATz, e.x, e.xs, e.c, e.l, e.u, e.par, e.upd}; }

template <class T, int W, class E>
cudaError_t launch_panels(const PanelMat<T>& a, int ctas, const PanelSize& most, const T* xin, const PanelWork<W>* work,
                          const int* active, const E& step, cudaStream_t st) {
    const size_t smem = panel_smem<T, W>(most.cols, most.rows, most.nlong);
    const cudaError_t e = allow_launches(reinterpret_cast<const void*>(&k_panel<T, T, W, E>),
                                         panel_smem<T, W>(kPanelCols, kPanelRows, kPanelRows));
    if (e != cudaSuccess) return e;
    return launch_early(k_panel<T, T, W, E>, ctas, kPanelThreads, smem, st, a, xin, work, active, step);
}

}  // namespace taral
