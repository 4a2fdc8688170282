// Test shim over the host side of panels.cuh: the plan of a matrix, its product formed on the host from the plan alone
// (as k_panel_fill and k_panel read it), and the rules. Allocations can be made to fail after a number of them.
#include "panels.cuh"

extern "C" void fail_allocations_after(int64_t count);

using namespace taral;

// y = A x by the plan; sizes: panels, most columns, rows and long rows of a panel, columns listed, entries stored.
// Returns 0 without panels, -1 where the plan is not one of this matrix, else 1.
extern "C" int panel_product(int rows, int cols, const int64_t* ptr, const int32_t* idx, const double* val, const double* x,
                             int target, int max_cols, int threads, int64_t allocs, double* y, int64_t* sizes) {
    fail_allocations_after(allocs);
    const PanelPlan p = build_panels(ptr, idx, rows, cols, target, max_cols, threads);
    fail_allocations_after(-1);
    if (p.empty()) return 0;
    for (int r = 0; r < rows; ++r) y[r] = -1e300;
    int next = 0;
    int64_t most[3] = {0, 0, 0};
    for (const Panel& h : p.panels) {
        if (h.row0 != next || h.rows < 1 || h.rows > kPanelRows || h.cols > max_cols) return -1;
        next += h.rows;
        const int size[3] = {h.cols, h.rows, h.nlong};
        for (int k = 0; k < 3; ++k) most[k] = std::max<int64_t>(most[k], size[k]);
        const int* list = p.cols.data() + h.col0;
        for (int i = 1; i < h.cols; ++i)
            if (list[i - 1] >= list[i]) return -1;
        auto sum = [&](int row, int64_t stored) {  // the row's entries, each found in the column list
            const int64_t b = ptr[h.row0 + row], e = ptr[h.row0 + row + 1];
            if (e - b > stored) return false;
            double s = 0;
            for (int64_t k = b; k < e; ++k) {
                const int* at = std::lower_bound(list, list + h.cols, idx[k]);
                if (at == list + h.cols || *at != idx[k]) return false;
                s += val[k] * x[*at];
            }
            y[h.row0 + row] = s;
            return true;
        };
        for (int q = 0; q < h.nlong; ++q) {
            const int4 r = p.longrow[size_t(h.long0 + q)];
            if (r.y <= kShort || r.x < 0 || r.x + r.y > p.long_entries) return -1;
            if (r.y != ptr[h.row0 + r.z + 1] - ptr[h.row0 + r.z]) return -1;
            if (!sum(r.z, r.y)) return -1;
        }
        for (int s = 0; s < h.slices; ++s) {
            const int2 sl = p.slice[size_t(h.slice0 + s)];
            if (sl.x < 0 || sl.x + sl.y > p.groups) return -1;
            for (int l = 0; l < 32; ++l) {
                const int row = p.order[size_t(32 * (h.slice0 + s) + l)];
                if (row == 0xffff) continue;
                if (row >= h.rows || !sum(row, 4 * sl.y)) return -1;
            }
        }
    }
    if (next != rows) return -1;
    if (most[0] != p.most.cols || most[1] != p.most.rows || most[2] != p.most.nlong) return -1;
    if (int64_t(p.cols.size()) != p.listed) return -1;
    const int64_t out[6] = {int64_t(p.panels.size()), most[0], most[1], most[2], p.listed, p.padded};
    std::copy(out, out + 6, sizes);
    return 1;
}

extern "C" int panels_suit_sizes(int64_t nnz, int64_t m, int64_t n, int64_t panels_a, int64_t panels_t, int sms, int fp64) {
    return panels_suit(nnz, m, n, panels_a, panels_t, sms, fp64 != 0);
}
extern "C" int64_t least_panels_of(int64_t nnz, int64_t rows, int target) { return least_panels(nnz, rows, target); }
