// Phase-reduced Kirchhoff sum on a rectangular screen as a tensor-core
// product (xk_grid.cu).
#pragma once

#include <climits>
#include <vector>

#include "xk_internal.cuh"

namespace xk {

// What the device finds out about the order of a solve's screen points: point
// i * len + l has one coordinate that depends on l alone (the inner axis), at
// most one that depends on i alone (the outer axis), the rest constant, bit
// for bit. extent[axis][k]: largest half-extent of a tile of kGridSpan << k
// consecutive points of the axis (0 outer, 1 inner), as the bits of a double.
constexpr int kGridSpan = 32;  // fewest rows or columns of a tile in use
constexpr int kGridSizes = 4;  // tile sizes, kGridSpan << 0 .. 3 (256)

// The product's forms: 128 columns per tile, 256, and 256 with the second order.
enum GridForm { kFormNarrow, kFormWide, kFormSecond };

struct GridProbe {
    int len;         // inner length; 0 if there is no such order
    int bad;         // a point breaks the order
    int inner;       // coordinate index (0 x, 1 y, 2 z) of the inner axis
    int outer_mask;  // coordinates that vary with i
    // Largest half extent (bits of a double) of kGridSpan << k points, outer and inner.
    unsigned long long extent[2][kGridSizes];
};

// Ranges of a solve's inputs (from the planner's summary).
struct GridRanges {
    double rlo[3], rhi[3];  // rays
    double plo[3], phi[3];  // screen
    double nlo[3], nhi[3];  // normals
    double nl_lo, nl_hi;
    double rc[3], pc[3];    // centroids
    double spread2;         // mean squared ray distance from the centroid
    double max_amp[2];      // largest component of either amplitude column summed
    double k;
};

// Everything the product of one solve needs besides the workspace.
struct GridPlan {
    int m_axis = 0, n_axis = 0, c_axis = 0;  // coordinates of the product's rows, columns, the rest
    bool rows_outer = true;                  // rows are the outer screen axis
    size_t nm = 0, nn = 0;                   // rows, columns (screen points along the axes)
    size_t inner_len = 0;
    int form = kFormNarrow;                  // GridForm
    int span_m = 0, span_n = 0;              // rows and columns of a tile in use
    int m_tiles = 0, n_tiles = 0, columns = 1;  // tiles of 256 rows and 128 or 256 columns; amplitude columns
    int ray_blocks = 0, splits = 1, seg = 0;
    size_t n = 0, chunk_rays = 0;            // rays, rays per product launch
    bool amp = false;                        // amplitude varies along a tile
    double c0 = 0.0, h0 = 0.0, k = 0.0, kt = 0.0, kt_lo = 0.0;
    double unit = 1.0;  // the kernels' lengths are mm times this power of two
    double inv_scale[2] = {1.0, 1.0}, e_bound = 0.0;
    RaysDev rays{};
    PixDev pix{};
    FieldDev out{};
    const double* amps[2][2] = {{nullptr, nullptr}, {nullptr, nullptr}};  // [column][re, im]
    double pes[2] = {1.0, 0.0}, pep[2] = {0.0, 0.0};  // one column: (Es, Ep) = (pes, pep) A
    double* axes = nullptr;  // nm + nn coordinates, then m_tiles + n_tiles tile references
};

struct GridWorkspace {
    DevBuf recs, partial;
};

// Below these the general kernel's whole solve is a few tens of microseconds
// of work; a screen of at most 1024 points fills four of its tiles.
constexpr size_t kGridMinRays = 1024, kGridMinPoints = 1025;

// Doubles `axes` of a plan for m screen points may need.
inline size_t grid_axes_doubles(size_t m) { return 2 * (m + 2) + 4; }

// Launches `kernel` over the solves' blocks, N solves at a time.
template <int N, class Batch, class Args>
Status launch_solves(void (*kernel)(Batch), std::vector<Args>& solves, cudaStream_t stream,
                     int* kernels) {
    for (size_t i0 = 0; i0 < solves.size(); i0 += N) {
        Batch b{};
        int blocks = 0;
        for (int i = 0; i < N; ++i) {
            b.s[i].first = INT_MAX;
            if (i0 + i >= solves.size()) continue;
            b.s[i] = solves[i0 + i];
            b.s[i].first = blocks;
            blocks += b.s[i].blocks;
        }
        kernel<<<blocks, 256, 0, stream>>>(b);
        XK_CUDA_TRY(cudaGetLastError());
        ++*kernels;
    }
    return Status::Ok();
}

// Checks the order of one screen. `first_change`: the candidate for the inner
// length (device). `probe` is zeroed by an earlier kernel on the stream,
// `host_probe` (pinned) by the caller; the kernel writes both. `ticket`: see
// last_block.
struct ProbeArgs {
    PixDev pix;
    int m;
    int first, blocks;  // of the grid's blocks; set by the launch
    const double* first_change;
    GridProbe* probe;
    unsigned* ticket;
    GridProbe* host_probe;
};
Status grid_probe_enqueue(std::vector<ProbeArgs>& screens, cudaStream_t stream, int* kernels);

// Decides whether the product takes the solve and fills `g` (without device
// pointers); `columns` amplitude columns; `tolerance` as requested.
bool grid_plan(const GridProbe& probe, const GridRanges& r, size_t n, size_t m, int columns,
               double tolerance, int num_sms, GridPlan* g);

// Gathers the axes into g.axes.
Status grid_axes_enqueue(const GridPlan& g, cudaStream_t stream);

// Raises `recs` and `partial` [bytes] to what the product needs; allocates them.
void grid_sizes(const GridPlan& g, size_t* recs, size_t* partial);
Status grid_reserve(size_t recs, size_t partial, GridWorkspace& ws);

// Enqueues the product (allocates nothing beyond grid_reserve). `err`: error
// word the kernels can write (device or pinned). `stall`: test hook, the first
// stage never completes.
Status grid_enqueue(const GridPlan& g, GridWorkspace& ws, int* err, uint32_t wait_limit,
                    bool stall, cudaStream_t stream, int* kernels);

}  // namespace xk
