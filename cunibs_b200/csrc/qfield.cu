// The reciprocity field on a grid (reference adm/reciprocity.py:173-213):
//     Q_d(g) = mu0/4pi sum_n W_dn x (g - r_n) / |g - r_n|^3,  mesh nodes r_n, up to three directions d.
//
// With w_gn = 1/|g - r_n|^3 and c the centre of a tile of grid points, W x (g - r) splits into
// W x (g - c) - W x (r - c), so
//     Q_d(g) = (sum_n w_gn W_dn) x (g - c) - sum_n w_gn (W_dn x (r_n - c)):
// per pair of a grid point and a node the distance and six multiply-adds a direction, 8 + 6 n_dir FP32 operations and one
// reciprocal square root, where the cross product of every pair takes 8 + 9 n_dir. The products W x (r - c) are formed
// once per block and node.
//
// Precision: g - c, r - c and W x (r - c) are taken in FP64 before they are rounded to FP32; both sums carry the same w. A
// block's sums over kStage nodes are added to running sums of their own, so that rounding does not grow with the number
// of nodes. What the rounding of the places and the cancellation of the two sums cost grows as |g - c| / |g - r|, so the
// nodes within 1 / kNear of the tile's half diagonal of its box take a cross product a point, with g - r and w from both
// parts that FP32 makes of g - c and r - c. Relative to 64 bits over eleven grids of 3 mm (nodes 3 to 10 mm apart): 1.8e-7 to
// 2.2e-7. A cross product a pair with grid-centred coordinates left 5.7e-7 to 1.2e-5; pairs nearer than an eighth of
// the half diagonal kept apart, but with the rounded places, 4.3e-7 to 6.8e-6.
//
// Bound: the FP32 pipe. 301k points by 179k nodes with three directions: 49.8 ms (26 operations a pair at the pipe's
// rate: 39 ms), one direction 28.9, against 73.7 and 35.0 for a cross product a pair and 50.6 and 29.8 with near pairs
// tested for in the loop over the nodes: sorted apart while they are staged, the far ones need no test. The matrix
// w on the tensor cores (tcgen05 kind::tf32, w in two terms from tensor memory, the weights in three) took 48.9 and,
// for 332k points by 52k nodes and one direction, 13.8 ms, where this form took 47.7 and 8.5 before near nodes were
// told apart: a block there forms w, hands it over and waits in step, and with one matrix instruction a chunk left it took 46.
#include <algorithm>
#include <cmath>

#include "internal.hpp"

namespace cunibs {
namespace {

constexpr int kThreads = 128;
constexpr int kPerThread = 4;                     // grid points a thread, as two pairs for the packed instructions
constexpr int kPoints = kThreads * kPerThread;    // points of a block's tile
constexpr int kStage = kThreads;                  // nodes staged at once, one a thread
constexpr int kMaxGroups = 16;                    // groups of threads that share a small tile's nodes
constexpr int kResident = 4;                      // blocks an SM
// Nodes within 1 / kNear of the tile's half diagonal of its box are near: 8 leaves 2.6e-7 to 4.8e-7 on the 6 and 10 mm heads
// with tiles of 8 x 8 x 8 and 3 x 15 x 11 points (restated on the CPU), 6 at most 3.0e-7 and 4 at most 3.6e-7, where a
// dearer cross product takes twice the nodes (1.4% of a 179k-node head's for a tile in its middle).
constexpr double kNear = 6.0;

// A staged node: -(r - c) and one unused word, then W and W x (r - c) of each direction; a near node holds the part
// of -(r - c) that FP32 leaves in place of the first direction's W x (r - c).
template <int ND>
constexpr int record_words() {
    return (4 + 6 * ND + 3) / 4 * 4;
}
// The staged nodes, the running sums, and the part of the points' places that FP32 leaves.
template <int ND>
constexpr int smem_bytes() {
    return static_cast<int>(sizeof(float)) * (kStage * record_words<ND>() + kPoints * (6 * ND + 3));
}

__device__ __forceinline__ float rsqrt_fast(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Boxes of t[0] x t[1] x t[2] <= kPoints / groups grid points; n[a] of them along axis a.
struct QTiles {
    int t[3];
    int n[3];
    int groups;
};

// Sources as the kernel reads them, one array per axis: positions in metres (3, n), then the weights of each
// direction (n_dir, 3, n).
__global__ void sources_kernel(const double* __restrict__ nodes_mm, const double* __restrict__ W, int n, int n_dir,
                               double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    for (int a = 0; a < 3; ++a) out[static_cast<long>(a) * n + i] = nodes_mm[3 * static_cast<long>(i) + a] * 1e-3;
    for (int d = 0; d < n_dir; ++d)
        for (int a = 0; a < 3; ++a)
            out[(3L + 3 * d + a) * n + i] = W[3 * (static_cast<long>(d) * n + i) + a];
}

// Work item = (tile of grid points, run of sources): item = run * n_tiles + tile. With one run the scaled
// field goes to out; with several the run's unscaled partial goes to part[run], and partial_sum_kernel
// adds the runs in order. The runs depend on the sizes only, never on ND, and a direction's sums are the same
// operations whatever ND. A tile of at most half the block's points (GROUPED) is held by 2 to 16 groups of
// threads, each with every point and its share of the staged nodes; their sums are added in order at the end.
template <int ND, bool GROUPED>
__global__ void __launch_bounds__(kThreads, kResident)
    qfield_kernel(AdmGrid gr, QTiles tiles, int n_tiles, const double* __restrict__ src, int n_src, int run, float scale,
                  float* __restrict__ out, float* __restrict__ part) {
    constexpr int kWords = record_words<ND>(), kPairs = 3 * ND;
    extern __shared__ __align__(16) float rec[];
    __shared__ int far_in_warp[kThreads / 32];
    float2* total = reinterpret_cast<float2*>(rec + kStage * kWords);  // [point][pair of sums][thread]
    float* low = reinterpret_cast<float*>(total + kPerThread * kPairs * kThreads);  // [axis][point][thread]
    const int groups = GROUPED ? tiles.groups : 1;
    const int width = kThreads / groups;  // threads a group
    const int group = GROUPED ? threadIdx.x / width : 0, lane = GROUPED ? threadIdx.x % width : threadIdx.x;
    const int tile = blockIdx.x % n_tiles, r0 = blockIdx.x / n_tiles;
    const int at[3] = {tile / (tiles.n[1] * tiles.n[2]) * tiles.t[0], tile / tiles.n[2] % tiles.n[1] * tiles.t[1],
                       tile % tiles.n[2] * tiles.t[2]};
    double center[3];
    float half[3];        // of the tile's box
    double lever2 = 0.0;  // |g - c|^2 of the tile's corners
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int extent = min(tiles.t[a], gr.shape[a] - at[a]);
        const double h = gr.spacing_mm[a] * 0.5 * (extent - 1) * 1e-3;
        half[a] = static_cast<float>(h);
        lever2 += h * h;
        center[a] = (gr.origin_mm[a] + gr.spacing_mm[a] * (at[a] + 0.5 * (extent - 1))) * 1e-3;
    }
    // Point p of the tile: its place relative to the centre, and its index in the grid (-1 past the tile).
    auto point = [&](int p, double (&g)[3]) {
        const int in[3] = {p / (tiles.t[1] * tiles.t[2]), p / tiles.t[2] % tiles.t[1], p % tiles.t[2]};
        bool inside = p < tiles.t[0] * tiles.t[1] * tiles.t[2];
        long index = 0;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const int extent = min(tiles.t[a], gr.shape[a] - at[a]);
            inside = inside && in[a] < extent;
            const int i = at[a] + min(in[a], extent - 1);
            g[a] = (gr.origin_mm[a] + gr.spacing_mm[a] * i) * 1e-3 - center[a];
            index = index * gr.shape[a] + i;
        }
        return inside ? index : -1L;
    };
    const float near2 = static_cast<float>(lever2 / (kNear * kNear));
    float2 gx[2], gy[2], gz[2];
#pragma unroll
    for (int u = 0; u < kPerThread; ++u) {
        double g[3];
        point(lane + u * width, g);
        const float h[3] = {static_cast<float>(g[0]), static_cast<float>(g[1]), static_cast<float>(g[2])};
#pragma unroll
        for (int a = 0; a < 3; ++a) low[(a * kPerThread + u) * kThreads + threadIdx.x] = static_cast<float>(g[a] - h[a]);
        (u % 2 ? gx[u / 2].y : gx[u / 2].x) = h[0];
        (u % 2 ? gy[u / 2].y : gy[u / 2].x) = h[1];
        (u % 2 ? gz[u / 2].y : gz[u / 2].x) = h[2];
    }
    for (int c = 0; c < kPerThread * kPairs; ++c) total[c * kThreads + threadIdx.x] = make_float2(0.f, 0.f);
    const int j_begin = r0 * run, j_end = min(n_src, j_begin + run);
    float2 acc[kPerThread][kPairs];
    int turn = 0;  // stages since the sums in acc began
    for (int j0 = j_begin; j0 < j_end; j0 += kStage) {
        const int nt = min(kStage, j_end - j0);
        // The far nodes go to the front of the stage, the near ones to its end.
        const int j = j0 + threadIdx.x;
        double x[3];
        float hi[3], box2 = 0.0f;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            x[a] = threadIdx.x < nt ? src[static_cast<long>(a) * n_src + j] - center[a] : 0.0;
            hi[a] = static_cast<float>(x[a]);
            const float past = fmaxf(fabsf(hi[a]) - half[a], 0.0f);
            box2 = fmaf(past, past, box2);
        }
        const bool is_near = box2 < near2;
        const unsigned staged = __ballot_sync(0xffffffffu, threadIdx.x < nt);
        const unsigned far = __ballot_sync(0xffffffffu, threadIdx.x < nt && !is_near);
        if (threadIdx.x % 32 == 0) far_in_warp[threadIdx.x / 32] = __popc(far);
        __syncthreads();
        int n_far = 0, far_before = 0;
#pragma unroll
        for (int w = 0; w < kThreads / 32; ++w) {
            if (w < threadIdx.x / 32) far_before += far_in_warp[w];
            n_far += far_in_warp[w];
        }
        if (threadIdx.x < nt) {
            const unsigned below = (1u << threadIdx.x % 32) - 1;
            const int near_before = threadIdx.x / 32 * 32 - far_before + __popc(staged & ~far & below);
            float* r = rec + (is_near ? n_far + near_before : far_before + __popc(far & below)) * kWords;
#pragma unroll
            for (int a = 0; a < 3; ++a) r[a] = -hi[a];
#pragma unroll
            for (int d = 0; d < ND; ++d) {
                double m[3];
#pragma unroll
                for (int a = 0; a < 3; ++a) m[a] = src[(3L + 3 * d + a) * n_src + j];
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    const int u = (a + 1) % 3, v = (a + 2) % 3;
                    r[4 + 6 * d + a] = static_cast<float>(m[a]);
                    r[7 + 6 * d + a] = static_cast<float>(m[u] * x[v] - m[v] * x[u]);
                }
            }
            if (is_near)
#pragma unroll
                for (int a = 0; a < 3; ++a) r[7 + a] = static_cast<float>(hi[a] - x[a]);
        }
        __syncthreads();
        if (turn == 0) {
#pragma unroll
            for (int u = 0; u < kPerThread; ++u)
#pragma unroll
                for (int c = 0; c < kPairs; ++c) acc[u][c] = make_float2(0.f, 0.f);
        }
#pragma unroll 1
        for (int i = group; i < n_far; i += groups) {
            const float* r = rec + i * kWords;
            const float4 at4 = *reinterpret_cast<const float4*>(r);
            float wu[kPerThread];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const float2 dx = __fadd2_rn(gx[q], make_float2(at4.x, at4.x));
                const float2 dy = __fadd2_rn(gy[q], make_float2(at4.y, at4.y));
                const float2 dz = __fadd2_rn(gz[q], make_float2(at4.z, at4.z));
                float2 d2 = __fmul2_rn(dx, dx);
                d2 = __ffma2_rn(dy, dy, d2);
                d2 = __ffma2_rn(dz, dz, d2);
                const float2 inv = make_float2(rsqrt_fast(d2.x), rsqrt_fast(d2.y));
                const float2 w = __fmul2_rn(__fmul2_rn(inv, inv), inv);
                wu[2 * q] = w.x;
                wu[2 * q + 1] = w.y;
            }
#pragma unroll
            for (int c = 0; c < kPairs; ++c) {
                const float2 m = *reinterpret_cast<const float2*>(r + 4 + 2 * c);
#pragma unroll
                for (int u = 0; u < kPerThread; ++u) acc[u][c] = __ffma2_rn(make_float2(wu[u], wu[u]), m, acc[u][c]);
            }
        }
        // The near nodes: g - r to FP32's last place from both parts, and the cross product itself, into the second sum.
#pragma unroll 1
        for (int i = n_far + group; i < nt; i += groups) {
            const float* r = rec + i * kWords;
#pragma unroll
            for (int u = 0; u < kPerThread; ++u) {
                const float* lo = low + u * kThreads + threadIdx.x;
                const float dx = ((u % 2 ? gx[u / 2].y : gx[u / 2].x) + r[0]) + (lo[0] + r[7]);
                const float dy = ((u % 2 ? gy[u / 2].y : gy[u / 2].x) + r[1]) + (lo[kPoints] + r[8]);
                const float dz = ((u % 2 ? gz[u / 2].y : gz[u / 2].x) + r[2]) + (lo[2 * kPoints] + r[9]);
                const float inv = rsqrt_fast(fmaf(dz, dz, fmaf(dy, dy, dx * dx)));
                const float w = -(inv * inv * inv);
#pragma unroll
                for (int d = 0; d < ND; ++d) {
                    const float mx = r[4 + 6 * d], my = r[5 + 6 * d], mz = r[6 + 6 * d];
                    float2* t = &acc[u][3 * d];
                    t[1].y = fmaf(w, fmaf(my, dz, -mz * dy), t[1].y);
                    t[2].x = fmaf(w, fmaf(mz, dx, -mx * dz), t[2].x);
                    t[2].y = fmaf(w, fmaf(mx, dy, -my * dx), t[2].y);
                }
            }
        }
        if (++turn == groups || j0 + kStage >= j_end) {
            turn = 0;
#pragma unroll
            for (int u = 0; u < kPerThread; ++u)
#pragma unroll
                for (int c = 0; c < kPairs; ++c) {
                    float2* t = total + (u * kPairs + c) * kThreads + threadIdx.x;
                    *t = __fadd2_rn(*t, acc[u][c]);
                }
        }
    }
    if (GROUPED) __syncthreads();
    const long count = static_cast<long>(gr.shape[0]) * gr.shape[1] * gr.shape[2];
    float* o = part ? part + static_cast<long>(r0) * ND * count * 3 : out;
    const float sc = part ? 1.0f : scale;
#pragma unroll 1
    for (int p = threadIdx.x; p < kPerThread * width; p += kThreads) {
        double gd[3];
        const long index = point(p, gd);
        if (index < 0) continue;
        const float g[3] = {static_cast<float>(gd[0]), static_cast<float>(gd[1]), static_cast<float>(gd[2])};
        const int u = p / width;
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            const float2* t = total + (u * kPairs + 3 * d) * kThreads + p % width;
            float2 t0 = t[0], t1 = t[kThreads], t2 = t[2 * kThreads];
            for (int h = 1; h < groups; ++h) {
                t0 = __fadd2_rn(t0, t[h * width]);
                t1 = __fadd2_rn(t1, t[kThreads + h * width]);
                t2 = __fadd2_rn(t2, t[2 * kThreads + h * width]);
            }
            const float m[3] = {t0.x, t0.y, t1.x}, w[3] = {t1.y, t2.x, t2.y};
            float* q = o + (static_cast<long>(d) * count + index) * 3;
            q[0] = sc * (fmaf(m[1], g[2], -m[2] * g[1]) - w[0]);
            q[1] = sc * (fmaf(m[2], g[0], -m[0] * g[2]) - w[1]);
            q[2] = sc * (fmaf(m[0], g[1], -m[1] * g[0]) - w[2]);
        }
    }
}

// out = scale * (the runs' partials added in order).
__global__ void partial_sum_kernel(long count, int runs, const float* __restrict__ part, float scale,
                                   float* __restrict__ out) {
    const long q = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (q >= count) return;
    float v = part[q];
#pragma unroll 8
    for (int c = 1; c < runs; ++c) v += part[c * count + q];
    out[q] = scale * v;
}

// The tiles that cover the grid at the least cost: per tile a stage's nodes over the groups that share them
// (with the staging worth kStageNodes more), and the near nodes kNearCost dearer (they take 14 + 9 n_dir operations a
// pair), where they are the share that the box and its near shell have of a ball of the mesh's reach. So a thick grid takes
// compact full tiles, a plane full tiles of one layer, and a line or a handful of points a few points held by many groups.
// One direction by 179k nodes, in ms: boxes near a cube's diagonal by one group and at most 16 runs; this rule; a cross
// product for every pair over the points in order:
//     200 x 200 points 9.78, 4.42, 4.75;    4096 in a line 6.31, 0.55, 0.56;    10^3 0.94, 0.18, 0.22;
//     16^3 0.94, 0.48, 0.56;    74 x 74 x 55 28.6, 28.9, 35.0.
// At 20 mm between points near shells take most of the head: 60^3 points by 121k nodes 15.2 ms, three directions 26.1 (25.3
// with the pairs tested one by one, 36.5 with a cross product for every pair).
constexpr double kStageNodes = 4.0;
constexpr double kNearCost = 1.0;
constexpr int kMaxSide = 64;

QTiles choose_tiles(const AdmGrid& gr, double reach_mm) {
    QTiles best{};
    double best_cost = INFINITY;
    const double ball = 4.18879 * reach_mm * reach_mm * reach_mm;
    for (int groups = 1; groups <= kMaxGroups; groups *= 2) {
        const int points = kPoints / groups;
        const double stage = static_cast<double>(kStage) / groups + kStageNodes;
        for (int x = 1; x <= std::min({points, kMaxSide, gr.shape[0]}); ++x)
            for (int y = 1; y <= std::min({points / x, kMaxSide, gr.shape[1]}); ++y) {
                const int t[3] = {x, y, std::min({points / (x * y), kMaxSide, gr.shape[2]})};
                double cost = stage;
                for (int a = 0; a < 3; ++a) cost *= (gr.shape[a] + t[a] - 1) / t[a];
                if (cost >= best_cost) continue;
                double side[3], lever2 = 0.0, box = 1.0;
                for (int a = 0; a < 3; ++a) {
                    side[a] = gr.spacing_mm[a] * (t[a] - 1);
                    lever2 += 0.25 * side[a] * side[a];
                }
                const double shell = 2.0 * std::sqrt(lever2) / kNear;
                for (int a = 0; a < 3; ++a) box *= side[a] + shell;
                cost *= 1.0 + kNearCost * std::min(1.0, box / ball);
                if (cost >= best_cost) continue;
                best_cost = cost;
                best.groups = groups;
                for (int a = 0; a < 3; ++a) best.t[a] = t[a];
            }
    }
    for (int a = 0; a < 3; ++a) best.n[a] = (gr.shape[a] + best.t[a] - 1) / best.t[a];
    return best;
}

// Nodes of a run: the fewest runs of sources whose waves of blocks (kResident per SM) take within 2% of the least time, a
// run's partial field counted with the nodes whose time it takes to write and to add.
int choose_run(int n_tiles, double points, int n_nodes, int slots) {
    const int stages = (n_nodes + kStage - 1) / kStage;
    const int most = std::min(stages, std::max(16, slots / n_tiles));
    const double partial = 0.5 + points / 4e4;
    auto cost = [&](int runs) {
        const int each = (stages + runs - 1) / runs;
        const double blocks = static_cast<double>(n_tiles) * ((stages + each - 1) / each);
        return std::ceil(blocks / slots) * each * kStage + (runs > 1 ? runs * partial : 0.0);
    };
    double least = INFINITY;
    for (int runs = 1; runs <= most; ++runs) least = std::min(least, cost(runs));
    int runs = 1;
    while (cost(runs) > 1.02 * least) ++runs;
    return (stages + runs - 1) / runs * kStage;
}

}  // namespace

void qfield_sample(const Mesh& m, const AdmGrid& gr, const double* W, int n_dir, float* Q, DevArray<double>& sources,
                   DevArray<float>& scratch, int sm_count, double reach_mm, cudaStream_t s) {
    if (n_dir < 1 || n_dir > kAdmMaxDir) fail(kEInval, "between 1 and 3 adjoint directions");
    sources.reserve(3 * static_cast<std::size_t>(m.n_nodes) * (1 + n_dir));
    sources_kernel<<<grid_for(m.n_nodes), kBlock, 0, s>>>(m.nodes.get(), W, m.n_nodes, n_dir, sources.get());
    count_launch();
    const QTiles tiles = choose_tiles(gr, reach_mm);
    const int n_tiles = tiles.n[0] * tiles.n[1] * tiles.n[2];
    const double points = static_cast<double>(gr.shape[0]) * gr.shape[1] * gr.shape[2];
    const int run = choose_run(n_tiles, points, m.n_nodes, sm_count * kResident);
    const int runs = (m.n_nodes + run - 1) / run;
    const long count = static_cast<long>(gr.shape[0]) * gr.shape[1] * gr.shape[2] * 3 * n_dir;
    if (runs > 1) scratch.reserve(static_cast<std::size_t>(count) * runs);
    float* part = runs > 1 ? scratch.get() : nullptr;
    auto go = [&](auto nd, auto grouped) {
        constexpr int ND = decltype(nd)::value;
        const auto kernel = qfield_kernel<ND, decltype(grouped)::value>;
        CUNIBS_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes<ND>()));
        kernel<<<n_tiles * runs, kThreads, smem_bytes<ND>(), s>>>(gr, tiles, n_tiles, sources.get(), m.n_nodes, run, 1e-7f,
                                                                  Q, part);
        count_launch();
    };
    auto pick = [&](auto nd) {
        if (tiles.groups > 1) go(nd, std::true_type{});
        else go(nd, std::false_type{});
    };
    if (n_dir == 1) pick(std::integral_constant<int, 1>{});
    else if (n_dir == 2) pick(std::integral_constant<int, 2>{});
    else pick(std::integral_constant<int, 3>{});
    CUNIBS_LAUNCH_CHECK("reciprocity field");
    if (runs > 1) {
        partial_sum_kernel<<<grid_for(count), kBlock, 0, s>>>(count, runs, part, 1e-7f, Q);
        count_launch();
    }
    CUNIBS_LAUNCH_CHECK("reciprocity field sum");
}

}  // namespace cunibs
