// APR tree means and APR isotropic convolution on the GPU.
//
// Tree means (APRTreeNumerics::fill_tree_mean, APRTreeNumerics.hpp:63-203):
// every node sums its children in the reference's order -- particle children
// first, then tree children, z then x then y within each -- with the
// reference's boundary scale factors (:97-110).  Levels run from fine to coarse.
//
// Row words: for every row of every level, one entry per 32 cells in y: a bit
// per cell that holds an element of the row, and the row offset of the first
// of them.  A cell's value is then one entry read and a population count away,
// so the convolution gathers the cells it needs and reads no y coordinates.
//
// Convolution (APRFilter::convolve_pencil, APRFilter.hpp:1094-1216), per level
// from fine to coarse, in two kernels.  level_image writes the level's
// isotropic neighbourhood image -- the values the reference gathers into its
// pencil buffer (update_dense_array, :825-849): same-level particles, parents
// one level coarser (piecewise constant, :766-793) and tree means of the same
// level (:802-818), with the reflective or zero boundary (:287-504) around
// them -- to HBM, a run of planes at a time.  conv_block then sums the 27 / 125
// taps of every particle of the level from that image, eight neighbours a
// lane, in the stencil's memory order without contraction
// (run_convolution_pencil, :706-736).  A cell no particle covers holds a
// sentinel; reading it is counted as a stale read (the reference would read a
// stale pencil buffer there) and contributes 0.
#include "kernels.cuh"

namespace aprb {

namespace {

constexpr uint32_t kMissingBits = 0x7fbadbadu;               // NaN payload marking an uncovered cell
constexpr uint64_t kMissingBits64 = 0x7ff7badbadbadbadull;  // the same for double values

// Value type of the filter: float, or double for the FP64 instantiation of
// richardson_lucy.  Arithmetic goes through the round-to-nearest intrinsics
// so no contraction can change a result.
template <typename T>
struct VT;
template <>
struct VT<float> {
    static __device__ __forceinline__ float miss() { return __uint_as_float(kMissingBits); }
    static __device__ __forceinline__ bool is_miss(float v) { return __float_as_uint(v) == kMissingBits; }
    static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
    static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
    static __device__ __forceinline__ float div(float a, float b) { return __fdiv_rn(a, b); }
};
template <>
struct VT<double> {
    static __device__ __forceinline__ double miss() { return __longlong_as_double((long long)kMissingBits64); }
    static __device__ __forceinline__ bool is_miss(double v) {
        return (uint64_t)__double_as_longlong(v) == kMissingBits64;
    }
    static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
    static __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
    static __device__ __forceinline__ double div(double a, double b) { return __ddiv_rn(a, b); }
};

struct LD {
    int yn, xn, zn;
};
LD ld(const Geom &g, int l) { return LD{g.y_num[l], g.x_num[l], g.z_num[l]}; }
uint64_t nrow(const Geom &g, int l) { return (uint64_t)g.x_num[l] * g.z_num[l]; }
__host__ __device__ __forceinline__ int nword(int yn) { return (yn + 31) / 32; }

// words[row * nw + w] = (bits, offset) of the cells [32 w, 32 w + 32) of the
// row: bit b set when cell 32 w + b holds an element, offset = position in the
// row of the first of them.  Entries of empty words stay as cleared by the
// caller.  One warp per row, 32 elements a step: y ascends, so a word's
// elements are neighbours and the word's bits are one warp reduction (a dense
// row has one or two words a step).
__global__ void row_words_kernel(const uint64_t *__restrict__ xz_end, uint64_t row_base,
                                 const uint16_t *__restrict__ y_vec, uint64_t rows, int nw,
                                 uint2 *__restrict__ words) {
    const uint64_t row = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (row >= rows) return;
    const uint64_t b = xz_end[row_base + row - 1], e = xz_end[row_base + row];
    const int n = (int)(e - b);
    uint2 *W = words + row * (uint64_t)nw;
    int cur = -1, off = 0;   // the word being filled and its first element
    unsigned bits = 0;
    for (int i0 = 0; i0 < n; i0 += 32) {
        const int i = i0 + lane;
        const int y = i < n ? (int)y_vec[b + i] : -1;
        const int w = y >> 5;  // -1 past the end
        unsigned todo = __ballot_sync(0xffffffffu, y >= 0);
        while (todo) {
            const int lead = __ffs(todo) - 1;
            const int lw = __shfl_sync(0xffffffffu, w, lead);
            if (lw != cur) {
                if (cur >= 0 && cur < nw && lane == 0) W[cur] = make_uint2(bits, (unsigned)off);
                cur = lw;
                off = i0 + lead;
                bits = 0;
            }
            bits |= __reduce_or_sync(0xffffffffu, w == lw ? 1u << (y & 31) : 0u);
            todo &= ~__ballot_sync(0xffffffffu, w == lw);
        }
    }
    if (cur >= 0 && cur < nw && lane == 0) W[cur] = make_uint2(bits, (unsigned)off);
}

// ---------------------------------------------------------------------------
// tree means of tree level t (children at level t+1)
// ---------------------------------------------------------------------------
struct TreeLevelArgs {
    LD dt;                  // tree level t dims (== APR level t dims)
    LD dc;                  // child level dims
    uint64_t t_row_base;    // tree level_xz[t]
    uint64_t c_row_base;    // APR level_xz[t+1]
    uint64_t ct_row_base;   // tree level_xz[t+1] (0 when t+1 has no tree level)
    const uint2 *tw;        // row words of the parents
    const uint2 *cw, *ctw;  // row words of the children (ctw null: no tree level)
};

// One warp per parent row, or per part of `per` words of one where rows are long
// and few, a lane per cell of a parent word.  The parent's word gives the node's
// index, the words of the four child rows each child pair's source and index, so
// every load of a node's eight children follows from words alone (a row's nodes
// are neighbours, and so are their children): no y coordinates; two words a step
// keep sixteen children a lane in flight.
// Bound by latency: the words come to shared memory 32 at a time, so a step
// waits for its children only.  512 x 2048 x 2048 APR, all levels: 1.8 ms (words
// read in each step 3.9, one step ahead in registers 3.2, child rows staged in
// shared memory cell by cell 3.8).  65535 cells in one row: 75 us in parts, 349
// row by row; 9 x 200 x 4100: 75 against 127 us.
// SUB: the children may be tree nodes too (not on the finest tree level, whose
// instance keeps half the row pointers).
template <bool SUB>
struct TreeWords {
    uint2 node[32], w[4][64], ws[SUB ? 4 : 1][SUB ? 64 : 1];
};
template <bool SUB, typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 4 : 2) tree_mean_kernel(TreeLevelArgs a,
                                                                                const uint64_t *__restrict__ xz_end,
                                                                                const T *__restrict__ parts,
                                                                                const uint64_t *__restrict__ t_xz_end,
                                                                                T *tree, int per) {
    __shared__ TreeWords<SUB> words[8];
    TreeWords<SUB> &sm = words[threadIdx.x >> 5];
    const uint64_t prow = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;  // z * xt + x
    const int lane = threadIdx.x & 31;
    if (prow >= (uint64_t)a.dt.xn * a.dt.zn) return;
    const uint64_t pb = t_xz_end[a.t_row_base + prow - 1], pe = t_xz_end[a.t_row_base + prow];
    if (pb == pe) return;
    const int xp = (int)(prow % (uint64_t)a.dt.xn), zp = (int)(prow / (uint64_t)a.dt.xn);
    const int first = (int)blockIdx.y * per;  // of the warp's words; counted from there below
    const int end = min(per, nword(a.dt.yn) - first), nw = nword(a.dc.yn) - 2 * first;
    const uint2 *WN = a.tw + prow * nword(a.dt.yn) + first;
    const uint2 *W[4], *WT[4];
    const T *own[4], *sub[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int cz = 2 * zp + (q >> 1), cx = 2 * xp + (q & 1);
        W[q] = WT[q] = nullptr;
        own[q] = sub[q] = nullptr;
        if (cz < a.dc.zn && cx < a.dc.xn) {
            const uint64_t row = (uint64_t)cz * a.dc.xn + cx;
            W[q] = a.cw + row * nword(a.dc.yn) + 2 * first;
            own[q] = parts + xz_end[a.c_row_base + row - 1];
            if (SUB) {
                WT[q] = a.ctw + row * nword(a.dc.yn) + 2 * first;
                sub[q] = tree + t_xz_end[a.ct_row_base + row - 1];
            }
        }
    }
    float sxz = (float)((((2 * a.dt.xn != a.dc.xn) && (xp == a.dt.xn - 1)) +
                         ((2 * a.dt.zn != a.dc.zn) && (zp == a.dt.zn - 1))) * 2);
    if (sxz == 0) sxz = 1;
    const float syxz = (2 * a.dt.yn != a.dc.yn) ? sxz * 2 : sxz;
    // x / 8 == x * 0.125 exactly: both are the correctly rounded x / 8
    const T eighth = T(0.125);
    const unsigned bit = 1u << lane, b = 2 * (lane & 15), low = (1u << b) - 1u;
    constexpr int U = SUB ? 1 : 2;
    for (int c0 = 0; c0 < end; c0 += 32) {
        // the words of 32 parent words, and of the two child words under each
        __syncwarp();
        sm.node[lane] = c0 + lane < end ? WN[c0 + lane] : make_uint2(0u, 0u);
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int k = lane; k < 64; k += 32) {
                const int j = 2 * c0 + k;
                const bool in = W[q] && j < nw;
                sm.w[q][k] = in ? W[q][j] : make_uint2(0u, 0u);
                if (SUB) sm.ws[SUB ? q : 0][SUB ? k : 0] = in ? WT[q][j] : make_uint2(0u, 0u);
            }
        __syncwarp();
        for (int j0 = 0; j0 < 32 && c0 + j0 < end; j0 += U) {
            uint2 node[U];
            T v[U][8], vs[U][8];
            unsigned has[U], hast[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                node[u] = sm.node[j0 + u];
                has[u] = hast[u] = 0;
                if (!(node[u].x & bit)) continue;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const uint2 w = sm.w[q][2 * (j0 + u) + (lane >> 4)];
                    const unsigned two = (w.x >> b) & 3u;
                    const T *p = own[q] + (w.y + __popc(w.x & low));
                    if (two & 1u) v[u][2 * q] = __ldg(p);
                    if (two & 2u) v[u][2 * q + 1] = __ldg(p + (two & 1u));
                    has[u] |= two << (2 * q);
                    if (SUB) {
                        const uint2 ws = sm.ws[q][2 * (j0 + u) + (lane >> 4)];
                        const unsigned twos = (ws.x >> b) & 3u;
                        const T *ps = sub[q] + (ws.y + __popc(ws.x & low));
                        if (twos & 1u) vs[u][2 * q] = ps[0];
                        if (twos & 2u) vs[u][2 * q + 1] = ps[twos & 1u];
                        hast[u] |= twos << (2 * q);
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (!(node[u].x & bit)) continue;
                const T s = T((32 * (first + c0 + j0 + u) + lane == a.dt.yn - 1) ? syxz : sxz);
                T acc = T(0);
                // particles first, then tree nodes, each in z, x, y order
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    if ((has[u] >> c) & 1u) acc = VT<T>::add(VT<T>::mul(VT<T>::mul(s, v[u][c]), eighth), acc);
                if (SUB) {
#pragma unroll
                    for (int c = 0; c < 8; ++c)
                        if ((hast[u] >> c) & 1u) acc = VT<T>::add(VT<T>::mul(VT<T>::mul(s, vs[u][c]), eighth), acc);
                }
                tree[pb + node[u].y + __popc(node[u].x & (bit - 1u))] = acc;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// convolution of one level
// ---------------------------------------------------------------------------
struct ConvLevelArgs {
    LD d;                 // level dims
    LD dp;                // parent level dims
    uint64_t row_base;    // APR level_xz[l]
    uint64_t prow_base;   // APR level_xz[l-1] (0: no parents used)
    uint64_t trow_base;   // tree level_xz[l] (0: no tree level)
    int reflect;
    const uint2 *w, *pw, *tw;  // row words of the level, the parents (null: unused) and the tree (null: no level)
};

// ---------------------------------------------------------------------------
// convolution of one level: its neighbourhood image, then 2 x 2 x 2 blocks
// ---------------------------------------------------------------------------
// Level image of a run of planes [z0, z1): planes z0 - R .. z1 + R, rows
// -R .. xn + R and cells -R .. yn + R with the boundary folded in -- a cell
// outside the level holds the value of its reflection, or 0 with the zero pad
// and where the reflection leaves the level too (an axis of one cell, or of two at
// R = 2; such taps are stale reads, and outside_taps counts them) -- so the sums
// need no boundary case.  Cell y of a row sits at index y + PADY; pitch and PADY
// keep the pair (2j - R, 2j - R + 1) aligned.  One plane, row and cell more
// than the taps of the last cell need: an odd extent's last block reads them.
template <int R, typename T>
struct ImageShape {
    static constexpr int PADY = R == 1 ? 3 : 4;
    int xn, yn, z0, z1;
    int xp;            // rows of a plane
    int pitch;         // elements of a row
    uint64_t plane;    // elements of a plane
    int halo;          // planes before z0; 0: the image of a single plane alone
    __host__ ImageShape(const LD &d, int z0_, int z1_, bool flat = false)
        : xn(d.xn), yn(d.yn), z0(z0_), z1(z1_), halo(flat ? 0 : R) {
        xp = xn + 2 * R + 1;
        pitch = (PADY + yn + R + 1 + 3) & ~3;
        plane = (uint64_t)xp * pitch;
    }
    __host__ __device__ int planes() const { return halo ? z1 - z0 + 2 * R + 1 : z1 - z0; }
    __host__ uint64_t elems() const { return (uint64_t)planes() * plane; }
};

constexpr int kTX = 16, kTZ = 8;   // rows of a block-sum tile, planes at most
constexpr int kTY = 128;           // cells of its rows

// source index of index i of an axis of length n: i itself, its reflection
// about the edge sample, or -1 (zero pad, or a reflection that leaves the axis)
__host__ __device__ __forceinline__ int src_index(int i, int n, int reflect) {
    if (i >= 0 && i < n) return i;
    if (!reflect) return -1;
    const int r = i < 0 ? -i : 2 * (n - 1) - i;
    return (r >= 0 && r < n) ? r : -1;
}

template <typename T>
struct Pair2;
template <>
struct Pair2<float> {
    using type = float2;
};
template <>
struct Pair2<double> {
    using type = double2;
};

// What an uncovered cell copies: the sentinel.
__device__ const uint32_t g_cell_f32 = kMissingBits;
__device__ const uint64_t g_cell_f64 = kMissingBits64;
template <typename T>
__device__ __forceinline__ const T *no_cell() {
    if constexpr (sizeof(T) == 4)
        return reinterpret_cast<const T *>(&g_cell_f32);
    else
        return reinterpret_cast<const T *>(&g_cell_f64);
}

// The level image: one warp per row (PARTS: per part of `per` cells, where rows
// are long and few), a lane per pair of cells (2j, 2j + 1), which share their
// parent.  The row words say which source holds a cell (particle, parent, tree
// mean) and at which index, so every cell is one load and one store, with no
// prefill and no y coordinates read.  Rows that no particle of the level is within
// R of are not written (nothing reads them).
// Bound by latency and issue slots: 3.7 ms for all levels of the 512 x 2048 x
// 2048 APR.  The words of 2048 cells come to shared memory at once, so a step
// waits for its values only (words read in each step: 4.6 ms; one step ahead in
// registers: 5.2; a word of 32 cells a step instead of 64 in pairs: 5.6).
template <int R, typename T, bool PARTS>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 5 : 4) level_image_kernel(ConvLevelArgs a, ImageShape<R, T> m,
                                                          const uint64_t *__restrict__ xz_end,
                                                          const T *__restrict__ in,
                                                          const uint64_t *__restrict__ t_xz_end,
                                                          const T *__restrict__ tree, T *__restrict__ D, int per) {
    __shared__ uint2 sm[8][160];
    const int lane = threadIdx.x & 31;
    const unsigned nb = (unsigned)(m.xp + 7) / 8, ip = blockIdx.x / nb;  // plane of the image
    const int pr = (int)(blockIdx.x - ip * nb) * 8 + (threadIdx.x >> 5);  // row of the plane
    if (pr >= m.xp) return;
    const int xn = a.d.xn, yn = a.d.yn, zn = a.d.zn;
    const int z = m.z0 - m.halo + (int)ip, x = pr - R;
    {
        constexpr int S = 2 * R + 1;
        const int k = lane;
        const int zz = z + k / S - R, xx = x + k % S - R;
        bool any = false;
        if (k < S * S && zz >= 0 && zz < zn && xx >= 0 && xx < xn) {
            const uint64_t r = a.row_base + (uint64_t)zz * xn + xx;
            any = xz_end[r] > xz_end[r - 1];
        }
        if (!__any_sync(0xffffffffu, any)) return;
    }
    T *row = D + (uint64_t)ip * m.plane + (uint64_t)pr * m.pitch + m.PADY;
    const int zs = src_index(z, zn, a.reflect), xs = src_index(x, xn, a.reflect);
    const bool row_in = zs >= 0 && xs >= 0;
    const int first = PARTS ? (int)blockIdx.y * per : 0, end = PARTS ? min(first + per, yn) : yn;  // the warp's cells
    if (!row_in) {
        for (int y = first + lane - R; y < end + R; y += 32) row[y] = T(0);
        return;
    }
    const int nw = nword(yn), nwp = nword(a.dp.yn);
    const uint64_t srow = (uint64_t)zs * xn + xs, prow = (uint64_t)(zs >> 1) * a.dp.xn + (xs >> 1);
    const uint2 *W = a.w + srow * nw;
    const uint2 *WT = a.tw ? a.tw + srow * nw : nullptr;
    const uint2 *WP = a.pw ? a.pw + prow * nwp : nullptr;
    const T *own = in + xz_end[a.row_base + srow - 1];
    const T *tr = a.tw ? tree + t_xz_end[a.trow_base + srow - 1] : nullptr;
    const T *par = a.pw ? in + xz_end[a.prow_base + prow - 1] : nullptr;
    const T *nowhere = no_cell<T>();
    const unsigned b2 = 2 * (lane & 15), low2 = (1u << b2) - 1u, bit = 1u << lane, low = bit - 1u;
    constexpr int U = 4;  // steps of 64 cells with their loads in flight
    const uint2 zero = make_uint2(0u, 0u);
    uint2 *sw = sm[threadIdx.x >> 5], *swp = sw + 64, *swt = sw + 96;  // a row's words: own, parents, tree
    for (int c0 = first; c0 < end; c0 += 2048) {
        __syncwarp();
#pragma unroll
        for (int k = lane; k < 64; k += 32) {
            const int j = c0 / 32 + k;
            sw[k] = j < nw ? W[j] : zero;
            if (WT) swt[k] = j < nw ? WT[j] : zero;
        }
        swp[lane] = WP && c0 / 64 + lane < nwp ? WP[c0 / 64 + lane] : zero;
        __syncwarp();
        for (int y0 = c0; y0 < min(c0 + 2048, end); y0 += 64 * U) {
            uint2 w[U], wp[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                w[u] = sw[(y0 - c0) / 32 + 2 * u + (lane >> 4)];
                wp[u] = swp[(y0 - c0) / 64 + u];
            }
            T v[U][2];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const T *p0 = nowhere, *p1 = nowhere;
                if (wp[u].x & bit) p0 = p1 = par + (wp[u].y + __popc(wp[u].x & low));
                if (WT) {
                    const uint2 wt = swt[(y0 - c0) / 32 + 2 * u + (lane >> 4)];
                    const unsigned two = wt.x >> b2;
                    const T *p = tr + (wt.y + __popc(wt.x & low2));
                    if (two & 1u) p0 = p;
                    if (two & 2u) p1 = p + (two & 1u);
                }
                const unsigned two = w[u].x >> b2;
                const T *p = own + (w[u].y + __popc(w[u].x & low2));
                if (two & 1u) p0 = p;
                if (two & 2u) p1 = p + (two & 1u);
                v[u][0] = __ldg(p0);
                v[u][1] = __ldg(p1);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int y = y0 + 64 * u + 2 * lane;
                if (m.PADY % 2 == 0 && y + 1 < yn) {
                    typename Pair2<T>::type t;
                    t.x = v[u][0];
                    t.y = v[u][1];
                    *reinterpret_cast<typename Pair2<T>::type *>(row + y) = t;
                } else {
                    if (y < yn) row[y] = v[u][0];
                    if (y + 1 < yn) row[y + 1] = v[u][1];
                }
            }
        }
    }
    if (first == 0 && lane < 2 * R) {
        // the R cells before and after the row
        const int y = lane < R ? -1 - lane : yn + lane - R;
        const int ys = src_index(y, yn, a.reflect);
        T v = T(0);
        if (ys >= 0) {
            const int j = ys >> 5;
            const unsigned b = 1u << (ys & 31);
            const uint2 w = W[j];
            const uint2 wt = WT ? WT[j] : make_uint2(0u, 0u);
            const uint2 wp = WP ? WP[ys >> 6] : make_uint2(0u, 0u);
            const unsigned pb = 1u << ((ys >> 1) & 31);
            v = VT<T>::miss();
            if (w.x & b)
                v = own[w.y + __popc(w.x & (b - 1u))];
            else if (wt.x & b)
                v = tr[wt.y + __popc(wt.x & (b - 1u))];
            else if (wp.x & pb)
                v = par[wp.y + __popc(wp.x & (pb - 1u))];
        }
        row[y] = v;
    }
}

template <int R, typename T>
struct StencilArg {
    T w[(2 * R + 1) * (2 * R + 1) * (2 * R + 1)];
};

// Weights in shared memory: a tap row of 2R + 1, padded to kWRow for vector loads.
template <int R>
constexpr int kWRow = R == 1 ? 4 : 8;
template <int R, typename T>
__device__ __forceinline__ void load_weights(const T *__restrict__ p, T (&w)[kWRow<R>]) {
    if constexpr (sizeof(T) == 4) {
        const float4 a = *reinterpret_cast<const float4 *>(p);
        w[0] = a.x, w[1] = a.y, w[2] = a.z, w[3] = a.w;
        if constexpr (R == 2) w[4] = p[4];
    } else {
        const double2 a = *reinterpret_cast<const double2 *>(p);
        w[0] = a.x, w[1] = a.y;
        if constexpr (R == 1) {
            w[2] = p[2];
        } else {
            const double2 b = *reinterpret_cast<const double2 *>(p + 2);
            w[2] = b.x, w[3] = b.y, w[4] = p[4];
        }
    }
}

template <typename T, int N>
__device__ __forceinline__ void load_row(const T *__restrict__ P, T (&d)[N]) {
    using T2 = typename Pair2<T>::type;
#pragma unroll
    for (int k = 0; k < N; k += 2) {
        const T2 t = __ldg(reinterpret_cast<const T2 *>(P + k));
        d[k] = t.x;
        d[k + 1] = t.y;
    }
}

// Where the weights come from, and whether a plane's first row is loaded during
// the plane before.  3^3 float: constant operands from the kernel's parameters,
// no.  Wider: the 50 weights a plane step needs do not stay constant operands
// (the plane loop is rolled) and spilled as registers, so a tap row's weights
// are read from shared memory where they are used (5^3, 250 x 1000 x 1013: 2.85
// -> 2.49 ms; 3^3 float that way: 11.5 against 11.3 ms on 512 x 2048 x 2048).
template <int R, typename T>
constexpr bool kSharedWeights = R == 2 || sizeof(T) == 8;

// Plane p of a block's neighbourhood (P: its first cell): the taps that the
// block's cells of its lower plane (DZ0: tap plane p) and of its upper plane
// (DZ1: tap plane p - 1) have there.  One row ahead is in flight, and no
// further: more rows only cost registers.  With kSharedWeights, v[0] holds row 0
// on entry and, where there is a next plane, its row 0 on return.
template <int R, typename T, bool DZ0, bool DZ1>
__device__ __forceinline__ void plane_taps(const T *__restrict__ P, const T *__restrict__ next, int pitch, int p,
                                           const StencilArg<R, T> &sw, const T *__restrict__ ws,
                                           T (&v)[2][2 * R + 2], T (&acc)[2][2][2]) {
    constexpr int S = 2 * R + 1, N = 2 * R + 2, WR = kWRow<R>;
    constexpr bool SW = kSharedWeights<R, T>;
    if (!SW) load_row<T, N>(P, v[0]);
#pragma unroll
    for (int q = 0; q < N; ++q) {
        P += pitch;
        if (q + 1 < N)
            load_row<T, N>(P, v[(q + 1) & 1]);
        else if (SW && DZ0)
            load_row<T, N>(next, v[0]);
        asm volatile("" ::: "memory");
        if constexpr (SW) {
#pragma unroll
            for (int dz = 0; dz < 2; ++dz) {
                if (dz ? !DZ1 : !DZ0) continue;
#pragma unroll
                for (int dx = 0; dx < 2; ++dx) {
                    const int ix = q - dx;
                    if (ix < 0 || ix >= S) continue;
                    T w[WR];
                    load_weights<R, T>(ws + ((p - dz) * S + ix) * WR, w);
#pragma unroll
                    for (int iy = 0; iy < S; ++iy)
#pragma unroll
                        for (int dy = 0; dy < 2; ++dy)
                            acc[dz][dx][dy] = VT<T>::add(acc[dz][dx][dy], VT<T>::mul(v[q & 1][iy + dy], w[iy]));
                }
            }
        } else {
#pragma unroll
            for (int iy = 0; iy < S; ++iy)
#pragma unroll
                for (int dz = 0; dz < 2; ++dz) {
                    if (dz ? !DZ1 : !DZ0) continue;
#pragma unroll
                    for (int dx = 0; dx < 2; ++dx) {
                        const int ix = q - dx;
                        if (ix < 0 || ix >= S) continue;
                        const T w = sw.w[((p - dz) * S + ix) * S + iy];
#pragma unroll
                        for (int dy = 0; dy < 2; ++dy)
                            acc[dz][dx][dy] = VT<T>::add(acc[dz][dx][dy], VT<T>::mul(v[q & 1][iy + dy], w));
                    }
                }
        }
    }
}

// The occupied 2 x 2 x 2 blocks of a tile of kTZ planes x kTX rows x kTY cells
// (any particle of the level in it), packed into one list so that lanes are
// full whatever the rows' shapes; the tile's row words and row starts stay in
// shared memory for the epilogue.
struct BlockTile {
    uint2 cen[kTZ][kTX][kTY / 32];
    uint64_t beg[kTZ][kTX];
    uint16_t list[kTZ / 2 * kTX / 2 * kTY / 2];  // layer << 9 | row pair << 6 | cell pair
    unsigned n;
};
template <int NT>
__device__ __forceinline__ int pack_blocks(BlockTile &t, const ConvLevelArgs &a, const uint64_t *__restrict__ xz_end,
                                           int z0, int x0, int y0, int ze, int tz) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nw = nword(a.d.yn);
    if (tid == 0) t.n = 0;
    for (int k = tid; k < tz * kTX * (kTY / 32); k += NT) {
        const int j = k % (kTY / 32), r = k / (kTY / 32) % kTX, p = k / (kTY / 32) / kTX;
        uint2 w = make_uint2(0u, 0u);
        if (z0 + p < ze && x0 + r < a.d.xn && y0 / 32 + j < nw)
            w = a.w[((uint64_t)(z0 + p) * a.d.xn + x0 + r) * nw + y0 / 32 + j];
        t.cen[p][r][j] = w;
    }
    for (int k = tid; k < tz * kTX; k += NT) {
        const int r = k % kTX, p = k / kTX;
        uint64_t b = 0;
        if (z0 + p < ze && x0 + r < a.d.xn) b = xz_end[a.row_base + (uint64_t)(z0 + p) * a.d.xn + x0 + r - 1];
        t.beg[p][r] = b;
    }
    __syncthreads();
    for (int k = warp; k < tz / 2 * (kTX / 2); k += NT / 32) {
        const int p = k / (kTX / 2), rp = k % (kTX / 2);
#pragma unroll
        for (int h = 0; h < kTY / 64; ++h) {
            const int j = 2 * h + (lane >> 4);
            const unsigned u = t.cen[2 * p][2 * rp][j].x | t.cen[2 * p][2 * rp + 1][j].x |
                               t.cen[2 * p + 1][2 * rp][j].x | t.cen[2 * p + 1][2 * rp + 1][j].x;
            const bool on = ((u >> (2 * (lane & 15))) & 3u) != 0u;
            const unsigned mk = __ballot_sync(0xffffffffu, on);
            unsigned at = 0;
            if (lane == 0 && mk) at = atomicAdd(&t.n, (unsigned)__popc(mk));
            at = __shfl_sync(0xffffffffu, at, 0);
            if (on) t.list[at + __popc(mk & ((1u << lane) - 1u))] = (uint16_t)(p << 9 | rp << 6 | (32 * h + lane));
        }
    }
    __syncthreads();
    return (int)t.n;
}

// One tap in the sentinel's presence: 0, counted as a stale read.
template <typename T>
__device__ __forceinline__ T covered(T v, unsigned &nstale) {
    if (!VT<T>::is_miss(v)) return v;
    nstale++;
    return T(0);
}

// Sums of a level from its image: a lane takes one 2 x 2 x 2 block of cells,
// reads the (2R + 2)^3 cells around it once (through L1, where the tile's rows
// meet) and sums the taps of all eight cells, each in the stencil's memory
// order, a separate multiply and add per tap, the weights constant operands
// from the kernel's parameters.  A NaN sum (a sentinel was read, or a NaN
// value) is redone tap by tap.  The loop over the inner planes stays rolled:
// unrolled whole, the weights are hoisted out of the block loop and spill.  (A
// paired f32x2 multiply followed by a paired add is contracted into a fused
// multiply-add by the code generator, so scalar operations it is.)
//
// What bounds it: issue slots, most of them the multiplies and adds (54 / 250
// per particle).  Blocks of 2 x 2 x 2 because level l_max comes in whole
// sibling groups: per particle 8 (3^3) or 27 (5^3) values are read instead of
// 27 or 125, and the eight chains are independent.
// 3^3 on the 512 x 2048 x 2048 APR (1.1e9 particles): 5.4 ms of 11.0 ms a
// convolution, 70 % of the issue slots, 64 % of L1's data pipe (the z-streaming
// shared-memory kernel this replaces: 13.5 of 19.4 ms); 5^3 on 250 x 1000 x
// 1013 (1.3e8): 1.5 of 2.4 ms (5.1 of 5.65).  Four CTAs per SM: 5.8 ms against
// 6.5 with three and 8.4 with two.  The epilogue is compiled per mode and stores
// a pair of particles without tests of its own: 11.2 -> 11.0 ms, 10 iterations
// of Richardson-Lucy on 128 x 512 x 512 9.18 -> 8.56 ms.
//
// threads of a conv_block CTA: 128 in double (96 x 250 x 260 Richardson-Lucy 2.47
// -> 2.33 ms), 256 in float (5^3 on 250 x 1000 x 1013: 2.86 ms against 2.97)
template <typename T>
constexpr int kConvThreads = sizeof(T) == 8 ? 128 : 256;
// MODE: 0 out = sum, 1 out = rl_in / sum, 2 out *= sum
// FLAT: a level of one plane.  The planes beside it are all 0, so their taps
// (finite weights: each adds +-0 to a sum that began at +0) and their part of the
// image are left out (2048 x 2048: 3^3 201 -> 175, 5^3 262 -> 213 us a call).
template <int R, typename T, int MODE, bool FLAT>
__global__ void __launch_bounds__(kConvThreads<T>, 4) conv_block_kernel(
    ConvLevelArgs a, const __grid_constant__ StencilArg<R, T> sw, ImageShape<R, T> m,
    const uint64_t *__restrict__ xz_end, const T *__restrict__ D, T *__restrict__ out,
    const uint16_t *__restrict__ rl_in, unsigned long long *stale, int tz) {
    constexpr int S = 2 * R + 1, N = 2 * R + 2;
    __shared__ BlockTile t;
    __shared__ __align__(16) T ws[kSharedWeights<R, T> ? S * S * kWRow<R> : 1];
    const int x0 = blockIdx.x * kTX, y0 = blockIdx.y * kTY, z0 = m.z0 + blockIdx.z * tz;
    for (int k = threadIdx.x; k < (kSharedWeights<R, T> ? S * S * kWRow<R> : 0); k += kConvThreads<T>) {
        const int iy = k % kWRow<R>;
        ws[k] = iy < S ? sw.w[k / kWRow<R> * S + iy] : T(0);
    }
    const int n = pack_blocks<kConvThreads<T>>(t, a, xz_end, z0, x0, y0, m.z1, tz);
    unsigned nstale = 0;
    for (int k = threadIdx.x; k < n; k += kConvThreads<T>) {
        const int e = t.list[k], lay = e >> 9, rp = (e >> 6) & 7, cp = e & 63;
        const T *base = D + (uint64_t)(z0 - m.z0 + 2 * lay) * m.plane + (uint64_t)(x0 + 2 * rp) * m.pitch +
                        (y0 + 2 * cp - R + m.PADY);
        T acc[2][2][2];
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[c >> 2][(c >> 1) & 1][c & 1] = T(0);
        T rows[2][N];
        if (kSharedWeights<R, T>) load_row<T, N>(base, rows[0]);
        if constexpr (FLAT) {
            plane_taps<R, T, true, false>(base, base, m.pitch, R, sw, ws, rows, acc);
        } else {
            const T *P = base + m.plane;
            plane_taps<R, T, true, false>(base, P, m.pitch, 0, sw, ws, rows, acc);
#pragma unroll 1
            for (int p = 1; p < N - 1; ++p, P += m.plane)
                plane_taps<R, T, true, true>(P, P + m.plane, m.pitch, p, sw, ws, rows, acc);
            plane_taps<R, T, false, true>(P, nullptr, m.pitch, N - 1, sw, ws, rows, acc);
        }
#pragma unroll
        for (int c = 0; c < (FLAT ? 2 : 4); ++c) {
            const int dz = c >> 1, dx = c & 1;
            const uint2 w = t.cen[2 * lay + dz][2 * rp + dx][cp >> 4];
            const unsigned b = 2 * (cp & 15), two = (w.x >> b) & 3u;
            const uint64_t o = t.beg[2 * lay + dz][2 * rp + dx] + w.y + __popc(w.x & ((1u << b) - 1u));
            T v[2] = {acc[dz][dx][0], acc[dz][dx][1]};
#pragma unroll
            for (int dy = 0; dy < 2; ++dy) {
                if (v[dy] == v[dy] || !((two >> dy) & 1u)) continue;
                T r = T(0);
                int cnt = FLAT ? R * S * S : 0;
                for (int iz = 0; iz < (FLAT ? 1 : S); ++iz)
                    for (int ix = 0; ix < S; ++ix) {
                        const T *q = base + (uint64_t)(iz + dz) * m.plane + (uint64_t)(ix + dx) * m.pitch + dy;
                        for (int iy = 0; iy < S; ++iy)
                            r = VT<T>::add(r, VT<T>::mul(covered(q[iy], nstale), sw.w[cnt++]));
                    }
                v[dy] = r;
            }
            auto put = [&](uint64_t i, T r) {
                if (MODE == 0)
                    out[i] = r;
                else if (MODE == 1)
                    out[i] = VT<T>::div((T)rl_in[i], r);
                else
                    out[i] = VT<T>::mul(out[i], r);
            };
            if (two == 3u) {  // on level l_max always, or the row has no block here
                put(o, v[0]);
                put(o + 1, v[1]);
            } else if (two) {
                put(o, two & 1u ? v[0] : v[1]);
            }
        }
    }
    if (nstale) atomicAdd(stale, (unsigned long long)nstale);
}

// Planes of a run: its image, halo planes included, takes at most 1 GiB, so
// that the scratch of a large level stays a fraction of its particles'; whole
// tiles, one at least, so levels of more than 2^30 / (kTZ + 2R + 1) bytes a plane
// (4900^2 floats at 3^3) take kTZ + 2R + 1 planes.  whole: all planes.
template <int R, typename T>
int image_run(const LD &d, bool whole) {
    const int64_t halo = 2 * R + 1;
    const int64_t fit = (int64_t)((uint64_t(1) << 30) / (ImageShape<R, T>(d, 0, 1).plane * sizeof(T))) - halo;
    if (whole || fit >= d.zn) return d.zn;
    return (int)std::min<int64_t>(d.zn, std::max<int64_t>(kTZ, fit / kTZ * kTZ));
}

// Taps of a particle's (2R + 1)^3 whose reflection leaves the level: as many for
// every particle of it, so those of its first cell are counted.  used[k]: tap k
// counts (null: all do).
uint64_t outside_taps(const LD &d, int R, const bool *used = nullptr) {
    const int S = 2 * R + 1;
    uint64_t out = 0;
    for (int k = 0; k < S * S * S; ++k)
        out += (!used || used[k]) && (src_index(k / (S * S) - R, d.zn, 1) < 0 ||
                                      src_index(k / S % S - R, d.xn, 1) < 0 || src_index(k % S - R, d.yn, 1) < 0);
    return out;
}

// What a warp takes of `rows` rows of n units: the whole row, or halves of it
// (whole steps, down to one) while there are fewer than `warps` warps, the SMs'
// fill.  A row is a serial walk, so on few long rows its length is the kernel's
// time.
int row_part(uint64_t rows, int n, int step, uint64_t warps) {
    int per = (n + step - 1) / step;
    while (per > 1 && rows * (uint64_t)((n + per * step - 1) / (per * step)) < warps) per = (per + 1) / 2;
    return per * step;
}

template <int R, typename T>
T *launch_level_image(const ConvLevelArgs &a, const ImageShape<R, T> &m, const uint64_t *xz_end, const T *in,
                      const uint64_t *t_xz_end, const T *tree, FilterBuffers &fb, cudaStream_t s) {
    APRB_PROF("level_image", s);
    T *D = (T *)fb.dense.get(m.elems() * sizeof(T));
    // whole steps of 256 cells, as many warps as the SMs hold: 3^3 on one row of
    // 65535 cells 474 -> 250 us
    const int per = row_part((uint64_t)m.xp * m.planes(), m.yn, 256, 148 * 40);
    const dim3 grid((unsigned)((m.xp + 7) / 8) * (unsigned)m.planes(), (unsigned)((m.yn + per - 1) / per));
    if (grid.y > 1)
        level_image_kernel<R, T, true><<<grid, 256, 0, s>>>(a, m, xz_end, in, t_xz_end, tree, D, per);
    else
        level_image_kernel<R, T, false><<<grid, 256, 0, s>>>(a, m, xz_end, in, t_xz_end, tree, D, per);
    count_launch();
    APRB_CHECK_LAUNCH();
    return D;
}

// Tiles of tz planes: kTZ, fewer (down to one layer of blocks) while that
// leaves the SMs under four waves of their four CTAs.  More planes fill the
// list's last round better (512 x 2048 x 2048, 3^3 sums: 5.8 ms against 6.6 with
// 4); on 64 x 128 x 128 cells they only leave SMs idle (35 us against 50 with 8).
template <int R, typename T>
dim3 block_grid(const ConvLevelArgs &a, const ImageShape<R, T> &m, int &tz) {
    const unsigned gx = (unsigned)((a.d.xn + kTX - 1) / kTX), gy = (unsigned)((a.d.yn + kTY - 1) / kTY);
    tz = kTZ;
    while (tz > 2 && (uint64_t)gx * gy * ((m.z1 - m.z0 + tz - 1) / tz) < 4ull * 4 * 148) tz /= 2;
    return dim3(gx, gy, (unsigned)((m.z1 - m.z0 + tz - 1) / tz));
}

template <int R, typename T>
void launch_conv_level(const ConvLevelArgs &a, const ConvPlan &plan, int sn, int mode, const uint64_t *xz_end, const T *in,
                       const uint64_t *t_xz_end, const T *tree, T *out, const uint16_t *rl_in,
                       unsigned long long *stale, FilterBuffers &fb, cudaStream_t s) {
    StencilArg<R, T> sw;
    for (int t = 0; t < (int)(sizeof(sw.w) / sizeof(T)); ++t) sw.w[t] = (T)plan.values[plan.offsets[sn] + t];
    bool flat = a.d.zn == 1;
    for (const T w : sw.w) flat = flat && std::isfinite(w);
    // in place, the whole level is read before any of it is written
    const int run = image_run<R, T>(a.d, (const void *)in == (const void *)out);
    for (int z0 = 0; z0 < a.d.zn; z0 += run) {
        const ImageShape<R, T> m(a.d, z0, std::min(z0 + run, a.d.zn), flat);
        const T *D = launch_level_image<R, T>(a, m, xz_end, in, t_xz_end, tree, fb, s);
        APRB_PROF("conv_block", s);
        int tz;
        const dim3 grid = block_grid(a, m, tz);
        auto run = [&](auto kern) {
            kern<<<grid, kConvThreads<T>, 0, s>>>(a, sw, m, xz_end, D, out, rl_in, stale, tz);
        };
        if (mode == 0)
            flat ? run(conv_block_kernel<R, T, 0, true>) : run(conv_block_kernel<R, T, 0, false>);
        else if (mode == 1)
            flat ? run(conv_block_kernel<R, T, 1, true>) : run(conv_block_kernel<R, T, 1, false>);
        else
            flat ? run(conv_block_kernel<R, T, 2, true>) : run(conv_block_kernel<R, T, 2, false>);
        count_launch();
        APRB_CHECK_LAUNCH();
    }
}

// Gradient magnitude of one level (APRNumerics::gradient_magnitude_cfd /
// _sobel, APRNumerics.hpp:227-287) from the level image, a lane per 2 x 2 x 2
// block as in conv_block_kernel: the three directions' sums share the block's
// cells, then y^2 (+ x^2) (+ z^2) and the square root, as the per-direction
// path (one convolution per direction, squares and a root) computes them.
// FULL: direction d's taps are the 18 cells off its centre plane (Sobel), else
// its two cells along d (central differences).  A tap of the pattern whose
// weight is zero (2-D Sobel) adds +-0 to a finite sum, which changes the sum
// only when it is itself zero, and then only its sign, which the square
// removes; cells of the block that no tap has are not read.
// Central differences on the 256 x 1024 x 1024 APR (1.4e8 particles): 0.52 ms
// of 1.38 ms a call, against 1.27 of 2.33 ms for a gather per particle.
struct GradArg {
    float w[3][27];  // weights of the directions in memory order
    int active[3];   // direction enters the magnitude
    int zuse[3];     // some weight of tap plane iz is not zero
};

constexpr int kGradThreads = 128;  // 256 x 1024 x 1024: 1.38 ms against 1.41 with 256
template <bool FULL>
__global__ void __launch_bounds__(kGradThreads, 6) grad_block_kernel(ConvLevelArgs a, const __grid_constant__ GradArg gw,
                                                                  ImageShape<1, float> m,
                                                                  const uint64_t *__restrict__ xz_end,
                                                                  const float *__restrict__ D, float *__restrict__ out,
                                                                  unsigned long long *stale, int tz) {
    __shared__ BlockTile t;
    const int x0 = blockIdx.x * kTX, y0 = blockIdx.y * kTY, z0 = m.z0 + blockIdx.z * tz;
    const int n = pack_blocks<kGradThreads>(t, a, xz_end, z0, x0, y0, m.z1, tz);
    unsigned nstale = 0;
    for (int k = threadIdx.x; k < n; k += kGradThreads) {
        const int e = t.list[k], lay = e >> 9, rp = (e >> 6) & 7, cp = e & 63;
        const float *base = D + (uint64_t)(z0 - m.z0 + 2 * lay) * m.plane + (uint64_t)(x0 + 2 * rp) * m.pitch +
                            (y0 + 2 * cp - 1 + m.PADY);
        float g[8][3];
#pragma unroll
        for (int c = 0; c < 8; ++c) g[c][0] = g[c][1] = g[c][2] = 0.0f;
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const bool pin = p == 1 || p == 2, qin = q == 1 || q == 2;
                if (!FULL && !pin && !qin) continue;
                const float *P = base + (uint64_t)p * m.plane + (uint64_t)q * m.pitch;
                float v[4] = {0, 0, 0, 0};
                if (FULL || (pin && qin)) {
                    const float2 f0 = __ldg(reinterpret_cast<const float2 *>(P));
                    const float2 f1 = __ldg(reinterpret_cast<const float2 *>(P + 2));
                    v[0] = f0.x, v[1] = f0.y, v[2] = f1.x, v[3] = f1.y;
                } else {
                    v[1] = __ldg(P + 1);
                    v[2] = __ldg(P + 2);
                }
#pragma unroll
                for (int iy = 0; iy < 3; ++iy)
#pragma unroll
                    for (int dz = 0; dz < 2; ++dz)
#pragma unroll
                        for (int dx = 0; dx < 2; ++dx) {
                            const int iz = p - dz, ix = q - dx;
                            if (iz < 0 || iz > 2 || ix < 0 || ix > 2) continue;
                            if (FULL && !gw.zuse[iz]) continue;
#pragma unroll
                            for (int d = 0; d < 3; ++d) {
                                const int id[3] = {iy, ix, iz};
                                const bool off = id[d] != 1;
                                const bool axis = off && id[(d + 1) % 3] == 1 && id[(d + 2) % 3] == 1;
                                if (!(FULL ? off : axis) || (d > 0 && !gw.active[d])) continue;
                                const float w = gw.w[d][(iz * 3 + ix) * 3 + iy];
#pragma unroll
                                for (int dy = 0; dy < 2; ++dy) {
                                    float &acc = g[(dz * 2 + dx) * 2 + dy][d];
                                    acc = __fadd_rn(acc, __fmul_rn(v[iy + dy], w));
                                }
                            }
                        }
            }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int dz = c >> 1, dx = c & 1;
            const uint2 w = t.cen[2 * lay + dz][2 * rp + dx][cp >> 4];
            const unsigned b = 2 * (cp & 15), two = (w.x >> b) & 3u;
            uint64_t o = t.beg[2 * lay + dz][2 * rp + dx] + w.y + __popc(w.x & ((1u << b) - 1u));
#pragma unroll
            for (int dy = 0; dy < 2; ++dy) {
                if (!((two >> dy) & 1u)) continue;
                float gv[3] = {g[2 * c + dy][0], g[2 * c + dy][1], g[2 * c + dy][2]};
                if (gv[0] != gv[0] || gv[1] != gv[1] || gv[2] != gv[2]) {
                    // a sentinel was read (or a NaN value): tap by tap, sentinels as 0 and counted
                    for (int d = 0; d < 3; ++d) {
                        float acc = 0.0f;
                        for (int tap = 0; tap < 27; ++tap) {
                            const float wt = gw.w[d][tap];
                            if (wt == 0.0f || !gw.active[d]) continue;
                            const float *P = base + (uint64_t)(tap / 9 + dz) * m.plane +
                                             (uint64_t)(tap / 3 % 3 + dx) * m.pitch + tap % 3 + dy;
                            acc = __fadd_rn(acc, __fmul_rn(covered(*P, nstale), wt));
                        }
                        if (d == 0) gv[0] = acc;
                        if (d == 1) gv[1] = acc;
                        if (d == 2) gv[2] = acc;
                    }
                }
                float r = __fmul_rn(gv[0], gv[0]);
                if (gw.active[1]) r = __fadd_rn(r, __fmul_rn(gv[1], gv[1]));
                if (gw.active[2]) r = __fadd_rn(r, __fmul_rn(gv[2], gv[2]));
                out[o] = __fsqrt_rn(r);
                ++o;
            }
        }
    }
    if (nstale) atomicAdd(stale, (unsigned long long)nstale);
}

}  // namespace

void build_filter_index(const Geom &g, const uint64_t *xz_end, const uint16_t *y_vec, const Geom &tg,
                        const uint64_t *t_xz_end, const uint16_t *t_y_vec, FilterIndex &fi, cudaStream_t s) {
    APRB_PROF("filter_index", s);
    uint64_t wtotal = 0;
    for (int l = g.l_min; l <= g.l_max; ++l) {
        fi.apr_woff[l] = wtotal;
        wtotal += nrow(g, l) * (uint64_t)nword(g.y_num[l]);
    }
    for (int t = tg.l_min; t <= tg.l_max; ++t) {
        fi.tree_woff[t] = wtotal;
        wtotal += nrow(tg, t) * (uint64_t)nword(tg.y_num[t]);
    }
    uint2 *words = fi.words.as_pooled<uint2>(wtotal ? wtotal : 1, s);
    APRB_CUDA(cudaMemsetAsync(words, 0, wtotal * sizeof(uint2), s));
    for (int l = g.l_min; l <= g.l_max; ++l) {
        const uint64_t rows = nrow(g, l);
        if (!rows) continue;
        row_words_kernel<<<blocks_for(rows * 32, 256), 256, 0, s>>>(xz_end, g.level_xz[l], y_vec, rows,
                                                                   nword(g.y_num[l]), words + fi.apr_woff[l]);
        count_launch();
    }
    for (int t = tg.l_min; t <= tg.l_max; ++t) {
        const uint64_t rows = nrow(tg, t);
        if (!rows) continue;
        row_words_kernel<<<blocks_for(rows * 32, 256), 256, 0, s>>>(t_xz_end, tg.level_xz[t], t_y_vec, rows,
                                                                   nword(tg.y_num[t]), words + fi.tree_woff[t]);
        count_launch();
    }
    APRB_CHECK_LAUNCH();
    uint64_t ends[33] = {};  // where level l - 1 ends
    for (int l = g.l_min; l <= g.l_max + 1; ++l)
        APRB_CUDA(cudaMemcpyAsync(&ends[l], xz_end + g.level_xz[l] - 1, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
    APRB_CUDA(cudaStreamSynchronize(s));
    for (int l = 0; l < 32; ++l) fi.level_count[l] = l < g.l_min || l > g.l_max ? 0 : ends[l + 1] - ends[l];
    fi.built = true;
}

// Tree means of every tree level, fine to coarse.
template <typename T>
static void tree_means_all(const Geom &g, const uint64_t *xz_end, const Geom &tg, const uint64_t *t_xz_end,
                           const FilterIndex &fi, const T *in, T *tree, cudaStream_t s) {
    APRB_PROF("tree_mean", s);
    const int L = g.l_max;
    const uint2 *words = (const uint2 *)fi.words.p;
    for (int t = tg.l_max; t >= tg.l_min; --t) {
        const int l = t + 1;  // child level
        if (l > L || l < g.l_min) continue;
        TreeLevelArgs ta;
        ta.dt = ld(tg, t);
        ta.dc = ld(g, l);
        ta.t_row_base = tg.level_xz[t];
        ta.c_row_base = g.level_xz[l];
        ta.ct_row_base = (l <= tg.l_max) ? tg.level_xz[l] : 0;
        ta.tw = words + fi.tree_woff[t];
        ta.cw = words + fi.apr_woff[l];
        ta.ctw = (l <= tg.l_max) ? words + fi.tree_woff[l] : nullptr;
        const uint64_t rows = (uint64_t)ta.dt.xn * ta.dt.zn;
        if (rows == 0) continue;
        // eight warps an SM: with 32, the 4096 rows of 4 words of a 128 x 512 x 512 APR
        // are halved too, and a part's staging costs more than its walk (10 iterations
        // of Richardson-Lucy 8.71 against 8.55 ms)
        const int nwt = nword(ta.dt.yn), per = row_part(rows, nwt, 2, 148 * 8);
        const dim3 grid(blocks_for(rows * 32, 256), (unsigned)((nwt + per - 1) / per));
        if (ta.ctw)
            tree_mean_kernel<true, T><<<grid, 256, 0, s>>>(ta, xz_end, in, t_xz_end, tree, per);
        else
            tree_mean_kernel<false, T><<<grid, 256, 0, s>>>(ta, xz_end, in, t_xz_end, tree, per);
        count_launch();
    }
    APRB_CHECK_LAUNCH();
}

// Neighbourhood arguments of level l for a stencil of the given side
// (parents used up to ceil(log2(r + 2) - 1) levels coarser, APRFilter.hpp:1118-1124).
static ConvLevelArgs conv_level_args(const Geom &g, const Geom &tg, const FilterIndex &fi, int l, int side,
                                     int reflect) {
    const int r = (side - 1) / 2;
    const int max_npl = (int)std::ceil(std::log2((double)(r + 2)) - 1);
    const int npl = std::min(max_npl, l - g.l_min);
    ConvLevelArgs a;
    a.d = ld(g, l);
    a.dp = l > g.l_min ? ld(g, l - 1) : LD{1, 1, 1};
    a.row_base = g.level_xz[l];
    a.prow_base = npl >= 1 ? g.level_xz[l - 1] : 0;
    a.trow_base = l <= tg.l_max ? tg.level_xz[l] : 0;
    a.reflect = reflect;
    const uint2 *wbase = (const uint2 *)fi.words.p;
    a.w = wbase + fi.apr_woff[l];
    a.pw = npl >= 1 ? wbase + fi.apr_woff[l - 1] : nullptr;
    a.tw = l <= tg.l_max ? wbase + fi.tree_woff[l] : nullptr;
    return a;
}

template <typename T>
void filter_apply(const Geom &g, const uint64_t *xz_end, const Geom &tg, const uint64_t *t_xz_end,
                  const FilterIndex &fi, const T *in, T *tree,
                  const ConvPlan *plan, T *out, int mode, const uint16_t *rl_in,
                  FilterBuffers &fb, cudaStream_t s) {
    APRB_PROF(plan ? "convolve" : "fill_tree_mean", s);
    const int L = g.l_max;
    unsigned long long *stale = fb.stale.as<unsigned long long>(1);
    APRB_CUDA(cudaMemsetAsync(stale, 0, sizeof(unsigned long long), s));
    fb.outside = 0;
    tree_means_all<T>(g, xz_end, tg, t_xz_end, fi, in, tree, s);
    if (!plan) return;
    for (int l = L; l >= g.l_min; --l) {
        if (fi.level_count[l] == 0) continue;
        const int sn = std::min(plan->nstencils - 1, L - l);
        const int side = plan->sides[sn];
        const ConvLevelArgs a = conv_level_args(g, tg, fi, l, side, plan->reflect);
        if (plan->reflect) fb.outside += fi.level_count[l] * outside_taps(a.d, side / 2);
        if (side == 3)
            launch_conv_level<1, T>(a, *plan, sn, mode, xz_end, in, t_xz_end, tree, out, rl_in, stale, fb, s);
        else
            launch_conv_level<2, T>(a, *plan, sn, mode, xz_end, in, t_xz_end, tree, out, rl_in, stale, fb, s);
    }
}

template void filter_apply<float>(const Geom &, const uint64_t *, const Geom &, const uint64_t *, const FilterIndex &,
                                  const float *, float *, const ConvPlan *, float *, int, const uint16_t *,
                                  FilterBuffers &, cudaStream_t);
template void filter_apply<double>(const Geom &, const uint64_t *, const Geom &, const uint64_t *, const FilterIndex &,
                                  const double *, double *, const ConvPlan *, double *, int, const uint16_t *,
                                  FilterBuffers &, cudaStream_t);

void filter_gradient_magnitude(const Geom &g, const uint64_t *xz_end, const Geom &tg,
                               const uint64_t *t_xz_end, const FilterIndex &fi,
                               const float *in, float *tree, const float *const stencils[3], const int active[3],
                               int nstencils, float *out, FilterBuffers &fb, cudaStream_t s) {
    APRB_PROF("gradient_magnitude", s);
    const int L = g.l_max;
    unsigned long long *stale = fb.stale.as<unsigned long long>(1);
    APRB_CUDA(cudaMemsetAsync(stale, 0, sizeof(unsigned long long), s));
    fb.outside = 0;
    tree_means_all<float>(g, xz_end, tg, t_xz_end, fi, in, tree, s);
    for (int l = L; l >= g.l_min; --l) {
        if (fi.level_count[l] == 0) continue;
        const int sn = std::min(nstencils - 1, L - l);
        const ConvLevelArgs a = conv_level_args(g, tg, fi, l, 3, 1);
        GradArg gw{};
        bool full = false;  // some tap lies off the axes
        for (int d = 0; d < 3; ++d) {
            gw.active[d] = active[d];
            bool used[27];
            for (int k = 0; k < 27; ++k) {
                const float w = active[d] ? stencils[d][27 * sn + k] : 0.0f;
                gw.w[d][k] = w;
                used[k] = w != 0.0f;
                if (w == 0.0f) continue;
                const int id[3] = {k % 3, k / 3 % 3, k / 9};
                full = full || id[(d + 1) % 3] != 1 || id[(d + 2) % 3] != 1;
                gw.zuse[k / 9] = 1;
            }
            fb.outside += fi.level_count[l] * outside_taps(a.d, 1, used);
        }
        // in place, the whole level is read before any of it is written
        const int run = image_run<1, float>(a.d, in == out);
        for (int z0 = 0; z0 < a.d.zn; z0 += run) {
            const ImageShape<1, float> m(a.d, z0, std::min(z0 + run, a.d.zn));
            const float *D = launch_level_image<1, float>(a, m, xz_end, in, t_xz_end, tree, fb, s);
            APRB_PROF("grad_block", s);
            int tz;
            const dim3 grid = block_grid(a, m, tz);
            if (full)
                grad_block_kernel<true><<<grid, kGradThreads, 0, s>>>(a, gw, m, xz_end, D, out, stale, tz);
            else
                grad_block_kernel<false><<<grid, kGradThreads, 0, s>>>(a, gw, m, xz_end, D, out, stale, tz);
            count_launch();
            APRB_CHECK_LAUNCH();
        }
    }
}

uint64_t filter_stale_count(FilterBuffers &fb, cudaStream_t s) {
    unsigned long long v = 0;
    APRB_CUDA(cudaMemcpyAsync(&v, fb.stale.as<unsigned long long>(1), sizeof(v), cudaMemcpyDeviceToHost, s));
    APRB_CUDA(cudaStreamSynchronize(s));
    return v + fb.outside;
}

}  // namespace aprb
