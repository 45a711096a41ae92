// The sum over loops and images by cells.
//
// Away from a loop its displacement is smooth, and nearly all of the sum's
// (source, image) pairs are far from any given atom.  So the atoms' bounding
// box is cut into cells, level by level; a pair that is far from a cell (but
// was not far from the cell around it on the level before) is evaluated, by
// the same closed form in FP64, at the q^3 Chebyshev points of that cell
// instead of at every atom in it.  The values are interpolated from each level
// to the next, last to small cells whose Chebyshev coefficients every atom
// evaluates once.  What is far from no cell around the atom is summed at the
// atom itself, exactly as the plain kernels do it.
//
// A source is a line piece, or a square of a loop's loopons (quadtree): the
// field is as smooth in the loopon's place, so from afar a square acts as
// q x q equivalent loopons.  The squares shrink with the cells, and at the
// atoms themselves the squares that are far enough from a final cell for
// their equivalents are taken first, the rest loopon by loopon.
//
// "Far" is per axis: |cell centre - source centre - image shift| >
// theta(q) h + rho along some axis, with h the cell's half width (the largest
// over the axes) and rho the radius of the ball that holds the source (a line
// piece's apex and vertices, a square's loopons); for equivalent loopons also
// > h + theta(q) A, A the square's half extent.  The near images of a source
// are then a box of indices, (2I + 1)^3 cut by three intervals, and a cell's
// table holds one packed box per source.  The boxes are nested by intersection
// (cell in cell, square in square), so every (atom, term, image) enters exactly
// once, on whatever level.
//
// theta(q): interpolation at q Chebyshev points converges like the Bernstein
// ellipse's parameter to the power -q, and theta is where the measured worst
// truncation over loops of 25 and 40 A radius, directions and cells of 12 to 30 A
// half width falls below 4e-15 A for |b| = 2.5 A (plus 3 to 10 %).  With the
// rounding of the node values, which the weights of many nodes add up, q = 21
// reaches 6e-15 A for loops as large as the cell and 1.2e-14 A for loops 60 times
// as large; the direct sum's own rounding is 1e-14 A.
//
// FP64 tables only.  The FP32 compensated form would gain as well (FCC 40^3
// cells, 12 loops, +-2: 25.1 -> 5.3 ms) and come closer to the exact sum (1.9e-6
// -> 6e-7 A), but its results would move by up to 1.8e-6 A.
//
// Measured against the plain kernel on one B200 (ms a call): FCC 100^3 cells
// (4.0 M atoms), 16 loops, +-2 images 986 -> 14.7; BCC 61 x 47 x 33 (184 k
// atoms), 9 loops, +-3 76 -> 8.3; BCC 40^3 (128 k), 4 loops of 64 segments,
// +-1 4.93 -> 3.10; loopons: BCC 40^3 (127 k), 8 prismatic loops of R 20 to 50
// (39 k loopons), +-1 255 -> 57.  A sum too small to gain stays with the plain
// kernel (worth_cells).
//
// The same atoms in the same order give the same bits, whatever the order of the
// blocks.  In another order an atom can have other warp mates, which choose the
// series of their near terms together, and the cells follow the bounding box and
// the number of all atoms: then results agree to rounding.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "common.cuh"
#include "field.cuh"
#include "field_device.cuh"
#include "tree.cuh"

namespace disco {

int choose_split(int64_t n, int nimg, int resident_ctas);

namespace {

// ---- orders ----------------------------------------------------------------------------

constexpr int kOrders = 9;
constexpr int kOrderQ[kOrders] = { 9, 10, 11, 12, 13, 15, 17, 19, 21 };
constexpr double kOrderTheta[kOrders] = { 18.0, 13.2, 10.2, 8.2, 6.9, 5.1, 4.15, 3.55, 3.1 };
constexpr int kMaxRefine = 8;                  // final cells per axis in a cell of the last level, at most
constexpr int kMaxFinalQ = 13;                 // the atoms' cells hold three components in shared memory
constexpr int kWarps = 4;                      // warps per CTA of the tile kernels
constexpr int kMaxCells = 1 << 18;
constexpr double kClip = 2.0;                  // atoms within +-2 box lengths are sorted into cells

__host__ __device__ constexpr int padded(int q) { return (q + 1) & ~1; }

// ---- device arguments ------------------------------------------------------------------

struct LevelArgs {
    int32_t m[3];
    int32_t q, q3, split;
    int32_t r[3];             // cells per axis of this level in a cell of the level before
    int32_t tiles;            // warp tiles per cell
    int64_t tile0;            // first warp tile of the level
    int64_t cell0;            // first cell of the level (tables, occupancy)
    double theta, cut;
    int32_t np;               // sources of the level
    int64_t near0;            // first entry in the table of near boxes: [cell][source]
    int64_t list0;            // first entry in the lists of sources
    double* val;              // [cell][3][q3]
    LooponRec* eq;            // [source][q q]: equivalent loopons
};

struct TreeArgs {
    FieldArgs f;
    const TreePiece* pieces;
    int32_t nodes;            // tree pieces
    int32_t* list;            // [level][source]: tree piece
    int32_t* up;              // [level][source]: the source on the level before that holds it
    int32_t* pos;             // [level][tree piece]: its place in the level's list
    int32_t levels, total;    // levels of cells; with the levels summed at the atoms
    LevelArgs lv[TreeShape::kMaxLevels];
    int32_t mf[3], qf;        // final cells
    int32_t rf[3];            // final cells per axis in a cell of the last level
    int32_t cells_s, cells_f; // cells of the last level, final cells
    int32_t cells_n, near_rr; // cells of the near pass, final cells in each of them
    int32_t near_split;
    int32_t images;
    int64_t level_cells;      // cells over all levels
    unsigned long long* box;  // 8: ordered bits of min x, y, z and max x, y, z; sorted atoms; 0: all to the plain kernel
    int32_t from, least;      // that is for `from` sorted atoms up to 1 / least of all
    uint64_t* near;           // [level cell][source]: packed box of near images
    int64_t near_size;
    uint8_t* occ;             // [level cell]: holds atoms
    uint32_t* key[2];         // [atom], [slot]: final cell, the sort's two buffers
    int32_t* idx[2];          // the atoms that go with them
    uint32_t* digits;         // [256][sort tile]
    uint32_t* digit_total;    // [256]
    int32_t sort_tiles;
    uint32_t* start;          // [final cell + 2]: first sorted slot
    uint32_t* near_tile;      // [near cell + 2]: first warp tile of the near pass
    const int32_t* perm;      // sorted slot -> atom
    double* mat;              // interpolation matrices, transition by transition
    int32_t mat_off[TreeShape::kMaxLevels + 1][3];
};

// Order-preserving bits of a double.
__device__ __forceinline__ unsigned long long ord_bits(double v)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double ord_value(unsigned long long k)
{
    return __longlong_as_double((long long)((k >> 63) ? (k & 0x7FFFFFFFFFFFFFFFull) : ~k));
}

// An atom that is sorted into a cell (a NaN or a far outlier is not: it takes
// every pair itself).
__device__ __forceinline__ bool sorted_in(const FieldArgs& f, double x, double y, double z)
{
    return fabs(x) <= kClip * f.Lx && fabs(y) <= kClip * f.Ly && fabs(z) <= kClip * f.Lz;
}

struct Geo {
    double lo[3], ext[3];
    bool few;               // too few atoms to sort: every atom is left to the plain kernel
};

// The cells' grid: the bounding box of the sorted atoms, no axis thinner than
// a thousandth of the longest.
__device__ __forceinline__ Geo load_geo(const TreeArgs& a)
{
    Geo g;
    g.few = a.box[6] >= (unsigned long long)a.from && a.box[6] * (unsigned long long)a.least < (unsigned long long)a.f.n;
    double hi[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        g.lo[d] = ord_value(a.box[d]);
        hi[d] = ord_value(a.box[3 + d]);
    }
    if (!(g.lo[0] <= hi[0])) {                       // no sorted atom
#pragma unroll
        for (int d = 0; d < 3; ++d) { g.lo[d] = 0.0; g.ext[d] = 1.0; }
        return g;
    }
    double big = 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) big = fmax(big, hi[d] - g.lo[d]);
    const double least = fmax(1e-3 * big, 1e-6);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double e = hi[d] - g.lo[d];
        if (e < least) g.lo[d] -= 0.5 * (least - e);
        g.ext[d] = fmax(e, least);
    }
    return g;
}

// Final-cell coordinates of a sorted atom.
__device__ __forceinline__ void final_coord(const TreeArgs& a, const Geo& g, double x, double y, double z, int (&c)[3])
{
    const double p[3] = { x, y, z };
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const int i = (int)((p[d] - g.lo[d]) * ((double)a.mf[d] / g.ext[d]));
        c[d] = min(max(i, 0), a.mf[d] - 1);
    }
}

// Index of a final cell: the cell of the last level first, so that each of
// those owns a contiguous run of final cells (and of sorted slots).
__device__ __forceinline__ int last_index(const TreeArgs& a, const int (&c)[3])
{
    const LevelArgs& L = a.lv[a.levels - 1];
    return ((c[0] / a.rf[0]) * L.m[1] + c[1] / a.rf[1]) * L.m[2] + c[2] / a.rf[2];
}
__device__ __forceinline__ int final_index(const TreeArgs& a, const int (&c)[3])
{
    const int sub = ((c[0] % a.rf[0]) * a.rf[1] + c[1] % a.rf[1]) * a.rf[2] + c[2] % a.rf[2];
    return last_index(a, c) * (a.rf[0] * a.rf[1] * a.rf[2]) + sub;
}
__device__ __forceinline__ void final_cell(const TreeArgs& a, int index, int (&c)[3])
{
    const LevelArgs& L = a.lv[a.levels - 1];
    const int rr = a.rf[0] * a.rf[1] * a.rf[2], s = index / rr, sub = index % rr;
    c[0] = (s / (L.m[1] * L.m[2])) * a.rf[0] + sub / (a.rf[1] * a.rf[2]);
    c[1] = (s / L.m[2] % L.m[1]) * a.rf[1] + sub / a.rf[2] % a.rf[1];
    c[2] = (s % L.m[2]) * a.rf[2] + sub % a.rf[2];
}
__device__ __forceinline__ int cell_of(const TreeArgs& a, const Geo& g, double x, double y, double z)
{
    if (g.few || !sorted_in(a.f, x, y, z)) return a.cells_f;
    int c[3];
    final_coord(a, g, x, y, z, c);
    return final_index(a, c);
}

// ---- sorting ----------------------------------------------------------------------------

__global__ void __launch_bounds__(256) tree_box_kernel(const TreeArgs a)
{
    unsigned long long k[6] = { ~0ull, ~0ull, ~0ull, 0ull, 0ull, 0ull };
    unsigned in = 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < a.f.n; i += (int64_t)gridDim.x * blockDim.x) {
        const double p[3] = { a.f.x[i], a.f.y[i], a.f.z[i] };
        if (!sorted_in(a.f, p[0], p[1], p[2])) continue;
        ++in;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const unsigned long long b = ord_bits(p[d]);
            k[d] = min(k[d], b);
            k[3 + d] = max(k[3 + d], b);
        }
    }
#pragma unroll
    for (int d = 0; d < 6; ++d)
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long t = __shfl_xor_sync(0xffffffffu, k[d], o);
            k[d] = d < 3 ? min(k[d], t) : max(k[d], t);
        }
    in = __reduce_add_sync(0xffffffffu, in);
    __shared__ unsigned long long part[8][7];
    if ((threadIdx.x & 31) == 0) {
        for (int d = 0; d < 6; ++d) part[threadIdx.x >> 5][d] = k[d];
        part[threadIdx.x >> 5][6] = in;
    }
    __syncthreads();
    if (threadIdx.x < 7) {
        const int d = threadIdx.x;
        unsigned long long v = part[0][d];
        for (int w = 1; w < 8; ++w) v = d < 3 ? min(v, part[w][d]) : d < 6 ? max(v, part[w][d]) : v + part[w][d];
        if (d < 3) atomicMin(&a.box[d], v);
        else if (d < 6) atomicMax(&a.box[d], v);
        else atomicAdd(&a.box[d], v);
    }
}

__global__ void tree_init_kernel(const TreeArgs a)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    if (t < 7) a.box[t] = t < 3 ? ~0ull : 0ull;
    for (int64_t i = t; i < a.level_cells; i += step) a.occ[i] = 0;
}

// Stable radix sort of the atoms by final cell, 8 bits a pass: which atoms
// share a warp decides the series that a piece takes there, so the order
// within a cell is fixed (ascending atoms) to keep results reproducible.
// Tiles of 2048 atoms; warp w of a tile owns 256 consecutive ones.
constexpr int kSortThreads = 256, kSortItems = 8, kSortTile = kSortThreads * kSortItems;

template <bool kFirst>
__global__ void __launch_bounds__(kSortThreads) tree_digits_kernel(const TreeArgs a, const uint32_t* key_in, int shift)
{
    __shared__ uint32_t hist[256];
    hist[threadIdx.x] = 0;
    __syncthreads();
    Geo g;
    if (kFirst) g = load_geo(a);
    const int64_t base = (int64_t)blockIdx.x * kSortTile;
    for (int r = 0; r < kSortItems; ++r) {
        const int64_t i = base + r * kSortThreads + threadIdx.x;
        if (i >= a.f.n) break;
        uint32_t key;
        if (kFirst) {
            key = (uint32_t)cell_of(a, g, a.f.x[i], a.f.y[i], a.f.z[i]);
            a.key[0][i] = key;
        } else {
            key = key_in[i];
        }
        atomicAdd(&hist[(key >> shift) & 255u], 1u);
    }
    __syncthreads();
    a.digits[(int64_t)threadIdx.x * a.sort_tiles + blockIdx.x] = hist[threadIdx.x];
}

// One CTA per digit: exclusive sums over its tiles, the total behind them.
__global__ void __launch_bounds__(256) tree_digit_scan_kernel(const TreeArgs a);

template <bool kFirst>
__global__ void __launch_bounds__(kSortThreads) tree_reorder_kernel(const TreeArgs a, const uint32_t* key_in,
                                                                    const int32_t* idx_in, uint32_t* key_out,
                                                                    int32_t* idx_out, int shift);

// Exclusive scan over one CTA of v per thread; *total = the sum.
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t* total)
{
    __shared__ uint32_t warp_sum[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t inc = v;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) warp_sum[w] = inc;
    __syncthreads();
    if (w == 0) {
        uint32_t s = lane < (int)(blockDim.x >> 5) ? warp_sum[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += t;
        }
        warp_sum[lane] = s;
    }
    __syncthreads();
    const uint32_t base = w ? warp_sum[w - 1] : 0;
    *total = warp_sum[(blockDim.x >> 5) - 1];
    __syncthreads();
    return base + inc - v;
}

__global__ void __launch_bounds__(256) tree_digit_scan_kernel(const TreeArgs a)
{
    uint32_t* row = a.digits + (int64_t)blockIdx.x * a.sort_tiles;
    uint32_t carry = 0;
    for (int t0 = 0; t0 < a.sort_tiles; t0 += 256) {
        const int t = t0 + threadIdx.x;
        const uint32_t v = t < a.sort_tiles ? row[t] : 0u;
        uint32_t tot;
        const uint32_t ex = block_scan(v, &tot);
        if (t < a.sort_tiles) row[t] = carry + ex;
        carry += tot;
    }
    if (threadIdx.x == 0) a.digit_total[blockIdx.x] = carry;
}

template <bool kFirst>
__global__ void __launch_bounds__(kSortThreads) tree_reorder_kernel(const TreeArgs a, const uint32_t* key_in,
                                                                    const int32_t* idx_in, uint32_t* key_out,
                                                                    int32_t* idx_out, int shift)
{
    __shared__ uint32_t at[kSortThreads / 32][256];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int e = threadIdx.x; e < 256 * (kSortThreads / 32); e += kSortThreads) at[e >> 8][e & 255] = 0;
    uint32_t tot;
    const uint32_t digit_base = block_scan(a.digit_total[threadIdx.x], &tot);   // its barriers cover the clearing
    const int64_t base = (int64_t)blockIdx.x * kSortTile + w * (32 * kSortItems);
    uint32_t key[kSortItems], rank[kSortItems];
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const int64_t i = base + r * 32 + lane;
        const bool valid = i < a.f.n;
        key[r] = valid ? key_in[i] : 0u;
        const uint32_t d = valid ? (key[r] >> shift) & 255u : 256u + lane;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        uint32_t before = 0;
        if (valid) before = at[w][d];
        __syncwarp();
        if (valid && lane == __ffs(peers) - 1) at[w][d] = before + (uint32_t)__popc(peers);
        __syncwarp();
        rank[r] = before + (uint32_t)__popc(peers & ((1u << lane) - 1u));
    }
    __syncthreads();
    uint32_t sum = digit_base + a.digits[(int64_t)threadIdx.x * a.sort_tiles + blockIdx.x];
#pragma unroll
    for (int k = 0; k < kSortThreads / 32; ++k) {
        const uint32_t c = at[k][threadIdx.x];
        at[k][threadIdx.x] = sum;
        sum += c;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const int64_t i = base + r * 32 + lane;
        if (i >= a.f.n) break;
        const uint32_t slot = at[w][(key[r] >> shift) & 255u] + rank[r];
        key_out[slot] = key[r];
        idx_out[slot] = kFirst ? (int32_t)i : idx_in[i];
    }
}

// First sorted slot of every final cell (and of the atoms outside the grid,
// one more cell at the end).
__global__ void __launch_bounds__(256) tree_starts_kernel(const TreeArgs a, const uint32_t* key)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= a.f.n; i += (int64_t)gridDim.x * blockDim.x) {
        const int lo = i == 0 ? -1 : (int)key[i - 1], hi = i == a.f.n ? a.cells_f + 1 : (int)key[i];
        for (int c = lo + 1; c <= hi; ++c) a.start[c] = (uint32_t)i;
    }
}

// Warp tiles of the near pass, by its cells (plus the outside cell), and which
// cells of each level hold atoms; one CTA.
__global__ void __launch_bounds__(1024) tree_scan_kernel(const TreeArgs a)
{
    const int rr = a.rf[0] * a.rf[1] * a.rf[2];
    const LevelArgs& E = a.lv[a.levels - 1];
    for (int s = threadIdx.x; s < a.cells_s; s += 1024) {
        if (a.start[(s + 1) * rr] == a.start[s * rr]) continue;
        const int c[3] = { s / (E.m[1] * E.m[2]), s / E.m[2] % E.m[1], s % E.m[2] };
        for (int l = 0; l < a.levels; ++l) {
            const LevelArgs& L = a.lv[l];
            const int lc = ((c[0] / (E.m[0] / L.m[0])) * L.m[1] + c[1] / (E.m[1] / L.m[1])) * L.m[2] +
                           c[2] / (E.m[2] / L.m[2]);
            a.occ[L.cell0 + lc] = 1;
        }
    }
    const bool few = load_geo(a).few;
    if (threadIdx.x == 0) a.box[7] = few ? 0 : 1;
    const int ns = a.cells_n + 1, per = (ns + 1023) / 1024;
    const int s0 = min(ns, (int)threadIdx.x * per), s1 = min(ns, s0 + per);
    const uint32_t per_tile = 32u / (uint32_t)a.near_split;
    auto tiles_of = [&](int s) {
        const uint32_t k = a.start[s < a.cells_n ? (s + 1) * a.near_rr : a.cells_f + 1] - a.start[s * a.near_rr];
        if (s == a.cells_n && few) return 0u;                                // the plain kernel's
        return (k + per_tile - 1) / per_tile;
    };
    uint32_t mine = 0, tot;
    for (int s = s0; s < s1; ++s) mine += tiles_of(s);
    uint32_t at = block_scan(mine, &tot);
    if (threadIdx.x == 0) a.near_tile[ns] = tot;
    for (int s = s0; s < s1; ++s) {
        a.near_tile[s] = at;
        at += tiles_of(s);
    }
}

// ---- near boxes --------------------------------------------------------------------------

// Packed box of image indices: lo and hi per axis, offset by 16, one byte
// each; an empty box is 0.
__host__ __device__ __forceinline__ uint64_t full_box(int images)
{
    uint64_t w = 0;
    for (int d = 0; d < 3; ++d) {
        w |= (uint64_t)(uint8_t)(16 - images) << (16 * d);
        w |= (uint64_t)(uint8_t)(16 + images) << (16 * d + 8);
    }
    return w;
}
struct ImgBox {
    int lo[3], n[3];
    __device__ __forceinline__ explicit ImgBox(uint64_t w)
    {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            lo[d] = (int)((w >> (16 * d)) & 0xFF) - 16;
            n[d] = (int)((w >> (16 * d + 8)) & 0xFF) - 16 - lo[d] + 1;
        }
    }
    __device__ __forceinline__ int count() const { return n[0] * n[1] * n[2]; }
    __device__ __forceinline__ void at(int idx, int& i, int& j, int& k) const
    {
        const int yz = n[1] * n[2];
        const int qi = idx / yz, r = idx - qi * yz;
        const int qj = r / n[2];
        i = lo[0] + qi;
        j = lo[1] + qj;
        k = lo[2] + (r - qj * n[2]);
    }
};

// The images of a box U outside a box O inside it (O may be empty), counted and
// numbered: the planes of U before and after O along x, then along y within
// O's x range, then along z.
struct ImgShell {
    ImgBox U, O;
    int a0, a1, b0, b1, c0, total;      // ends of the x-, x+, y-, y+ and z- parts
    bool whole;
    __device__ __forceinline__ ImgShell(uint64_t u, uint64_t o) : U(u), O(o == 0 ? u : o), whole(o == 0)
    {
        const int yz = U.n[1] * U.n[2];
        if (whole) { a0 = a1 = b0 = b1 = c0 = total = U.count(); return; }
        a0 = (O.lo[0] - U.lo[0]) * yz;
        a1 = a0 + (U.lo[0] + U.n[0] - O.lo[0] - O.n[0]) * yz;
        b0 = a1 + O.n[0] * (O.lo[1] - U.lo[1]) * U.n[2];
        b1 = b0 + O.n[0] * (U.lo[1] + U.n[1] - O.lo[1] - O.n[1]) * U.n[2];
        c0 = b1 + O.n[0] * O.n[1] * (O.lo[2] - U.lo[2]);
        total = c0 + O.n[0] * O.n[1] * (U.lo[2] + U.n[2] - O.lo[2] - O.n[2]);
    }
    __device__ __forceinline__ void at(int idx, int& i, int& j, int& k) const
    {
        int x = U.lo[0], y = U.lo[1], z = U.lo[2], ny = U.n[1], nz = U.n[2];
        if (idx >= a0) {
            if (idx < a1) { idx -= a0; x = O.lo[0] + O.n[0]; }
            else {
                x = O.lo[0];
                if (idx < b0) { idx -= a1; ny = O.lo[1] - U.lo[1]; }
                else if (idx < b1) { idx -= b0; y = O.lo[1] + O.n[1]; ny = U.lo[1] + U.n[1] - y; }
                else {
                    y = O.lo[1];
                    ny = O.n[1];
                    if (idx < c0) { idx -= b1; nz = O.lo[2] - U.lo[2]; }
                    else { idx -= c0; z = O.lo[2] + O.n[2]; nz = U.lo[2] + U.n[2] - z; }
                }
            }
        }
        const int yz = ny * nz, q = idx / yz, r = idx - q * yz, p = r / nz;
        i = x + q;
        j = y + p;
        k = z + (r - p * nz);
    }
};

// A tree piece is a source of a level whose cut its square fits and the one
// above it does not.
__device__ __forceinline__ bool in_cut(const TreeArgs& a, const TreePiece& t, int self, double cut)
{
    const bool fits = t.size <= cut || t.leaf0 == self;
    return fits && (t.parent < 0 || a.pieces[t.parent].size > cut);
}

// One CTA per level: its sources in order.
__global__ void __launch_bounds__(1024) tree_list_kernel(const TreeArgs a)
{
    const LevelArgs& v = a.lv[blockIdx.x];
    uint32_t at = 0;
    for (int n0 = 0; n0 < a.nodes; n0 += 1024) {
        const int n = n0 + threadIdx.x;
        const bool in = n < a.nodes && in_cut(a, a.pieces[n], n, v.cut);
        uint32_t tot;
        const uint32_t k = at + block_scan(in ? 1u : 0u, &tot);
        if (in && k < (uint32_t)v.np) {
            a.list[v.list0 + k] = n;
            a.pos[(int64_t)blockIdx.x * a.nodes + n] = (int32_t)k;
        }
        at += tot;
    }
}

// The tree piece that holds n (or n itself) among the sources of a level with
// a coarser (or the same) cut.
__device__ __forceinline__ int holder(const TreeArgs& a, int n, double cut)
{
    for (;;) {
        const int up = a.pieces[n].parent;
        if (up < 0 || a.pieces[up].size > cut) return n;
        n = up;
    }
}

// Whether a source is summed through its q x q equivalent loopons: a square
// that holds others, or a leaf with more loopons than that.
__device__ __forceinline__ bool uses_eq(const LevelArgs& v, const TreePiece& t, int self)
{
    return v.eq != nullptr && (t.leaf0 != self || t.terms > v.q * v.q);
}

// One thread per (level cell, source): the intersection of the near boxes of
// the cell and of the cells around it on the levels before, each for the
// source there that holds this one.  Equivalent loopons hold from
// theta(q) half extents of the square on, so where they are used the cell has
// to be that far as well; a level summed at the atoms asks for nothing else.
__global__ void __launch_bounds__(256) tree_near_kernel(const TreeArgs a)
{
    const Geo g = load_geo(a);
    if (g.few) return;
    const double L[3] = { a.f.Lx, a.f.Ly, a.f.Lz };
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < a.near_size;
         t += (int64_t)gridDim.x * blockDim.x) {
        int k = a.total - 1;
        while (a.lv[k].near0 > t) --k;
        const int64_t local = t - a.lv[k].near0;
        const int c = (int)(local / a.lv[k].np), e = (int)(local % a.lv[k].np);
        int ci[3];
        if (k < a.levels) {
            ci[0] = c / (a.lv[k].m[1] * a.lv[k].m[2]);
            ci[1] = c / a.lv[k].m[2] % a.lv[k].m[1];
            ci[2] = c % a.lv[k].m[2];
        } else {
            final_cell(a, c, ci);
        }
        int lo[3], hi[3];
        for (int d = 0; d < 3; ++d) { lo[d] = -a.images; hi[d] = a.images; }
        int n = a.list[a.lv[k].list0 + e];
        for (int j = k; j >= 0; --j) {
            const LevelArgs& v = a.lv[j];
            n = holder(a, n, v.cut);
            if (j == k - 1 && c == 0) a.up[a.lv[k].list0 + e] = a.pos[(int64_t)j * a.nodes + n];
            const TreePiece& tp = a.pieces[n];
            double h = 0.0;
            for (int d = 0; d < 3; ++d) h = fmax(h, 0.5 * g.ext[d] / v.m[d]);
            const bool eq = uses_eq(v, tp, n);
            if (j >= a.levels && !eq) continue;           // summed at the atoms one by one
            double R = j < a.levels ? v.theta * h + tp.rho : 0.0;
            if (eq) R = fmax(R, h + v.theta * fmax(tp.a1, tp.a2));
            const double s[3] = { tp.x, tp.y, tp.z };
            for (int d = 0; d < 3; ++d) {
                const int cj = ci[d] / (a.lv[k].m[d] / v.m[d]);
                const double cc = g.lo[d] + (cj + 0.5) * (g.ext[d] / v.m[d]) - s[d];
                // |cc - i L| <= R; clamped before the conversion to int
                lo[d] = max(lo[d], (int)fmin(fmax(ceil((cc - R) / L[d]), -64.0), 64.0));
                hi[d] = min(hi[d], (int)fmin(fmax(floor((cc + R) / L[d]), -64.0), 64.0));
            }
        }
        uint64_t w = 0;
        if (lo[0] <= hi[0] && lo[1] <= hi[1] && lo[2] <= hi[2])
            for (int d = 0; d < 3; ++d) {
                w |= (uint64_t)(uint8_t)(16 + lo[d]) << (16 * d);
                w |= (uint64_t)(uint8_t)(16 + hi[d]) << (16 * d + 8);
            }
        a.near[t] = w;
    }
}

// Equivalent loopons of a square: the field is smooth in the loopon's place
// too, so from afar the square's loopons act as q x q loopons at the Chebyshev
// points of its extent, weighted by the sums of the interpolation weights of
// all its loopons: with the moments M_ab = sum T_a(x) T_b(y) over the loopons,
// w_ij = sum_ab c_a T_a(x_i) c_b T_b(x_j) M_ab, c_0 = 1/q, c_a = 2/q.  One CTA
// per source, a moment per thread; the loopons come in batches of 64.
constexpr int kMaxQ = 21;
constexpr int kEqThreads = 448;                    // 21 x 21 and whole warps
__global__ void __launch_bounds__(kEqThreads) tree_equivalent_kernel(const TreeArgs a)
{
    const LevelArgs& v = a.lv[blockIdx.y];
    if (v.eq == nullptr || blockIdx.x >= (unsigned)v.np || a.box[7] == 0) return;
    const int self = a.list[v.list0 + blockIdx.x];
    const TreePiece& tp = a.pieces[self];
    if (!uses_eq(v, tp, self)) return;
    constexpr int kBatch = 64;
    __shared__ double cq[4 * kMaxQ], T1[kBatch][kMaxQ], T2[kBatch][kMaxQ];
    const int q = v.q, t = threadIdx.x, ma = t / q, mb = t % q;
    for (int e = t; e < 4 * q; e += kEqThreads) cq[e] = cospi(e / (2.0 * q));
    const LooponPiece& pc = *reinterpret_cast<const LooponPiece*>(a.f.table + tp.piece);
    const double ox = tp.x - pc.cx, oy = tp.y - pc.cy, oz = tp.z - pc.cz;
    const double i1 = tp.a1 > 0.0 ? 1.0 / tp.a1 : 0.0, i2 = tp.a2 > 0.0 ? 1.0 / tp.a2 : 0.0;
    double acc = 0.0;
    for (int leaf = tp.leaf0; leaf < tp.leaf0 + tp.leaves; ++leaf) {
        const LooponRec* rec = reinterpret_cast<const LooponRec*>(a.f.table + a.pieces[leaf].rec);
        const int terms = a.pieces[leaf].terms;
        for (int k0 = 0; k0 < terms; k0 += kBatch) {
            const int nb = min(kBatch, terms - k0);
            __syncthreads();
            if (t < 2 * nb) {
                const bool y = t >= nb;
                const int k = y ? t - nb : t;
                const LooponRec& r = rec[k0 + k];
                const double* d = y ? tp.e2 : tp.e1;
                double x = (d[0] * (r.x - ox) + d[1] * (r.y - oy) + d[2] * (r.z - oz)) * (y ? i2 : i1);
                x = fmin(fmax(x, -1.0), 1.0);
                double* T = y ? T2[k] : T1[k];
                double t0 = 1.0, t1 = x;
                for (int i = 0; i < q; ++i) {
                    T[i] = t0;
                    const double t2 = fma(2.0 * x, t1, -t0);
                    t0 = t1;
                    t1 = t2;
                }
            }
            __syncthreads();
            if (ma < q)
                for (int k = 0; k < nb; ++k) acc = fma(T1[k][ma], T2[k][mb], acc);
        }
    }
    __syncthreads();
    // c_a T_a(x_i), the moments over b, then over a
    double (*M)[kMaxQ] = T1, (*R)[kMaxQ] = T2;
    if (ma < q) M[ma][mb] = acc;
    __syncthreads();
    const int wi = ma, wj = mb;
    if (ma < q) {
        double s = 0.0;
        for (int b = 0; b < q; ++b) s = fma((b ? 2.0 : 1.0) / q * cq[(b * (2 * wj + 1)) % (4 * q)], M[ma][b], s);
        R[ma][wj] = s;
    }
    __syncthreads();
    if (wi < q) {
        double s = 0.0;
        for (int k = 0; k < q; ++k) s = fma((k ? 2.0 : 1.0) / q * cq[(k * (2 * wi + 1)) % (4 * q)], R[k][wj], s);
        const double t1 = tp.a1 * cq[2 * wi + 1], t2 = tp.a2 * cq[2 * wj + 1];
        LooponRec r;
        r.x = ox + t1 * tp.e1[0] + t2 * tp.e2[0];
        r.y = oy + t1 * tp.e1[1] + t2 * tp.e2[1];
        r.z = oz + t1 * tp.e1[2] + t2 * tp.e2[2];
        r.ml = pc.mx * r.x + pc.my * r.y + pc.mz * r.z;
        r.nl = pc.nx * r.x + pc.ny * r.y + pc.nz * r.z;
        r.w = s;
        v.eq[(int64_t)blockIdx.x * q * q + t] = r;
    }
}

// ---- node sums ---------------------------------------------------------------------------

// One warp: 32 / split nodes of one cell; its far pairs are those in the near
// boxes of the level before and not in its own.  FP64 bound like the plain
// line kernel (records are read through L1 as warp-uniform 16-byte loads).
template <int kKind>
__global__ void __launch_bounds__(32 * kWarps, 4) tree_node_kernel(const TreeArgs a)
{
    const int lane = threadIdx.x & 31;
    const int64_t w = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5);
    int k = a.levels - 1;
    while (k > 0 && a.lv[k].tile0 > w) --k;
    const LevelArgs& v = a.lv[k];
    const int64_t local = w - v.tile0;
    const int64_t cells = (int64_t)v.m[0] * v.m[1] * v.m[2];
    if (local >= cells * v.tiles) return;
    const int cell = (int)(local / v.tiles), tile = (int)(local % v.tiles);
    if (!a.occ[v.cell0 + cell]) return;
    const Geo g = load_geo(a);
    const int split = v.split;
    const int node = tile * (32 / split) + lane / split, part = lane % split;
    const bool valid = node < v.q3;
    const int nd = valid ? node : v.q3 - 1;
    const int ci[3] = { cell / (v.m[1] * v.m[2]), cell / v.m[2] % v.m[1], cell % v.m[2] };
    const int ni[3] = { nd / (v.q * v.q), nd / v.q % v.q, nd % v.q };
    double P[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double e = g.ext[d] / v.m[d];
        P[d] = g.lo[d] + (ci[d] + 0.5) * e + 0.5 * e * cospi((2 * ni[d] + 1) / (2.0 * v.q));
    }
    const uint64_t* own = a.near + v.near0 + (int64_t)cell * v.np;
    const uint64_t* up = nullptr;
    if (k > 0) {
        const LevelArgs& u = a.lv[k - 1];
        const int uc = ((ci[0] / v.r[0]) * u.m[1] + ci[1] / v.r[1]) * u.m[2] + ci[2] / v.r[2];
        up = a.near + u.near0 + (int64_t)uc * u.np;
    }
    const uint64_t all = full_box(a.images);
    const double cJK = a.f.cJ / a.f.cK;
    double ux = 0.0, uy = 0.0, uz = 0.0;
    bool plane = false;
    for (int base = 0; base < v.np; base += 32) {
        uint64_t wu = 0, wo = 0;
        if (base + lane < v.np) {
            wu = up ? up[a.up[v.list0 + base + lane]] : all;
            wo = own[base + lane];
        }
        unsigned todo = __ballot_sync(0xffffffffu, wu != 0 && wu != wo);
        while (todo) {
            const int b = __ffs(todo) - 1;
            todo &= todo - 1;
            const uint64_t bu = __shfl_sync(0xffffffffu, wu, b), bo = __shfl_sync(0xffffffffu, wo, b);
            const int self = a.list[v.list0 + base + b];
            const TreePiece& tp = a.pieces[self];
            const ImgShell far(bu, bo);
            if constexpr (kKind == kLineKind) {
                const LinePiece& pc = *reinterpret_cast<const LinePiece*>(a.f.table + tp.piece);
                const LineSeg* seg = reinterpret_cast<const LineSeg*>(a.f.table + tp.rec);
                for (int idx = part; idx < far.total; idx += split) {
                    int i, j, l;
                    far.at(idx, i, j, l);
                    line_piece_fp64<true>(pc, seg, P[0] - a.f.Lx * i, P[1] - a.f.Ly * j, P[2] - a.f.Lz * l, cJK, ux,
                                          uy, uz, plane);
                }
            } else {
                const LooponPiece& pc = *reinterpret_cast<const LooponPiece*>(a.f.table + tp.piece);
                const bool eq = uses_eq(v, tp, self);
                const LooponRec* rec = eq ? v.eq + (int64_t)(base + b) * v.q * v.q
                                          : reinterpret_cast<const LooponRec*>(a.f.table + tp.rec);
                const int n = eq ? v.q * v.q : tp.terms;
                const double qx = P[0] - pc.cx, qy = P[1] - pc.cy, qz = P[2] - pc.cz;
                for (int idx = 0; idx < far.total; ++idx) {
                    int i, j, l;
                    far.at(idx, i, j, l);
                    loopon_terms_fp64<true>(pc, rec, n, qx - a.f.Lx * i, qy - a.f.Ly * j, qz - a.f.Lz * l, a.f.c2, ux,
                                            uy, uz, part, split);
                }
            }
        }
    }
    for (int o = split / 2; o > 0; o >>= 1) {
        ux += __shfl_xor_sync(0xffffffffu, ux, o);
        uy += __shfl_xor_sync(0xffffffffu, uy, o);
        uz += __shfl_xor_sync(0xffffffffu, uz, o);
    }
    if (valid && part == 0) {
        double* out = v.val + (int64_t)cell * 3 * v.q3 + node;
        out[0] = ux;
        out[v.q3] = uy;
        out[2 * v.q3] = uz;
    }
}

// ---- interpolation -----------------------------------------------------------------------

// Matrices of transition t (level t-1 -> t, or last level -> final cells for
// t = levels): for axis d and sub-position s of r, M[s][i][j] takes the
// parent's value at its node i to the child's node j (final: to the child's
// Chebyshev coefficient j).  Interpolation at q Chebyshev points is
// f(x) = sum_i f_i (1/q) (1 + 2 sum_k T_k(x_i) T_k(x)).
// cq[t] = cos(pi t / (2 q)), t < 4 q
__device__ __forceinline__ double interp_weight(const double* cq, int q, int i, double x)
{
    double t0 = 1.0, t1 = x, s = 0.5;
    int ph = 0;
    for (int k = 1; k < q; ++k) {
        ph += 2 * i + 1;
        if (ph >= 4 * q) ph -= 4 * q;
        s = fma(cq[ph], t1, s);
        const double t2 = fma(2.0 * x, t1, -t0);
        t0 = t1;
        t1 = t2;
    }
    return 2.0 * s / q;
}

__global__ void __launch_bounds__(128) tree_matrix_kernel(const TreeArgs a)
{
    __shared__ double cp[4 * kMaxQ], cc[4 * kMaxQ];
    const int t = blockIdx.x + 1, d = blockIdx.y;      // transitions 1..levels
    const bool last = t == a.levels;
    const int qp = a.lv[t - 1].q, qc = last ? a.qf : a.lv[t].q, r = last ? a.rf[d] : a.lv[t].r[d];
    for (int e = threadIdx.x; e < 4 * qp; e += blockDim.x) cp[e] = cospi(e / (2.0 * qp));
    for (int e = threadIdx.x; e < 4 * qc; e += blockDim.x) cc[e] = cospi(e / (2.0 * qc));
    __syncthreads();
    double* M = a.mat + a.mat_off[t][d];
    for (int e = blockIdx.z * blockDim.x + threadIdx.x; e < r * qp * qc; e += gridDim.z * blockDim.x) {
        const int s = e / (qp * qc), i = e / qc % qp, j = e % qc;
        const double x0 = (2.0 * s + 1.0) / r - 1.0;
        double v = 0.0;
        if (!last) {
            v = interp_weight(cp, qp, i, x0 + cc[2 * j + 1] / r);
        } else {
            for (int n = 0; n < qc; ++n)
                v = fma(interp_weight(cp, qp, i, x0 + cc[2 * n + 1] / r), cc[(j * (2 * n + 1)) % (4 * qc)], v);
            v *= (j ? 2.0 : 1.0) / qc;
        }
        M[e] = v;
    }
}

// One axis of the tensor interpolation: in[a][i][b] -> out[a][j][b] for
// na x nb columns, each thread one column with the QC sums in registers.
template <int QC>
__device__ __forceinline__ void contract(const double* in, const double* M, double* out, int na, int qp, int nb)
{
    for (int c = threadIdx.x; c < na * nb; c += blockDim.x) {
        const int ia = c / nb, ib = c - ia * nb;
        const double* src = in + ia * qp * nb + ib;
        double acc[QC];
#pragma unroll
        for (int j = 0; j < QC; ++j) acc[j] = 0.0;
#pragma unroll 2
        for (int i = 0; i < qp; ++i) {
            const double f = src[i * nb];
#pragma unroll
            for (int j = 0; j < QC; ++j) acc[j] = fma(M[i * QC + j], f, acc[j]);
        }
        double* dst = out + ia * QC * nb + ib;
#pragma unroll
        for (int j = 0; j < QC; ++j) dst[j * nb] = acc[j];
    }
}

// Level t - 1 -> t: one CTA adds one component of one cell's values, read
// from the cell around it (in L2: its children read it together).
template <int QC>
__global__ void __launch_bounds__(256) tree_down_kernel(const TreeArgs a, int t)
{
    extern __shared__ double sm[];
    const LevelArgs& up = a.lv[t - 1];
    const LevelArgs& v = a.lv[t];
    const int qp = up.q, comp = blockIdx.y, cell = blockIdx.x;
    if (!a.occ[v.cell0 + cell]) return;
    const int ci[3] = { cell / (v.m[1] * v.m[2]), cell / v.m[2] % v.m[1], cell % v.m[2] };
    const int pc = ((ci[0] / v.r[0]) * up.m[1] + ci[1] / v.r[1]) * up.m[2] + ci[2] / v.r[2];
    double* b0 = sm;                                   // [QC][qp][qp], then [QC][QC][QC]
    double* b1 = b0 + max(QC * qp * qp, QC * QC * QC); // [QC][QC][qp]
    double* M = b1 + QC * QC * qp;
    for (int d = 0; d < 3; ++d) {
        const double* m = a.mat + a.mat_off[t][d] + (ci[d] % v.r[d]) * qp * QC;
        for (int e = threadIdx.x; e < qp * QC; e += blockDim.x) M[d * qp * QC + e] = m[e];
    }
    __syncthreads();
    contract<QC>(up.val + ((int64_t)pc * 3 + comp) * up.q3, M, b0, 1, qp, qp * qp);
    __syncthreads();
    contract<QC>(b0, M + qp * QC, b1, QC, qp, qp);
    __syncthreads();
    contract<QC>(b1, M + 2 * qp * QC, b0, QC * QC, qp, 1);
    __syncthreads();
    double* out = v.val + ((int64_t)cell * 3 + comp) * (QC * QC * QC);
    for (int e = threadIdx.x; e < QC * QC * QC; e += blockDim.x) out[e] += b0[e];
}

// One axis of the tensor interpolation with the matrix rows padded to QP and
// read as pairs: in[c][i] at stride `in_step` -> QC sums in registers.
template <int QC>
__device__ __forceinline__ void column(const double* src, int step, const double* M, int qp, double (&acc)[padded(QC)])
{
    constexpr int QP = padded(QC);
#pragma unroll
    for (int j = 0; j < QP; ++j) acc[j] = 0.0;
#pragma unroll 6
    for (int i = 0; i < qp; ++i) {
        const double f = src[i * step];
        const double2* m = reinterpret_cast<const double2*>(M + i * QP);
#pragma unroll
        for (int j = 0; j < QP / 2; ++j) {
            const double2 w = m[j];
            acc[2 * j] = fma(w.x, f, acc[2 * j]);
            if (2 * j + 1 < QC) acc[2 * j + 1] = fma(w.y, f, acc[2 * j + 1]);
        }
    }
}

// Last level -> atoms: one CTA per (cell of the last level, x and y
// sub-position, component) interpolates along x and y once for the rf[2] final
// cells of that column; for each of them it makes the Chebyshev coefficients
// in shared memory (the transform is folded into the matrices) and evaluates
// them at the cell's atoms, 64 atoms (two per lane) and a share of the x orders
// per warp; u += the sum.  Bound by FP64 multiply-adds: QC qp^3 + QC^2 qp^2 per
// column, QC^3 qp per cell, QC^3 per atom; a pair of coefficients loaded from
// shared memory feeds four of them.  One component per CTA keeps the shared
// memory at 40 to 70 KB (three CTAs per SM; one with all three components).
template <int QC>
__global__ void __launch_bounds__(256, 3) tree_leaf_kernel(const TreeArgs a)
{
    extern __shared__ double sm[];
    constexpr int QP = padded(QC), kWarpsPerCta = 8;
    const int t = a.levels;
    const LevelArgs& up = a.lv[t - 1];
    const int qp = up.q, comp = blockIdx.y;
    const int rxy = a.rf[0] * a.rf[1], rz = a.rf[2];
    const int s = blockIdx.x / rxy, sub = blockIdx.x % rxy;
    const int bx = sub / a.rf[1], by = sub % a.rf[1];
    const int cell0 = (s * rxy + sub) * rz;             // the column's first final cell
    if (a.start[cell0] == a.start[cell0 + rz]) return;
    double* coef = sm;                                  // [QC][QC][QP]
    double* b1 = coef + QC * QC * QP;                   // [QC][QC][qp]
    double* b0 = b1 + padded(QC * QC * qp);             // [QC][qp][qp]; later the atoms' partial sums
    double* M = b0 + padded(max(QC * qp * qp, 8 * 64)); // x, y and the rz matrices of z, [qp][QP] each
    for (int k = 0; k < 2 + rz; ++k) {
        const int d = min(k, 2), b = k == 0 ? bx : k == 1 ? by : k - 2;
        const double* m = a.mat + a.mat_off[t][d] + b * qp * QC;
        for (int e = threadIdx.x; e < qp * QP; e += 256)
            M[k * qp * QP + e] = e % QP < QC ? m[(e / QP) * QC + e % QP] : 0.0;
    }
    __syncthreads();
    {
        double acc[QP];
        const double* val = up.val + ((int64_t)s * 3 + comp) * up.q3;
        for (int c = threadIdx.x; c < qp * qp; c += 256) {
            column<QC>(val + c, qp * qp, M, qp, acc);
#pragma unroll
            for (int j = 0; j < QC; ++j) b0[j * qp * qp + c] = acc[j];
        }
        __syncthreads();
        for (int c = threadIdx.x; c < QC * qp; c += 256) {
            const int ia = c / qp, ib = c - ia * qp;
            column<QC>(b0 + ia * qp * qp + ib, qp, M + qp * QP, qp, acc);
#pragma unroll
            for (int j = 0; j < QC; ++j) b1[(ia * QC + j) * qp + ib] = acc[j];
        }
        __syncthreads();
    }
    const Geo g = load_geo(a);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int cx = (s / (up.m[1] * up.m[2])) * a.rf[0] + bx, cy = (s / up.m[2] % up.m[1]) * a.rf[1] + by;
    double* uo = comp == 0 ? a.f.ux : comp == 1 ? a.f.uy : a.f.uz;
    double* red = b0;                                   // [warp][2][32]
    for (int bz = 0; bz < rz; ++bz) {
        const uint32_t s0 = a.start[cell0 + bz];
        const int cnt = (int)(a.start[cell0 + bz + 1] - s0);
        if (cnt == 0) continue;
        for (int c = threadIdx.x; c < QC * QC; c += 256) {
            double acc[QP];
            column<QC>(b1 + c * qp, 1, M + (2 + bz) * qp * QP, qp, acc);
            double2* dst = reinterpret_cast<double2*>(coef + c * QP);
#pragma unroll
            for (int j = 0; j < QP / 2; ++j) dst[j] = make_double2(acc[2 * j], acc[2 * j + 1]);
        }
        __syncthreads();
        const int ci[3] = { cx, cy, (s % up.m[2]) * rz + bz };
        // groups of G warps per 64 atoms, each warp QC / G of the x orders
        const int G = cnt <= 64 ? 8 : cnt <= 128 ? 4 : cnt <= 256 ? 2 : 1;
        const int part = w % G, i0 = QC * part / G, i1 = QC * (part + 1) / G;
        const int step = 64 * (kWarpsPerCta / G);
        for (int base = 0; base < cnt; base += step) {
            const int first = base + 64 * (w / G);
            int32_t atom[2];
            double X[2], Y[2], Tz[2][QC];
            double u[2] = {};
            if (first < cnt) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    atom[h] = a.perm[s0 + min(first + lane + 32 * h, cnt - 1)];
                    const double p[3] = { a.f.x[atom[h]], a.f.y[atom[h]], a.f.z[atom[h]] };
                    double tt[3];
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        const double e = g.ext[d] / a.mf[d];
                        tt[d] = fmin(fmax((p[d] - (g.lo[d] + (ci[d] + 0.5) * e)) * (2.0 / e), -1.0), 1.0);
                    }
                    X[h] = tt[0];
                    Y[h] = tt[1];
                    Tz[h][0] = 1.0;
                    Tz[h][1] = tt[2];
#pragma unroll
                    for (int i = 2; i < QC; ++i) Tz[h][i] = fma(2.0 * tt[2], Tz[h][i - 1], -Tz[h][i - 2]);
                }
                double ax0 = 1.0, bx0 = X[0], ax1 = 1.0, bx1 = X[1];        // T_i, T_{i+1}
                for (int i = 0; i < i1; ++i) {
                    if (i >= i0) {
                        double ay0 = 1.0, by0 = Y[0], ay1 = 1.0, by1 = Y[1];
                        double sy0 = 0.0, sy1 = 0.0;
#pragma unroll 2
                        for (int j = 0; j < QC; ++j) {
                            const double2* C = reinterpret_cast<const double2*>(coef + (i * QC + j) * QP);
                            double v0 = 0.0, v1 = 0.0;
#pragma unroll
                            for (int k = 0; k < QP / 2; ++k) {
                                const double2 c = C[k];
                                v0 = fma(c.x, Tz[0][2 * k], v0);
                                v1 = fma(c.x, Tz[1][2 * k], v1);
                                if (2 * k + 1 < QC) {
                                    v0 = fma(c.y, Tz[0][2 * k + 1], v0);
                                    v1 = fma(c.y, Tz[1][2 * k + 1], v1);
                                }
                            }
                            sy0 = fma(ay0, v0, sy0);
                            sy1 = fma(ay1, v1, sy1);
                            const double n0 = fma(2.0 * Y[0], by0, -ay0), n1 = fma(2.0 * Y[1], by1, -ay1);
                            ay0 = by0; by0 = n0;
                            ay1 = by1; by1 = n1;
                        }
                        u[0] = fma(ax0, sy0, u[0]);
                        u[1] = fma(ax1, sy1, u[1]);
                    }
                    const double n0 = fma(2.0 * X[0], bx0, -ax0), n1 = fma(2.0 * X[1], bx1, -ax1);
                    ax0 = bx0; bx0 = n0;
                    ax1 = bx1; bx1 = n1;
                }
            }
            if (G > 1) {
                // the shares of the x orders, added in order by the group's first warp
                red[(w * 2) * 32 + lane] = u[0];
                red[(w * 2 + 1) * 32 + lane] = u[1];
                __syncthreads();
                if (part == 0)
                    for (int k = 1; k < G; ++k) {
                        u[0] += red[((w + k) * 2) * 32 + lane];
                        u[1] += red[((w + k) * 2 + 1) * 32 + lane];
                    }
            }
            if (part == 0) {
                if (first + lane < cnt) uo[atom[0]] += u[0];
                if (first + lane + 32 < cnt) uo[atom[1]] += u[1];
            }
            if (G > 1) __syncthreads();
        }
        __syncthreads();                                // the coefficients are free again
    }
}

// The cell of a tile, by bisection of the tiles' prefix sums.
__device__ __forceinline__ int cell_of_tile(const uint32_t* first, int cells, uint32_t tile)
{
    int lo = 0, hi = cells;                    // first[lo] <= tile < first[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (first[mid] <= tile) lo = mid; else hi = mid;
    }
    return lo;
}

// ---- near pairs --------------------------------------------------------------------------

// The sources of the last level with near images of one near cell, 32 at a time;
// F(tree piece, box) for each.
template <class F>
__device__ __forceinline__ void for_near(const TreeArgs& a, int cell, F f)
{
    const int lane = threadIdx.x & 31;
    const uint64_t all = full_box(a.images);
    const LevelArgs& v = a.lv[a.total - 1];
    // boxes by final cell on the levels summed at the atoms, by the last level's
    // cell where there are none
    const int row = a.total > a.levels ? cell : cell / (a.cells_n / a.cells_s);
    const uint64_t* own = cell < a.cells_n ? a.near + v.near0 + (int64_t)row * v.np : nullptr;
    for (int base = 0; base < v.np; base += 32) {
        uint64_t w = 0;
        if (base + lane < v.np) w = own ? own[base + lane] : all;
        unsigned todo = __ballot_sync(0xffffffffu, w != 0);
        while (todo) {
            const int b = __ffs(todo) - 1;
            todo &= todo - 1;
            f(a.pieces[a.list[v.list0 + base + b]], ImgBox(__shfl_sync(0xffffffffu, w, b)));
        }
    }
}

// One warp: 32 / near_split atoms of one near cell (or atoms outside the grid,
// which take every image), lanes of an atom splitting the images of each
// piece (line) or the loopons of each source.
template <int kKind>
__global__ void __launch_bounds__(32 * kWarps, 4) tree_near_sum_kernel(const TreeArgs a)
{
    const int lane = threadIdx.x & 31;
    const uint32_t w = blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (w >= a.near_tile[a.cells_n + 1]) return;
    const int cell = cell_of_tile(a.near_tile, a.cells_n + 1, w);
    const int split = a.near_split, part = lane % split;
    const uint32_t s1 = a.start[cell < a.cells_n ? (cell + 1) * a.near_rr : a.cells_f + 1];
    const uint32_t slot = a.start[cell * a.near_rr] + (w - a.near_tile[cell]) * (32 / split) + lane / split;
    const bool valid = slot < s1;
    const int64_t atom = a.perm[valid ? slot : s1 - 1];
    const double px = a.f.x[atom], py = a.f.y[atom], pz = a.f.z[atom];
    double ux = 0.0, uy = 0.0, uz = 0.0;
    if constexpr (kKind == kLineKind) {
        const double cJK = a.f.cJ / a.f.cK;
        bool plane = false;
        for_near(a, cell, [&](const TreePiece& tp, const ImgBox& B) {
            const LinePiece& pc = *reinterpret_cast<const LinePiece*>(a.f.table + tp.piece);
            const LineSeg* seg = reinterpret_cast<const LineSeg*>(a.f.table + tp.rec);
            const int cnt = B.count();
            for (int idx = part; idx < cnt; idx += split) {
                int i, j, k;
                B.at(idx, i, j, k);
                line_piece_fp64(pc, seg, px - a.f.Lx * i, py - a.f.Ly * j, pz - a.f.Lz * k, cJK, ux, uy, uz, plane);
            }
        });
        if (__any_sync(0xffffffffu, plane)) {         // atoms in a loop's plane band: the reference's solid angle
            for_near(a, cell, [&](const TreePiece& tp, const ImgBox& B) {
                const LinePiece& pc = *reinterpret_cast<const LinePiece*>(a.f.table + tp.piece);
                const int cnt = B.count();
                for (int idx = part; idx < cnt; idx += split) {
                    int i, j, k;
                    B.at(idx, i, j, k);
                    if (plane)
                        line_piece_plane(pc, a.f.raw, px - a.f.Lx * i, py - a.f.Ly * j, pz - a.f.Lz * k, ux, uy, uz);
                }
            });
        }
    } else {
        // squares far enough from the cell for their equivalent loopons
        for (int l = a.levels; l < a.total && cell < a.cells_n; ++l) {
            const LevelArgs &v = a.lv[l], &u = a.lv[l - 1];
            const uint64_t* own = a.near + v.near0 + (int64_t)cell * v.np;
            const uint64_t* up = a.near + u.near0 + (int64_t)(l > a.levels ? cell : cell / (a.cells_n / a.cells_s)) * u.np;
            const int q2 = v.q * v.q;
            for (int base = 0; base < v.np; base += 32) {
                uint64_t wu = 0, wo = 0;
                if (base + lane < v.np) {
                    wu = up[a.up[v.list0 + base + lane]];
                    wo = own[base + lane];
                }
                unsigned todo = __ballot_sync(0xffffffffu, wu != 0 && wu != wo);
                while (todo) {
                    const int b = __ffs(todo) - 1;
                    todo &= todo - 1;
                    const ImgShell far(__shfl_sync(0xffffffffu, wu, b), __shfl_sync(0xffffffffu, wo, b));
                    const int self = a.list[v.list0 + base + b];
                    const TreePiece& tp = a.pieces[self];
                    const bool eq = uses_eq(v, tp, self);
                    const LooponRec* rec = eq ? v.eq + (int64_t)(base + b) * q2
                                              : reinterpret_cast<const LooponRec*>(a.f.table + tp.rec);
                    const int n = eq ? q2 : tp.terms;
                    const LooponPiece& pc = *reinterpret_cast<const LooponPiece*>(a.f.table + tp.piece);
                    const double qx = px - pc.cx, qy = py - pc.cy, qz = pz - pc.cz;
                    for (int idx = 0; idx < far.total; ++idx) {
                        int i, j, k;
                        far.at(idx, i, j, k);
                        loopon_terms_fp64<true>(pc, rec, n, qx - a.f.Lx * i, qy - a.f.Ly * j, qz - a.f.Lz * k,
                                                a.f.c2, ux, uy, uz, part, split);
                    }
                }
            }
        }
        // what is left: the squares' loopons one by one
        for_near(a, cell, [&](const TreePiece& tp, const ImgBox& B) {
            const LooponPiece& pc = *reinterpret_cast<const LooponPiece*>(a.f.table + tp.piece);
            const double qx = px - pc.cx, qy = py - pc.cy, qz = pz - pc.cz;
            const int cnt = B.count();
            for (int leaf = tp.leaf0; leaf < tp.leaf0 + tp.leaves; ++leaf) {
                const LooponRec* rec = reinterpret_cast<const LooponRec*>(a.f.table + a.pieces[leaf].rec);
                const int n = a.pieces[leaf].terms;
                for (int idx = 0; idx < cnt; ++idx) {
                    int i, j, k;
                    B.at(idx, i, j, k);
                    loopon_terms_fp64(pc, rec, n, qx - a.f.Lx * i, qy - a.f.Ly * j, qz - a.f.Lz * k, a.f.c2, ux, uy,
                                      uz, part, split);
                }
            }
        });
    }
    for (int o = split / 2; o > 0; o >>= 1) {
        ux += __shfl_xor_sync(0xffffffffu, ux, o);
        uy += __shfl_xor_sync(0xffffffffu, uy, o);
        uz += __shfl_xor_sync(0xffffffffu, uz, o);
    }
    if (valid && part == 0) {
        a.f.ux[atom] += ux;
        a.f.uy[atom] += uy;
        a.f.uz[atom] += uz;
    }
}

// ---- host: choice of the cells -----------------------------------------------------------

int order_for(double theta)
{
    for (int i = 0; i < kOrders; ++i)
        if (kOrderTheta[i] <= theta) return i;
    return -1;
}

// One loop (line: one piece) by the depths of its quadtree: half edge, radius
// and count of its squares there, and its terms.
struct Depth { double size, rho; int squares; };
struct Root { double terms; std::vector<Depth> depth; };

std::vector<Root> roots_of(const HostTable& T)
{
    std::vector<Root> out;
    std::vector<int> root(T.tree.size()), level(T.tree.size());
    for (size_t k = 0; k < T.tree.size(); ++k) {
        const TreePiece& t = T.tree[k];
        if (t.parent < 0) {
            root[k] = (int)out.size();
            level[k] = 0;
            out.push_back({ (double)t.terms, {} });
        } else {
            root[k] = root[t.parent];
            level[k] = level[t.parent] + 1;
        }
        std::vector<Depth>& d = out[root[k]].depth;
        if ((int)d.size() <= level[k]) d.push_back({ t.size, 0.0, 0 });
        Depth& e = d[level[k]];
        e.rho = std::max(e.rho, t.rho);
        e.squares++;
    }
    return out;
}

// The depth a cut takes a loop at.
const Depth& depth_at(const Root& r, double cut)
{
    size_t k = 0;
    while (k + 1 < r.depth.size() && r.depth[k].size > cut) ++k;
    return r.depth[k];
}

// What the choice below settled on, in FP64 operations.
struct Choice {
    double cost, node, near, fill;      // all of it; the nodes; the near pass, and the lanes it starts for one it uses
    double node_lanes, sources;         // lanes of the node kernel; sources that a warp of the near pass looks at
    double node_scans;                  // (warp, source) pairs of the node kernel
    int near_split, levels;
};

// Whether the chosen cells beat the plain sum.  The operation counts rank cells
// against cells; against the plain sum, what they leave out decides, so both
// sides are turned into times: the plain kernel's rounds of tiles; for the
// cells the warps that are missing to fill the GPU (16 an SM), the sources
// looked at, and the launches.  The weights are fitted to 414 random plans (500
// to 2.6 M atoms, 1 to 256 loops, 0 to 4 shells) on both sides of the line.  Of
// 190 that the operation counts alone sent to the cells 29 lost by it, up to 2.5
// times (16 loopon loops of R 6, 2 000 atoms, +-4: 7.2 ms plain, 17.7 by cells);
// by this rule 4 lose, by 1 to 4 and 12 %, and of the gains that it passes up one
// is above 10 % (22 %: 32 loopon loops of R 7, 1.1 M atoms, no images).
bool worth_cells(const Choice& c, bool line, int64_t n, double terms, double nimg, double e64, double us, int sm_count)
{
    const int S = choose_split(n, (int)nimg, sm_count * 2);
    const double tiles = std::ceil((double)n * S / kThreads);
    const double rounds = 0.5 * std::ceil(tiles / sm_count);          // two CTAs an SM; one alone has all of it
    const double plain = rounds * 2.0 * sm_count * kThreads * std::ceil(nimg / S) * terms * e64;
    const double full = 16.0 * sm_count;
    const double near_warps = (double)n * c.near_split / 32.0 * c.fill;
    const double node_part = c.node * (1.0 + (line ? 0.92 : 0.21) * full / (c.node_lanes / 32.0));
    const double near_part = c.near * (1.0 + (line ? 0.22 : 0.47) * full / near_warps);
    const double rest = std::max(0.0, c.cost - c.node - c.near * c.fill);
    if (line)
        return 30.0 * us + 0.573 * node_part + 1.05 * near_part + 1.06 * rest + 38.0 * us * c.levels <
               0.97 * (18.0 * us + 1.054 * plain);
    return 120.0 * us + 1.129 * node_part + 0.877 * near_part + 0.758 * rest +
               (0.00118 * c.node_scans + 0.00116 * near_warps * c.sources) * us <
           1.05 * (10.0 * us + 0.938 * plain);
}

} // namespace

void append_tree_pieces(HostTable& T)
{
    if (T.fp32 || T.chunks.empty()) { T.tree.clear(); return; }
    if (T.kind == kLineKind) {
        T.tree.clear();
        for (const Chunk& c : T.chunks) {
            const unsigned char* base = T.bytes.data() + c.offset;
            for (int i = 0; i < c.npieces; ++i) {
                LinePiece p;
                std::memcpy(&p, base + i * sizeof(p), sizeof(p));
                TreePiece t;
                std::memset(&t, 0, sizeof(t));
                t.piece = (uint32_t)(c.offset + i * sizeof(p));
                t.rec = (uint32_t)(c.offset + c.npieces * sizeof(p) + p.rec * sizeof(LineSeg));
                t.x = p.cx; t.y = p.cy; t.z = p.cz;
                t.rho = p.rho;
                t.terms = p.nseg;
                t.parent = -1;
                t.leaf0 = (int32_t)T.tree.size();
                t.leaves = 1;
                T.tree.push_back(t);
            }
        }
    }
    // a ball the far rule cannot use, or offsets past 32 bits: no cells
    bool ok = !T.tree.empty() && T.bytes.size() <= 0xFFFFFFFFull;
    for (const TreePiece& t : T.tree)
        ok = ok && std::isfinite(t.rho + std::fabs(t.x) + std::fabs(t.y) + std::fabs(t.z));
    if (!ok) { T.tree.clear(); return; }
    while (T.bytes.size() % 16) T.bytes.push_back(0);
    T.aux_tree = T.bytes.size();
    const unsigned char* s = reinterpret_cast<const unsigned char*>(T.tree.data());
    T.bytes.insert(T.bytes.end(), s, s + T.tree.size() * sizeof(TreePiece));
}

TreeShape tree_shape(const HostTable& T, int64_t n, const double box[3], int images, int sm_count)
{
    TreeShape S;
    if (!T.aux_tree || T.tree.empty() || n > 0x7FFFFFFF - 64) return S;
    const bool line = T.kind == kLineKind;
    // FP64 operations of a term, and a microsecond of the GPU in them (18.6e12
    // per second at the 75 % that the field kernels reach)
    const double e64 = line ? 78.0 : 34.0, us = 1.4e7;
    const double W = (double)(2 * images + 1), nimg = W * W * W;
    const std::vector<Root> roots = roots_of(T);
    double terms = 0.0;
    for (const Root& r : roots) terms += r.terms;
    const double all = terms * nimg;
    S.direct = (double)n * all * e64 + 5.0 * us;
    // the boxes' aspect: axes get m0 2^k cells
    const double lmin = std::min(box[0], std::min(box[1], box[2]));
    int m0[3];
    for (int d = 0; d < 3; ++d) m0[d] = (int)std::min(8.0, std::max(1.0, std::round(box[d] / lmin)));
    struct State {
        double cost, near, h, cells, cut;
        int a, o, prev, np;
        bool eq;
        std::vector<double> v;       // near images of a source, per loop
    };
    std::vector<State> st;
    constexpr int kDepth = 6;
    for (int a = 0; a < kDepth; ++a) {
        double h = 0.0, cells = 1.0;
        for (int d = 0; d < 3; ++d) {
            const int m = m0[d] << a;
            h = std::max(h, 0.5 * box[d] / m);
            cells *= m;
        }
        if (cells > 32768.0) break;
        for (int ob = 0; ob < kOrders * (line ? 1 : 2); ++ob) {
            const int o = ob % kOrders;
            const double q = kOrderQ[o], q3 = q * q * q, theta = kOrderTheta[o];
            if (cells * q3 > 1.5 * (double)n + 1e5) continue;
            State s;
            s.h = h; s.cells = cells; s.a = a; s.o = o; s.prev = -1; s.np = 0; s.eq = false;
            s.cut = ob < kOrders ? h : 0.5 * h;      // squares as large as the cells, or half
            s.near = 0.0;
            std::vector<double> far(roots.size());       // far terms per image pair of the loop
            for (size_t l = 0; l < roots.size(); ++l) {
                const Depth& d = depth_at(roots[l], s.cut);
                const bool leaf = &d == &roots[l].depth.back();
                const double raw = roots[l].terms / d.squares;
                const bool eq = !line && (!leaf || raw > q * q);
                double R = theta * h + d.rho;
                if (eq) R = std::max(R, h + theta * d.size);
                double v = 1.0;
                for (int k = 0; k < 3; ++k) v *= std::min(W, 2.0 * R / box[k]);
                s.v.push_back(v);
                s.near += v * roots[l].terms;
                far[l] = d.squares * (eq ? q * q : raw);
                s.eq = s.eq || eq;
                s.np += d.squares;
            }
            if (s.near > 0.97 * all || cells * s.np > 1.6e7) continue;
            double best = 1e300;
            for (int p = -1; p < (int)st.size(); ++p) {
                if (p >= 0 && (st[p].near < s.near * 1.02 || st[p].cut < s.cut || (st[p].a == a && st[p].o >= o)))
                    continue;
                double pairs = 0.0;
                for (size_t l = 0; l < roots.size(); ++l)
                    pairs += std::max(0.0, (p < 0 ? nimg : st[p].v[l]) - s.v[l]) * far[l];
                double c = (p < 0 ? 0.0 : st[p].cost) + pairs * cells * q3 * e64 * 1.1 + 3.0 * us +
                           cells * q3 * s.np * 0.5 + (line ? 0.0 : terms * q * q * 2.0 + 10.0 * us);
                if (p >= 0) {
                    const double qp = kOrderQ[st[p].o];
                    c += 3.0 * cells * (q * qp * qp * qp + q * q * qp * qp + q3 * qp) * 2.0 + 4.0 * us;
                }
                if (c < best) { best = c; s.prev = p; }
            }
            if (best >= 1e299) continue;
            int depth = 1;
            for (int p = s.prev; p >= 0; p = st[p].prev) ++depth;
            if (depth >= TreeShape::kMaxLevels) continue;
            s.cost = best;
            st.push_back(std::move(s));
        }
    }
    // what is left at the atoms of a last level: its near terms one by one, or
    // (loopons) first the squares that are far enough from the cell for their
    // equivalent loopons, by falling size and rising order
    struct Step { double cost, cut; int o, prev, np; bool eq; std::vector<double> v; };
    auto near_steps = [&](const State& p, double h, double cells, std::vector<Step>& steps, int& end) {
        auto rest = [&](const std::vector<double>& v) {
            double t = 0.0;
            for (size_t l = 0; l < roots.size(); ++l) t += v[l] * roots[l].terms;
            return (double)n * t * e64 * 1.1;
        };
        double least = rest(p.v);
        end = -1;
        if (line) return least;
        double smallest = 1e300;
        for (const Root& r : roots) smallest = std::min(smallest, r.depth.back().size);
        for (double cut = p.cut; cut > 0.5 * smallest; cut *= 0.5)
            for (int o = 0; o < kOrders; ++o) {
                const double q2 = (double)kOrderQ[o] * kOrderQ[o];
                Step s;
                s.cut = cut; s.o = o; s.prev = -1; s.np = 0; s.eq = false;
                s.cost = 1e300;
                std::vector<double> own(roots.size()), far(roots.size());
                for (size_t l = 0; l < roots.size(); ++l) {
                    const Depth& d = depth_at(roots[l], cut);
                    const bool leaf = &d == &roots[l].depth.back();
                    const bool eq = !leaf || roots[l].terms / d.squares > q2;
                    own[l] = 1e300;
                    far[l] = d.squares * q2;
                    s.np += d.squares;
                    if (!eq) continue;
                    s.eq = true;
                    own[l] = 1.0;
                    for (int k = 0; k < 3; ++k) own[l] *= std::min(W, 2.0 * (h + kOrderTheta[o] * d.size) / box[k]);
                }
                if (!s.eq || cells * s.np > 1.6e7) continue;
                for (int b = -1; b < (int)steps.size(); ++b) {
                    if (b >= 0 && steps[b].cut <= cut && steps[b].o >= o) continue;
                    const std::vector<double>& before = b < 0 ? p.v : steps[b].v;
                    double pairs = 0.0;
                    for (size_t l = 0; l < roots.size(); ++l) pairs += std::max(0.0, before[l] - own[l]) * far[l];
                    const double c = (b < 0 ? 0.0 : steps[b].cost) + (double)n * pairs * e64 * 1.13 +
                                     (double)n * s.np * 0.5 + terms * q2 * 2.0 + 15.0 * us;
                    if (c < s.cost) { s.cost = c; s.prev = b; }
                }
                int depth = 1;
                for (int b = s.prev; b >= 0; b = steps[b].prev) ++depth;
                if (depth > 6) continue;
                s.v = s.prev < 0 ? p.v : steps[s.prev].v;
                for (size_t l = 0; l < roots.size(); ++l) s.v[l] = std::min(s.v[l], own[l]);
                steps.push_back(std::move(s));
                const double c = steps.back().cost + rest(steps.back().v);
                if (c < least) { least = c; end = (int)steps.size() - 1; }
            }
        return least;
    };
    double best = S.direct;
    int pick = -1, pick_r = 1, pick_q = 0, pick_end = -1;
    Choice chosen = {};
    std::vector<Step> pick_steps;
    for (int p = 0; p < (int)st.size(); ++p) {
        const double theta = kOrderTheta[st[p].o];
        if (st[p].cost >= best) continue;
        int levels = 1, end = -1;
        for (int b = st[p].prev; b >= 0; b = st[b].prev) ++levels;
        if (levels + 6 > TreeShape::kMaxLevels) continue;
        for (int r = 1; r <= kMaxRefine; r *= 2) {
            const double cells = st[p].cells * r * r * r;
            if (cells > (line ? kMaxCells : 32768)) break;
            const int o = order_for((theta - 1.0) * r + 1.0);
            const double q = kOrderQ[o], q3 = q * q * q, qp = kOrderQ[st[p].o];
            if (kOrderQ[o] > kMaxFinalQ) continue;
            const double atoms = std::max(1.0, (double)n / cells);
            const double fill = (std::floor(atoms / 64.0) + 1.0) * 64.0 / atoms;
            std::vector<Step> steps;
            const double near = near_steps(st[p], st[p].h / r, cells, steps, end);
            const double part = line ? 1.0 : (std::floor(atoms / 16.0) + 1.0) * 16.0 / atoms;     // partly filled warps
            const double c = st[p].cost + near * part + (double)n * st[p].np * 0.5 +
                             3.0 * cells * ((q * qp * qp * qp + q * q * qp * qp) / r + q3 * qp) * 2.5 +
                             (double)n * 3.0 * q3 * 2.0 * std::min(fill, 64.0) + 60.0 * us + (double)n * 60.0;
            if (c < best) {
                best = c; pick = p; pick_r = r; pick_q = o; pick_end = end;
                pick_steps = steps;
                chosen.near = near;
                chosen.fill = part;
            }
        }
    }
    S.cost = best;
    if (pick < 0) return S;
    std::vector<int> chain;
    for (int p = pick; p >= 0; p = st[p].prev) chain.push_back(p);
    std::reverse(chain.begin(), chain.end());
    S.levels = (int)chain.size();
    // far images per source of a level, and those that each lane would sum if all
    // lanes of the GPU (16 warps an SM) shared them evenly
    auto pairs = [&](int k) {
        double p = 0.0;
        for (size_t l = 0; l < roots.size(); ++l) p += (k ? st[chain[k - 1]].v[l] : nimg) - st[chain[k]].v[l];
        return p;
    };
    const double gpu_lanes = 16.0 * 32.0 * sm_count;
    double fair = 0.0;
    for (int k = 0; k < S.levels; ++k) {
        const double q = kOrderQ[st[chain[k]].o];
        fair += st[chain[k]].cells * q * q * q * pairs(k) / gpu_lanes;
    }
    // lanes per node of a line level: many images per source for each lane, or their
    // uneven shares idle lanes (BCC 61 x 47 x 33, 9 loops, +-3: 8.69 ms with 6 images
    // a lane, 8.27 with 48, 8.81 with one lane everywhere).  Where some lane's chain
    // is over twice an even share, a small sum waits for it: then the level with the
    // longest chain gets more lanes until none is over 1.8 shares (32 loops of R 13,
    // 11 206 atoms, +-2: 9.7 ms without, 5.8 with; every level to 1.5 shares: sums of
    // 30 000 atoms lose 4 to 9 %; only levels over two shares: 10 % of a sum whose
    // next level is just below)
    std::vector<int> lanes((size_t)S.levels, 1);
    auto longest = [&] {
        int worst = 0;
        for (int k = 1; k < S.levels; ++k)
            if (pairs(k) / lanes[k] > pairs(worst) / lanes[worst]) worst = k;
        return worst;
    };
    if (line) {
        const double loops = (double)roots.size();
        for (int k = 0; k < S.levels; ++k)
            while (lanes[k] < 32 && pairs(k) / loops >= 48.0 * lanes[k]) lanes[k] *= 2;
        int k = longest();
        if (pairs(k) / lanes[k] > 2.0 * fair)
            for (; pairs(k) / lanes[k] > 1.8 * fair && lanes[k] < 32 && pairs(k) / loops >= 4.0 * lanes[k]; k = longest())
                lanes[k] *= 2;
    }
    for (int k = 0; k < S.levels; ++k) {
        const State& s = st[chain[k]];
        for (int d = 0; d < 3; ++d) S.m[k][d] = m0[d] << s.a;
        S.q[k] = kOrderQ[s.o];
        S.theta[k] = kOrderTheta[s.o];
        S.cut[k] = s.cut;
        S.np[k] = s.np;
        S.eq[k] = s.eq;
        const int q3 = S.q[k] * S.q[k] * S.q[k];
        int split = lanes[k];
        if (!line)
            while (split < 8 && s.cells * q3 * split < 300000.0) split *= 2;
        chosen.node_lanes += s.cells * q3 * split;
        chosen.node_scans += s.cells * q3 * split / 32.0 * s.np;
        S.split[k] = split;
    }
    S.total = S.levels;
    std::vector<int> tail;
    for (int b = pick_end; b >= 0; b = pick_steps[b].prev) tail.push_back(b);
    for (auto it = tail.rbegin(); it != tail.rend(); ++it, ++S.total) {
        const Step& s = pick_steps[*it];
        for (int d = 0; d < 3; ++d) S.m[S.total][d] = S.m[S.levels - 1][d] * pick_r;
        S.q[S.total] = kOrderQ[s.o];
        S.theta[S.total] = kOrderTheta[s.o];
        S.cut[S.total] = s.cut;
        S.np[S.total] = s.np;
        S.eq[S.total] = s.eq;
        S.split[S.total] = 1;
    }
    for (int d = 0; d < 3; ++d) S.mf[d] = S.m[S.levels - 1][d] * pick_r;
    S.qf = kOrderQ[pick_q];
    S.fine = !line;
    // lanes per atom: as many as the near images (or the loopons) feed, while the
    // atoms alone do not fill the GPU several times
    const double per_atom = st[pick].near / terms;
    if (line) while (S.near_split < 32 && per_atom >= 4.0 * S.near_split && n * S.near_split < 600000) S.near_split *= 2;
    else while (S.near_split < 8 && n * S.near_split < 600000) S.near_split *= 2;
    chosen.cost = best;
    chosen.node = st[pick].cost;
    chosen.levels = S.levels;
    chosen.near_split = S.near_split;
    chosen.sources = st[pick].np;
    for (int k = S.levels; k < S.total; ++k) chosen.sources += S.np[k];
    S.use = worth_cells(chosen, line, n, terms, nimg, e64, us, sm_count);
    return S;
}

// ---- host: scratch and launches ----------------------------------------------------------

namespace {

// Shared memory of one CTA for parent cells of qp nodes per axis (and rz final
// cells along z).
template <int QC>
constexpr size_t down_smem(int qp)
{
    return ((size_t)(qp > QC ? QC * qp * qp : QC * QC * QC) + (size_t)QC * QC * qp + 3 * (size_t)qp * QC) * sizeof(double);
}
template <int QC>
constexpr size_t leaf_smem(int qp, int rz)
{
    return ((size_t)QC * QC * padded(QC) + padded(QC * QC * qp) +
            padded(QC * qp * qp > 8 * 64 ? QC * qp * qp : 8 * 64) + (size_t)(2 + rz) * qp * padded(QC)) * sizeof(double);
}

// A kernel's limit of dynamic shared memory holds for the whole process, so it
// is set to the largest size of any shape, never to one call's: another thread
// may launch a larger one in between.
template <int QC>
cudaError_t down(const TreeArgs& a, int t, int cells, cudaStream_t s)
{
    constexpr size_t most = down_smem<QC>(kMaxQ);
    static_assert(most <= kSmemLimit, "one CTA's shared memory");
    const cudaError_t e = cudaFuncSetAttribute(tree_down_kernel<QC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)most);
    if (e != cudaSuccess) return e;
    tree_down_kernel<QC><<<dim3((unsigned)cells, 3), 256, down_smem<QC>(a.lv[t - 1].q), s>>>(a, t);
    return cudaGetLastError();
}

template <int QC>
cudaError_t leaf(const TreeArgs& a, cudaStream_t s)
{
    constexpr size_t most = leaf_smem<QC>(kMaxQ, kMaxRefine);
    static_assert(most <= kSmemLimit, "one CTA's shared memory");
    const cudaError_t e = cudaFuncSetAttribute(tree_leaf_kernel<QC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)most);
    if (e != cudaSuccess) return e;
    tree_leaf_kernel<QC><<<dim3((unsigned)(a.cells_f / a.rf[2]), 3), 256, leaf_smem<QC>(a.lv[a.levels - 1].q, a.rf[2]),
                           s>>>(a);
    return cudaGetLastError();
}

cudaError_t down_any(const TreeArgs& a, int t, int cells, cudaStream_t s)
{
    switch (a.lv[t].q) {
    case 9:  return down<9>(a, t, cells, s);
    case 10: return down<10>(a, t, cells, s);
    case 11: return down<11>(a, t, cells, s);
    case 12: return down<12>(a, t, cells, s);
    case 13: return down<13>(a, t, cells, s);
    case 15: return down<15>(a, t, cells, s);
    case 17: return down<17>(a, t, cells, s);
    case 19: return down<19>(a, t, cells, s);
    default: return down<21>(a, t, cells, s);
    }
}

cudaError_t leaf_any(const TreeArgs& a, cudaStream_t s)
{
    switch (a.qf) {
    case 9:  return leaf<9>(a, s);
    case 10: return leaf<10>(a, s);
    case 11: return leaf<11>(a, s);
    case 12: return leaf<12>(a, s);
    default: return leaf<13>(a, s);
    }
}

} // namespace

int launch_tree(const FieldArgs& f, const HostTable& T, const TreeShape& S, int sm_count,
                cudaStream_t s, int* launches, std::string& err)
{
    *launches = 0;
    OutsideCapture relaxed;
    TreeArgs a;
    std::memset(&a, 0, sizeof(a));
    a.f = f;
    a.pieces = reinterpret_cast<const TreePiece*>(f.table + T.aux_tree);
    a.nodes = (int32_t)T.tree.size();
    a.levels = S.levels;
    a.total = S.total;
    a.images = f.images;
    a.near_split = S.near_split;
    a.qf = S.qf;
    // scratch layout
    size_t at = 0;
    auto take = [&](size_t bytes) { const size_t o = at; at += (bytes + 255) & ~size_t(255); return o; };
    const size_t o_box = take(8 * sizeof(unsigned long long));
    int64_t lcells = 0, tiles = 0;
    size_t o_val[TreeShape::kMaxLevels], o_eq[TreeShape::kMaxLevels], mats = 0;
    int64_t sources = 0;
    int lvcells[TreeShape::kMaxLevels];
    for (int k = 0; k < S.total; ++k) {
        LevelArgs& v = a.lv[k];
        const bool nodes = k < S.levels;
        int64_t cells = 1;
        for (int d = 0; d < 3; ++d) {
            v.m[d] = S.m[k][d];
            v.r[d] = k ? S.m[k][d] / S.m[k - 1][d] : 1;
            cells *= v.m[d];
        }
        v.q = S.q[k];
        v.q3 = v.q * v.q * v.q;
        v.split = S.split[k];
        v.theta = S.theta[k];
        v.cut = S.cut[k];
        v.np = S.np[k];
        v.near0 = a.near_size;
        v.list0 = sources;
        a.near_size += cells * v.np;
        sources += v.np;
        o_eq[k] = !S.eq[k] ? 0 : take((size_t)v.np * v.q * v.q * sizeof(LooponRec));
        if (!nodes) continue;
        v.tiles = (v.q3 * v.split + 31) / 32;
        v.tile0 = tiles;
        v.cell0 = lcells;
        tiles += cells * v.tiles;
        lcells += cells;
        lvcells[k] = (int)cells;
        o_val[k] = take((size_t)cells * 3 * v.q3 * sizeof(double));
    }
    a.level_cells = lcells;
    int64_t cf = 1;
    for (int d = 0; d < 3; ++d) {
        a.mf[d] = S.mf[d];
        a.rf[d] = S.mf[d] / S.m[S.levels - 1][d];
        cf *= a.mf[d];
    }
    a.cells_s = lvcells[S.levels - 1];
    a.cells_f = (int32_t)cf;
    a.near_rr = S.fine ? 1 : a.rf[0] * a.rf[1] * a.rf[2];
    a.cells_n = a.cells_f / a.near_rr;
    for (int t = 1; t <= S.levels; ++t) {
        const bool last = t == S.levels;
        const int qp = a.lv[t - 1].q, qc = last ? a.qf : a.lv[t].q;
        for (int d = 0; d < 3; ++d) {
            a.mat_off[t][d] = (int32_t)mats;
            mats += (size_t)(last ? a.rf[d] : a.lv[t].r[d]) * qp * qc;
        }
    }
    const size_t o_near = take((size_t)a.near_size * sizeof(uint64_t));
    const size_t o_list = take((size_t)sources * 2 * sizeof(int32_t));
    const size_t o_pos = take((size_t)S.total * a.nodes * sizeof(int32_t));
    const size_t o_occ = take((size_t)lcells);
    const size_t o_start = take((size_t)(cf + 2) * sizeof(uint32_t));
    const size_t o_ntile = take((size_t)(a.cells_n + 2) * sizeof(uint32_t));
    a.sort_tiles = (int32_t)((f.n + kSortTile - 1) / kSortTile);
    const size_t o_sort = take((size_t)f.n * 4 * sizeof(uint32_t));
    const size_t o_digits = take(((size_t)a.sort_tiles * 256 + 256) * sizeof(uint32_t));
    const size_t o_mat = take(mats * sizeof(double));
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); return DISCO_OK; }
    cudaMemPool_t pool = scratch_pool(dev);
    if (!pool) return DISCO_OK;
    unsigned char* ws = nullptr;
    if (cudaMallocFromPoolAsync(reinterpret_cast<void**>(&ws), at, pool, s) != cudaSuccess) {
        cudaGetLastError();
        return DISCO_OK;
    }
    a.box = reinterpret_cast<unsigned long long*>(ws + o_box);
    int most = 0;
    for (int k = 0; k < S.total; ++k) {
        if (k < S.levels) a.lv[k].val = reinterpret_cast<double*>(ws + o_val[k]);
        if (o_eq[k]) a.lv[k].eq = reinterpret_cast<LooponRec*>(ws + o_eq[k]);
        most = std::max(most, S.np[k]);
    }
    a.list = reinterpret_cast<int32_t*>(ws + o_list);
    a.up = a.list + sources;
    a.pos = reinterpret_cast<int32_t*>(ws + o_pos);
    a.near = reinterpret_cast<uint64_t*>(ws + o_near);
    a.occ = ws + o_occ;
    a.start = reinterpret_cast<uint32_t*>(ws + o_start);
    a.near_tile = reinterpret_cast<uint32_t*>(ws + o_ntile);
    for (int b = 0; b < 2; ++b) {
        a.key[b] = reinterpret_cast<uint32_t*>(ws + o_sort) + (size_t)b * f.n;
        a.idx[b] = reinterpret_cast<int32_t*>(ws + o_sort) + (size_t)(2 + b) * f.n;
    }
    a.digits = reinterpret_cast<uint32_t*>(ws + o_digits);
    a.digit_total = a.digits + (size_t)a.sort_tiles * 256;
    a.mat = reinterpret_cast<double*>(ws + o_mat);

    const bool line = T.kind == kLineKind;
    // Atoms away from the box (unwrapped trajectories) take every image in the
    // near pass, beside the others.  Where nearly all of them are away, the nodes
    // still work for all atoms, on cells as large as the few inside spread, and
    // the plain kernel is faster: 864 k atoms, 5 % inside, 8 line loops, +-2: 121 ms
    // against 137; 53 k atoms, 4 loopon loops, 5 %: 16.3 against 18.3, none: 16.3
    // against 18.7 (line loops, none: 115 ms in the near pass, 120 plain).
    a.from = line ? 1 : 0;
    a.least = line ? 8 : 4;
    auto queue = [&]() -> cudaError_t {
        const int64_t sweep = std::min<int64_t>((f.n + 255) / 256, (int64_t)sm_count * 8);
        cudaError_t e;
        int passes = 0;
        tree_init_kernel<<<(unsigned)std::min<int64_t>((lcells + 255) / 256, sm_count * 4), 256, 0, s>>>(a);
        tree_box_kernel<<<(unsigned)sweep, 256, 0, s>>>(a);
        const unsigned nt = (unsigned)a.sort_tiles;
        int in = 0;
        for (int shift = 0; shift == 0 || (cf >> shift) > 0; shift += 8) {
            if (shift == 0) {
                tree_digits_kernel<true><<<nt, kSortThreads, 0, s>>>(a, nullptr, shift);
                tree_digit_scan_kernel<<<256, 256, 0, s>>>(a);
                tree_reorder_kernel<true><<<nt, kSortThreads, 0, s>>>(a, a.key[0], nullptr, a.key[1], a.idx[1], shift);
            } else {
                tree_digits_kernel<false><<<nt, kSortThreads, 0, s>>>(a, a.key[in], shift);
                tree_digit_scan_kernel<<<256, 256, 0, s>>>(a);
                tree_reorder_kernel<false><<<nt, kSortThreads, 0, s>>>(a, a.key[in], a.idx[in], a.key[in ^ 1],
                                                                       a.idx[in ^ 1], shift);
            }
            in ^= 1;
            ++passes;
        }
        a.perm = a.idx[in];
        tree_starts_kernel<<<(unsigned)((f.n + 256) / 256), 256, 0, s>>>(a, a.key[in]);
        tree_scan_kernel<<<1, 1024, 0, s>>>(a);
        tree_list_kernel<<<(unsigned)S.total, 1024, 0, s>>>(a);
        tree_near_kernel<<<(unsigned)std::min<int64_t>((a.near_size + 255) / 256, (int64_t)sm_count * 16), 256, 0, s>>>(a);
        if (!line) tree_equivalent_kernel<<<dim3((unsigned)most, (unsigned)S.total), kEqThreads, 0, s>>>(a);
        tree_matrix_kernel<<<dim3((unsigned)S.levels, 3, 8), 128, 0, s>>>(a);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        const unsigned nodes = (unsigned)((tiles + kWarps - 1) / kWarps);
        if (line) tree_node_kernel<kLineKind><<<nodes, 32 * kWarps, 0, s>>>(a);
        else tree_node_kernel<kLooponKind><<<nodes, 32 * kWarps, 0, s>>>(a);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        for (int t = 1; t < S.levels; ++t)
            if ((e = down_any(a, t, lvcells[t], s)) != cudaSuccess) return e;
        if ((e = leaf_any(a, s)) != cudaSuccess) return e;
        const int64_t ntiles = f.n * S.near_split / 32 + a.cells_n + 2;
        const unsigned ngrid = (unsigned)((ntiles + kWarps - 1) / kWarps);
        if (line) tree_near_sum_kernel<kLineKind><<<ngrid, 32 * kWarps, 0, s>>>(a);
        else tree_near_sum_kernel<kLooponKind><<<ngrid, 32 * kWarps, 0, s>>>(a);
        // init, box, three per sorting pass, starts, scan, list, near, (equivalent),
        // matrix, node, one down per further level, leaf, near_sum
        *launches = 2 + 3 * passes + 4 + (line ? 0 : 1) + 2 + (S.levels - 1) + 2;
        return cudaGetLastError();
    };
    const cudaError_t e = queue();
    int plain = DISCO_OK;
    if (e == cudaSuccess) {
        FieldArgs out = a.f;
        out.near_mode = 3;
        out.near_count = reinterpret_cast<unsigned int*>(a.box + 7);
        plain = launch_field(out, T.kind, false, sm_count, 0, 0, s, err);
        ++*launches;
    }
    const cudaError_t ef = cudaFreeAsync(ws, s);
    if (e != cudaSuccess) { err = cudaGetErrorString(e); return DISCO_ECUDA; }
    if (ef != cudaSuccess) { err = cudaGetErrorString(ef); return DISCO_ECUDA; }
    return plain;
}

} // namespace disco
