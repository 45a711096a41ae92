// Displacement-sum kernels (sm_100a) and their table builder / launcher.
//
// What is summed is the reference's: for every atom, every loop, every periodic
// image and every segment (Barnett line integral, Code/barnett.hpp:44-107) or
// loopon (Kroupa pair term, Code/kroupa.hpp:52-73); Code/backend_cpu.cpp:28-99
// is the loop nest.  How it is summed is B200-specific:
//   - one launch covers all loops and all images (the reference launches and
//     synchronises once per loop, Code/backend_cuda.cu:646-704);
//   - persistent CTAs walk atom tiles; the loop table is cut into chunks that a
//     single thread stages into shared memory with bulk async copies completed
//     on an mbarrier (double-buffered when the table does not fit at once), and
//     every warp reads each record as a shared-memory broadcast;
//   - image shifts are enumerated in registers; when there are too few atoms
//     to fill the GPU, S consecutive lanes share an atom and split its images,
//     and a fixed-order warp butterfly sums their parts;
//   - everything that does not depend on the atom (unit tangent, length,
//     w = b x t per segment; m.l, n.l per loopon; Kroupa prefactors) is
//     computed once on the host;
//   - line method: the solid angle of the fan is the argument of the running
//     complex product of the Van Oosterom-Strackee terms (one atan2 per atom,
//     piece and image instead of one per segment); the line integrals use one
//     rsqrt per vertex, J0 = ln((RA+RB+L)/(RA+RB-L)) and K0 d^2 = sB/RB - sA/RA,
//     all cancellation-free in the product that enters u.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>

#include "common.cuh"
#include "field.cuh"
#include "field_device.cuh"

namespace disco {

// Appends the raw vertex triplets to the table bytes (16-byte aligned).
void append_raw(HostTable& T, const std::vector<double>& raw)
{
    while (T.bytes.size() % 16) T.bytes.push_back(0);
    T.aux_raw = T.bytes.size();
    const unsigned char* s = reinterpret_cast<const unsigned char*>(raw.data());
    T.bytes.insert(T.bytes.end(), s, s + raw.size() * sizeof(double));
}

namespace {

// Quadtree order of one loop's loopons: squares of the loop's plane halved
// until a leaf holds about 200, numbered along the Z curve, so that every
// square's loopons are consecutive.  order[k] = the loopon at place k;
// nodes: the squares that hold any, parents first (parent, leaf0, leaves and
// terms relative to this loop; `rec` holds a leaf's first place).  False where
// the loopons do not lie in one plane normal to n (or are not finite): no tree.
bool quadtree(const disco_loop& lp, std::vector<int32_t>& order, std::vector<TreePiece>& nodes)
{
    const int np = lp.n_loopons;
    const disco_loop_phys& ph = lp.phys;
    double n[3] = { ph.nx, ph.ny, ph.nz };
    const double nn = std::sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
    if (!(nn > 0.5) || !std::isfinite(nn)) return false;
    for (double& v : n) v /= nn;
    int ax = 0;
    for (int d = 1; d < 3; ++d)
        if (std::fabs(n[d]) < std::fabs(n[ax])) ax = d;
    double e1[3] = { -n[ax] * n[0], -n[ax] * n[1], -n[ax] * n[2] };      // axis ax, made normal to n
    e1[ax] += 1.0;
    const double l1 = std::sqrt(e1[0] * e1[0] + e1[1] * e1[1] + e1[2] * e1[2]);
    for (double& v : e1) v /= l1;
    const double e2[3] = { n[1] * e1[2] - n[2] * e1[1], n[2] * e1[0] - n[0] * e1[2], n[0] * e1[1] - n[1] * e1[0] };
    const double o[3] = { lp.x[0], lp.y[0], lp.z[0] };
    std::vector<double> a((size_t)np), b((size_t)np);
    double lo[2] = { 0, 0 }, hi[2] = { 0, 0 }, off = 0.0, big = 0.0;
    for (int k = 0; k < np; ++k) {
        const double r[3] = { lp.x[k] - o[0], lp.y[k] - o[1], lp.z[k] - o[2] };
        a[k] = e1[0] * r[0] + e1[1] * r[1] + e1[2] * r[2];
        b[k] = e2[0] * r[0] + e2[1] * r[1] + e2[2] * r[2];
        off = std::max(off, std::fabs(n[0] * r[0] + n[1] * r[1] + n[2] * r[2]));
        big = std::max(big, std::fabs(lp.x[k]) + std::fabs(lp.y[k]) + std::fabs(lp.z[k]));
        lo[0] = std::min(lo[0], a[k]); hi[0] = std::max(hi[0], a[k]);
        lo[1] = std::min(lo[1], b[k]); hi[1] = std::max(hi[1], b[k]);
    }
    // rounding of the positions' own sums, nothing more
    if (!std::isfinite(big) || !(off <= 1e-14 * (big + 10.0))) return false;
    const double half = 0.5 * std::max(hi[0] - lo[0], hi[1] - lo[1]) * (1.0 + 1e-12) + 1e-9;
    const double mid[2] = { 0.5 * (lo[0] + hi[0]), 0.5 * (lo[1] + hi[1]) };
    int depth = 0;
    while (depth < 8 && (double)np / std::ldexp(1.0, 2 * depth) > 256.0) ++depth;
    const int side = 1 << depth;
    // extents of the squares of every depth, the finest from the loopons
    struct Extent { double l[2], h[2]; };
    std::vector<std::vector<Extent>> ext((size_t)depth + 1);
    for (int t = 0; t <= depth; ++t) ext[t].assign((size_t)1 << (2 * t), { { 1e300, 1e300 }, { -1e300, -1e300 } });
    auto widen = [](Extent& e, const double (&l)[2], const double (&h)[2]) {
        for (int d = 0; d < 2; ++d) { e.l[d] = std::min(e.l[d], l[d]); e.h[d] = std::max(e.h[d], h[d]); }
    };
    std::vector<int32_t> spread((size_t)side, 0);                // bit t of a number at bit 2 t
    for (int i = 0; i < side; ++i)
        for (int t = 0; t < depth; ++t) spread[i] |= (i >> t & 1) << (2 * t);
    std::vector<int32_t> code((size_t)np), first((size_t)side * side + 1, 0);
    for (int k = 0; k < np; ++k) {
        const int i = std::min(side - 1, std::max(0, (int)((a[k] - mid[0] + half) / (2.0 * half) * side)));
        const int j = std::min(side - 1, std::max(0, (int)((b[k] - mid[1] + half) / (2.0 * half) * side)));
        const int c = spread[i] << 1 | spread[j];
        code[k] = c;
        ++first[c + 1];
        const double p[2] = { a[k], b[k] };
        widen(ext[depth][c], p, p);
    }
    for (int t = depth; t > 0; --t)
        for (size_t c = 0; c < ext[t].size(); ++c) widen(ext[t - 1][c >> 2], ext[t][c].l, ext[t][c].h);
    for (int c = 0; c < side * side; ++c) {
        if (first[c + 1] > kMaxLooponPiece) return false;
        first[c + 1] += first[c];
    }
    order.resize((size_t)np);
    std::vector<int32_t> at(first.begin(), first.end() - 1);
    for (int k = 0; k < np; ++k) order[at[code[k]]++] = k;
    // squares that hold loopons, from the whole loop down
    std::vector<int32_t> above(1, -1), mine;
    for (int t = 0; t <= depth; ++t) {
        const int cells = 1 << (2 * t), span = 1 << (2 * (depth - t));
        mine.assign((size_t)cells, -1);
        for (int c = 0; c < cells; ++c) {
            const int k0 = first[c * span], k1 = first[(c + 1) * span];
            if (k0 == k1) continue;
            const double (&l)[2] = ext[t][c].l, (&h)[2] = ext[t][c].h;
            TreePiece q;
            std::memset(&q, 0, sizeof(q));
            const double ca = 0.5 * (l[0] + h[0]), cb = 0.5 * (l[1] + h[1]);
            q.x = o[0] + ca * e1[0] + cb * e2[0];
            q.y = o[1] + ca * e1[1] + cb * e2[1];
            q.z = o[2] + ca * e1[2] + cb * e2[2];
            q.a1 = 0.5 * (h[0] - l[0]);
            q.a2 = 0.5 * (h[1] - l[1]);
            q.rho = std::sqrt(q.a1 * q.a1 + q.a2 * q.a2) * (1.0 + 1e-12) + 1e-9;
            for (int d = 0; d < 3; ++d) { q.e1[d] = e1[d]; q.e2[d] = e2[d]; }
            q.size = half / (1 << t);
            q.terms = k1 - k0;
            q.rec = (uint32_t)k0;
            q.parent = t ? above[c >> 2] : -1;
            q.leaf0 = -1;
            mine[c] = (int32_t)nodes.size();
            nodes.push_back(q);
        }
        above.swap(mine);
    }
    // leaves are the last depth, in order: count them up the tree
    const int total = (int)nodes.size();
    for (int k = total - 1; k >= 0; --k) {
        TreePiece& q = nodes[k];
        if (q.leaves == 0) { q.leaf0 = k; q.leaves = 1; }
        if (q.parent >= 0) {
            TreePiece& up = nodes[q.parent];
            up.leaf0 = q.leaf0;                 // children come last to first
            up.leaves += q.leaves;
        }
    }
    return true;
}

} // namespace

int build_table(const disco_loop* loops, int nloops, int kind, int precision, double nu,
                HostTable& T, std::string& err, uint32_t stage_cap, bool tree)
{
    T = HostTable();
    T.kind = kind;
    T.fp32 = precision == DISCO_FP32C;
    T.loop_evals.assign((size_t)nloops, 0.0);
    if (T.fp32) { err = "FP32 tables are built by build_table_fp32"; return DISCO_EINVAL; }
    const double k1 = 1.0 / (8.0 * M_PI * (1.0 - nu));          // Code/kroupa.hpp:38-41
    if (kind == kLineKind) {
        PieceList<LinePiece, LineSeg> L;
        std::vector<double> raw;
        for (int l = 0; l < nloops; ++l) {
            const disco_loop& lp = loops[l];
            if (!lp.line) continue;
            const int nv = lp.n_vertices;
            if (nv <= 0) continue;
            if (!lp.vx || !lp.vy || !lp.vz) { err = "line loop without vertices"; return DISCO_EINVAL; }
            // b = (|b|_x m_x, |b|_y m_y, |b|_z m_z): Code/backend_cpu.cpp:44-45
            const double bx = lp.phys.bx * lp.phys.mx, by = lp.phys.by * lp.phys.my,
                         bz = lp.phys.bz * lp.phys.mz;
            T.loop_evals[l] = nv;
            T.n_segments += nv;
            for (int k0 = 0; k0 < nv; k0 += kMaxLinePiece) {
                const int k1e = std::min(nv, k0 + kMaxLinePiece);
                LinePiece p;
                std::vector<LineSeg> recs;
                make_line_piece(lp, k0, k1e, bx, by, bz, k1, p, recs, raw);
                L.pieces.push_back(p);
                L.recs.push_back(std::move(recs));
            }
        }
        pack_chunks(L, T, stage_cap);
        if (!T.chunks.empty()) append_raw(T, raw);
    } else {
        PieceList<LooponPiece, LooponRec> L;
        // tree pieces; a leaf's `piece` and `rec` hold its table piece and its
        // place in it until the chunks have their offsets
        std::vector<TreePiece> nodes, mine;
        std::vector<int32_t> order;
        for (int l = 0; l < nloops; ++l) {
            const disco_loop& lp = loops[l];
            if (lp.line) continue;
            const int np = lp.n_loopons;
            if (np <= 0) continue;
            if (!lp.x || !lp.y || !lp.z) { err = "loopon loop without loopons"; return DISCO_EINVAL; }
            const disco_loop_phys& ph = lp.phys;
            T.loop_evals[l] = np;
            T.n_loopons += np;
            double cx = 0.0, cy = 0.0, cz = 0.0;
            for (int k = 0; k < np; ++k) { cx += lp.x[k]; cy += lp.y[k]; cz += lp.z[k]; }
            cx /= np; cy /= np; cz /= np;
            mine.clear();
            order.clear();
            if (tree && !quadtree(lp, order, mine)) { tree = false; order.clear(); mine.clear(); }
            // a piece ends at kMaxLooponPiece loopons, with a tree before the
            // leaf that would pass them
            size_t leaf = 0;
            while (leaf < mine.size() && mine[leaf].leaf0 != (int32_t)leaf) ++leaf;
            const int32_t base = (int32_t)nodes.size();
            int k0 = 0;
            while (k0 < np) {
                int k1e = std::min(np, k0 + kMaxLooponPiece);
                for (; leaf < mine.size() && (int)mine[leaf].rec + mine[leaf].terms <= k1e; ++leaf) {
                    mine[leaf].piece = (uint32_t)L.pieces.size();
                    mine[leaf].rec -= (uint32_t)k0;
                }
                if (leaf < mine.size()) k1e = (int)mine[leaf].rec;
                LooponPiece p;
                std::memset(&p, 0, sizeof(p));
                p.cx = cx; p.cy = cy; p.cz = cz;
                p.fbx = -k1 * ph.dS * ph.bx;
                p.fby = -k1 * ph.dS * ph.by;
                p.fbz = -k1 * ph.dS * ph.bz;
                p.mx = ph.mx; p.my = ph.my; p.mz = ph.mz;
                p.nx = ph.nx; p.ny = ph.ny; p.nz = ph.nz;
                p.b_n = ph.mx * ph.nx + ph.my * ph.ny + ph.mz * ph.nz;
                p.n = k1e - k0;
                std::vector<LooponRec> recs;
                recs.reserve((size_t)(k1e - k0));
                for (int k = k0; k < k1e; ++k) {
                    const int i = order.empty() ? k : order[k];
                    LooponRec r;
                    r.x = lp.x[i] - cx; r.y = lp.y[i] - cy; r.z = lp.z[i] - cz;
                    r.ml = ph.mx * r.x + ph.my * r.y + ph.mz * r.z;
                    r.nl = ph.nx * r.x + ph.ny * r.y + ph.nz * r.z;
                    r.w = 1.0;
                    recs.push_back(r);
                }
                L.pieces.push_back(p);
                L.recs.push_back(std::move(recs));
                k0 = k1e;
            }
            for (TreePiece q : mine) {
                if (q.parent >= 0) q.parent += base;
                q.leaf0 += base;
                nodes.push_back(q);
            }
        }
        pack_chunks(L, T, stage_cap);
        if (tree) {
            std::vector<uint32_t> at_piece, at_rec;
            for (const Chunk& c : T.chunks) {
                uint64_t rec = c.offset + (uint64_t)c.npieces * sizeof(LooponPiece);
                for (int i = 0; i < c.npieces; ++i) {
                    at_piece.push_back((uint32_t)(c.offset + i * sizeof(LooponPiece)));
                    at_rec.push_back((uint32_t)rec);
                    rec += (uint64_t)L.pieces[at_piece.size() - 1].n * sizeof(LooponRec);
                }
            }
            for (size_t k = 0; k < nodes.size(); ++k) {
                TreePiece& q = nodes[k];
                if (q.leaf0 != (int32_t)k) continue;
                const uint32_t i = q.piece;
                q.piece = at_piece[i];
                q.rec = at_rec[i] + q.rec * (uint32_t)sizeof(LooponRec);
            }
            for (TreePiece& q : nodes) q.piece = nodes[q.leaf0].piece;      // m, n and b are the loop's
            T.tree = std::move(nodes);
        }
    }
    return DISCO_OK;
}

// ---- host: launch ------------------------------------------------------------------------

namespace {

template <class Policy, int S>
int launch_one(const FieldArgs& a, int sm_count, size_t smem, cudaStream_t stream, std::string& err)
{
    auto kern = field_kernel<Policy, S>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit);
    if (e != cudaSuccess) { err = cudaGetErrorString(e); return DISCO_ECUDA; }
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, smem);
    if (e != cudaSuccess || per_sm < 1) { err = "kernel does not fit on an SM"; return DISCO_ECUDA; }
    const int64_t atoms_per_cta = kThreads / S;
    const int64_t ntiles = (a.n + atoms_per_cta - 1) / atoms_per_cta;
    const int64_t grid = std::min<int64_t>(ntiles, (int64_t)sm_count * per_sm);
    kern<<<(unsigned)grid, kThreads, smem, stream>>>(a);
    e = cudaGetLastError();
    if (e != cudaSuccess) { err = cudaGetErrorString(e); return DISCO_ECUDA; }
    return DISCO_OK;
}

template <class Policy>
int launch_kind(const FieldArgs& a, int S, int sm_count, size_t smem, cudaStream_t stream, std::string& err)
{
    switch (S) {
    case 1:  return launch_one<Policy, 1>(a, sm_count, smem, stream, err);
    case 2:  return launch_one<Policy, 2>(a, sm_count, smem, stream, err);
    case 4:  return launch_one<Policy, 4>(a, sm_count, smem, stream, err);
    case 8:  return launch_one<Policy, 8>(a, sm_count, smem, stream, err);
    case 16: return launch_one<Policy, 16>(a, sm_count, smem, stream, err);
    default: return launch_one<Policy, 32>(a, sm_count, smem, stream, err);
    }
}

} // namespace

// Image split S: the power of two (<= 32, <= images) that minimises
// rounds x images-per-lane, with rounds = ceil(tiles / resident CTAs).
int choose_split(int64_t n, int nimg, int resident_ctas)
{
    int best = 1;
    double best_cost = 1e300;
    for (int S = 1; S <= 32; S *= 2) {
        if (S > 1 && S > nimg) break;
        const int64_t ntiles = (n * S + kThreads - 1) / kThreads;
        const double rounds = std::ceil((double)ntiles / resident_ctas);
        const double cost = rounds * std::ceil((double)nimg / S);
        if (cost < best_cost * (1.0 - 1e-9)) { best_cost = cost; best = S; }
    }
    return best;
}

int launch_field(const FieldArgs& a, int kind, bool fp32, int sm_count, int threads_hint,
                 int split_hint, cudaStream_t stream, std::string& err)
{
    (void)threads_hint;
    if (a.n <= 0 || a.nchunks <= 0) return DISCO_OK;
    if (fp32) { err = "FP32 launch goes through launch_field_fp32"; return DISCO_EINVAL; }
    const size_t smem = kSmemHeader + (size_t)a.stage_bytes * (a.resident ? 1 : 2);
    const int S = split_hint > 0 ? split_hint : choose_split(a.n, a.nimg, sm_count * 2);
    return kind == kLineKind ? launch_kind<LineFp64>(a, S, sm_count, smem, stream, err)
                             : launch_kind<LooponFp64>(a, S, sm_count, smem, stream, err);
}

} // namespace disco

// ---- self-test of the kernels' own FP64 math routines -------------------------------------

namespace {

__global__ void math_check_kernel(int fn, const double* x, double* y, int64_t n)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double v = x[i];
        double r;
        switch (fn) {
        case 0: r = disco::rsqrt_nr(v); break;
        case 1: r = disco::rcp_nr(v); break;
        case 2: r = 2.0 * disco::half_j0_series<8>(v); break;
        case 3: r = 2.0 * disco::half_j0_series<6>(v); break;
        default: r = 2.0 * disco::half_j0_series<4>(v); break;
        }
        y[i] = r;
    }
}

} // namespace

extern "C" int disco_b200_math_check(int32_t fn, const double* x, double* y, int64_t n, void* stream)
{
    if (fn < 0 || fn > 4 || n < 0 || (n > 0 && (!x || !y))) {
        disco::set_last_error("math_check: bad argument");
        return DISCO_EINVAL;
    }
    if (n == 0) return DISCO_OK;
    const int grid = (int)std::min<int64_t>((n + 255) / 256, 4096);
    math_check_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(fn, x, y, n);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        disco::set_last_error(std::string("math_check: ") + cudaGetErrorString(e));
        return DISCO_ECUDA;
    }
    return DISCO_OK;
}
