// Text output of the final positions on the device: the atom lines of the
// reference's XYZ writer (Code/main.cpp:826-831) and LAMMPS writer
// (Code/main.cpp:86-92, orthorhombic box), formatted as the C++ stream does
// with `fixed << setprecision(8)`: each coordinate rounded to 8 decimals from
// its exact binary value, ties to even, sign kept for negative values that
// round to zero.
//
// Rounding: a = m 2^k (m the 53-bit significand), so a 1e8 = m 1e8 2^k exactly,
// with m 1e8 < 2^80 held in a 128-bit integer; shifting by -k with round-half-
// even gives the 8-decimal integer R exactly (64 bits: |v| below 1.8e11).
//
// A coordinate's length needs no rounding: it grows where |v| reaches the
// smallest double that rounds to 10^k, found once on the host by the rounding
// itself, so the first kernel compares (and reads 24 B an atom).  Its last CTA
// turns the tile sums into offsets.  The second kernel formats 256 lines at a
// time into shared memory, at the alignment of their place in the text, and
// copies them out 16 bytes a thread: the text is written once, in whole
// sectors (single bytes per thread to global memory: 352 us for 1.0 M atoms,
// 45 MB; 50 us staged, bound by integer work).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>

#include <cuda_runtime.h>

#include "common.cuh"

namespace {

constexpr int kThreads = 256;
constexpr int kPerThread = 4;
constexpr int kTile = kThreads * kPerThread;
constexpr int kMaxPrefix = 64;            // bytes of the XYZ element name
constexpr int kMaxWhole = 12;             // digits before the point: |v| < 1.8e11
// the longest line: element or index, three coordinates, four separators
constexpr int kMaxLine = kMaxPrefix + 3 * (1 + kMaxWhole + 1 + 8) + 4;

struct Fixed8 {
    unsigned long long R;                 // round(|v| 1e8)
    bool neg, ok;
};

__host__ __device__ __forceinline__ Fixed8 fixed8(double v)
{
    Fixed8 f;
    unsigned long long bits;
    memcpy(&bits, &v, sizeof(bits));
    f.neg = (bits >> 63) != 0;
    const int ex = (int)((bits >> 52) & 0x7FF);
    const unsigned long long mant = bits & ((1ull << 52) - 1);
    f.ok = ex != 0x7FF;
    f.R = 0;
    if (!f.ok) return f;
    const unsigned long long m = ex == 0 ? mant : (mant | (1ull << 52));
    const int k = ex == 0 ? -1074 : ex - 1075;
    const unsigned __int128 P = (unsigned __int128)m * 100000000ull;
    if (k >= 0) {
        if (k > 10 || (P << k) >> 64) { f.ok = false; return f; }
        f.R = (unsigned long long)(P << k);
        return f;
    }
    const int s = -k;
    if (s > 100) return f;                // |v| 1e8 < 2^-20: rounds to 0
    const unsigned __int128 q = P >> s;
    const unsigned __int128 r = P - (q << s);
    const unsigned __int128 half = (unsigned __int128)1 << (s - 1);
    unsigned __int128 R = q;
    if (r > half || (r == half && (q & 1))) R += 1;
    if (R >> 64) { f.ok = false; return f; }
    f.R = (unsigned long long)R;
    return f;
}

// Whole digits of a coordinate by its magnitude: reach[k] is the smallest
// double that rounds to 10^(k + 1) or more, bad the smallest that does not fit.
struct Lengths {
    double reach[kMaxWhole - 1], bad;
};

__device__ __forceinline__ int ndigits(unsigned long long v)
{
    int d = 1;
    while (v >= 10) { v /= 10; ++d; }
    return d;
}

// Two decimal digits at o.
__device__ __forceinline__ void put2(char* o, unsigned v)
{
    const unsigned t = v * 103u >> 10;                // v / 10 for v < 100
    o[0] = (char)('0' + t);
    o[1] = (char)('0' + (v - 10u * t));
}

__device__ __forceinline__ char* put_uint(char* o, unsigned long long v)
{
    if (v < 100ull) {                                 // most coordinates and many indices
        const unsigned w = (unsigned)v;
        if (w >= 10u) { put2(o, w); return o + 2; }
        *o = (char)('0' + w);
        return o + 1;
    }
    const int d = ndigits(v);
    int i = d;
    while (v >= 100ull) {
        i -= 2;
        put2(o + i, (unsigned)(v % 100ull));
        v /= 100ull;
    }
    if (v >= 10ull) put2(o, (unsigned)v); else *o = (char)('0' + (unsigned)v);
    return o + d;
}

__device__ __forceinline__ char* put_fixed8(char* o, double v)
{
    const Fixed8 f = fixed8(v);
    if (f.neg) *o++ = '-';
    const unsigned long long whole = f.R / 100000000ull;
    o = put_uint(o, whole);
    *o++ = '.';
    const unsigned fr = (unsigned)(f.R - whole * 100000000ull), hi = fr / 10000u, lo = fr - hi * 10000u;
    put2(o, hi / 100u);
    put2(o + 2, hi % 100u);
    put2(o + 4, lo / 100u);
    put2(o + 6, lo % 100u);
    return o + 8;
}

struct WriterArgs {
    const double *x, *y, *z;
    int64_t n;
    int32_t lammps;                       // 0: "<element> x y z", 1: "<k+1> 1 x y z"
    int32_t plen;
    char prefix[kMaxPrefix];
    Lengths len;
    int64_t ntiles;
    int64_t* tile_len;                    // per tile, then exclusive offsets; [ntiles] the total
    unsigned int* bad;                    // [0] a coordinate does not fit, [1] tiles done
    char* out;
};

__device__ __forceinline__ int coord_len(const Lengths& L, double v, bool& ok)
{
    const double m = fabs(v);
    ok = ok && m < L.bad;                 // false for a NaN
    int d = 10 + (__double_as_longlong(v) < 0 ? 1 : 0);
#pragma unroll
    for (int k = 0; k < kMaxWhole - 1; ++k) d += m >= L.reach[k] ? 1 : 0;
    return d;
}

__device__ __forceinline__ int line_len(const WriterArgs& a, int64_t i, double x, double y, double z, bool& ok)
{
    const int head = a.lammps ? ndigits((unsigned long long)(i + 1)) + 3 : a.plen + 1;
    return head + coord_len(a.len, x, ok) + 1 + coord_len(a.len, y, ok) + 1 + coord_len(a.len, z, ok) + 1;
}

// Exclusive scan of one value per thread over the CTA; returns the CTA total.
__device__ __forceinline__ long long cta_scan(long long v, long long& excl)
{
    __shared__ long long warp_tot[kThreads / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    long long inc = v;
    for (int o = 1; o < 32; o <<= 1) {
        const long long t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) warp_tot[w] = inc;
    __syncthreads();
    long long base = 0, tot = 0;
    for (int k = 0; k < kThreads / 32; ++k) {
        if (k < w) base += warp_tot[k];
        tot += warp_tot[k];
    }
    __syncthreads();
    excl = base + inc - v;
    return tot;
}

__global__ void __launch_bounds__(kThreads) len_kernel(const WriterArgs a)
{
    const int64_t t0 = (int64_t)blockIdx.x * kTile + threadIdx.x;
    long long mine = 0;
    bool ok = true;
#pragma unroll
    for (int j = 0; j < kPerThread; ++j) {
        const int64_t i = t0 + j * kThreads;
        if (i < a.n) mine += line_len(a, i, a.x[i], a.y[i], a.z[i], ok);
    }
    if (!ok) atomicExch(&a.bad[0], 1u);
    long long excl;
    const long long tot = cta_scan(mine, excl);
    __shared__ bool last;
    if (threadIdx.x == 0) {
        a.tile_len[blockIdx.x] = tot;
        __threadfence();
        last = atomicAdd(&a.bad[1], 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    // the last tile to finish: exclusive offsets, the total behind them
    __threadfence();
    long long carry = 0;
    for (int64_t b0 = 0; b0 < a.ntiles; b0 += kTile) {
        long long v[kPerThread], sum = 0;
#pragma unroll
        for (int j = 0; j < kPerThread; ++j) {
            const int64_t b = b0 + (int64_t)threadIdx.x * kPerThread + j;
            v[j] = b < a.ntiles ? *(volatile int64_t*)(a.tile_len + b) : 0;
            sum += v[j];
        }
        const long long all = cta_scan(sum, excl);
        long long at = carry + excl;
#pragma unroll
        for (int j = 0; j < kPerThread; ++j) {
            const int64_t b = b0 + (int64_t)threadIdx.x * kPerThread + j;
            if (b < a.ntiles) a.tile_len[b] = at;
            at += v[j];
        }
        carry += all;
    }
    if (threadIdx.x == 0) a.tile_len[a.ntiles] = carry;
}

__global__ void __launch_bounds__(kThreads) write_kernel(const WriterArgs a)
{
    __shared__ __align__(16) char text[16 + kThreads * kMaxLine];
    long long at = a.tile_len[blockIdx.x];
    for (int j = 0; j < kPerThread; ++j) {
        const int64_t i = (int64_t)blockIdx.x * kTile + j * kThreads + threadIdx.x;
        double c[3] = { 0.0, 0.0, 0.0 };
        long long len = 0, excl;
        bool ok = true;
        if (i < a.n) {
            c[0] = a.x[i]; c[1] = a.y[i]; c[2] = a.z[i];
            len = line_len(a, i, c[0], c[1], c[2], ok);
        }
        const int tot = (int)cta_scan(len, excl);
        // the lines at the 16-byte phase of their place in the text
        char* const dst = a.out + at;
        const int skew = (int)(reinterpret_cast<uintptr_t>(dst) & 15);
        char* o = text + skew + excl;
        if (i < a.n) {
            if (a.lammps) {
                o = put_uint(o, (unsigned long long)(i + 1));
                *o++ = ' '; *o++ = '1'; *o++ = ' ';
            } else {
                for (int p = 0; p < a.plen; ++p) *o++ = a.prefix[p];
                *o++ = ' ';
            }
            o = put_fixed8(o, c[0]);
            *o++ = ' ';
            o = put_fixed8(o, c[1]);
            *o++ = ' ';
            o = put_fixed8(o, c[2]);
            *o++ = '\n';
        }
        __syncthreads();
        const int b0 = min(tot, (16 - skew) & 15), b1 = b0 + (tot - b0) / 16 * 16;
        if ((int)threadIdx.x < b0) dst[threadIdx.x] = text[skew + threadIdx.x];
        for (int b = b0 + 16 * threadIdx.x; b < b1; b += 16 * kThreads)
            *reinterpret_cast<uint4*>(dst + b) = *reinterpret_cast<const uint4*>(text + skew + b);
        if (b1 + (int)threadIdx.x < tot) dst[b1 + threadIdx.x] = text[skew + b1 + threadIdx.x];
        at += tot;
        __syncthreads();
    }
}

// The smallest double in (lo, hi] for which `holds` (false at lo, true at hi,
// monotone), by bisection of the ordered bits of positive doubles.
template <class F>
double smallest(double lo, double hi, F holds)
{
    unsigned long long a, b;
    std::memcpy(&a, &lo, 8);
    std::memcpy(&b, &hi, 8);
    while (b - a > 1) {
        const unsigned long long m = a + (b - a) / 2;
        double v;
        std::memcpy(&v, &m, 8);
        if (holds(v)) b = m; else a = m;
    }
    double v;
    std::memcpy(&v, &b, 8);
    return v;
}

const Lengths& lengths()
{
    static const Lengths L = [] {
        Lengths t;
        unsigned long long ten = 1000000000ull;       // 10 with 8 decimals
        double p = 10.0;
        for (int k = 0; k < kMaxWhole - 1; ++k, p *= 10.0) {
            if (p > 1e11) { t.reach[k] = HUGE_VAL; continue; }
            t.reach[k] = smallest(0.5 * p, p, [&](double v) { return fixed8(v).R >= ten; });
            ten *= 10ull;
        }
        t.bad = smallest(1e11, 1e12, [](double v) { return !fixed8(v).ok; });
        return t;
    }();
    return L;
}

int wfail(int code, const std::string& msg)
{
    disco::set_last_error(msg);
    return code;
}

} // namespace

extern "C" int disco_b200_format_atoms(int32_t format, const char* element, const double* x, const double* y,
                                       const double* z, int64_t n, char* out, int64_t capacity,
                                       int64_t* bytes, void* stream)
{
    if (!bytes || n < 0 || (format != 0 && format != 1) || (n > 0 && (!x || !y || !z)))
        return wfail(DISCO_EINVAL, "format_atoms: bad argument");
    *bytes = 0;
    WriterArgs a;
    std::memset(&a, 0, sizeof(a));
    a.lammps = format;
    if (format == 0) {
        const size_t L = element ? std::strlen(element) : 0;
        if (L == 0 || L > (size_t)kMaxPrefix) return wfail(DISCO_EINVAL, "format_atoms: element name of 1..64 bytes");
        std::memcpy(a.prefix, element, L);
        a.plen = (int32_t)L;
    }
    if (n == 0) return DISCO_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int64_t ntiles = (n + kTile - 1) / kTile;
    if (ntiles > 0x7FFFFFFF) return wfail(DISCO_ELIMIT, "format_atoms: too many atoms");
    a.x = x; a.y = y; a.z = z; a.n = n;
    a.len = lengths();
    a.ntiles = ntiles;
    void* scratch = nullptr;
    cudaError_t e = disco::scratch_alloc(&scratch, (size_t)(ntiles + 2) * sizeof(int64_t), s);
    if (e != cudaSuccess) return wfail(DISCO_ENOMEM, std::string("format_atoms: ") + cudaGetErrorString(e));
    a.tile_len = static_cast<int64_t*>(scratch);
    a.bad = reinterpret_cast<unsigned int*>(a.tile_len + ntiles + 1);
    int64_t got[2] = { 0, 0 };                        // the total, then bad and the tiles done
    e = cudaMemsetAsync(a.bad, 0, sizeof(int64_t), s);
    if (e == cudaSuccess) {
        len_kernel<<<(unsigned)ntiles, kThreads, 0, s>>>(a);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(got, a.tile_len + ntiles, sizeof(got), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    int st = DISCO_OK;
    const int64_t total = got[0];
    if (e != cudaSuccess) {
        st = wfail(DISCO_ECUDA, std::string("format_atoms: ") + cudaGetErrorString(e));
    } else if ((uint32_t)got[1] != 0u) {
        st = wfail(DISCO_EINVAL, "format_atoms: a coordinate is not finite or |v| >= 1.8e11");
    } else {
        *bytes = total;
        if (total > capacity || !out) {
            st = wfail(DISCO_ELIMIT, "format_atoms: output buffer too small (*bytes holds the size needed)");
        } else {
            a.out = out;
            write_kernel<<<(unsigned)ntiles, kThreads, 0, s>>>(a);
            e = cudaGetLastError();
            if (e != cudaSuccess) st = wfail(DISCO_ECUDA, std::string("format_atoms: ") + cudaGetErrorString(e));
        }
    }
    cudaFreeAsync(scratch, s);
    return st;
}
