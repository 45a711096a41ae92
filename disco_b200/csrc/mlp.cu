// The learned far-image surrogate's network: 14 -> 128 -> 128 -> 128 -> 3,
// SiLU, BF16 weights and activations on the tensor cores, FP32 accumulation,
// FP32 master weights and Adam.
//
// net_kernel does a whole forward pass, or forward and backward, for 128 rows
// at a time in one CTA of 256 threads (row r is tensor-memory lane r; warps w
// and w + 4 read the same lanes and split the columns).  Weights, activations
// and their transposes sit in shared memory as BF16 K-major tiles (tcgen05.cuh;
// 224 KB in all), the three layers' FP32 pre-activations stay in tensor memory
// until the backward pass has used them, and their columns then take the weight
// gradients:
//
//     columns    0..127   pre-activation 1, then dW1
//              128..255   pre-activation 2, then dW2
//              256..383   pre-activation 3, then dW3
//              384..511   output, dW4, then dh3, dh2, dh1
//
// dh = dpre W needs W transposed, dW = dpre^T h both operands: the epilogues
// write each tile in both orders (a transposed tile of h makes room for the
// transposed dpre of the layer above), and W3, W2 are staged again transposed
// over themselves (bulk copies of BF16 tiles that Adam writes with the weights).
// Each CTA keeps its own partial gradient in global memory;
// sum_kernel adds the partials in order, so a gradient is the same in every run.
// The latency of one tile's chain of layers bounds a step (4096 rows are 32
// tiles; their SMs issue on 19 % of the cycles, waiting for L2 and for
// barriers): 0.40 ms with one launch per product and reduction (18 launches),
// 0.050 ms with this kernel (37 us alone; 50 with the weights converted in it), the
// sum (10 us) and Adam (4).
//
// Inputs are padded to 16 features and outputs to 16 (the MMA's N >= 16 for
// M = 128); the padding columns of W1 and rows of W4 are zero and stay zero
// (their gradients are masked).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "common.cuh"
#include "mlp.cuh"
#include "tcgen05.cuh"

namespace disco {
namespace mlp {

constexpr int kNetThreads = 256;
constexpr int kRows = 128;                        // rows per tile
constexpr uint32_t kTile = kRows * kHid * 2;      // a 128 x 128 BF16 tile
constexpr uint32_t kThin = kRows * kIn * 2;       // a 128 x 16 (or 16 x 128) one
// Transposed activations are written 2 bytes at a time, 32 rows (K values) of a
// column by a warp: 16 bytes more between K blocks than their core matrices
// take puts the four blocks on different banks (four-way conflicts without).
constexpr uint32_t kTransLbo = (kHid / 8) * 128 + 16, kTrans = kTransLbo * (kRows / 8);
constexpr uint32_t kThinLbo = (kIn / 8) * 128 + 16, kThinTrans = kThinLbo * (kRows / 8);
constexpr uint32_t oSW1 = 0;                      // [128 x 16]
constexpr uint32_t oSW2 = oSW1 + kThin;           // [128 x 128], in the backward pass transposed
constexpr uint32_t oSW3 = oSW2 + kTile;
constexpr uint32_t oSW4 = oSW3 + kTile;           // [16 x 128]
constexpr uint32_t oSW4T = oSW4 + kThin;          // [128 x 16]
constexpr uint32_t oSX = oSW4T + kThin;           // [rows x 16]
constexpr uint32_t oSXT = oSX + kThin;            // [16 x rows], padded
constexpr uint32_t oSH = oSXT + kThinTrans;       // activations, then dpre: [rows x 128]
constexpr uint32_t oST = oSH + kTile;             // three padded tiles [128 x rows]: h1, h2, h3 transposed, then dpre
constexpr uint32_t oSDy = oST + 3 * kTrans;       // [rows x 16]
constexpr uint32_t oSDyT = oSDy + kThin;          // [16 x rows], padded
constexpr uint32_t oSBias = oSDyT + kThinTrans;   // b1, b2, b3, b4 (FP32)
constexpr uint32_t oSLoss = oSBias + (3 * kHid + kOut) * 4;     // the warps' losses
constexpr uint32_t oSBar = oSLoss + 32;           // products, weights; the tensor-memory slot
constexpr uint32_t kNetSmem = oSBar + 32;
static_assert(kNetSmem <= 227 * 1024, "one CTA's shared memory");
static_assert(oSH % 16 == 0 && oSBar % 8 == 0, "tile and barrier alignment");
// The weights as the tiles the kernel stages: W1, W2, W3, W4, then W4, W3 and W2
// transposed, K-major BF16 (written by Adam, or by pack_kernel for new weights).
constexpr uint32_t kImg = 3 * kThin + 4 * kTile;
constexpr uint32_t oIW1 = 0, oIW2 = oIW1 + kThin, oIW3 = oIW2 + kTile, oIW4 = oIW3 + kTile, oIW4T = oIW4 + kThin,
                   oIW3T = oIW4T + kThin, oIW2T = oIW3T + kTile;
static_assert(oIW2T + kTile == kImg && oIW1 == oSW1 && oIW4T == oSW4T, "weight image layout");
constexpr uint32_t kLbo = (kRows / 8) * 128, kOutLbo = (kOut / 8) * 128;      // K blocks of 128 and 16 rows
constexpr int kPart = kParams + 4;                // a partial gradient and its loss

struct NetArgs {
    const float* P;
    const unsigned char* img; // BF16 tiles of the weights
    const float* X;           // [n x 16]
    const float* T;           // [n x 3], null: forward only
    float* Y;                 // [n x 16], forward only
    float* part;              // [CTA][kPart]
    float* dpre;              // [3][n x 128]
    float* dy;                // [n x 4]
    int64_t n;
    int32_t tiles;
    int32_t x16, y16;         // X, Y 16-byte aligned
    int* status;
};

__device__ __forceinline__ uint32_t bf16x2(float lo, float hi)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// Parameter i's places in the weight image (biases have none).
__device__ __forceinline__ void put_weight(unsigned char* img, int i, float v)
{
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    auto put = [&](uint32_t tile, int r, int k, int rows) {
        *reinterpret_cast<__nv_bfloat16*>(img + tile + tc::kmajor_offset(r, k, rows)) = h;
    };
    if (i < ob1) {
        put(oIW1, (i - oW1) / kIn, (i - oW1) % kIn, kHid);
    } else if (i >= oW2 && i < ob2) {
        const int r = (i - oW2) / kHid, k = (i - oW2) % kHid;
        put(oIW2, r, k, kHid);
        put(oIW2T, k, r, kHid);
    } else if (i >= oW3 && i < ob3) {
        const int r = (i - oW3) / kHid, k = (i - oW3) % kHid;
        put(oIW3, r, k, kHid);
        put(oIW3T, k, r, kHid);
    } else if (i >= oW4 && i < ob4) {
        const int r = (i - oW4) / kHid, k = (i - oW4) % kHid;
        put(oIW4, r, k, kOut);
        put(oIW4T, k, r, kHid);
    }
}

__global__ void pack_kernel(const float* P, unsigned char* img)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kParams) put_weight(img, i, P[i]);
}

// One product D (+)= A B^T over K = 16 nk, issued by the calling thread; alb,
// blb: bytes between the operands' K blocks.
__device__ __forceinline__ void product(uint32_t tmem, uint32_t a, uint32_t alb, uint32_t b, uint32_t blb, int nk, int N)
{
    const uint32_t id = tc::idesc_bf16(kRows, N);
    for (int j = 0; j < nk; ++j)
        tc::mma_bf16(tmem, tc::smem_desc(a + j * 2 * alb, alb, 128), tc::smem_desc(b + j * 2 * blb, blb, 128), id, j > 0);
}

// Publishes every thread's tile writes and finished tensor-memory loads, has
// one thread issue the products and waits for them (bounded); false, agreed by
// the whole CTA, on a timeout.
template <class Issue>
__device__ __forceinline__ bool products(uint64_t* bar, uint32_t& phase, Issue issue)
{
    fence_proxy_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    if (threadIdx.x == 0) {
        tc::fence_after_sync();
        issue();
        tc::commit(bar);
    }
    const bool mine = mbar_wait_bounded(bar, phase);
    phase ^= 1;
    const bool bad = __syncthreads_or(!mine);
    tc::fence_after_sync();
    return !bad;
}

// Element (r, k) of a transposed tile, K blocks lbo bytes apart.
__device__ __forceinline__ uint32_t trans_offset(int r, int k, uint32_t lbo)
{
    return (uint32_t)(k >> 3) * lbo + (uint32_t)((r >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2);
}

// 32 consecutive columns of one row into a transposed tile [columns x rows].
__device__ __forceinline__ void put_transposed(unsigned char* tile, const float (&h)[32], int row, int c0)
{
#pragma unroll
    for (int i = 0; i < 32; ++i)
        *reinterpret_cast<__nv_bfloat16*>(tile + trans_offset(c0 + i, row, kTransLbo)) = __float2bfloat16_rn(h[i]);
}
__device__ __forceinline__ void put_row(unsigned char* tile, const float (&h)[32], int row, int c0)
{
#pragma unroll
    for (int q = 0; q < 4; ++q)
        *reinterpret_cast<uint4*>(tile + tc::kmajor_offset(row, c0 + 8 * q, kRows)) =
            make_uint4(bf16x2(h[8 * q], h[8 * q + 1]), bf16x2(h[8 * q + 2], h[8 * q + 3]),
                       bf16x2(h[8 * q + 4], h[8 * q + 5]), bf16x2(h[8 * q + 6], h[8 * q + 7]));
}

template <bool kTrain>
__global__ void __launch_bounds__(kNetThreads, 1) net_kernel(const NetArgs a)
{
    extern __shared__ __align__(128) unsigned char sm[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + oSBar);
    uint32_t* slot = reinterpret_cast<uint32_t*>(sm + oSBar + 16);
    float* bias = reinterpret_cast<float*>(sm + oSBias);
    float* losses = reinterpret_cast<float*>(sm + oSLoss);
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int row = t & 127, half = t >> 7;
    if (warp == 0) tc::alloc(slot, 512);
    if (t == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_mbar_init();
    }
    for (int e = t; e < 3 * kHid + kOut; e += kNetThreads)
        bias[e] = a.P[e < kHid ? ob1 + e : e < 2 * kHid ? ob2 + e - kHid : e < 3 * kHid ? ob3 + e - 2 * kHid
                                                                                     : ob4 + e - 3 * kHid];
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *slot;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;             // this warp's tensor-memory lanes
    const uint32_t s0 = smem_addr(sm);
    const int c0 = half * (kHid / 2);
    uint32_t phase = 0, wphase = 0;
    bool ok = true;
    float loss = 0.0f;
    // weight tiles by bulk copy, `bytes` of the image at `from` to `to`; every
    // copy in flight completes the phase of bar[1] that its wait names
    auto fetch = [&](uint32_t to, uint32_t from, uint32_t bytes) { stage_load(sm + to, a.img + from, bytes, &bar[1]); };
    auto fetched = [&]() {
        const bool mine = mbar_wait_bounded(&bar[1], wphase);
        wphase ^= 1;
        return mine;
    };
    if (t == 0) fetch(oSW1, oIW1, oSX - oSW1);
    bool staged = false;                          // the first copy has been waited for
    float* const part = kTrain ? a.part + (int64_t)blockIdx.x * kPart : nullptr;

    // a hidden layer's activations from its pre-activation in columns `col`
    auto activate = [&](uint32_t col, const float* b, unsigned char* T) {
#pragma unroll 1
        for (int c = c0; c < c0 + kHid / 2; c += 32) {
            float v[32];
            tc::ld32(tmem + lanes + col + c, v);
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = silu_half(0.5f * (v[i] + b[c + i]));
            put_row(sm + oSH, v, row, c);
            if (kTrain) put_transposed(T, v, row, c);
        }
    };
    for (int tile = blockIdx.x; ok && tile < a.tiles; tile += gridDim.x) {
        const int64_t r = (int64_t)tile * kRows + row;
        const bool valid = r < a.n;
        const bool first = tile == (int)blockIdx.x;
        if (kTrain && staged && t == 0) fetch(oSW2, oIW2, 2 * kTile);    // over the last tile's transposed ones
        {
            float x[kIn];
#pragma unroll
            for (int k = 0; k < kIn; ++k) x[k] = 0.0f;
            if (valid) {
                const float* src = a.X + r * kIn;
                if (a.x16) {
#pragma unroll
                    for (int q = 0; q < kIn / 4; ++q) {
                        const float4 f = reinterpret_cast<const float4*>(src)[q];
                        x[4 * q] = f.x; x[4 * q + 1] = f.y; x[4 * q + 2] = f.z; x[4 * q + 3] = f.w;
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < kIn; ++k) x[k] = src[k];
                }
            }
            if (half == 0) {
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    *reinterpret_cast<uint4*>(sm + oSX + tc::kmajor_offset(row, 8 * q, kRows)) =
                        make_uint4(bf16x2(x[8 * q], x[8 * q + 1]), bf16x2(x[8 * q + 2], x[8 * q + 3]),
                                   bf16x2(x[8 * q + 4], x[8 * q + 5]), bf16x2(x[8 * q + 6], x[8 * q + 7]));
            } else if (kTrain) {
#pragma unroll
                for (int k = 0; k < kIn; ++k)
                    *reinterpret_cast<__nv_bfloat16*>(sm + oSXT + trans_offset(k, row, kThinLbo)) = __float2bfloat16_rn(x[k]);
            }
        }
        if (!staged || kTrain) ok = fetched();
        staged = true;
        if (__syncthreads_or(!ok)) { ok = false; break; }
        // forward
        ok = products(bar, phase, [&] { product(tmem, s0 + oSX, kLbo, s0 + oSW1, kLbo, kIn / 16, kHid); });
        if (!ok) break;
        activate(0, bias, sm + oST);
        ok = products(bar, phase, [&] { product(tmem + 128, s0 + oSH, kLbo, s0 + oSW2, kLbo, kHid / 16, kHid); });
        if (!ok) break;
        activate(128, bias + kHid, sm + oST + kTrans);
        ok = products(bar, phase, [&] { product(tmem + 256, s0 + oSH, kLbo, s0 + oSW3, kLbo, kHid / 16, kHid); });
        if (!ok) break;
        // the weights of dh2 and dh1 over those the forward pass is done with
        if (kTrain && t == 0) {
            mbar_arrive_expect_tx(&bar[1], 2 * kTile);
            bulk_load(sm + oSW3, a.img + oIW3T, kTile, &bar[1]);
            bulk_load(sm + oSW2, a.img + oIW2T, kTile, &bar[1]);
        }
        activate(256, bias + 2 * kHid, sm + oST + 2 * kTrans);
        ok = products(bar, phase, [&] { product(tmem + 384, s0 + oSH, kLbo, s0 + oSW4, kOutLbo, kHid / 16, kOut); });
        if (!ok) break;
        if (!kTrain) {
            if (half == 0) {
                float y[16];
                tc::ld16(tmem + lanes + 384, y);
                if (valid) {
                    float* o = a.Y + r * kOut;
#pragma unroll
                    for (int k = 0; k < kOut; ++k) y[k] += bias[3 * kHid + k];
                    if (a.y16) {
#pragma unroll
                        for (int q = 0; q < kOut / 4; ++q)
                            reinterpret_cast<float4*>(o)[q] = make_float4(y[4 * q], y[4 * q + 1], y[4 * q + 2], y[4 * q + 3]);
                    } else {
#pragma unroll
                        for (int k = 0; k < kOut; ++k) o[k] = y[k];
                    }
                }
            }
            continue;
        }
        // dy = 2 (y - t) / n on the real outputs, 0 on padding and past the last row
        if (half == 0) {
            float y[16], g[kOutReal];
            tc::ld16(tmem + lanes + 384, y);
#pragma unroll
            for (int k = 0; k < kOutReal; ++k) {
                g[k] = 0.0f;
                if (valid) {
                    const float d = (y[k] + bias[3 * kHid + k]) - a.T[r * kOutReal + k];
                    loss += d * d;
                    g[k] = 2.0f * d / (float)a.n;
                }
            }
            *reinterpret_cast<uint4*>(sm + oSDy + tc::kmajor_offset(row, 0, kRows)) =
                make_uint4(bf16x2(g[0], g[1]), bf16x2(g[2], 0.0f), 0u, 0u);
            *reinterpret_cast<uint4*>(sm + oSDy + tc::kmajor_offset(row, 8, kRows)) = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
            for (int k = 0; k < kOut; ++k)
                *reinterpret_cast<__nv_bfloat16*>(sm + oSDyT + trans_offset(k, row, kThinLbo)) =
                    __float2bfloat16_rn(k < kOutReal ? g[k] : 0.0f);
            if (valid) reinterpret_cast<float4*>(a.dy)[r] = make_float4(g[0], g[1], g[2], 0.0f);
        }
        auto put = [&](float* dst, float v) { *dst = first ? v : *dst + v; };
        auto put4 = [&](float* dst, float x, float y, float z, float w) {
            float4* d = reinterpret_cast<float4*>(dst);
            float4 o = make_float4(x, y, z, w);
            if (!first) {
                const float4 p = *d;
                o.x = p.x + x; o.y = p.y + y; o.z = p.z + z; o.w = p.w + w;
            }
            *d = o;
        };
        // 64 columns of this thread's row of a 128 x 128 weight gradient
        auto put_gradient = [&](uint32_t col, int off) {
#pragma unroll 1
            for (int c = c0; c < c0 + kHid / 2; c += 32) {
                float v[32];
                tc::ld32(tmem + lanes + col + c, v);
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    put4(part + off + row * kHid + c + 4 * q, v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
            }
        };
        // dpre = dh dSiLU(pre) of one layer: its tiles, and its FP32 rows for db
        auto dpre = [&](uint32_t col, const float* b, unsigned char* T, int layer, bool rows) {
#pragma unroll 1
            for (int c = c0; c < c0 + kHid / 2; c += 32) {
                float p[32], v[32];
                tc::ld32(tmem + lanes + col + c, p);
                tc::ld32(tmem + lanes + 384 + c, v);
#pragma unroll
                for (int i = 0; i < 32; ++i) v[i] *= dsilu(p[i] + b[c + i]);
                if (rows) put_row(sm + oSH, v, row, c);
                put_transposed(T, v, row, c);
                if (valid) {
                    float4* o = reinterpret_cast<float4*>(a.dpre + ((int64_t)layer * a.n + r) * kHid + c);
#pragma unroll
                    for (int q = 0; q < 8; ++q) o[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                }
            }
        };
        // dW4 = (h3^T dy)^T
        ok = products(bar, phase, [&] {
            product(tmem + 384, s0 + oST + 2 * kTrans, kTransLbo, s0 + oSDyT, kThinLbo, kRows / 16, kOut);
        });
        if (!ok) break;
        if (half == 0) {
            float v[16];
            tc::ld16(tmem + lanes + 384, v);
#pragma unroll
            for (int k = 0; k < kOut; ++k) put(part + oW4 + k * kHid + row, k < kOutReal ? v[k] : 0.0f);
        }
        // dh3 = dy W4
        ok = products(bar, phase, [&] { product(tmem + 384, s0 + oSDy, kLbo, s0 + oSW4T, kLbo, kOut / 16, kHid); });
        if (!ok) break;
        dpre(256, bias + 2 * kHid, sm + oST + 2 * kTrans, 2, true);
        // dh2 = dpre3 W3, dW3 = dpre3^T h2
        ok = fetched();
        if (__syncthreads_or(!ok)) { ok = false; break; }
        ok = products(bar, phase, [&] {
            product(tmem + 384, s0 + oSH, kLbo, s0 + oSW3, kLbo, kHid / 16, kHid);
            product(tmem + 256, s0 + oST + 2 * kTrans, kTransLbo, s0 + oST + kTrans, kTransLbo, kRows / 16, kHid);
        });
        if (!ok) break;
        dpre(128, bias + kHid, sm + oST + kTrans, 1, true);
        put_gradient(256, oW3);
        // dh1 = dpre2 W2, dW2 = dpre2^T h1
        ok = products(bar, phase, [&] {
            product(tmem + 384, s0 + oSH, kLbo, s0 + oSW2, kLbo, kHid / 16, kHid);
            product(tmem + 128, s0 + oST + kTrans, kTransLbo, s0 + oST, kTransLbo, kRows / 16, kHid);
        });
        if (!ok) break;
        dpre(0, bias, sm + oST, 0, false);
        put_gradient(128, oW2);
        // dW1 = dpre1^T x
        ok = products(bar, phase, [&] { product(tmem, s0 + oST, kTransLbo, s0 + oSXT, kThinLbo, kRows / 16, kIn); });
        if (!ok) break;
        if (half == 0) {
            float v[16];
            tc::ld16(tmem + lanes, v);
            v[14] = v[15] = 0.0f;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                put4(part + oW1 + row * kIn + 4 * q, v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
        }
    }
    if (!ok && t == 0) {
        report(a.status, DISCO_ETIMEOUT);
        mbar_wait_bounded(&bar[0], phase ^ 1);
        mbar_wait_bounded(&bar[1], wphase);
    }
    if (kTrain) {
        for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
        if (lane == 0) losses[warp] = loss;
        __syncthreads();
        if (t == 0) part[kParams] = ((losses[0] + losses[1]) + losses[2]) + losses[3];
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::dealloc(tmem, 512);
}

// grads += the gradients of one call, loss = its mean squared error.  Blocks
// below kWeightBlocks add the CTAs' partial weight gradients and losses (FP64, in
// CTA order); the others the biases' column sums, eight columns of one
// layer's dpre (or the output's dy) each: row k, k + 256, ... per thread, then
// the threads.
constexpr int kWeightBlocks = (kParams + 1 + 255) / 256;
constexpr int kBiasBlocks = 3 * (kHid / 8) + 1;
__global__ void __launch_bounds__(256) sum_kernel(const float* part, const float* dpre, const float* dy, int ctas,
                                                  int64_t n, float* grads, float* loss)
{
    const int t = threadIdx.x;
    if (blockIdx.x < kWeightBlocks) {
        const int i = blockIdx.x * 256 + t;
        const bool bias = (i >= ob1 && i < oW2) || (i >= ob2 && i < oW3) || (i >= ob3 && i < oW4) ||
                          (i >= ob4 && i < kParams);
        if (i > kParams || bias) return;
        double s = 0.0;
#pragma unroll 8
        for (int c = 0; c < ctas; ++c) s += (double)part[(int64_t)c * kPart + i];
        if (i < kParams) grads[i] += (float)s;
        else *loss = (float)(s / (double)n);
        return;
    }
    const int b = blockIdx.x - kWeightBlocks, layer = b / (kHid / 8), c0 = (b % (kHid / 8)) * 8;
    float v[8] = {};
    if (layer < 3) {
#pragma unroll 4
        for (int64_t r = t; r < n; r += 256) {
            const float4* q = reinterpret_cast<const float4*>(dpre + ((int64_t)layer * n + r) * kHid + c0);
            const float4 x = q[0], y = q[1];
            v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
            v[4] += y.x; v[5] += y.y; v[6] += y.z; v[7] += y.w;
        }
    } else {
#pragma unroll 4
        for (int64_t r = t; r < n; r += 256) {
            const float4 x = reinterpret_cast<const float4*>(dy)[r];
            v[0] += x.x; v[1] += x.y; v[2] += x.z;
        }
    }
    __shared__ float part8[8][8];
#pragma unroll
    for (int k = 0; k < 8; ++k)
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    if ((t & 31) == 0)
#pragma unroll
        for (int k = 0; k < 8; ++k) part8[k][t >> 5] = v[k];
    __syncthreads();
    if (t < 8) {
        const float* s = part8[t];
        const float sum = ((s[0] + s[4]) + (s[2] + s[6])) + ((s[1] + s[5]) + (s[3] + s[7]));
        if (layer == 0) grads[ob1 + c0 + t] += sum;
        else if (layer == 1) grads[ob2 + c0 + t] += sum;
        else if (layer == 2) grads[ob3 + c0 + t] += sum;
        else if (t < kOutReal) grads[ob4 + t] += sum;
    }
}

__global__ void adam_kernel(float* p, float* g, float* m, float* v, int n, float lr, float b1, float b2,
                            float eps, float bc1, float bc2, float wd, unsigned char* img)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float upd = (mi / bc1) / (sqrtf(vi / bc2) + eps) + wd * p[i];
    const float pi = p[i] - lr * upd;
    p[i] = pi;
    put_weight(img, i, pi);
    g[i] = 0.0f;
}

} // namespace mlp
} // namespace disco

// ---- host ---------------------------------------------------------------------------------


namespace {

using namespace disco::mlp;

int mfail(int code, const std::string& msg)
{
    disco::set_last_error(msg);
    return code;
}

int mcuda(cudaError_t e, const char* what)
{
    disco::set_last_error(std::string(what) + ": " + cudaGetErrorString(e));
    return e == cudaErrorMemoryAllocation ? DISCO_ENOMEM : DISCO_ECUDA;
}

void free_mlp(disco_mlp* p)
{
    if (!p) return;
    if (p->part) cudaFree(p->part);
    if (p->packed) cudaFree(p->packed);
    if (p->img) cudaFree(p->img);
    delete p;
}

// The tiles of new weights, complete when this returns: every later launch, and
// every replay of a captured one, reads them whatever its stream.
cudaError_t pack_weights(disco_mlp* p)
{
    pack_kernel<<<(kParams + 255) / 256, 256>>>(p->params, p->img);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? cudaStreamSynchronize(nullptr) : e;
}

// Queues the network over n rows of X: forward into Y (T null), or forward and
// backward into the gradients and the loss.
int run_net(disco_mlp* p, const float* X, const float* T, int64_t n, float* Y, cudaStream_t s)
{
    if (n > (int64_t)0x7FFFFFFF * kRows) return mfail(DISCO_ELIMIT, "too many rows");
    if (!p->sms) {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&p->sms, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(net_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kNetSmem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(net_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kNetSmem);
        if (e != cudaSuccess) { p->sms = 0; return mcuda(e, "network setup"); }
    }
    NetArgs a;
    std::memset(&a, 0, sizeof(a));
    a.P = p->params;
    a.img = p->img;
    a.X = X; a.T = T; a.Y = Y;
    a.n = n;
    a.tiles = (int32_t)((n + kRows - 1) / kRows);
    a.x16 = (reinterpret_cast<uintptr_t>(X) & 15) == 0;
    a.y16 = (reinterpret_cast<uintptr_t>(Y) & 15) == 0;
    a.status = p->status;
    const int grid = std::min(a.tiles, p->sms);
    if (T && n > p->cap) {
        // partial gradients, and dpre and dy of n rows
        if (p->part) cudaFree(p->part);
        const size_t floats = (size_t)p->sms * kPart + (size_t)n * (3 * kHid + 4);
        const cudaError_t e = cudaMalloc(&p->part, floats * sizeof(float));
        if (e != cudaSuccess) { p->part = nullptr; p->cap = 0; return mcuda(e, "MLP workspace"); }
        p->cap = n;
    }
    a.part = p->part;
    a.dpre = p->part ? p->part + (size_t)p->sms * kPart : nullptr;
    a.dy = a.dpre ? a.dpre + (size_t)n * 3 * kHid : nullptr;
    if (T) {
        net_kernel<true><<<grid, kNetThreads, kNetSmem, s>>>(a);
        sum_kernel<<<kWeightBlocks + kBiasBlocks, 256, 0, s>>>(a.part, a.dpre, a.dy, grid, n, p->grads, p->loss);
    } else {
        net_kernel<false><<<grid, kNetThreads, kNetSmem, s>>>(a);
    }
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? DISCO_OK : mcuda(e, "network launch");
}

} // namespace

extern "C" {

int disco_b200_mlp_create(uint64_t seed, disco_mlp** out)
{
    if (!out) return mfail(DISCO_EINVAL, "null out");
    *out = nullptr;
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0) return mfail(DISCO_ENODEV, "no CUDA device");
    disco_mlp* p = new disco_mlp();
    cudaError_t e = cudaSuccess;
    // one block: weight image, weights, gradients, Adam's moments, loss, status
    constexpr size_t kVec = ((size_t)kParams * sizeof(float) + 255) / 256 * 256;
    e = cudaMalloc(&p->img, kImg + 4 * kVec + 512);
    if (e != cudaSuccess) { p->img = nullptr; free_mlp(p); return mcuda(e, "MLP allocation"); }
    float** bufs[] = { &p->params, &p->grads, &p->m, &p->v };
    for (int k = 0; k < 4; ++k) *bufs[k] = reinterpret_cast<float*>(p->img + kImg + k * kVec);
    p->loss = reinterpret_cast<float*>(p->img + kImg + 4 * kVec);
    p->status = reinterpret_cast<int*>(p->img + kImg + 4 * kVec + 256);
    // Kaiming-uniform weights (a SplitMix64 stream), zero biases and padding
    std::vector<float> h(kParams, 0.0f);
    uint64_t st = seed * 0x9E3779B97F4A7C15ull + 1;
    auto next = [&]() {
        st += 0x9E3779B97F4A7C15ull;
        uint64_t z = st;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        return (double)(z >> 11) * (1.0 / 9007199254740992.0);
    };
    auto fill = [&](int off, int rows, int cols, int rows_real, int cols_real) {
        const double bound = std::sqrt(6.0 / cols_real);
        for (int r = 0; r < rows; ++r)
            for (int c = 0; c < cols; ++c)
                h[off + r * cols + c] = (r < rows_real && c < cols_real) ? (float)((2.0 * next() - 1.0) * bound) : 0.0f;
    };
    fill(oW1, kHid, kIn, kHid, kInReal);
    fill(oW2, kHid, kHid, kHid, kHid);
    fill(oW3, kHid, kHid, kHid, kHid);
    fill(oW4, kOut, kHid, kOutReal, kHid);
    e = cudaMemcpy(p->params, h.data(), kParams * sizeof(float), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(p->grads, 0, 3 * kVec + 512);
    if (e == cudaSuccess) e = pack_weights(p);
    if (e != cudaSuccess) { free_mlp(p); return mcuda(e, "MLP init"); }
    *out = p;
    return DISCO_OK;
}

int disco_b200_mlp_destroy(disco_mlp* p)
{
    free_mlp(p);
    return DISCO_OK;
}

int disco_b200_mlp_param_count(void) { return kParams; }

int disco_b200_mlp_get_params(const disco_mlp* p, float* host)
{
    if (!p || !host) return mfail(DISCO_EINVAL, "null argument");
    const cudaError_t e = cudaMemcpy(host, p->params, kParams * sizeof(float), cudaMemcpyDeviceToHost);
    return e == cudaSuccess ? DISCO_OK : mcuda(e, "params download");
}

int disco_b200_mlp_set_params(disco_mlp* p, const float* host)
{
    if (!p || !host) return mfail(DISCO_EINVAL, "null argument");
    cudaError_t e = cudaMemcpy(p->params, host, kParams * sizeof(float), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = pack_weights(p);
    return e == cudaSuccess ? DISCO_OK : mcuda(e, "params upload");
}

int disco_b200_mlp_get_grads(const disco_mlp* p, float* host)
{
    if (!p || !host) return mfail(DISCO_EINVAL, "null argument");
    const cudaError_t e = cudaMemcpy(host, p->grads, kParams * sizeof(float), cudaMemcpyDeviceToHost);
    return e == cudaSuccess ? DISCO_OK : mcuda(e, "grads download");
}

int disco_b200_mlp_forward(disco_mlp* p, const float* X, int64_t n, float* Y, void* stream)
{
    if (!p || n < 0 || (n > 0 && (!X || !Y))) return mfail(DISCO_EINVAL, "bad argument");
    if (n == 0) return DISCO_OK;
    return run_net(p, X, nullptr, n, Y, static_cast<cudaStream_t>(stream));
}

// Forward + backward of the MSE loss over n rows; gradients accumulate in the
// model (zeroed by disco_b200_mlp_adam); *loss = mean squared error.
int disco_b200_mlp_grad(disco_mlp* p, const float* X, const float* T, int64_t n, float* loss, void* stream)
{
    if (!p || n <= 0 || !X || !T) return mfail(DISCO_EINVAL, "bad argument");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int st = run_net(p, X, T, n, nullptr, s);
    if (st) return st;
    cudaError_t e;
    if (loss) {
        e = cudaMemcpyAsync(loss, p->loss, sizeof(float), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return mcuda(e, "loss read");
    }
    return DISCO_OK;
}

int disco_b200_mlp_adam(disco_mlp* p, float lr, float beta1, float beta2, float eps, float weight_decay,
                        void* stream)
{
    if (!p) return mfail(DISCO_EINVAL, "null model");
    p->step++;
    const float bc1 = 1.0f - std::pow(beta1, (float)p->step), bc2 = 1.0f - std::pow(beta2, (float)p->step);
    adam_kernel<<<(kParams + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        p->params, p->grads, p->m, p->v, kParams, lr, beta1, beta2, eps, bc1, bc2, weight_decay, p->img);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? DISCO_OK : mcuda(e, "adam");
}

int disco_b200_mlp_status(disco_mlp* p)
{
    if (!p) return mfail(DISCO_EINVAL, "null model");
    int st = 0;
    cudaError_t e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpy(&st, p->status, sizeof(int), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return mcuda(e, "status");
    if (st) { cudaMemset(p->status, 0, sizeof(int)); return mfail(st, "an MLP kernel's bounded wait gave up"); }
    return DISCO_OK;
}

} // extern "C"
