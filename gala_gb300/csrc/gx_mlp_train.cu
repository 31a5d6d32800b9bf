// gx_mlp_train.cu -- training of the potential surrogate (gx_mlp.cuh) on the GPU.
//
// The loss fits both the value and the input gradient of the target:
//   L = alpha * mean_b (y_b - y*_b)^2 + beta * mean_b |G_b - G*_b|^2,  G = d y / d xh,
// so the parameter gradient needs the derivative of the input gradient with
// respect to the parameters ("double backward").  One training step runs, in
// FP32 on the CUDA cores:
//   forward      Z_l = A_{l-1} W_l^T + b_l, A_l = silu(Z_l), keeping S_l = silu'(Z_l), T_l = silu''(Z_l)
//   input grad   D_4 = w5 * S_4, U_l = D_{l+1} W_{l+1}, D_l = U_l * S_l, G = D_1 W_1
//   adjoint      E = dL/dG, e = dL/dy;  back through the input-gradient pass
//                (W1g += D_1^T E, Dbar_1 = E W_1^T, Ubar_l = Dbar_l * S_l,
//                 Zbar_l = Dbar_l * U_l * T_l, W_{l+1}g += D_{l+1}^T Ubar_l,
//                 Dbar_{l+1} = Ubar_l W_{l+1}^T, w5g += sum Dbar_4 * S_4,
//                 Zbar_4 = Dbar_4 * w5 * T_4), then ordinary backprop of the
//                forward pass (Zbar_4 += e w5 * S_4, W_l g += Zbar_l^T A_{l-1},
//                Abar = Zbar_l W_l, Zbar_{l-1} += Abar * S_{l-1}).
// Parameter gradients are written to `grads`; gx_mlp_adam applies Adam.
// Every 256-wide product is a tiled FP32 kernel (rows_kernel, with the elementwise pass
// that follows it in its epilogue; grads_kernel for the weights); the products with the
// 3-wide input or gradient are row and column reductions of their own.  Most of a step is
// 18 products of batch x 256 x 256 at about half the rate of the FP32 pipe: two 128 x 64
// tiles on an SM (84 % of the slots at batch 8,192) that wait for their slabs and for one
// another, and the start and end of each of 42 launches.  Batch 8,192, 16 steps: 21.1 ->
// 12.6 ms.
#include <algorithm>
#include <cooperative_groups.h>

#include "gx_host.h"
#include "gx_mlp.cuh"

namespace cg = cooperative_groups;

namespace gx {
namespace mlp {

// What happens to a product d on its way out:
//   EPI_ACT   z = d + bias -> C = silu(z), p = silu'(z), q = silu''(z)
//   EPI_UD    C = d, p = d * S
//   EPI_ADJ   C = d * S, p = d * U * T
//   EPI_LAST  C = d * S, p = bias (d * T + e S)            (bias the output weights, e per row)
//   EPI_MAC   C += d * S
enum { EPI_ACT, EPI_UD, EPI_ADJ, EPI_LAST, EPI_MAC };

static inline unsigned nblk(int64_t n, int bs) { return (unsigned)((n + bs - 1) / bs); }

struct Epi {
    const float *bias, *S, *U, *T, *e;
    float *p, *q;
};

// two FP32 multiply-adds (each rounded as fmaf) in one instruction
__device__ __forceinline__ void fma2(uint64_t &c, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint64_t twice(float x) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float2 halves(uint64_t x) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(x));
    return r;
}
// four floats into shared memory (zeros unless `in`); VEC: both addresses are multiples of 16 bytes
template <bool VEC>
__device__ __forceinline__ void copy4(float *dst, const float *src, bool in) {
    const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
    if (VEC) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(in ? 16 : 0) : "memory");
    } else {
#pragma unroll
        for (int i = 0; i < 4; i++)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d + 4 * i), "l"(src + i), "r"(in ? 4 : 0)
                         : "memory");
    }
}
__device__ __forceinline__ void copies_end() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void copies_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory");
}

template <bool VEC>
__device__ __forceinline__ float4 load4(const float *p) {
    if (VEC) return *reinterpret_cast<const float4 *>(p);
    return make_float4(p[0], p[1], p[2], p[3]);
}
template <bool VEC>
__device__ __forceinline__ void store4(float *p, float4 v) {
    if (VEC) {
        *reinterpret_cast<float4 *>(p) = v;
    } else {
        p[0] = v.x; p[1] = v.y; p[2] = v.z; p[3] = v.w;
    }
}
__device__ __forceinline__ float4 operator*(float4 a, float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }

// Both products run 128 x 64 tiles, 256 threads of 8 x 4 outputs, two CTAs per SM, over
// K slabs of 16 held [k][row] and [k][column] in three stages of shared memory.  A slab
// is a thousand cycles of the FP32 pipe, about a read that misses L2, so two of them are
// in flight (one slab ahead, 128 x 128 tiles and one CTA per SM left the FP32 pipe 60%
// idle, half of that waiting for global memory).  One instruction multiplies two
// neighbouring rows; with two neighbouring k instead, which needs no transposing, there
// were not the registers to read ahead and rows_kernel took 39 to 60 us for 34 to 38.
constexpr int BM = 128, BN = 64, BK = 16, STAGES = 3;
constexpr int LDM = BM + 4, LDN = BN + 4;
typedef float SlabA[BK][LDM];
typedef float SlabB[BK][LDN];

__device__ __forceinline__ void slab_product(uint64_t (&acc)[4][4], const SlabA &As, const SlabB &Bs, int tx, int ty) {
#pragma unroll
    for (int kk = 0; kk < BK; kk++) {
        const ulonglong2 a0 = *reinterpret_cast<const ulonglong2 *>(&As[kk][ty * 4]);
        const ulonglong2 a1 = *reinterpret_cast<const ulonglong2 *>(&As[kk][64 + ty * 4]);
        const float4 bv = *reinterpret_cast<const float4 *>(&Bs[kk][tx * 4]);
        const uint64_t a[4] = {a0.x, a0.y, a1.x, a1.y};
        const uint64_t b[4] = {twice(bv.x), twice(bv.y), twice(bv.z), twice(bv.w)};
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) fma2(acc[i][j], a[i], b[j]);
    }
}
// the tile's row of acc[i], half r, and its four values
__device__ __forceinline__ int tile_row(int i, int r, int ty) { return (i < 2 ? 0 : 60) + ty * 4 + 2 * i + r; }
__device__ __forceinline__ float4 tile_values(const uint64_t (&c)[4], int r) {
    const float2 v0 = halves(c[0]), v1 = halves(c[1]), v2 = halves(c[2]), v3 = halves(c[3]);
    return r ? make_float4(v0.y, v1.y, v2.y, v3.y) : make_float4(v0.x, v1.x, v2.x, v3.x);
}

// C[M,H] = A[M,H] op(W) and the epilogue; A and C are [M][H], W is [n][k] with TB, else
// [k][n].  What is stored k-contiguous passes through registers and is transposed on the
// way to shared memory (two lanes to a row of 8 k, 4 LDM = 4 LDN = 16 mod 32: no bank
// conflicts), the rest is copied there.
// 8,192 x 256 x 256: 38 -> 34 to 38 us, with the elementwise pass that followed
// it (8-9 us) inside.
template <bool TB, int EPI, bool VEC>
__global__ void __launch_bounds__(256, 2) rows_kernel(int M, const float *__restrict__ A, const float *__restrict__ W,
                                                      float *C, Epi ep) {
    constexpr int SLABS = H / BK;
    __shared__ __align__(16) SlabA As[STAGES];
    __shared__ __align__(16) SlabB Bs[STAGES];
    const int tid = threadIdx.x;
    const int tx = tid % 16, ty = tid / 16;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    // what this thread brings in: rows `row` and row + 64, four k from kq
    const int kq = (tid % 2 + 2 * (tid / 128)) * 4, row = tid % 128 / 2;
    float4 ra[2], rb;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    auto fetch = [&](int slab) {
        const int k0 = slab * BK;
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int gm = m0 + row + 64 * q;
            ra[q] = gm < M ? load4<VEC>(A + (int64_t)gm * H + k0 + kq) : zero;
        }
        if (TB) {
            rb = load4<VEC>(W + (int64_t)(n0 + row) * H + k0 + kq);
        } else {
            copy4<VEC>(&Bs[slab % STAGES][tid / 16][tx * 4], W + (int64_t)(k0 + tid / 16) * H + n0 + tx * 4, true);
            copies_end();
        }
    };
    auto settle = [&](int slab) {
        const int st = slab % STAGES;
#pragma unroll
        for (int q = 0; q < 2; q++) {
            As[st][kq][row + 64 * q] = ra[q].x;
            As[st][kq + 1][row + 64 * q] = ra[q].y;
            As[st][kq + 2][row + 64 * q] = ra[q].z;
            As[st][kq + 3][row + 64 * q] = ra[q].w;
        }
        if (TB) {
            Bs[st][kq][row] = rb.x;
            Bs[st][kq + 1][row] = rb.y;
            Bs[st][kq + 2][row] = rb.z;
            Bs[st][kq + 3][row] = rb.w;
        }
    };
    uint64_t acc[4][4] = {};
#pragma unroll
    for (int s = 0; s < 2; s++) {
        fetch(s);
        settle(s);
    }
    for (int s = 0; s < SLABS; s++) {
        if (!TB) copies_wait<1>();
        __syncthreads();
        if (s + 2 < SLABS) fetch(s + 2);
        else if (!TB) copies_end();
        slab_product(acc, As[s % STAGES], Bs[s % STAGES], tx, ty);
        if (s + 2 < SLABS) settle(s + 2);
    }
    const int gn = n0 + tx * 4;
    const float4 bias = EPI == EPI_ACT || EPI == EPI_LAST ? load4<VEC>(ep.bias + gn) : zero;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        // both rows' operands are read before either is stored: the compiler may not do so
        float4 s[2], t[2], u[2];
        float e[2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const int gm = m0 + tile_row(i, r, ty);
            if (gm >= M) continue;
            const int64_t o = (int64_t)gm * H + gn;
            if (EPI != EPI_ACT) s[r] = load4<VEC>(ep.S + o);
            if (EPI == EPI_ADJ || EPI == EPI_LAST) t[r] = load4<VEC>(ep.T + o);
            if (EPI == EPI_ADJ) u[r] = load4<VEC>(ep.U + o);
            if (EPI == EPI_MAC) u[r] = load4<VEC>(C + o);
            if (EPI == EPI_LAST) e[r] = ep.e[gm];
        }
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const int gm = m0 + tile_row(i, r, ty);
            if (gm >= M) continue;
            const int64_t o = (int64_t)gm * H + gn;
            const float4 d = tile_values(acc[i], r);
            if (EPI == EPI_ACT) {
                float4 a, p, q;
                silu3(d.x + bias.x, a.x, p.x, q.x);
                silu3(d.y + bias.y, a.y, p.y, q.y);
                silu3(d.z + bias.z, a.z, p.z, q.z);
                silu3(d.w + bias.w, a.w, p.w, q.w);
                store4<VEC>(C + o, a);
                store4<VEC>(ep.p + o, p);
                store4<VEC>(ep.q + o, q);
            } else if (EPI == EPI_UD) {
                store4<VEC>(C + o, d);
                store4<VEC>(ep.p + o, d * s[r]);
            } else if (EPI == EPI_ADJ) {
                store4<VEC>(C + o, d * s[r]);
                store4<VEC>(ep.p + o, d * u[r] * t[r]);
            } else if (EPI == EPI_LAST) {
                store4<VEC>(C + o, d * s[r]);
                store4<VEC>(ep.p + o, make_float4(bias.x * (d.x * t[r].x + e[r] * s[r].x), bias.y * (d.y * t[r].y + e[r] * s[r].y),
                                                  bias.z * (d.z * t[r].z + e[r] * s[r].z), bias.w * (d.w * t[r].w + e[r] * s[r].w)));
            } else {
                store4<VEC>(C + o, make_float4(u[r].x + d.x * s[r].x, u[r].y + d.y * s[r].y, u[r].z + d.z * s[r].z,
                                               u[r].w + d.w * s[r].w));
            }
        }
    }
}

// C[H,H] += sum over the rows b of the batch of A[b,:]^T B[b,:], each CTA of a tile over
// its share of the batch (gridDim.z shares, so that the 8 tiles fill two CTAs on every
// SM). Two CTAs of a cluster add their tiles before they add to C, four columns at a
// time: half the additions in a row, whose rounding is most of the error (relative to
// 64 bits, batch 4,096: 1.9e-7 alone, 1.5e-7 in pairs).
// 256 x 256 x 8,192: 56 -> 26 us.
template <bool VEC>
__global__ void __cluster_dims__(1, 1, 2) __launch_bounds__(256, 2) grads_kernel(int64_t batch, int share, const float *__restrict__ A,
                                                       const float *__restrict__ B, float *__restrict__ C) {
    __shared__ __align__(16) union {
        struct {
            SlabA As[STAGES];
            SlabB Bs[STAGES];
        } in;
        float4 tile[BM][BN / 4];
    } sh;
    SlabA *const As = sh.in.As;
    SlabB *const Bs = sh.in.Bs;
    const int tid = threadIdx.x;
    const int tx = tid % 16, ty = tid / 16;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int64_t kbeg = (int64_t)blockIdx.z * share;
    const int64_t kend = min(batch, kbeg + share);
    const int slabs = kbeg < kend ? (int)((kend - kbeg + BK - 1) / BK) : 0;
    auto fetch = [&](int slab) {
        const int64_t k0 = kbeg + (int64_t)slab * BK;
        const int st = slab % STAGES;
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int e = tid + 256 * q, kk = e / 32, mm = e % 32 * 4;
            const bool in = k0 + kk < kend;
            copy4<VEC>(&As[st][kk][mm], A + (in ? k0 + kk : 0) * H + m0 + mm, in);
        }
        const bool in = k0 + ty < kend;
        copy4<VEC>(&Bs[st][ty][tx * 4], B + (in ? k0 + ty : 0) * H + n0 + tx * 4, in);
        copies_end();
    };
    uint64_t acc[4][4] = {};
#pragma unroll
    for (int s = 0; s < 2; s++) {
        if (s < slabs) fetch(s);
        else copies_end();
    }
    for (int s = 0; s < slabs; s++) {
        copies_wait<1>();
        __syncthreads();
        if (s + 2 < slabs) fetch(s + 2);
        else copies_end();
        slab_product(acc, As[s % STAGES], Bs[s % STAGES], tx, ty);
    }
    copies_wait<0>();
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int r = 0; r < 2; r++) sh.tile[tile_row(i, r, ty)][tx] = tile_values(acc[i], r);
    // each CTA adds up half of the rows
    cg::cluster_group pair = cg::this_cluster();
    pair.sync();
    const unsigned rank = pair.block_rank();
    const float4(*const theirs)[BN / 4] = pair.map_shared_rank(sh.tile, rank ^ 1);
#pragma unroll
    for (int q = 0; q < BM / 2 / 16; q++) {
        const int row = rank * (BM / 2) + 16 * q + ty;
        const float4 a = sh.tile[row][tx], b = theirs[row][tx];
        const float4 d = make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
        float *c = C + (int64_t)(m0 + row) * H + n0 + tx * 4;
        if (VEC) {
            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(c), "f"(d.x), "f"(d.y), "f"(d.z), "f"(d.w)
                         : "memory");
        } else {
            atomicAdd(c, d.x);
            atomicAdd(c + 1, d.y);
            atomicAdd(c + 2, d.z);
            atomicAdd(c + 3, d.w);
        }
    }
    pair.sync();  // the other CTA has read this one's tile
}

template <typename... P>
static bool aligned16(const P *...p) {
    return ((... | reinterpret_cast<uintptr_t>(p)) & 15) == 0;
}

// C = A op(W) with its epilogue
template <bool TB, int EPI>
static void rows(cudaStream_t st, int64_t batch, const float *A, const float *W, float *C, const Epi &ep) {
    const dim3 grid(H / BN, nblk(batch, BM));
    if (aligned16(A, W, C, ep.bias, ep.S, ep.U, ep.T, ep.p, ep.q))
        rows_kernel<TB, EPI, true><<<grid, 256, 0, st>>>((int)batch, A, W, C, ep);
    else
        rows_kernel<TB, EPI, false><<<grid, 256, 0, st>>>((int)batch, A, W, C, ep);
}

// C += A^T B over the batch
static void weight_grads(cudaStream_t st, int64_t batch, const float *A, const float *B, float *C) {
    constexpr int TILES = (H / BM) * (H / BN);
    // whole pairs of CTAs, no more than two CTAs on every SM: a pair beyond is a second wave
    const int64_t split = std::max(2 * gx::multiprocessors() / TILES / 2 * 2, 2);
    const int share = (int)(((batch + split - 1) / split + BK - 1) / BK * BK);
    const dim3 grid(H / BN, H / BM, (nblk(batch, share) + 1) / 2 * 2);
    if (aligned16(A, B, C))
        grads_kernel<true><<<grid, 256, 0, st>>>(batch, share, A, B, C);
    else
        grads_kernel<false><<<grid, 256, 0, st>>>(batch, share, A, B, C);
}

// G[b, 0..2] = D[b, :] W with W [H][3] (one warp per row; as a 128-wide tile 38 us, now 7)
__global__ void rows3_kernel(int64_t B, const float *__restrict__ D, const float *__restrict__ W, float *__restrict__ G) {
    const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32;
    const int lane = threadIdx.x & 31;
    if (row >= B) return;
    float g0 = 0.f, g1 = 0.f, g2 = 0.f;
    for (int k = lane; k < H; k += 32) {
        const float d = D[row * H + k];
        g0 = fmaf(d, W[3 * k], g0);
        g1 = fmaf(d, W[3 * k + 1], g1);
        g2 = fmaf(d, W[3 * k + 2], g2);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        g0 += __shfl_xor_sync(0xffffffffu, g0, o);
        g1 += __shfl_xor_sync(0xffffffffu, g1, o);
        g2 += __shfl_xor_sync(0xffffffffu, g2, o);
    }
    if (lane < 3) G[row * 3 + lane] = lane == 0 ? g0 : lane == 1 ? g1 : g2;
}

// The column reductions: a CTA takes 256 rows of the batch, four groups of 256 threads
// 64 each, and adds the groups' sums before it adds to the result: 32 additions in a row
// for 8,192 samples.  (With 256 rows to a thread a column sum took 21 us, now 8; with
// 32 rows to a thread and 256 CTAs 6 us, but twice the rounding error.)
constexpr int COL_GROUPS = 4, COL_ROWS = 64;

// W[k, 0..2] += sum_b X[b, k] Y[b, 0..2], and with `sum` sum[k] += sum_b X[b, k] (as
// 128-wide tiles 51 us, now 9)
__global__ void __launch_bounds__(COL_GROUPS *H) cols3_kernel(int64_t B, const float *__restrict__ X, const float *__restrict__ Y,
                                                              float *__restrict__ W, float *__restrict__ sum) {
    const int k = threadIdx.x % H, part = threadIdx.x / H;
    const int64_t c0 = (int64_t)blockIdx.x * COL_GROUPS * COL_ROWS, r0 = c0 + part * COL_ROWS;
    __shared__ float y[3 * COL_GROUPS * COL_ROWS], sums[COL_GROUPS][4][H];
    if (threadIdx.x < 3 * COL_GROUPS * COL_ROWS) y[threadIdx.x] = 3 * c0 + threadIdx.x < 3 * B ? Y[3 * c0 + threadIdx.x] : 0.f;
    __syncthreads();
    float w0 = 0.f, w1 = 0.f, w2 = 0.f, s = 0.f;
#pragma unroll 16
    for (int r = 0; r < COL_ROWS; r++) {
        const float x = r0 + r < B ? X[(r0 + r) * H + k] : 0.f;
        const float *yr = y + 3 * (part * COL_ROWS + r);
        w0 = fmaf(x, yr[0], w0);
        w1 = fmaf(x, yr[1], w1);
        w2 = fmaf(x, yr[2], w2);
        s += x;
    }
    sums[part][0][k] = w0;
    sums[part][1][k] = w1;
    sums[part][2][k] = w2;
    sums[part][3][k] = s;
    __syncthreads();
    const float total = (sums[0][part][k] + sums[1][part][k]) + (sums[2][part][k] + sums[3][part][k]);
    if (part < 3) atomicAdd(&W[3 * k + part], total);
    else if (sum) atomicAdd(&sum[k], total);
}

// The adjoint of G = D_1 W_1 for the first layer: d = E W_1^T, Ubar = d * S, Zbar = d * U * T
__global__ void adj1_kernel(int64_t n, const float *__restrict__ E, const float *__restrict__ W1, const float *__restrict__ S,
                            const float *__restrict__ U, const float *__restrict__ T, float *__restrict__ Ubar,
                            float *__restrict__ Zbar) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t b = i / H;
    const int k = (int)(i % H);
    const float d = fmaf(E[b * 3 + 2], W1[3 * k + 2], fmaf(E[b * 3 + 1], W1[3 * k + 1], E[b * 3] * W1[3 * k]));
    Ubar[i] = d * S[i];
    Zbar[i] = d * U[i] * T[i];
}

// out[b] = dot(A[b,:], w) + c  (one warp per row)
__global__ void rowdot_kernel(int64_t B, const float *__restrict__ A, const float *__restrict__ w,
                              const float *__restrict__ c, float *__restrict__ out) {
    const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32;
    const int lane = threadIdx.x & 31;
    if (row >= B) return;
    float acc = 0.f;
    for (int k = lane; k < H; k += 32) acc = fmaf(A[row * H + k], w[k], acc);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) out[row] = acc + (c ? *c : 0.f);
}

// D4 = w5 * S4 (row-broadcast)
__global__ void d4_kernel(int64_t n, const float *__restrict__ w5, const float *__restrict__ S4,
                          float *__restrict__ D4) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) D4[i] = w5[i % H] * S4[i];
}

// loss terms and their seeds: e = 2 alpha (y - y*) / B, E = 2 beta w (G - G*) / B
// (w = per-sample weight of the gradient term, 1 if wg is NULL)
__global__ void loss_kernel(int64_t B, float alpha, float beta, const float *__restrict__ y,
                            const float *__restrict__ ys, const float *__restrict__ G, const float *__restrict__ Gs,
                            const float *__restrict__ wg, float *__restrict__ e, float *__restrict__ E,
                            float *__restrict__ loss) {
    const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    float lv = 0.f, lg = 0.f;
    if (b < B) {
        const float dv = y[b] - ys[b];
        e[b] = 2.f * alpha * dv / (float)B;
        lv = dv * dv;
        const float wb = wg ? wg[b] : 1.f;
        for (int j = 0; j < 3; j++) {
            const float dg = G[b * 3 + j] - Gs[b * 3 + j];
            E[b * 3 + j] = 2.f * beta * wb * dg / (float)B;
            lg += wb * dg * dg;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lv += __shfl_xor_sync(0xffffffffu, lv, o);
        lg += __shfl_xor_sync(0xffffffffu, lg, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&loss[0], lv / (float)B);
        atomicAdd(&loss[1], lg / (float)B);
    }
}

// column sums over the batch: out[k] = sum_b X[b, k] (+ sum_b e[b] Y[b, k] if e)
__global__ void __launch_bounds__(COL_GROUPS *H) colsum_kernel(int64_t B, const float *__restrict__ X, const float *__restrict__ e,
                                                               const float *__restrict__ Y, float *__restrict__ out) {
    const int k = threadIdx.x % H, part = threadIdx.x / H;
    const int64_t r0 = ((int64_t)blockIdx.x * COL_GROUPS + part) * COL_ROWS;
    __shared__ float sums[COL_GROUPS][H];
    float acc = 0.f;
#pragma unroll 16
    for (int r = 0; r < COL_ROWS; r++) {
        const bool in = r0 + r < B;
        acc += in ? X[(r0 + r) * H + k] : 0.f;
        if (e) acc += in ? e[r0 + r] * Y[(r0 + r) * H + k] : 0.f;
    }
    sums[part][k] = acc;
    __syncthreads();
    if (part == 0) atomicAdd(&out[k], (sums[0][k] + sums[1][k]) + (sums[2][k] + sums[3][k]));
}

// out += sum_b x[b]
__global__ void sum_kernel(int64_t B, const float *__restrict__ x, float *__restrict__ out) {
    const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    float v = b < B ? x[b] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(out, v);
}

// layer-1 forward with K = 3 inputs
__global__ void layer1_kernel(int64_t B, const float *__restrict__ X, const float *__restrict__ P,
                              float *__restrict__ A, float *__restrict__ S, float *__restrict__ T) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= B * H) return;
    const int64_t b = i / H;
    const int o = (int)(i % H);
    const float *W1 = P + OFF_W1;
    const float z = W1[o * 3 + 0] * X[b * 3 + 0] + W1[o * 3 + 1] * X[b * 3 + 1] + W1[o * 3 + 2] * X[b * 3 + 2] +
                    P[OFF_B1 + o];
    float a, s1, s2;
    silu3(z, a, s1, s2);
    A[i] = a;
    S[i] = s1;
    T[i] = s2;
}

// Adam (bias-corrected), FP32 master weights
__global__ void adam_kernel(int64_t n, float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m,
                            float *__restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}


}  // namespace mlp
}  // namespace gx

using namespace gx::mlp;

extern "C" int64_t gx_mlp_param_count(void) { return NPARAM; }

extern "C" int64_t gx_mlp_train_workspace_floats(int64_t batch) { return batch * (26 * (int64_t)H + 16); }

extern "C" int gx_mlp_forward(const float *params, const float *xh, int64_t B, float *y, float *G, float *workspace,
                              void *stream) {
    GX_CHECK_ARG(params && xh && y && workspace && B > 0 && B < (1 << 26), "bad arguments");
    cudaStream_t st = gx::as_stream(stream);
    const int64_t n = B * H;
    float *w = workspace;
    float *A[5], *S[5], *T[5], *D[5], *U[4];
    for (int l = 1; l <= 4; l++) {
        A[l] = w; w += n;
        S[l] = w; w += n;
        T[l] = w; w += n;
        D[l] = w; w += n;
    }
    for (int l = 1; l <= 3; l++) { U[l] = w; w += n; }
    layer1_kernel<<<nblk(n, 256), 256, 0, st>>>(B, xh, params, A[1], S[1], T[1]);
    for (int l = 2; l <= 4; l++) {
        Epi ep = {};
        ep.bias = params + off_b(l);
        ep.p = S[l];
        ep.q = T[l];
        rows<true, EPI_ACT>(st, B, A[l - 1], params + off_W(l), A[l], ep);
    }
    rowdot_kernel<<<nblk(B * 32, 256), 256, 0, st>>>(B, A[4], params + OFF_W5, params + OFF_B5, y);
    if (G) {
        d4_kernel<<<nblk(n, 256), 256, 0, st>>>(n, params + OFF_W5, S[4], D[4]);
        for (int l = 3; l >= 1; l--) {
            Epi ep = {};
            ep.S = S[l];
            ep.p = D[l];
            rows<false, EPI_UD>(st, B, D[l + 1], params + off_W(l + 1), U[l], ep);
        }
        rows3_kernel<<<nblk(B * 32, 256), 256, 0, st>>>(B, D[1], params + OFF_W1, G);
    }
    return gx::check_launch("mlp_forward");
}

extern "C" int gx_mlp_train_step(const float *params, float *grads, const float *xh, const float *ystar,
                                 const float *Gstar, const float *gweight, int64_t B, float alpha, float beta,
                                 float *workspace, float *loss, void *stream) {
    GX_CHECK_ARG(params && grads && xh && ystar && Gstar && workspace && loss, "NULL pointer");
    GX_CHECK_ARG(B > 0 && B < (1 << 26), "batch out of range");
    cudaStream_t st = gx::as_stream(stream);
    const int64_t n = B * H;
    float *w = workspace;
    float *A[5], *S[5], *T[5], *D[5], *U[4];
    for (int l = 1; l <= 4; l++) {
        A[l] = w; w += n;
        S[l] = w; w += n;
        T[l] = w; w += n;
        D[l] = w; w += n;
    }
    for (int l = 1; l <= 3; l++) { U[l] = w; w += n; }
    float *Zb[5];
    for (int l = 1; l <= 4; l++) { Zb[l] = w; w += n; }
    w += n;
    float *Ubar = w; w += n;
    float *Abar = w; w += n;
    float *y = w; w += B;
    float *e = w; w += B;
    float *G = w; w += 3 * B;
    float *E = w; w += 3 * B;
    const float *W5 = params + OFF_W5;
    float *g = grads;

    GX_CUDA_TRY(cudaMemsetAsync(grads, 0, sizeof(float) * NPARAM, st));
    GX_CUDA_TRY(cudaMemsetAsync(loss, 0, sizeof(float) * 2, st));
    // forward and input gradient
    int rc = gx_mlp_forward(params, xh, B, y, G, workspace, stream);
    if (rc) return rc;
    loss_kernel<<<nblk(B, 256), 256, 0, st>>>(B, alpha, beta, y, ystar, G, Gstar, gweight, e, E, loss);

    // adjoint of the input-gradient pass
    const unsigned cols = nblk(B, COL_GROUPS * COL_ROWS);
    cols3_kernel<<<cols, COL_GROUPS * H, 0, st>>>(B, D[1], E, g + OFF_W1, nullptr);  // W1g += D1^T E
    adj1_kernel<<<nblk(n, 256), 256, 0, st>>>(n, E, params + OFF_W1, S[1], U[1], T[1], Ubar, Zb[1]);
    for (int l = 1; l <= 3; l++) {
        // W_{l+1} g += D_{l+1}^T Ubar_l  : [256 x B] x [B x 256]
        weight_grads(st, B, D[l + 1], Ubar, g + off_W(l + 1));
        // Dbar_{l+1} = Ubar_l W_{l+1}^T, and what follows it
        Epi ep = {};
        ep.S = S[l + 1];
        ep.T = T[l + 1];
        ep.p = Zb[l + 1];
        if (l < 3) {
            ep.U = U[l + 1];
            rows<true, EPI_ADJ>(st, B, Ubar, params + off_W(l + 1), Abar, ep);
            float *next = Ubar;
            Ubar = Abar;
            Abar = next;
        } else {
            // Abar = Dbar4 * S4 ; Zbar4 = w5 * (Dbar4 * T4 + e * S4)
            ep.bias = W5;
            ep.e = e;
            rows<true, EPI_LAST>(st, B, Ubar, params + off_W(4), Abar, ep);
        }
    }
    // w5g += colsum(Dbar4 * S4) + A4^T e
    colsum_kernel<<<cols, COL_GROUPS * H, 0, st>>>(B, Abar, e, A[4], g + OFF_W5);
    // b5g = sum e
    sum_kernel<<<nblk(B, 256), 256, 0, st>>>(B, e, g + OFF_B5);
    // backprop through the forward pass
    for (int l = 4; l >= 2; l--) {
        weight_grads(st, B, Zb[l], A[l - 1], g + off_W(l));  // W_l g += Zbar^T A
        colsum_kernel<<<cols, COL_GROUPS * H, 0, st>>>(B, Zb[l], nullptr, nullptr, g + off_b(l));
        Epi ep = {};
        ep.S = S[l - 1];
        rows<false, EPI_MAC>(st, B, Zb[l], params + off_W(l), Zb[l - 1], ep);  // Zbar_{l-1} += (Zbar_l W_l) * S
    }
    cols3_kernel<<<cols, COL_GROUPS * H, 0, st>>>(B, Zb[1], xh, g + OFF_W1, g + OFF_B1);  // W1g += Zbar1^T X, b1g
    return gx::check_launch("mlp_train_step");
}

extern "C" int gx_mlp_adam(float *params, const float *grads, float *m, float *v, int64_t n, float lr, float beta1,
                           float beta2, float eps, int64_t step, void *stream) {
    GX_CHECK_ARG(params && grads && m && v && n > 0 && step >= 1, "bad arguments");
    const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
    adam_kernel<<<nblk(n, 256), 256, 0, gx::as_stream(stream)>>>(n, params, grads, m, v, lr, beta1, beta2, eps, c1,
                                                                  c2);
    return gx::check_launch("mlp_adam");
}
