// fs_mlp_train.cu -- training of the learned bisection proposal's network on the tcgen05
// tensor cores (BF16 operands, FP32 accumulation in tensor memory), its Adam step and weight
// packing, and the C ABI of training and batched inference.  No counterpart in the
// reference.
//
// Parameters (FP32 master copy, one flat array, FS_MLP_NPARAM floats):
//   W1[128][16] b1[128] W2[128][128] b2[128] W3[128][128] b3[128] W4[16][128] b4[16]
// The forward pass keeps the BF16 activations in shared memory; the loss gradient is formed
// per row; the backward pass runs dA = dZ W and dW = dZ^T A and adds the weight / bias
// gradients to an FP32 gradient array with atomics, or leaves each CTA's own for the optimiser to
// add in order (the Adam kernel divides nothing: the loss is already a batch mean).
// The orders are different numbers: a gradient's last bit, through Adam's m / sqrt(v) and the BF16
// rounding of the weights, becomes 1e-4 of the parameters within some twenty steps.  The atomics have
// a few usual orders, so that four runs of five end within 1e-6 of another run's parameters (14
// batches of 683 to 4458 rows, 11 to 37 steps); the order of the CTAs' numbers is as exact but may
// be none of those (683 rows, 17 steps: 1.2e-4 from every one of 20 runs).
//
// Loss (per row, D degrees of freedom, z the midpoint's displacement from the endpoints'
// mean in units of sigma_1): sum_d 0.5 (z_d - o_d)^2 exp(-s_d) + 0.5 s_d with
// s_d = 4 tanh(o_{D+d} / 4): the Gaussian negative log-likelihood of z under N(o, exp(s)).
#include <cuda_runtime.h>

#include <stddef.h>

#include "../../include/feynsimul.h"
#include "fs_mlp.cuh"
#include "fs_tc.cuh"

#define FS_MLP_NPARAM (128 * 16 + 128 + 128 * 128 + 128 + 128 * 128 + 128 + 16 * 128 + 16)
#define P_W1 0
#define P_B1 (P_W1 + 128 * 16)
#define P_W2 (P_B1 + 128)
#define P_B2 (P_W2 + 128 * 128)
#define P_W3 (P_B2 + 128)
#define P_B3 (P_W3 + 128 * 128)
#define P_W4 (P_B3 + 128)
#define P_B4 (P_W4 + 16 * 128)
static_assert(P_W1 % 4 == 0 && P_W2 % 4 == 0 && P_W3 % 4 == 0, "16-byte gradient rows");

// BF16 weight copy used by training (row-major, same order as the FP32 weights, no biases)
#define Q_W1 0
#define Q_W2 (Q_W1 + 128 * 16)
#define Q_W3 (Q_W2 + 128 * 128)
#define Q_W4 (Q_W3 + 128 * 128)
#define Q_N (Q_W4 + 16 * 128)

extern int fsi_thread_error(int code, const char *msg);

__device__ __forceinline__ fs_bf16 f2bf(float x)
{
    unsigned r = fs_pack_bf16(x, 0.f);
    return (fs_bf16)(r & 0xFFFFu);
}

// ---------------------------------------------------------------- tcgen05 training
// The same forward pass, loss and backward pass on the fifth-generation tensor cores, with
// the same BF16 rounding points.  One CTA = 16 warps, persistent over 128-row tiles; a row of a
// tile (a tensor-memory lane) belongs to the four threads r + 128 k, which take a quarter of its
// columns each in every epilogue (a warp reads the 32 lanes of its number modulo 4).  The step is
// a chain of 8 MMA groups with an epilogue between.  With two threads a row, one tile took 34
// thousand cycles (42 with one, and gradients stored line by line): the MMAs and their waits about
// 7, the epilogues 15, the weights 5 and the gradient's way out 5.  So the epilogues have four
// threads a row, and the weight-gradient MMAs, which nothing in the tile waits for, run behind the
// next epilogue.  A step on 4096 rows, optimiser and gather included, took 105 us in ten launches;
// 31 in three launches with two threads a row, and 27 now, the optimiser's launch overlapped too.
// Rows of a training set are gathered in place by an index array.  Tensor memory (512 FP32
// columns): the layer accumulator F (a forward layer's output or a hidden gradient dA), and
// the weight gradients summed over the CTA's tiles: dW2 and dW3 (128 columns each), dW1 (16)
// and dW4 transposed (16; its M is the 128 inputs).  Shared memory holds BF16 tiles in the
// canonical layout of fs_tc.cuh: the activations a1..a3 and the hidden gradient (in g, then a3, then
// g again), 128 x 128 each with the tile's rows, the input x and the output gradient dz4 (128 x
// 16), and the weights W1..W4 ([out][in]).  The forward GEMMs read them K-major; dA = dZ W reads W
// MN-major, and dW = dZ^T A reads dZ and A MN-major (K = the tile's rows), so no tile is
// transposed.  The six 128-wide tiles come first and the allocation is padded, so every
// byte a descriptor can reach lies inside it under either reading of its byte offsets.
// Bias gradients are FP32 column sums of the unrounded gradients (warp butterflies, each quarter
// of the rows on its own, then the quarters in order).
// A CTA's gradient goes to its own row of `part` for the optimiser step to add up in order
// (fs_mlp_train_batch: the same training run gives the same bits), or, without one, to grad
// by atomics (fs_mlp_train_step, fs_mlp_train_rows).
#define TT_THREADS 512
#define TT_TMEM_COLS 512
#define TT_F 0u
#define TT_DW2 128u
#define TT_DW3 256u
#define TT_DW1 384u
#define TT_DW4 400u

struct TtSmem {
    alignas(1024) fs_bf16 a1[128 * 128];
    alignas(128) fs_bf16 a2[128 * 128];
    alignas(128) fs_bf16 w2[128 * 128];
    alignas(128) fs_bf16 w3[128 * 128];
    alignas(128) fs_bf16 w4[16 * 128];
    alignas(128) fs_bf16 a3[128 * 128];
    alignas(128) fs_bf16 g[128 * 128];
    alignas(128) fs_bf16 x[128 * 16];
    alignas(128) fs_bf16 dz4[128 * 16];
    alignas(128) fs_bf16 w1[128 * 16];
    float bias[128 * 3 + 16];
    float db[4][128 * 3 + 16];  // bias gradients of each quarter of a tile's rows
    float loss[4];
    alignas(8) unsigned long long mbar, mbar_last;
    unsigned tmem_base;
    int give_up;
};
// farthest byte a read of a 128-wide tile can reach from the tile's start: 8 K-steps of 16
// rows (4096 bytes each) plus 15 column blocks and one row block at the larger offset
#define TT_REACH (7 * 4096 + 15 * 2048 + 256)
#define TT_SMEM_BYTES \
    (offsetof(TtSmem, g) + TT_REACH > sizeof(TtSmem) ? offsetof(TtSmem, g) + TT_REACH : sizeof(TtSmem))

// A row of `part`: a gradient in the parameters' order, but W1..W3 by quads of inputs, (input / 4,
// output, input mod 4), so that a warp of tensor-memory lanes (outputs) writes 512 consecutive bytes
// (in the parameters' order each of its 16-byte stores is a line of its own, and the 144 KB took 12
// of the pass's 42 thousand cycles); then the loss, padded to 16 floats
__device__ __forceinline__ int tt_quad(int row, int col, int rows) { return (col >> 2) * 4 * rows + row * 4 + (col & 3); }
#define TT_PART ((FS_MLP_NPARAM + 1 + 15) / 16 * 16)

// column sums over the warp's 32 lanes of v[0..32) (one value per column and lane), added to
// dst[lane] for lane < ncols (no other warp adds there); v is consumed
__device__ __forceinline__ void tt_colsum32(float (&v)[32], float *dst, int lane, int ncols)
{
#pragma unroll
    for (int w = 16; w >= 1; w >>= 1) {
        const bool up = (lane & w) != 0;
#pragma unroll
        for (int i = 0; i < w; i++) {
            const float send = up ? v[i] : v[i + w];
            const float keep = up ? v[i + w] : v[i];
            v[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, w);
        }
    }
    if (lane < ncols) dst[lane] += v[0];
}

__global__ void __launch_bounds__(TT_THREADS, 1) fs_mlp_train_tc_kernel(
    const float *__restrict__ params, const fs_bf16 *__restrict__ wq, float *__restrict__ grad,
    const float *__restrict__ xin, const float *__restrict__ zin, const long long *__restrict__ pick, int n_rows,
    int dof, float inv_batch, float *loss_out, float *part)
{
    extern __shared__ __align__(1024) unsigned char tt_raw[];
    TtSmem &S = *reinterpret_cast<TtSmem *>(tt_raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int r = tid & 127, quarter = tid >> 7;  // row of the tile, quarter of its columns
    const int n_tiles = (n_rows + 127) / 128;
    const uint32_t mbar = tc_smem(&S.mbar);

    // ---- the first tile's rows, ahead of the weights ----
    const int row0 = (int)blockIdx.x * 128 + r;
    const bool valid0 = row0 < n_rows;
    size_t src = valid0 && pick ? (size_t)pick[row0] : (size_t)row0;
    // half a row of x (quarters 0 and 1), and the row's z (quarter 0)
    float4 xv[2], zv[2];
    auto fetch = [&](bool valid) {
        const float4 *xr = reinterpret_cast<const float4 *>(xin + src * 16 + 8 * (quarter & 1));
#pragma unroll
        for (int c = 0; c < 2; c++) xv[c] = valid && quarter < 2 ? xr[c] : make_float4(0.f, 0.f, 0.f, 0.f);
        float *z = reinterpret_cast<float *>(zv);
#pragma unroll
        for (int d = 0; d < 8; d++) z[d] = valid && quarter == 0 && d < dof ? zin[src * 8 + d] : 0.f;
    };
    // ---- weights (the BF16 training copy, [out][in]) into canonical tiles, eight
    // consecutive inputs (one core-matrix row, 16 bytes) per load and store; a warp takes 8
    // rows of 4 core matrices: 64 contiguous bytes of each row, 512 of the tile ----
    {
        const uint4 *q = reinterpret_cast<const uint4 *>(wq);
        const int lr = lane & 7, lk = lane >> 3;
        auto tile128 = [&](fs_bf16 *w, int off, int rows) {
#pragma unroll 8
            for (int i = warp; i < rows / 8 * 4; i += TT_THREADS / 32) {
                const int row = i / 4 * 8 + lr, k = i % 4 * 4 + lk;
                *reinterpret_cast<uint4 *>(w + tc_off(row, k * 8, 128)) = q[off / 8 + row * 16 + k];
            }
        };
        tile128(S.w2, Q_W2, 128);
        tile128(S.w3, Q_W3, 128);
        tile128(S.w4, Q_W4, 16);
        if (warp < 8) {
            const int row = warp * 16 + (lane & 15), k = lane >> 4;  // 16 rows of 2 core matrices a warp
            *reinterpret_cast<uint4 *>(S.w1 + tc_off(row, k * 8, 16)) = q[Q_W1 / 8 + row * 2 + k];
        }
    }
    fetch(valid0);
    for (int i = tid; i < 128; i += TT_THREADS) {
        S.bias[i] = params[P_B1 + i];
        S.bias[128 + i] = params[P_B2 + i];
        S.bias[256 + i] = params[P_B3 + i];
    }
    if (tid < 16) S.bias[384 + tid] = params[P_B4 + tid];
    for (int i = tid; i < 4 * (128 * 3 + 16); i += TT_THREADS) S.db[0][i] = 0.f;
    if (tid < 4) S.loss[tid] = 0.f;
    if (tid == 0) {
        S.give_up = 0;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&S.mbar_last)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(&S.tmem_base)),
                     "r"(TT_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = S.tmem_base;
    const uint32_t t_row = tmem + ((uint32_t)(32 * (warp & 3)) << 16);  // this warp's lanes
    uint32_t phase = 0;
    bool ok = true, first = true;
    float *const db = S.db[warp & 3];

    // the optimiser's CTAs may take their places now; they wait for this grid's end
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    // one step: the operands made visible to the tensor cores, thread 0 issues the MMAs and
    // commits, every thread waits (bounded) for them.  The MMAs of `after` run behind them, during
    // the epilogue: the next step's wait covers them.
    auto step = [&](auto &&issue, auto &&after) {
        tc_fence_async();
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        if (tid == 0) {
            issue();
            tc_commit(mbar);
            after();
        }
        if (!tc_wait(mbar, phase)) S.give_up = 1;
        phase ^= 1u;
        tc_fence_after();
        __syncthreads();
        ok = S.give_up == 0;
        return ok;
    };
    auto none = [] {};
    // forward epilogue: act = BF16(relu(F + b))
    auto relu_out = [&](fs_bf16 *act, const float *b) {
#pragma unroll 1
        for (int c0 = 32 * quarter; c0 < 32 * quarter + 32; c0 += 16) {
            float v[16];
            tc_ld16(t_row + TT_F + (uint32_t)c0, v);
#pragma unroll
            for (int i = 0; i < 16; i++) v[i] = fmaxf(v[i] + b[c0 + i], 0.f);
            tc_st8(act + tc_off(r, c0, 128), v);
            tc_st8(act + tc_off(r, c0 + 8, 128), v + 8);
        }
    };
    // backward epilogue: dZ = F * (act > 0) -> g as BF16, its FP32 column sums into dbl
    auto grad_out = [&](const fs_bf16 *act, fs_bf16 *g, float *dbl) {
        {
            const int c0 = 32 * quarter;
            float v[32];
            tc_ld16(t_row + TT_F + (uint32_t)c0, *reinterpret_cast<float(*)[16]>(v));
            tc_ld16(t_row + TT_F + (uint32_t)c0 + 16u, *reinterpret_cast<float(*)[16]>(v + 16));
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const uint4 u = *reinterpret_cast<const uint4 *>(act + tc_off(r, c0 + 8 * q, 128));
                const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    if (!(__uint_as_float(w[e] << 16) > 0.f)) v[8 * q + 2 * e] = 0.f;
                    if (!(__uint_as_float(w[e] & 0xFFFF0000u) > 0.f)) v[8 * q + 2 * e + 1] = 0.f;
                }
                tc_st8(g + tc_off(r, c0 + 8 * q, 128), v + 8 * q);
            }
            tt_colsum32(v, dbl + c0, lane, 32);
        }
    };

    for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
        const int row = tile * 128 + r;
        const bool valid = row < n_rows;
        if (tile != (int)blockIdx.x) {
            src = valid && pick ? (size_t)pick[row] : (size_t)row;
            fetch(valid);
        }
        if (quarter < 2) tc_st8(S.x + tc_off(r, 8 * quarter, 16), reinterpret_cast<const float *>(xv));
        // ---- forward ----
        if (!step([&] { tc_mma(tmem + TT_F, tc_desc(S.x, 16), tc_desc(S.w1, 16), tc_idesc(128, 128), 0); }, none))
            break;
        relu_out(S.a1, S.bias);
        if (!step([&] {
                for (int kk = 0; kk < 8; kk++)
                    tc_mma(tmem + TT_F, tc_desc(S.a1 + kk * 128, 128), tc_desc(S.w2 + kk * 128, 128),
                           tc_idesc(128, 128), kk > 0);
            }, none))
            break;
        relu_out(S.a2, S.bias + 128);
        if (!step([&] {
                for (int kk = 0; kk < 8; kk++)
                    tc_mma(tmem + TT_F, tc_desc(S.a2 + kk * 128, 128), tc_desc(S.w3 + kk * 128, 128),
                           tc_idesc(128, 128), kk > 0);
            }, none))
            break;
        relu_out(S.a3, S.bias + 256);
        if (!step([&] {
                for (int kk = 0; kk < 8; kk++)
                    tc_mma(tmem + TT_F, tc_desc(S.a3 + kk * 128, 128), tc_desc(S.w4 + kk * 128, 128),
                           tc_idesc(128, 16), kk > 0);
            }, none))
            break;
        // ---- loss and its gradient for this thread's row ----
        if (quarter == 0) {
            float z4[16], g[32];
            tc_ld16(t_row + TT_F, z4);
#pragma unroll
            for (int c = 0; c < 16; c++) z4[c] += S.bias[384 + c];
#pragma unroll
            for (int c = 0; c < 32; c++) g[c] = 0.f;
            float l = 0.f;
            if (valid) {
#pragma unroll
                for (int d = 0; d < 8; d++) {
                    if (d >= dof) break;
                    float sr = 0.f;
#pragma unroll
                    for (int c = 0; c < 16; c++) sr = c == dof + d ? z4[c] : sr;
                    const float o = z4[d];
                    const float th = tanhf(0.25f * sr);
                    const float s = 4.f * th;
                    const float e = expf(-s);
                    const float z = reinterpret_cast<const float *>(zv)[d];
                    const float df = z - o;
                    l += 0.5f * df * df * e + 0.5f * s;
                    g[d] = -df * e * inv_batch;
                    const float gs = (0.5f - 0.5f * df * df * e) * (1.f - th * th) * inv_batch;
#pragma unroll
                    for (int c = 0; c < 16; c++) g[c] = c == dof + d ? gs : g[c];
                }
            }
            tc_st8(S.dz4 + tc_off(r, 0, 16), g);
            tc_st8(S.dz4 + tc_off(r, 8, 16), g + 8);
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) l += __shfl_xor_sync(0xFFFFFFFFu, l, off);
            if (lane == 0) S.loss[warp] += l;
            tt_colsum32(g, db + 384, lane, 16);
        }
        // ---- backward ----
        const uint32_t acc0 = first ? 0u : 1u;
        if (!step([&] {  // dA3 = dZ4 W4
                tc_mma(tmem + TT_F, tc_desc(S.dz4, 16), tc_desc_mn(S.w4, 128), tc_idesc(128, 128, false, true), 0);
            }, [&] {
                for (int kk = 0; kk < 8; kk++)  // dW4^T += A3^T dZ4 (M = inputs, N = outputs)
                    tc_mma(tmem + TT_DW4, tc_desc_mn(S.a3 + kk * 2048, 128), tc_desc_mn(S.dz4 + kk * 256, 16),
                           tc_idesc(128, 16, true, true), acc0 | (kk > 0));
            }))
            break;
        grad_out(S.a3, S.g, db + 256);
        if (!step([&] {
                for (int kk = 0; kk < 8; kk++)  // dA2 = dZ3 W3
                    tc_mma(tmem + TT_F, tc_desc(S.g + kk * 128, 128), tc_desc_mn(S.w3 + kk * 2048, 128),
                           tc_idesc(128, 128, false, true), kk > 0);
            }, [&] {
                for (int kk = 0; kk < 8; kk++)  // dW3 += dZ3^T A2
                    tc_mma(tmem + TT_DW3, tc_desc_mn(S.g + kk * 2048, 128), tc_desc_mn(S.a2 + kk * 2048, 128),
                           tc_idesc(128, 128, true, true), acc0 | (kk > 0));
            }))
            break;
        // dW3 still reads g; a3 and its reader dW4 are done
        grad_out(S.a2, S.a3, db + 128);
        if (!step([&] {
                for (int kk = 0; kk < 8; kk++)  // dA1 = dZ2 W2
                    tc_mma(tmem + TT_F, tc_desc(S.a3 + kk * 128, 128), tc_desc_mn(S.w2 + kk * 2048, 128),
                           tc_idesc(128, 128, false, true), kk > 0);
            }, [&] {
                for (int kk = 0; kk < 8; kk++)  // dW2 += dZ2^T A1
                    tc_mma(tmem + TT_DW2, tc_desc_mn(S.a3 + kk * 2048, 128), tc_desc_mn(S.a1 + kk * 2048, 128),
                           tc_idesc(128, 128, true, true), acc0 | (kk > 0));
            }))
            break;
        grad_out(S.a1, S.g, db);
        if (!step([&] {
                for (int kk = 0; kk < 8; kk++)  // dW1 += dZ1^T X
                    tc_mma(tmem + TT_DW1, tc_desc_mn(S.g + kk * 2048, 128), tc_desc_mn(S.x + kk * 256, 16),
                           tc_idesc(128, 16, true, true), acc0 | (kk > 0));
            }, none))
            break;
        first = false;
    }
    if (ok && !first) {
        // the CTA's weight gradients out of tensor memory: lane r is output row r of dW1..dW3 and
        // input column r of dW4; the row's four threads take half of dW2 or dW3 each, two of them
        // dW1 and dW4 too
        // (16-byte vector atomics: the parameter offsets of W1..W3 are multiples of 4 floats)
        float *const out = part ? part + (size_t)blockIdx.x * TT_PART : grad;
        auto put4 = [&](float *dst, const float *v) {
            const float4 f = make_float4(v[0], v[1], v[2], v[3]);
            if (part) *reinterpret_cast<float4 *>(dst) = f;
            else atomicAdd(reinterpret_cast<float4 *>(dst), f);
        };
        auto put = [&](float *dst, float v) {
            if (part) *dst = v;
            else atomicAdd(dst, v);
        };
        const uint32_t t_dw = t_row + (quarter < 2 ? TT_DW2 : TT_DW3);
        const int p_w = quarter < 2 ? P_W2 : P_W3, first_c = 64 * (quarter & 1);
#pragma unroll 2
        for (int c0 = first_c; c0 < first_c + 64; c0 += 16) {
            float v[16];
            tc_ld16(t_dw + (uint32_t)c0, v);
#pragma unroll
            for (int i = 0; i < 16; i += 4) put4(out + p_w + (part ? tt_quad(r, c0 + i, 128) : r * 128 + c0 + i), v + i);
        }
        if (quarter % 2 == 0) {
            float v[16];
            tc_ld16(t_row + (quarter == 0 ? TT_DW1 : TT_DW4), v);
            if (quarter == 0) {
#pragma unroll
                for (int i = 0; i < 16; i += 4) put4(out + P_W1 + (part ? tt_quad(r, i, 128) : r * 16 + i), v + i);
            } else {
#pragma unroll
                for (int o = 0; o < 16; o++) put(out + P_W4 + o * 128 + r, v[o]);
            }
        }
        auto quarters = [&](int i) { return ((S.db[0][i] + S.db[1][i]) + S.db[2][i]) + S.db[3][i]; };
        if (tid < 128) {
            put(out + P_B1 + tid, quarters(tid));
            put(out + P_B2 + tid, quarters(128 + tid));
            put(out + P_B3 + tid, quarters(256 + tid));
        }
        if (tid < 16) put(out + P_B4 + tid, quarters(384 + tid));
        const float loss = ((S.loss[0] + S.loss[1]) + S.loss[2]) + S.loss[3];
        if (tid == 0 && part) out[FS_MLP_NPARAM] = loss;
        if (tid == 0 && !part && loss_out) atomicAdd(loss_out, loss);
    }
    if (!ok && tid == 0 && part) part[(size_t)blockIdx.x * TT_PART + FS_MLP_NPARAM] = __int_as_float(0x7FC00000);
    if (!ok && tid == 0 && !part && loss_out) atomicAdd(loss_out, __int_as_float(0x7FC00000));  // gave up: NaN loss
    // release the tensor memory once no MMA is in flight: after a give-up, one more commit behind
    // all of them, waited for (bounded) before freeing the columns
    if (!ok) {
        if (tid == 0) tc_commit(tc_smem(&S.mbar_last));
        tc_wait(tc_smem(&S.mbar_last), 0u);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TT_TMEM_COLS)
                     : "memory");
}

// one parameter's Adam step on the FP32 master weights; writes the BF16 training copy
__device__ __forceinline__ void adam_one(int i, float g, float w0, float m0, float v0, float *params, float *m,
                                         float *v, fs_bf16 *wq, float lr, float b1c, float b2c)
{
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float mi = b1 * m0 + (1.f - b1) * g;
    const float vi = b2 * v0 + (1.f - b2) * g * g;
    m[i] = mi;
    v[i] = vi;
    const float w = w0 - lr * (mi / b1c) / (sqrtf(vi / b2c) + eps);
    params[i] = w;
    int q = -1;
    if (i < P_B1) q = Q_W1 + (i - P_W1);
    else if (i >= P_W2 && i < P_B2) q = Q_W2 + (i - P_W2);
    else if (i >= P_W3 && i < P_B3) q = Q_W3 + (i - P_W3);
    else if (i >= P_W4 && i < P_B4) q = Q_W4 + (i - P_W4);
    if (q >= 0) wq[q] = f2bf(w);
}

// Adam step; clears the gradient.
__global__ void fs_mlp_adam_kernel(float *params, float *m, float *v, float *grad, fs_bf16 *wq, float lr,
                                   float b1c, float b2c)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= FS_MLP_NPARAM) return;
    adam_one(i, grad[i], params[i], m[i], v[i], params, m, v, wq, lr, b1c, b2c);
    grad[i] = 0.f;
}

// Adam step on the gradient that n_parts CTAs of the training pass left in their rows of part,
// added in the CTAs' order.  The last thread adds the losses.  A CTA that gave up has written no
// gradient, only a NaN for its loss: with any such loss the step leaves the parameters, moments and
// weights as they are.  Launched while the pass still runs
// (params, m and v are not its to write); part is no read-only memory, so no load of it may move
// above the wait.
__global__ void fs_mlp_adam_parts_kernel(const float *part, int n_parts, float *params, float *m, float *v,
                                         fs_bf16 *wq, float lr, float b1c, float b2c, float *loss_out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    // the parameter at place i of the row (tt_quad)
    int p = i;
    if (i < P_B1) p = P_W1 + (i - P_W1) % 512 / 4 * 16 + (i - P_W1) / 512 * 4 + i % 4;
    else if (i >= P_W2 && i < P_B2) p = P_W2 + (i - P_W2) % 512 / 4 * 128 + (i - P_W2) / 512 * 4 + i % 4;
    else if (i >= P_W3 && i < P_B3) p = P_W3 + (i - P_W3) % 512 / 4 * 128 + (i - P_W3) / 512 * 4 + i % 4;
    const bool param = i < FS_MLP_NPARAM;
    const float w0 = param ? params[p] : 0.f, m0 = param ? m[p] : 0.f, v0 = param ? v[p] : 0.f;
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the training pass has ended
    bool nan = false;
    for (int k = threadIdx.x; k < n_parts; k += blockDim.x) {
        const float loss = part[(size_t)k * TT_PART + FS_MLP_NPARAM];
        nan |= loss != loss;
    }
    nan = __syncthreads_or(nan);
    if (i > FS_MLP_NPARAM || (nan && param)) return;
    float g = 0.f;
#pragma unroll 16
    for (int k = 0; k < n_parts; k++) g = __fadd_rn(g, part[(size_t)k * TT_PART + i]);
    if (param) adam_one(p, g, w0, m0, v0, params, m, v, wq, lr, b1c, b2c);
    else if (loss_out) *loss_out = g;
}

// FP32 master weights -> BF16 training copy + inference fragments + biases
__global__ void fs_mlp_pack_kernel(const float *params, fs_bf16 *wq, uint2 *frag, float *bias)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < Q_N) {
        int p;
        if (i < Q_W2) p = P_W1 + i;
        else if (i < Q_W3) p = P_W2 + (i - Q_W2);
        else if (i < Q_W4) p = P_W3 + (i - Q_W3);
        else p = P_W4 + (i - Q_W4);
        wq[i] = f2bf(params[p]);
    }
    if (i < FS_MLP_FRAG_U2) {
        // which layer / tile / lane this fragment entry belongs to
        int off, K, N, pw;
        if (i < FS_MLP_OFF_W2) { off = FS_MLP_OFF_W1; K = 16; N = 128; pw = P_W1; }
        else if (i < FS_MLP_OFF_W3) { off = FS_MLP_OFF_W2; K = 128; N = 128; pw = P_W2; }
        else if (i < FS_MLP_OFF_W4) { off = FS_MLP_OFF_W3; K = 128; N = 128; pw = P_W3; }
        else { off = FS_MLP_OFF_W4; K = 128; N = 16; pw = P_W4; }
        const int e = i - off, lane = e & 31, t = e >> 5, NT = N / 8;
        const int kt = t / NT, nt = t % NT;
        const int n = nt * 8 + (lane >> 2), k = kt * 16 + (lane & 3) * 2;
        const float *W = params + pw;  // W[n][k], row stride K
        uint2 u;
        u.x = fs_pack_bf16(W[n * K + k], W[n * K + k + 1]);
        u.y = fs_pack_bf16(W[n * K + k + 8], W[n * K + k + 9]);
        frag[i] = u;
    }
    if (i < FS_MLP_NBIAS) {
        int p;
        if (i < FS_MLP_OFF_B2) p = P_B1 + i;
        else if (i < FS_MLP_OFF_B3) p = P_B2 + (i - FS_MLP_OFF_B2);
        else if (i < FS_MLP_OFF_B4) p = P_B3 + (i - FS_MLP_OFF_B3);
        else p = P_B4 + (i - FS_MLP_OFF_B4);
        bias[i] = params[p];
    }
}

// ------------------------------------------------------------------ C ABI
static int launch_check(const char *what)
{
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fsi_thread_error(FS_ERR_LAUNCH, cudaGetErrorString(e));
    (void)what;
    return FS_OK;
}

extern "C" int fs_mlp_sizes(int64_t *n_param, int64_t *n_bf16, int64_t *n_frag_u2, int64_t *n_bias)
{
    if (n_param) *n_param = FS_MLP_NPARAM;
    if (n_bf16) *n_bf16 = Q_N;
    if (n_frag_u2) *n_frag_u2 = FS_MLP_FRAG_U2;
    if (n_bias) *n_bias = FS_MLP_NBIAS;
    return FS_OK;
}

// CTAs of a pass over n_rows: one per 128-row tile, at most one per SM
static int train_ctas(int n_rows)
{
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int n_tiles = (n_rows + 127) / 128;
    return n_tiles < sms ? n_tiles : sms < 1 ? 1 : sms;
}

static int train_pass(const float *params, const uint16_t *wq, float *grad, const float *x, const float *z,
                      const long long *pick, int32_t n_rows, int32_t dof, float inv_batch, float *loss, float *part,
                      int ctas, void *stream)
{
    // per call: the attribute belongs to the current device (a process may use several)
    cudaError_t e = cudaFuncSetAttribute(fs_mlp_train_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)TT_SMEM_BYTES);
    if (e != cudaSuccess) return fsi_thread_error(FS_ERR_CUDA, cudaGetErrorString(e));
    fs_mlp_train_tc_kernel<<<ctas, TT_THREADS, TT_SMEM_BYTES, (cudaStream_t)stream>>>(
        params, (const fs_bf16 *)wq, grad, x, z, pick, n_rows, dof, inv_batch, loss, part);
    return launch_check("fs_mlp_train_tc_kernel");
}

extern "C" int fs_mlp_train_step(const float *params, const uint16_t *wq, float *grad, const float *x,
                                 const float *z, int32_t n_rows, int32_t dof, float inv_batch, float *loss,
                                 void *stream)
{
    if (dof < 1 || dof > 8 || n_rows < 1)
        return fsi_thread_error(FS_ERR_CONFIG, "fs_mlp_train_step: need 1 <= dof <= 8 and n_rows >= 1");
    if (((uintptr_t)wq | (uintptr_t)x | (uintptr_t)grad) & 15u)
        return fsi_thread_error(FS_ERR_CONFIG, "fs_mlp_train_step: wq, x and grad must be 16-byte aligned");
    return train_pass(params, wq, grad, x, z, nullptr, n_rows, dof, inv_batch, loss, nullptr, train_ctas(n_rows), stream);
}

extern "C" int fs_mlp_train_rows(const float *params, const uint16_t *wq, float *grad, const float *x, const float *z,
                                 const int64_t *rows, int32_t n_rows, int32_t dof, float inv_batch, float *loss,
                                 void *stream)
{
    if (dof < 1 || dof > 8 || n_rows < 1 || !rows)
        return fsi_thread_error(FS_ERR_CONFIG, "fs_mlp_train_rows: need rows, 1 <= dof <= 8 and n_rows >= 1");
    if (((uintptr_t)wq | (uintptr_t)x | (uintptr_t)grad) & 15u)
        return fsi_thread_error(FS_ERR_CONFIG, "fs_mlp_train_rows: wq, x and grad must be 16-byte aligned");
    static_assert(sizeof(long long) == sizeof(int64_t), "row numbers");
    return train_pass(params, wq, grad, x, z, (const long long *)rows, n_rows, dof, inv_batch, loss, nullptr,
                      train_ctas(n_rows), stream);
}

extern "C" int fs_mlp_adam(float *params, float *m, float *v, float *grad, uint16_t *wq, int32_t step, float lr,
                           void *stream)
{
    if (step < 1) return fsi_thread_error(FS_ERR_CONFIG, "fs_mlp_adam: step counts from 1");
    const float b1c = 1.f - powf(0.9f, (float)step), b2c = 1.f - powf(0.999f, (float)step);
    fs_mlp_adam_kernel<<<(FS_MLP_NPARAM + 255) / 256, 256, 0, (cudaStream_t)stream>>>(
        params, m, v, grad, (fs_bf16 *)wq, lr, b1c, b2c);
    return launch_check("fs_mlp_adam_kernel");
}

extern "C" int fs_mlp_workspace(int32_t n_rows, int64_t *n_floats)
{
    if (n_rows < 1 || !n_floats) return fsi_thread_error(FS_ERR_CONFIG, "fs_mlp_workspace: need n_rows >= 1");
    *n_floats = (int64_t)train_ctas(n_rows) * TT_PART;
    return FS_OK;
}

extern "C" int fs_mlp_train_batch(float *params, float *m, float *v, uint16_t *wq, const float *x, const float *z,
                                  const int64_t *rows, int32_t n_rows, int32_t dof, float *loss, int32_t step,
                                  float lr, float *workspace, int64_t n_workspace, void *stream)
{
    if (dof < 1 || dof > 8 || n_rows < 1 || step < 1 || !rows || !workspace)
        return fsi_thread_error(FS_ERR_CONFIG,
                                "fs_mlp_train_batch: need rows, a workspace, 1 <= dof <= 8, n_rows >= 1 and step >= 1");
    if (((uintptr_t)wq | (uintptr_t)x | (uintptr_t)workspace) & 15u)
        return fsi_thread_error(FS_ERR_CONFIG, "fs_mlp_train_batch: wq, x and workspace must be 16-byte aligned");
    const int ctas = train_ctas(n_rows);
    if (n_workspace < (int64_t)ctas * TT_PART)
        return fsi_thread_error(FS_ERR_CONFIG, "fs_mlp_train_batch: workspace smaller than fs_mlp_workspace asks for");
    int rc = train_pass(params, wq, nullptr, x, z, (const long long *)rows, n_rows, dof, (float)(1.0 / n_rows), nullptr,
                        workspace, ctas, stream);
    if (rc) return rc;
    const float b1c = 1.f - powf(0.9f, (float)step), b2c = 1.f - powf(0.999f, (float)step);
    cudaLaunchAttribute early = {};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t at = {};
    at.gridDim = dim3(FS_MLP_NPARAM / 128 + 1);
    at.blockDim = dim3(128);
    at.stream = (cudaStream_t)stream;
    at.attrs = &early;
    at.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&at, fs_mlp_adam_parts_kernel, (const float *)workspace, (int)ctas, params, m, v,
                                       (fs_bf16 *)wq, lr, b1c, b2c, loss);
    if (e != cudaSuccess) return fsi_thread_error(FS_ERR_LAUNCH, cudaGetErrorString(e));
    return launch_check("fs_mlp_adam_parts_kernel");
}

extern "C" int fs_mlp_pack(const float *params, uint16_t *wq, void *frag, float *bias, void *stream)
{
    int n = FS_MLP_FRAG_U2 > Q_N ? FS_MLP_FRAG_U2 : Q_N;
    fs_mlp_pack_kernel<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(params, (fs_bf16 *)wq, (uint2 *)frag,
                                                                           bias);
    return launch_check("fs_mlp_pack_kernel");
}

// batched inference on the tcgen05 tensor cores (fs_mlp_tc.cu)
extern int fsi_mlp_infer_tc(const void *frag, const float *bias, const float *x, float *y, int n_rows,
                            cudaStream_t s);

extern "C" int fs_mlp_infer(const void *frag, const float *bias, const float *x, float *y, int32_t n_rows,
                            void *stream)
{
    if (n_rows < 1) return FS_OK;
    return fsi_mlp_infer_tc(frag, bias, x, y, n_rows, (cudaStream_t)stream);
}
