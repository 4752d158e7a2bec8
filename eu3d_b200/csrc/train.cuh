// Training step of the learned chemistry surrogate: the network's forward
// pass, loss and backward pass of a minibatch in one kernel, and Adam with the
// sum over that kernel's blocks in a second.
//
// A block of 512 threads owns 128 samples at a time.  All products run on the
// tensor cores (BF16 operands in shared memory, FP32 accumulation in TMEM):
//     Z_l = H_{l-1} W_l,  dH_{l-1} = dZ_l W_l^T,  dW_l^T = dZ_l^T H_{l-1}
// with a row-major activation tile for the first two and transposed tiles for
// the third, written by the same epilogues.  The weight gradients stay in TMEM
// over all of a block's samples and leave once, as the block's partial; the
// second kernel adds the partials in block order, so a step's result does not
// depend on scheduling.  Small batches give a block 256 samples and their bias
// sums a kernel of their own (trn_paired).
//
// Why one kernel: the step's 1.8 GFLOP (batch 8192) take 1 us of tensor-core
// time; as some 30 kernels (a GEMM, an activation, a column sum, ... per
// layer) it took 480 us, each kernel a chain of global round trips: transposed
// activations in 2-byte scattered stores, uncoalesced GEMM epilogues and 32
// blocks of atomics per weight gradient.  Now 43 us: 33 for this kernel, 10 for
// the second, which also makes the next batch (FP64 targets; inside this
// kernel they took 5 us of its chain).  What bounds it is a tile's chain of
// eight tensor-core waits (1100 to 2000 cycles each) with an epilogue between
// them (4000 to 5700 cycles for 128 x 128 values), and the block's partial at
// its end (6000 cycles for 149 KB); 64 blocks leave 84 SMs idle at batch 8192 (a
// tile needs 128 rows).  Left out: 256 threads a block (52 us); layers unrolled
// (56 us with 256 threads: 9000 straight-line instructions a warp, stalled on
// their fetch).
#pragma once

#include "mlp.cuh"
#include "surrogate.cuh"

namespace eu3d {

// per-block partials: the flat gradient, then the loss
constexpr int TRN_PART = SUR_NPARAM + 16;
constexpr int TRN_THREADS = 512;
// floats of one block's pre-activations: 3 layers x 128 columns x 128 rows
constexpr int TRN_Z = 3 * SUR_H * 128;

struct TrainSmem {
    static constexpr uint32_t BIG = 128 * 128 * 2, SMALL = 128 * 16 * 2;
    // W_2^T (forward), then W_3 (backward); W_3^T, then W_2
    static constexpr uint32_t WA = 0, WB = WA + BIG;
    static constexpr uint32_t ACT = WB + BIG;                  // row-major H_1, H_2, H_3, dZ_3, dZ_2 in turn
    static constexpr uint32_t T1 = ACT + BIG, T2 = T1 + BIG;   // H_1^T, H_2^T
    static constexpr uint32_t T3 = T2 + BIG;                   // H_3^T, then dZ_3^T, dZ_2^T, dZ_1^T
    static constexpr uint32_t W1T = T3 + BIG, W4T = W1T + SMALL, W4 = W4T + SMALL;
    static constexpr uint32_t H0 = W4 + SMALL, H0T = H0 + SMALL, DZ4 = H0T + SMALL, DZ4T = DZ4 + SMALL;
    static constexpr uint32_t BIAS = DZ4T + SMALL;             // 3 x 128 + 16 floats
    static constexpr uint32_t YS = BIAS + 4 * 400;             // targets [10][128]
    static constexpr uint32_t RED = YS + 4 * 10 * 128;         // 8 floats
    static constexpr uint32_t MBAR = RED + 32, SLOT = MBAR + 8;
    static constexpr uint32_t BYTES = SLOT + 8;
};
static_assert(TrainSmem::BYTES + 128 <= 227 * 1024, "one block fits an SM");

__device__ __forceinline__ void trn_cp16(uint32_t dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void trn_cp_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// an R x K operand tile from row-major global memory, asynchronously
template <int R, int K>
__device__ __forceinline__ void trn_load_op(uint32_t dst, const __nv_bfloat16 *src, int tid)
{
    constexpr int VEC = K / 8;
#pragma unroll 1
    for (int v = tid; v < R * VEC; v += TRN_THREADS) {
        const int r = v / VEC, kk = (v % VEC) * 8;
        trn_cp16(dst + tc::op_off(R, r, kk), src + (size_t)r * K + kk);
    }
}

// D (+)= A B^T over `slabs` x 16 columns, issued by one thread; A has 128 rows,
// B has N
__device__ __forceinline__ void trn_mma(uint32_t tmem, uint32_t a, uint32_t b, int N, int slabs, bool accumulate)
{
    const uint32_t idesc = tc::idesc_bf16(128, N);
#pragma unroll 1
    for (int s = 0; s < slabs; s++)
        tc::mma(tmem, tc::sdesc(a + s * 128 * 32), tc::sdesc(b + s * N * 32), idesc, (accumulate || s > 0) ? 1u : 0u);
}

// 32 values of one row (packed pairs of columns c0 ..) into the row-major tile
// and, transposed, into a feature-major one.  The transposed stores pair two
// rows: neighbouring lanes swap halves, the even lane stores the even column's
// pair and the odd lane the odd one's.
__device__ __forceinline__ void trn_store_tile(unsigned char *act, unsigned char *tr, int row, int c0,
                                               const uint32_t h[16])
{
#pragma unroll
    for (int q = 0; q < 4; q++)
        *reinterpret_cast<uint4 *>(act + tc::op_off(128, row, c0 + 8 * q)) =
            make_uint4(h[4 * q], h[4 * q + 1], h[4 * q + 2], h[4 * q + 3]);
    const int odd = row & 1;
#pragma unroll
    for (int q = 0; q < 16; q++) {
        const uint32_t other = __shfl_xor_sync(0xffffffffu, h[q], 1);
        const uint32_t pair = odd ? __byte_perm(other, h[q], 0x7632) : __byte_perm(h[q], other, 0x5410);
        *reinterpret_cast<uint32_t *>(tr + tc::op_off(128, c0 + 2 * q + odd, row & ~1)) = pair;
    }
}

// column c, rows [32 quarter, 32 quarter + 32) of a transposed tile to global
// memory
__device__ __forceinline__ void trn_copy_col(__nv_bfloat16 *dst, const unsigned char *tr, int c, int quarter)
{
#pragma unroll
    for (int q = 0; q < 4; q++)
        reinterpret_cast<uint4 *>(dst)[q] = *reinterpret_cast<const uint4 *>(tr + tc::op_off(128, c, 32 * quarter + 8 * q));
}

// this thread's quarter of a column sum over a transposed tile: column c, rows
// [32 quarter, 32 quarter + 32)
__device__ __forceinline__ float trn_colsum(const unsigned char *tr, int c, int quarter)
{
    float s = 0.f;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const uint4 x = *reinterpret_cast<const uint4 *>(tr + tc::op_off(128, c, 32 * quarter + 8 * q));
        const uint32_t u[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int k = 0; k < 4; k++) s += __uint_as_float(u[k] << 16) + __uint_as_float(u[k] & 0xffff0000u);
    }
    return s;
}

// Xb, Yb: features and targets of the batch, B x 16 each (column 15 of Yb the
// sample's weight).  Block b takes the tiles b, b + gridDim.x, ...; PAIRED
// (trn_paired): the tiles 2 b and 2 b + 1, and it leaves dZ_l^T in dzt ([4][128][B])
// for k_sur_bias instead of summing the bias gradients.  A template, since the
// choice at run time costs the large batches 3 % (44 against 45.5 us a step).
template <bool PAIRED>
__global__ void __launch_bounds__(TRN_THREADS, 1) k_sur_train(const float *__restrict__ Xb, const float *__restrict__ Yb,
                                                             SurBf16 w, const float *__restrict__ p,
                                                             float *__restrict__ zbuf,
                                                             float *__restrict__ part, float *__restrict__ out4,
                                                             int B, __nv_bfloat16 *__restrict__ dzt,
                                                             int *__restrict__ err)
{
    using S = TrainSmem;
    extern __shared__ unsigned char trn_raw[];
    const uint32_t raw = tc::smem_u32(trn_raw);
    unsigned char *sm = trn_raw + (((raw + 127u) & ~127u) - raw);
    const uint32_t sb = tc::smem_u32(sm);
    float *bias = reinterpret_cast<float *>(sm + S::BIAS), *red = reinterpret_cast<float *>(sm + S::RED);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // four threads a row: columns [32 quarter, 32 quarter + 32) of every tile
    const int row = (warp & 3) * 32 + lane, quarter = warp >> 2, c0 = 32 * quarter;
    uint32_t *slot = reinterpret_cast<uint32_t *>(sm + S::SLOT);
    const uint32_t mbar = sb + S::MBAR;
    if (warp == 0) tc::tmem_alloc(slot, 512);
    if (tid == 0) {
        tc::mbar_init(mbar, 1);
        tc::fence_mbar_init();
    }
    for (int t = tid; t < 400; t += TRN_THREADS)
        bias[t] = p[t < 128 ? SUR_OFF_B1 + t : t < 256 ? SUR_OFF_B2 + t - 128 : t < 384 ? SUR_OFF_B3 + t - 256
                                                                               : SUR_OFF_B4 + t - 384];
    trn_load_op<128, 16>(sb + S::W1T, w.Wt[0], tid);
    trn_load_op<16, 128>(sb + S::W4T, w.Wt[3], tid);
    trn_load_op<128, 16>(sb + S::W4, w.W[3], tid);
    trn_load_op<128, 128>(sb + S::WA, w.Wt[1], tid);
    trn_load_op<128, 128>(sb + S::WB, w.Wt[2], tid);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = *slot, tl = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    constexpr uint32_t D2 = 128, D3 = 256, D1 = 384, D4 = 400;  // weight-gradient columns; 0 .. 127 work
    float *Z = zbuf + (size_t)blockIdx.x * TRN_Z;
    float dbs[3] = {0.f, 0.f, 0.f}, db4 = 0.f, loss = 0.f;
    const float scale = 1.0f / ((float)B * SUR_NOUT);
    uint32_t phase = 0;
    bool ok = true, first = true;
    // all threads: their shared-memory writes and copies reach the tensor core,
    // one thread issues and commits, everybody waits; false when the (bounded)
    // wait ran out for anyone
    auto run = [&](auto &&issue) -> bool {
        trn_cp_wait();
        tc::fence_async_smem();
        tc::fence_before();
        __syncthreads();
        if (tid == 0) {
            tc::fence_after();
            issue();
            tc::commit(mbar);
        }
        ok = tc::mbar_wait(mbar, phase) && ok;
        phase ^= 1;
        const bool all = !__syncthreads_or(!ok);
        tc::fence_after();
        return all;
    };
    // epilogue of layer l (0-based), forward: z = acc + b kept for the backward
    // pass, H = gelu(z) into the tiles; backward: dZ = dH gelu'(z)
    auto epilogue = [&](int l, bool back, uint32_t tr) {
        uint32_t h[16];
        float v[32];
        // four columns of a row together, rows consecutive across lanes
        float4 *zq = reinterpret_cast<float4 *>(Z) + (l * 32 + c0 / 4) * 128 + row;
        if (back) {
            float4 z[8];
#pragma unroll
            for (int k = 0; k < 8; k++) z[k] = zq[k * 128];
            tc::tmem_ld32(tl + c0, v);
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const __nv_bfloat162 g0 = __floats2bfloat162_rn(v[4 * k] * gelu_grad_f(z[k].x),
                                                                v[4 * k + 1] * gelu_grad_f(z[k].y));
                const __nv_bfloat162 g1 = __floats2bfloat162_rn(v[4 * k + 2] * gelu_grad_f(z[k].z),
                                                                v[4 * k + 3] * gelu_grad_f(z[k].w));
                h[2 * k] = *reinterpret_cast<const uint32_t *>(&g0);
                h[2 * k + 1] = *reinterpret_cast<const uint32_t *>(&g1);
            }
        } else {
            tc::tmem_ld32(tl + c0, v);
            const float4 *bq = reinterpret_cast<const float4 *>(bias + l * 128 + c0);
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const float4 b = bq[k];
                const float4 z = make_float4(v[4 * k] + b.x, v[4 * k + 1] + b.y, v[4 * k + 2] + b.z, v[4 * k + 3] + b.w);
                zq[k * 128] = z;
                h[2 * k] = gelu_bf16x2(z.x, z.y);
                h[2 * k + 1] = gelu_bf16x2(z.z, z.w);
            }
        }
        trn_store_tile(sm + S::ACT, sm + tr, row, c0, h);
    };
    float *ys = reinterpret_cast<float *>(sm + S::YS);
    const int tile_step = PAIRED ? 1 : gridDim.x, tile_end = PAIRED ? 2 * blockIdx.x + 2 : B / 128;
    // bias gradient of layer l (0-based) from the tile of dZ^T in T3
    auto bias_grad = [&](int l, int tile) -> float {
        if (!PAIRED) return trn_colsum(sm + S::T3, tid & 127, quarter);
        trn_copy_col(dzt + (size_t)(l * SUR_H + (tid & 127)) * B + tile * 128 + 32 * quarter, sm + S::T3, tid & 127, quarter);
        return 0.f;
    };
    for (int tile = PAIRED ? 2 * blockIdx.x : blockIdx.x; tile < tile_end; tile += tile_step) {
        const long long r = (long long)tile * 128 + row;
        float wt = 0.f;
        if (quarter == 0) {
            const float4 *xq = reinterpret_cast<const float4 *>(Xb + r * SUR_IN);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const float4 x = xq[q];
                const float f[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const __nv_bfloat16 b = __float2bfloat16_rn(f[i]);
                    *reinterpret_cast<__nv_bfloat16 *>(sm + S::H0 + tc::op_off(128, row, 4 * q + i)) = b;
                    *reinterpret_cast<__nv_bfloat16 *>(sm + S::H0T + tc::op_off(16, 4 * q + i, row)) = b;
                }
            }
        } else if (quarter == 3) {
#pragma unroll
            for (int k = 0; k < SUR_NOUT; k++) ys[k * 128 + row] = Yb[r * SUR_OUT + k];
            wt = Yb[r * SUR_OUT + 15];
        }
        bool good = true;
#pragma unroll 1
        for (int l = 0; l < 3 && good; l++) {
            const uint32_t a = l == 0 ? S::H0 : S::ACT, b = l == 0 ? S::W1T : l == 1 ? S::WA : S::WB;
            good = run([&] { trn_mma(tmem, sb + a, sb + b, 128, l == 0 ? 1 : 8, false); });
            if (!good) break;
            // the product has read its weights: the backward pass's take their place
            if (l > 0) trn_load_op<128, 128>(sb + b, l == 1 ? w.W[2] : w.W[1], tid);
            epilogue(l, false, S::T1 + l * S::BIG);
        }
        if (!good || !run([&] { trn_mma(tmem, sb + S::ACT, sb + S::W4T, 16, 8, false); })) break;
        // output layer and loss: sum over rows and output columns of
        // w (out - y)^2 / (B SUR_NOUT); dZ_4 = 2 w (out - y) / (B SUR_NOUT)
        if (quarter == 3) {
            float v[16];
            tc::tmem_ld16(tl, v);
#pragma unroll
            for (int c = 0; c < SUR_OUT; c++) {
                const float o = v[c] + bias[384 + c];
                if (out4) out4[r * SUR_OUT + c] = o;
                float g = 0.f;
                if (c < SUR_NOUT) {
                    const float d = o - ys[c * 128 + row];
                    loss += wt * d * d * scale;
                    g = 2.f * wt * d * scale;
                }
                const __nv_bfloat16 b = __float2bfloat16_rn(g);
                *reinterpret_cast<__nv_bfloat16 *>(sm + S::DZ4 + tc::op_off(128, row, c)) = b;
                *reinterpret_cast<__nv_bfloat16 *>(sm + S::DZ4T + tc::op_off(16, c, row)) = b;
            }
        }
        const bool more = tile + tile_step < tile_end;
        // l = 2, 1, 0: dH of layer l's output with the weight gradient above it,
        // then dZ_l.  dW_4 = H_3^T dZ_4, dW_{l+1}^T = dZ_{l+1}^T H_l
#pragma unroll 1
        for (int l = 2; l >= 0; l--) {
            const uint32_t wb = l == 1 ? S::WA : S::WB;
            good = run([&] {
                if (l == 2) {
                    trn_mma(tmem, sb + S::DZ4, sb + S::W4, 128, 1, false);
                    trn_mma(tmem + D4, sb + S::T3, sb + S::DZ4T, 16, 8, !first);
                } else {
                    trn_mma(tmem, sb + S::ACT, sb + wb, 128, 8, false);
                    trn_mma(tmem + (l == 1 ? D3 : D2), sb + S::T3, sb + S::T1 + l * S::BIG, 128, 8, !first);
                }
            });
            if (!good) break;
            if (l == 2) {
                // column tid & 15, rows 4 (tid >> 4) .. + 3
                const uint2 x = *reinterpret_cast<const uint2 *>(sm + S::DZ4T + tc::op_off(16, tid & 15, 4 * (tid >> 4)));
                if (PAIRED)
                    *reinterpret_cast<uint2 *>(dzt + (size_t)(3 * SUR_H + (tid & 15)) * B + tile * 128 + 4 * (tid >> 4)) = x;
                else
                    db4 += (__uint_as_float(x.x << 16) + __uint_as_float(x.x & 0xffff0000u)) +
                           (__uint_as_float(x.y << 16) + __uint_as_float(x.y & 0xffff0000u));
            } else {
                const float db = bias_grad(l + 1, tile);
                dbs[1] += l == 0 ? db : 0.f;
                dbs[2] += l == 1 ? db : 0.f;
                if (more) trn_load_op<128, 128>(sb + wb, l == 1 ? w.Wt[1] : w.Wt[2], tid);
                __syncthreads();  // the column sums have read dZ^T
            }
            epilogue(l, true, S::T3);
        }
        if (!good || !run([&] { trn_mma(tmem + D1, sb + S::T3, sb + S::H0T, 16, 8, !first); })) break;
        dbs[0] += bias_grad(0, tile);
        __syncthreads();
        first = false;
    }
    if (!ok) {
        // a wait ran out: record it and give the products in flight one more
        // bounded wait before the accumulators are freed
        atomicExch(err, 1);
        tc::mbar_wait(mbar, phase);
    }
    trn_cp_wait();
    __syncthreads();
    // the block's partial: D[o][i] for layers 1 to 3 (lane = output o, so that
    // lanes store consecutive floats), D[i][o] for layer 4
    float *pt = part + (size_t)blockIdx.x * TRN_PART;
    {
        float v[32];
        tc::tmem_ld32(tl + D2 + c0, v);
#pragma unroll
        for (int k = 0; k < 32; k++) pt[SUR_OFF_W2 + (c0 + k) * SUR_H + row] = v[k];
        tc::tmem_ld32(tl + D3 + c0, v);
#pragma unroll
        for (int k = 0; k < 32; k++) pt[SUR_OFF_W3 + (c0 + k) * SUR_H + row] = v[k];
    }
    if (quarter < 2) {
        float v[16];
        tc::tmem_ld16(tl + (quarter == 0 ? D1 : D4), v);
#pragma unroll
        for (int k = 0; k < 16; k++)
            pt[quarter == 0 ? SUR_OFF_W1 + k * SUR_H + row : SUR_OFF_W4 + row * SUR_OUT + k] = v[k];
    }
    // bias gradients: the quarters of each column sum meet in shared memory
    float *hs = reinterpret_cast<float *>(sm + S::ACT);
    for (int l = 0; l < 3; l++) hs[l * 512 + tid] = dbs[l];
    hs[3 * 512 + tid] = db4;
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_down_sync(0xffffffffu, loss, o);
    if (lane == 0 && quarter == 3) red[warp & 3] = loss;
    tc::fence_before();
    __syncthreads();
    if (tid < 384) {
        const int l = tid >> 7, c = tid & 127;
        const float *q = hs + l * 512 + c;
        pt[(l == 0 ? SUR_OFF_B1 : l == 1 ? SUR_OFF_B2 : SUR_OFF_B3) + c] = ((q[0] + q[128]) + q[256]) + q[384];
    }
    if (tid >= 384 && tid < 384 + SUR_OUT) {
        float q = 0.f;
        for (int k = 0; k < 32; k++) q += hs[3 * 512 + 16 * k + tid - 384];
        pt[SUR_OFF_B4 + tid - 384] = q;
    }
    if (tid == 0) pt[SUR_NPARAM] = ((red[0] + red[1]) + red[2]) + red[3];
    if (warp == 0) tc::tmem_free(tmem, 512);
}

// Batches under 16 chunks of 256 rows keep one order of sums: a chunk's weight
// gradients are one tensor-core accumulation over its rows, the chunks add in
// order, and a bias gradient is the sum over the chunks of each row, then a tree
// over the 256 rows.  Adam divides by the root of the second moment and rounds
// the weights to BF16 at each step, so that another order of the same sums moves
// losses and parameters by 1e-4 relative within 70 steps.  One or two chunks,
// whose sum has no other order, have always repeated bit for bit, and runs are
// compared with earlier ones.  More chunks once met in atomics: two such runs
// differ by 1e-7 to 5e-6 (parameters, 20 steps), this order differs from them by
// 4e-8 to 6e-6 at 1024 to 3072 rows where 128-row partials differ by 5e-6 to
// 2e-5, and at 4096 rows both differ by 4e-6.  From there on a block takes 128
// rows, which keeps twice the SMs busy: 43 us a step against 82 at 4096 and 8192
// rows (below 4096 rows 39 to 43 against the 76 to 84 us of this order).
constexpr int TRN_CHUNK = 256, TRN_CHUNKS = 16;
__host__ __device__ constexpr bool trn_paired(int B) { return B < TRN_CHUNKS * TRN_CHUNK; }

// bias gradients of a paired batch, into the first block's partial (the others
// hold zeros): one block per column of dzt
__global__ void __launch_bounds__(TRN_CHUNK) k_sur_bias(const __nv_bfloat16 *__restrict__ dzt, int B, float *__restrict__ part)
{
    const int c = blockIdx.x, l = c / SUR_H;
    float s = 0.f;
    for (int r = threadIdx.x; r < B; r += TRN_CHUNK) s += __bfloat162float(dzt[(size_t)c * B + r]);
    __shared__ float sm[TRN_CHUNK / 32];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        s = threadIdx.x < TRN_CHUNK / 32 ? sm[threadIdx.x] : 0.f;
        for (int o = TRN_CHUNK / 64; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (threadIdx.x == 0)
            part[(l == 0 ? SUR_OFF_B1 : l == 1 ? SUR_OFF_B2 : l == 2 ? SUR_OFF_B3 : SUR_OFF_B4) + c - l * SUR_H] = s;
    }
}

// The minibatch of one step: row r of B is a random sample of the training set
// (n x 12 features X, labels Lb), with replacement.
struct BatchSrc {
    const float *X, *Lb;
    long long n;
    unsigned long long seed;
    long long step;
    int B;
    float *Xb, *Yb;
};
constexpr int BATCH_TASKS = 11;  // threads a row: ten targets, the features

__device__ __forceinline__ void trn_batch_task(const BatchSrc &s, const SurNorm &nrm, int t)
{
    const int r = t / BATCH_TASKS, k = t - r * BATCH_TASKS;
    if (r >= s.B) return;
    const long long idx =
        (long long)(smix64(s.seed ^ smix64((unsigned long long)s.step * 0x100000001ull + (unsigned long long)r)) % s.n);
    const float *x = s.X + idx * 12, *lab = s.Lb + idx * 12;
    if (k < SUR_NOUT) {
        s.Yb[(long long)r * SUR_OUT + k] = sur_target(nrm, sur_target_scale(nrm, x), k, x, lab[k]);
        return;
    }
    float raw[SUR_NIN], f[SUR_IN];
#pragma unroll
    for (int i = 0; i < SUR_NIN; i++) raw[i] = x[i];
    sur_features(nrm, raw, f);
#pragma unroll
    for (int i = 0; i < SUR_IN; i++) s.Xb[(long long)r * SUR_IN + i] = f[i];
    s.Yb[(long long)r * SUR_OUT + 15] = lab[10];
}

__global__ void __launch_bounds__(256) k_sur_batch(BatchSrc s, const __grid_constant__ SurNorm nrm)
{
    trn_batch_task(s, nrm, blockIdx.x * blockDim.x + threadIdx.x);
}

// Gradient = sum of the blocks' partials in block order (to g when given);
// with `update` Adam with bias correction (t = step count, from 1), the BF16
// copies of the weights and the loss.  One thread per parameter; the partials
// of a batch of 8192 are 9.5 MB that the step before left in L2.
struct AdamCfg {
    float lr, b1, b2, eps;
    int t, update;
};

// 64 parameters a block, four threads each: a quarter of the partials, their
// loads issued together, the quarters added in order.  (The few partials of a
// paired batch are the first thread's, in order.)
constexpr int STEP_PARAMS = 64, STEP_BLOCKS = SUR_NPARAM / STEP_PARAMS + 1;

__global__ void __launch_bounds__(4 * STEP_PARAMS) k_sur_step(const float *__restrict__ part, int nparts,
                                                              float *__restrict__ p, float *__restrict__ m,
                                                              float *__restrict__ v, float *__restrict__ g,
                                                              float *__restrict__ loss, SurBf16 w, AdamCfg c,
                                                              BatchSrc next, const __grid_constant__ SurNorm nrm)
{
    // blocks past the parameters make the next step's batch meanwhile
    if (blockIdx.x >= STEP_BLOCKS) {
        trn_batch_task(next, nrm, (blockIdx.x - STEP_BLOCKS) * blockDim.x + threadIdx.x);
        return;
    }
    __shared__ float quarter[4][STEP_PARAMS];
    const int t = threadIdx.x % STEP_PARAMS, q = threadIdx.x / STEP_PARAMS;
    const int i = blockIdx.x * STEP_PARAMS + t;
    float s = 0.f;
    if (i <= SUR_NPARAM) {
        const int n4 = nparts < TRN_CHUNKS ? nparts : (nparts + 3) / 4, e = min(nparts, (q + 1) * n4);
        int b = q * n4;
        for (; b + 16 <= e; b += 16) {
            float x[16];
#pragma unroll
            for (int k = 0; k < 16; k++) x[k] = part[(size_t)(b + k) * TRN_PART + i];
#pragma unroll
            for (int k = 0; k < 16; k++) s += x[k];
        }
        for (; b < e; b++) s += part[(size_t)b * TRN_PART + i];
    }
    quarter[q][t] = s;
    __syncthreads();
    if (q || i > SUR_NPARAM) return;
    s = ((quarter[0][t] + quarter[1][t]) + quarter[2][t]) + quarter[3][t];
    if (i == SUR_NPARAM) {
        if (loss) *loss = s;
        return;
    }
    if (g) g[i] = s;
    if (!c.update) return;
    const float c1 = 1.f - powf(c.b1, (float)c.t), c2 = 1.f - powf(c.b2, (float)c.t);
    const float mi = c.b1 * m[i] + (1.f - c.b1) * s;
    const float vi = c.b2 * v[i] + (1.f - c.b2) * s * s;
    m[i] = mi;
    v[i] = vi;
    const float pn = p[i] - c.lr * (mi / c1) / (sqrtf(vi / c2) + c.eps);
    p[i] = pn;
    const __nv_bfloat16 h = __float2bfloat16_rn(pn);
#pragma unroll
    for (int l = 0; l < 4; l++) {
        int off, in, out;
        sur_weight_dims(l, off, in, out);
        const int t = i - off;
        if (t >= 0 && t < in * out) {
            w.W[l][t] = h;
            w.Wt[l][(t % out) * in + t / out] = h;
        }
    }
}

}  // namespace eu3d
