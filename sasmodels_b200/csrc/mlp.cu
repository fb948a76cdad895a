// Tensor-core MLP for the I(q) surrogate: 16 (7 used) -> 256 -> 256 -> 256
// -> 256 -> 1, SiLU, BF16 weights and activations, FP32 accumulation in TMEM
// (tcgen05.mma kind::f16, M = 128 rows per CTA, N = 256, K = 16 per MMA).
//
// Kernels
//   mlp_forward    all four hidden layers of 128 samples per CTA; the
//                  activations stay in shared memory as the next layer's A
//                  operand, weights stream through a 256 x 64 staging tile.
//                  Activations are kept as a compensated BF16 pair
//                  h = hi + lo (hi = bf16(h), lo = bf16(h - hi)) and each
//                  layer issues the MMAs of both halves into the same FP32
//                  accumulator, so the layer inputs carry ~16 significant
//                  bits instead of 8 while every operand stays BF16;
//                  bias + SiLU in the TMEM epilogue, the 256 -> 1 output layer
//                  as a per-row dot product in the last epilogue.  Optionally
//                  saves the pre-activations z and activations h for training.
//   mlp_backward   dZ3 = dout w_out * silu'(z3), then dZ(l-1) = (dZl W_l) *
//                  silu'(z(l-1)) through the three 256x256 layers, the same
//                  way (A = dZ in smem, B = W_l^T streamed).
//   mlp_infer,     persistent pipelined forms of the two (weights bulk-copied
//   mlp_backward_p through a shared-memory ring); they give the planes of
//                  mlp_forward / mlp_backward bit for bit.
//   mlp_serve      the forward with the tensor core and the epilogue working
//                  at once (a dedicated MMA warp, two TMEM accumulators,
//                  layer l+1's MMAs under layer l's epilogue chunk by chunk);
//                  serves inference and the training forward.
//   mlp_halves     few tiles: two SMs per tile; serving, or forward and backward of
//                  a training step (mlp_halves.cuh)
//   mlp_serve_pairs   inference over many tiles: pairs of SMs (cta_group::2), two
//                  tiles in flight on each (mlp_pairs.cuh).
//   mlp_backward_t, mlp_weight_grads   the training step's backward and weight
//                  gradients on tiled planes (mlp_train.cuh).
//   + the learning rate schedule, Adam, feature packing; column sums, loss
//     gradient and Adam of one tensor, which tests compare with.
//
// All launches return an error code; device-side waits are bounded and
// report through *err (0 = ok).
#include <cstdint>
#include <cstdio>
#include <type_traits>
#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_bf16.h>

#include "tc_ptx.cuh"

namespace mlp {

constexpr int HID = 256;
constexpr int NIN = 16;           // padded input features
constexpr int TM = 128;           // rows per CTA
constexpr int KC = 64;            // streamed K chunk
constexpr int THREADS = 128;
constexpr int ACT_BYTES = TM*HID*2;                // one 128 x 256 bf16 tile
constexpr int FWD_SMEM = 2*ACT_BYTES + HID*KC*2;   // act hi + lo + 32 KB weights
constexpr int BWD_SMEM = ACT_BYTES + HID*KC*2;     // dZ tile + 32 KB weights

struct Weights {
    const __nv_bfloat16 *w[4];    // w[0]: 256 x 16, w[1..3]: 256 x 256, [out][in]
    const float *b[4];
    const float *w_out;
    const float *b_out;           // device scalar
};

// silu(z) = z sigmoid(z) with sigmoid(z) = (1 + tanh(z/2))/2, i.e.
// h = z/2 + (z/2) tanh(z/2): one MUFU operation (tanh.approx.f32, documented
// maximum relative error about 2^-11) and two FP32 operations.  Every
// forward kernel (training and serving) uses this one function, so the
// network is served with the activation it was trained with.
__device__ __forceinline__ float silu(float z)
{
    const float hz = 0.5f*z;
    float t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(hz));
    return fmaf(hz, t, hz);
}

// silu'(z) = s (1 + z (1 - s)) with the sigmoid s = (1 + tanh(z/2))/2 taken
// as in silu above, so the backward pass differentiates the function the
// forward pass evaluates (one MUFU operation instead of an exp and a divide).
__device__ __forceinline__ float dsilu(float z)
{
    float t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(0.5f*z));
    const float s = fmaf(0.5f, t, 0.5f);
    return s*(1.0f + z*(1.0f - s));
}

__device__ __forceinline__ uint32_t pack2(float a, float b)
{
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t *>(&v);
}

__device__ __forceinline__ float bf_lo(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float bf_hi(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }

// Copy a ROWS x K (K-major, row stride ld elements) bf16 block starting at
// column k0 into a canonical K-major smem tile; rows >= nrows read as zero.
template <int ROWS, int K>
__device__ __forceinline__ void load_tile(uint8_t *tile, const __nv_bfloat16 *src, int ld,
                                          int k0, int nrows)
{
    constexpr int VEC = ROWS*(K/8);
    for (int i = threadIdx.x; i < VEC; i += THREADS) {
        const int r = i/(K/8), c = i % (K/8);
        uint4 v = make_uint4(0, 0, 0, 0);
        if (r < nrows)
            v = *reinterpret_cast<const uint4 *>(src + (size_t)r*ld + k0 + 8*c);
        *reinterpret_cast<uint4 *>(tile + tc::kmajor_offset<ROWS>(r, 8*c)) = v;
    }
}

struct Pipe {
    uint64_t *bar;
    uint32_t phase;
    bool ok;
};

// Issue the MMAs of one staged chunk (single thread), then wait (all).
// a_addr: canonical 128-row A tile holding the full K; a_step0: first K=16
// step of this chunk within A; b_addr: canonical NB-row tile of this chunk.
// a_lo_addr != 0 adds the MMAs of the low half of a compensated A.
template <int NB, int STEPS>
__device__ __forceinline__ void mma_chunk(Pipe &pp, uint32_t tmem, uint32_t a_addr, int a_step0,
                                          uint32_t b_addr, bool accumulate,
                                          uint32_t a_lo_addr = 0)
{
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (threadIdx.x == 0) {
        constexpr uint32_t idesc = tc::idesc_bf16(128, NB);
        #pragma unroll
        for (int s = 0; s < STEPS; ++s) {
            const uint64_t bdesc = tc::kmajor_desc<NB>(b_addr, s);
            tc::mma_bf16(tmem, tc::kmajor_desc<128>(a_addr, a_step0 + s), bdesc, idesc,
                         (accumulate || s > 0) ? 1u : 0u);
            if (a_lo_addr)
                tc::mma_bf16(tmem, tc::kmajor_desc<128>(a_lo_addr, a_step0 + s), bdesc, idesc, 1u);
        }
        tc::mma_commit(pp.bar);
    }
    const bool done = tc::mbar_wait(pp.bar, pp.phase);
    pp.phase ^= 1u;
    pp.ok = __syncthreads_and(done && pp.ok) != 0;
    tc::fence_after_sync();
}

// A (128 x 256, resident; plus its low half when act_lo != nullptr) times a
// streamed [256 x 256] weight (rows = N).
__device__ __forceinline__ void layer_256(Pipe &pp, uint32_t tmem, uint8_t *act, uint8_t *wbuf,
                                          const __nv_bfloat16 *w, uint8_t *act_lo = nullptr)
{
    const uint32_t a_addr = tc::smem_u32(act), b_addr = tc::smem_u32(wbuf);
    const uint32_t lo_addr = act_lo ? tc::smem_u32(act_lo) : 0u;
    for (int kc = 0; kc < HID/KC; ++kc) {
        if (!pp.ok) return;
        load_tile<HID, KC>(wbuf, w, HID, kc*KC, HID);
        mma_chunk<HID, KC/16>(pp, tmem, a_addr, kc*(KC/16), b_addr, kc > 0, lo_addr);
    }
}

// Read this thread's TMEM row (cols c0..c0+15) into floats.
__device__ __forceinline__ void tmem_row16(uint32_t tmem, int c0, float (&v)[16])
{
    uint32_t r[16];
    const uint32_t lane_base = (uint32_t)((threadIdx.x & ~31) << 16);
    tc::tmem_ld16(tmem + lane_base + (uint32_t)c0, r);
    tc::tmem_wait_ld();
    #pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
}

__device__ __forceinline__ void store16(uint8_t *act, int row, int c0, const float (&h)[16])
{
    uint4 lo, hi;
    lo.x = pack2(h[0], h[1]);   lo.y = pack2(h[2], h[3]);
    lo.z = pack2(h[4], h[5]);   lo.w = pack2(h[6], h[7]);
    hi.x = pack2(h[8], h[9]);   hi.y = pack2(h[10], h[11]);
    hi.z = pack2(h[12], h[13]); hi.w = pack2(h[14], h[15]);
    *reinterpret_cast<uint4 *>(act + tc::kmajor_offset<TM>(row, c0)) = lo;
    *reinterpret_cast<uint4 *>(act + tc::kmajor_offset<TM>(row, c0 + 8)) = hi;
}

// Compensated pair: hi = bf16(h) into act, lo = bf16(h - hi) into act_lo.
__device__ __forceinline__ void store16_split(uint8_t *act, uint8_t *act_lo, int row, int c0,
                                              const float (&h)[16])
{
    float hi[16], lo[16];
    #pragma unroll
    for (int j = 0; j < 16; ++j) {
        hi[j] = __bfloat162float(__float2bfloat16_rn(h[j]));
        lo[j] = h[j] - hi[j];
    }
    store16(act, row, c0, hi);
    store16(act_lo, row, c0, lo);
}

__device__ __forceinline__ void save16(__nv_bfloat16 *dst, const float (&h)[16])
{
    uint4 lo, hi;
    lo.x = pack2(h[0], h[1]);   lo.y = pack2(h[2], h[3]);
    lo.z = pack2(h[4], h[5]);   lo.w = pack2(h[6], h[7]);
    hi.x = pack2(h[8], h[9]);   hi.y = pack2(h[10], h[11]);
    hi.z = pack2(h[12], h[13]); hi.w = pack2(h[14], h[15]);
    reinterpret_cast<uint4 *>(dst)[0] = lo;
    reinterpret_cast<uint4 *>(dst)[1] = hi;
}

__device__ __forceinline__ void load16(const __nv_bfloat16 *src, float (&z)[16])
{
    const uint4 lo = reinterpret_cast<const uint4 *>(src)[0];
    const uint4 hi = reinterpret_cast<const uint4 *>(src)[1];
    const uint32_t u[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    #pragma unroll
    for (int j = 0; j < 8; ++j) { z[2*j] = bf_lo(u[j]); z[2*j + 1] = bf_hi(u[j]); }
}

// Epilogue of hidden layer l: z = acc + b, h = silu(z); h back into the
// activation tile (next A), z and h optionally to global; the last layer
// also forms out = h . w_out + b_out.
__device__ __forceinline__ void epilogue_hidden(uint32_t tmem, uint8_t *act, uint8_t *act_lo,
                                                const float *bias,
                                                const float *w_out, const float *b_out, bool last,
                                                int grow, int n, __nv_bfloat16 *zs,
                                                __nv_bfloat16 *hs, float *out)
{
    const int t = threadIdx.x;
    float dot = 0.0f;
    for (int c0 = 0; c0 < HID; c0 += 16) {
        float z[16], h[16];
        tmem_row16(tmem, c0, z);
        #pragma unroll
        for (int j = 0; j < 16; ++j) {
            z[j] += bias[c0 + j];
            h[j] = silu(z[j]);
        }
        if (last) {
            #pragma unroll
            for (int j = 0; j < 16; ++j) dot = fmaf(h[j], w_out[c0 + j], dot);
        } else {
            store16_split(act, act_lo, t, c0, h);
        }
        if (zs != nullptr) {          // every row of the padded batch (zero inputs)
            save16(zs + (size_t)grow*HID + c0, z);
            save16(hs + (size_t)grow*HID + c0, h);
        }
    }
    if (last && grow < n) out[grow] = dot + *b_out;
}

__global__ void __launch_bounds__(THREADS, 1)
mlp_forward(int n, const __nv_bfloat16 *__restrict__ x, const __nv_bfloat16 *__restrict__ x_lo,
            Weights wts, float *__restrict__ out,
            __nv_bfloat16 *__restrict__ z_save, __nv_bfloat16 *__restrict__ h_save,
            int *__restrict__ err)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t *act = smem;
    uint8_t *act_lo = smem + ACT_BYTES;
    uint8_t *wbuf = smem + 2*ACT_BYTES;
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_slot;
    const int t = threadIdx.x;
    const int row0 = blockIdx.x*TM;

    if (t < 32) {
        tc::tmem_alloc(&tmem_slot, HID);
        tc::tmem_relinquish();
    }
    if (t == 0) {
        tc::mbar_init(&bar, 1);
        tc::mbar_fence_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_slot;
    Pipe pp{&bar, 0u, true};

    // layer 0: K = 16 features (hi and lo halves)
    load_tile<TM, NIN>(act, x + (size_t)row0*NIN, NIN, 0, n - row0);
    load_tile<TM, NIN>(act_lo, x_lo + (size_t)row0*NIN, NIN, 0, n - row0);
    load_tile<HID, NIN>(wbuf, wts.w[0], NIN, 0, HID);
    mma_chunk<HID, 1>(pp, tmem, tc::smem_u32(act), 0, tc::smem_u32(wbuf), false,
                      tc::smem_u32(act_lo));
    const size_t plane = (size_t)gridDim.x*TM*HID;
    for (int l = 0; l < 4 && pp.ok; ++l) {
        if (l > 0) layer_256(pp, tmem, act, wbuf, wts.w[l], act_lo);
        if (!pp.ok) break;
        epilogue_hidden(tmem, act, act_lo, wts.b[l], wts.w_out, wts.b_out, l == 3, row0 + t, n,
                        z_save ? z_save + l*plane : nullptr,
                        h_save ? h_save + l*plane : nullptr, out);
        tc::fence_before_sync();
        __syncthreads();
        tc::fence_after_sync();
    }
    tc::fence_before_sync();
    __syncthreads();
    if (t < 32) tc::tmem_dealloc(tmem, HID);
    if (!pp.ok && t == 0) atomicExch(err, 1);
}

// Backward through the hidden layers of 128 samples.  wt[l] = W_l^T stored
// [in][out] (K-major B for dH = dZ W).  dz_save[l] receives dZ_l.
struct WeightsT {
    const __nv_bfloat16 *wt[4];   // wt[1..3] used
    const float *w_out;
};

__global__ void __launch_bounds__(THREADS, 1)
mlp_backward(int n, WeightsT wts, const float *__restrict__ dout,
             const __nv_bfloat16 *__restrict__ z_save, __nv_bfloat16 *__restrict__ dz_save,
             int *__restrict__ err)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t *act = smem;
    uint8_t *wbuf = smem + ACT_BYTES;
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_slot;
    const int t = threadIdx.x;
    const int row0 = blockIdx.x*TM;
    const int grow = row0 + t;
    const size_t plane = (size_t)gridDim.x*TM*HID;

    if (t < 32) {
        tc::tmem_alloc(&tmem_slot, HID);
        tc::tmem_relinquish();
    }
    if (t == 0) {
        tc::mbar_init(&bar, 1);
        tc::mbar_fence_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_slot;
    Pipe pp{&bar, 0u, true};

    // dZ3 = dout * w_out * silu'(z3)
    {
        const float d = grow < n ? dout[grow] : 0.0f;
        const __nv_bfloat16 *zrow = z_save + 3*plane + (size_t)grow*HID;
        __nv_bfloat16 *drow = dz_save + 3*plane + (size_t)grow*HID;
        for (int c0 = 0; c0 < HID; c0 += 16) {
            float z[16], g[16];
            load16(zrow + c0, z);
            #pragma unroll
            for (int j = 0; j < 16; ++j) g[j] = d*wts.w_out[c0 + j]*dsilu(z[j]);
            store16(act, t, c0, g);
            save16(drow + c0, g);
        }
    }
    for (int l = 3; l >= 1 && pp.ok; --l) {
        layer_256(pp, tmem, act, wbuf, wts.wt[l]);
        if (!pp.ok) break;
        const __nv_bfloat16 *zrow = z_save + (l - 1)*plane + (size_t)grow*HID;
        __nv_bfloat16 *drow = dz_save + (l - 1)*plane + (size_t)grow*HID;
        for (int c0 = 0; c0 < HID; c0 += 16) {
            float g[16], z[16];
            tmem_row16(tmem, c0, g);
            load16(zrow + c0, z);
            #pragma unroll
            for (int j = 0; j < 16; ++j) g[j] *= dsilu(z[j]);
            store16(act, t, c0, g);
            save16(drow + c0, g);
        }
        tc::fence_before_sync();
        __syncthreads();
        tc::fence_after_sync();
    }
    tc::fence_before_sync();
    __syncthreads();
    if (t < 32) tc::tmem_dealloc(tmem, HID);
    if (!pp.ok && t == 0) atomicExch(err, 1);
}

// ---- small CUDA-core kernels ------------------------------------------------

// Column sums of a row-major [rows x cols] bf16 matrix, each row weighted
// by v[row] when v is given (the bias gradients from the dZ planes, the
// output-layer gradient from the last h plane with v = dout).  Pass 1: one
// thread per column sums CS_ROWS consecutive rows (coalesced row reads, the
// loads of a block of rows in flight together, rows/CS_ROWS blocks); pass
// 2: one warp per column, lane j adding partials j, j + 32, ... in order and
// the lanes combined by a butterfly, so the result does not depend on
// scheduling.
constexpr int CS_ROWS = 64;
__global__ void col_sum_partial(int rows, int cols, const __nv_bfloat16 *__restrict__ M,
                                const float *__restrict__ v, float *__restrict__ part)
{
    const int c = blockIdx.y*blockDim.x + threadIdx.x;
    if (c >= cols) return;
    const int r0 = blockIdx.x*CS_ROWS, r1 = min(rows, r0 + CS_ROWS);
    float s = 0.0f;
    if (r1 - r0 == CS_ROWS) {
        float m[CS_ROWS/4];
        #pragma unroll
        for (int q = 0; q < 4; ++q) {
            #pragma unroll
            for (int j = 0; j < CS_ROWS/4; ++j)
                m[j] = __bfloat162float(M[(size_t)(r0 + q*(CS_ROWS/4) + j)*cols + c]);
            #pragma unroll
            for (int j = 0; j < CS_ROWS/4; ++j)
                s = fmaf(m[j], v ? v[r0 + q*(CS_ROWS/4) + j] : 1.0f, s);
        }
    } else {
        for (int r = r0; r < r1; ++r)
            s = fmaf(__bfloat162float(M[(size_t)r*cols + c]), v ? v[r] : 1.0f, s);
    }
    part[(size_t)blockIdx.x*cols + c] = s;
}

__global__ void col_sum_final(int nparts, int cols, const float *__restrict__ part,
                              float *__restrict__ out)
{
    const int c = blockIdx.x*(blockDim.x/32) + threadIdx.x/32;
    const int lane = threadIdx.x & 31;
    if (c >= cols) return;
    float s = 0.0f;
    for (int b = lane; b < nparts; b += 32) s += part[(size_t)b*cols + c];
    #pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (lane == 0) out[c] = s;
}

// Gradient of the mean loss over the first n rows (0 on padding) and the
// per-row loss: squared error for delta <= 0, else Huber with threshold
// delta (quadratic inside, linear outside), which keeps the few points
// near form-factor minima from dominating the fit.
__device__ __forceinline__ void loss_of(float d, float delta, float &g, float &l)
{
    if (delta <= 0.0f || fabsf(d) <= delta) {
        g = 2.0f*d;
        l = d*d;
    } else {
        g = 2.0f*delta*copysignf(1.0f, d);
        l = delta*(2.0f*fabsf(d) - delta);
    }
}

__global__ void loss_grad(int n, int n_pad, const float *__restrict__ out,
                          const float *__restrict__ y, float delta, float *__restrict__ dout,
                          float *__restrict__ loss)
{
    const int i = blockIdx.x*blockDim.x + threadIdx.x;
    if (i >= n_pad) return;
    float g, l;
    loss_of(i < n ? out[i] - y[i] : 0.0f, delta, g, l);
    dout[i] = i < n ? g/(float)n : 0.0f;
    loss[i] = l;
}

__device__ __forceinline__ void adam_update(float g, float &p, float &m, float &v, float lr,
                                            float b1, float b2, float eps, float bc1, float bc2)
{
    // the contractions are spelled out, so that every kernel rounds alike
    const float mi = fmaf(b1, m, (1.0f - b1)*g);
    const float vi = fmaf(b2, v, (1.0f - b2)*g*g);
    m = mi;
    v = vi;
    p = p - lr*(mi/bc1)/(sqrtf(vi/bc2) + eps);
}

// Adam on one FP32 master tensor; the gradient is the sum of its `splits` partials.
// Writes the BF16 copy and, if wt is given, its transpose (rows x cols).
__global__ void adam_step(int size, int splits, const float *__restrict__ grad, float *__restrict__ p,
                          float *__restrict__ m, float *__restrict__ v, float lr, float b1,
                          float b2, float eps, float bc1, float bc2, __nv_bfloat16 *__restrict__ w,
                          __nv_bfloat16 *__restrict__ wt, int rows, int cols)
{
    const int i = blockIdx.x*blockDim.x + threadIdx.x;
    if (i >= size) return;
    float g = 0.0f;
    for (int s = 0; s < splits; ++s) g += grad[(size_t)s*size + i];
    float pi = p[i];
    adam_update(g, pi, m[i], v[i], lr, b1, b2, eps, bc1, bc2);
    p[i] = pi;
    if (w) w[i] = __float2bfloat16_rn(pi);
    if (wt) {
        const int r = i/cols, c = i % cols;
        wt[(size_t)c*rows + r] = __float2bfloat16_rn(pi);
    }
}

// One training step's learning rate and Adam bias corrections from two
// device counters {schedule step s, Adam step count t}, then s and t advance:
// lr = lr0 min(1, (s + 1)/warmup) (1 + cos(pi s/total))/2 (linear warm-up,
// cosine decay), bc1 = 1 - b1^(t+1), bc2 = 1 - b2^(t+1).  One thread.
__device__ __forceinline__ void schedule_step(int *__restrict__ counters,
                                              float *__restrict__ sched, int total, int warmup,
                                              float lr0, float b1, float b2)
{
    const int s = counters[0], t = counters[1] + 1;
    const double frac = (double)s/(double)total;
    const double rate = (double)lr0*fmin(1.0, (double)(s + 1)/(double)warmup)
                      *0.5*(1.0 + cos(3.141592653589793*frac));
    sched[0] = (float)rate;
    sched[1] = 1.0f - powf(b1, (float)t);
    sched[2] = 1.0f - powf(b2, (float)t);
    counters[0] = s + 1;
    counters[1] = t;
}

__global__ void lr_schedule(int *__restrict__ counters, float *__restrict__ sched, int total,
                            int warmup, float lr0, float b1, float b2)
{
    if (threadIdx.x == 0 && blockIdx.x == 0)
        schedule_step(counters, sched, total, warmup, lr0, b1, b2);
}

// Surrogate input features, each mapped to about [-1, 1]: the seven model
// inputs -- log R on [log 10, log 300], log L on [log 20, log 3000], R_pd and
// L_pd on [0, 0.3], contrast on [-5, 5], log q on [log 1e-3, log 0.5], flag
// {0, 1} -- and four functions of them that carry the scattering physics in
// a form a small network represents easily: log(qR), log(qL/2) and the
// dispersity damping log(1 + R_pd qR), log(1 + L_pd qL/2), and the damped
// oscillations cos/sin(2qR) exp(-2 (R_pd qR)^2), cos/sin(qL) exp(-2 (L_pd qL/2)^2).
// Slot 15 is zero.
__device__ __forceinline__ void feature_row(double radius, double length, double rpd, double lpd,
                                            double drho, double q, double flag, float (&f)[16])
{
    // Three logarithms for the five, and products with the ranges' reciprocals, as a
    // division takes some 20 instructions: the kernels are bound by the issue of
    // FP64 arithmetic (1400 instructions per row before).  Both change a feature by
    // less than 1e-15, far below the floats they become.
    constexpr double LOG_10 = 2.302585092994046, LOG_20 = 2.995732273553991,
                     LOG_300 = 5.703782474656201, LOG_3000 = 8.006367567650246,
                     LOG_001 = -6.907755278982137, LOG_HALF = -0.6931471805599453;
    const double lr = log(radius), ll = log(length), lq = log(q);
    f[0] = (float)((lr - LOG_10)*(2.0/(LOG_300 - LOG_10)) - 1.0);
    f[1] = (float)((ll - LOG_20)*(2.0/(LOG_3000 - LOG_20)) - 1.0);
    f[2] = (float)(rpd*(2.0/0.3) - 1.0);
    f[3] = (float)(lpd*(2.0/0.3) - 1.0);
    f[4] = (float)(drho*0.2);
    f[5] = (float)((lq - LOG_001)*(2.0/(LOG_HALF - LOG_001)) - 1.0);
    f[6] = (float)(2.0*flag - 1.0);
    const double qr = q*radius, qh = 0.5*q*length;
    f[7] = (float)((lq + lr)*0.25);
    f[8] = (float)((lq + ll + LOG_HALF)*0.25);
    f[9] = (float)(log1p(rpd*qr)/2.0);
    f[10] = (float)(log1p(lpd*qh)/2.0);
    // oscillation of the cross-section and length factors (period pi in
    // qR and qL/2), damped as a gaussian size distribution damps them
    const double ar = exp(-2.0*(rpd*qr)*(rpd*qr));
    const double al = exp(-2.0*(lpd*qh)*(lpd*qh));
    double sr, cr, sh, ch;
    sincos(2.0*qr, &sr, &cr);
    sincos(2.0*qh, &sh, &ch);
    f[11] = (float)(ar*cr);
    f[12] = (float)(ar*sr);
    f[13] = (float)(al*ch);
    f[14] = (float)(al*sh);
}

__device__ __forceinline__ void save_features(const float (&f)[16], __nv_bfloat16 *x,
                                              __nv_bfloat16 *x_lo, int i)
{
    float lo[16];
    #pragma unroll
    for (int j = 0; j < 16; ++j) lo[j] = f[j] - __bfloat162float(__float2bfloat16_rn(f[j]));
    save16(x + (size_t)i*NIN, f);
    save16(x_lo + (size_t)i*NIN, lo);
}

// 500,009 rows 28.8 -> 17.9 us, 100,000 rows 8.6 -> 5.9 (the last wave of blocks of
// 256 threads cost 0.6 of it).
__global__ void __launch_bounds__(128)
features(int n, int n_pad, const double *__restrict__ radius,
                         const double *__restrict__ length, const double *__restrict__ rpd,
                         const double *__restrict__ lpd, const double *__restrict__ drho,
                         const double *__restrict__ q, const double *__restrict__ flag,
                         __nv_bfloat16 *__restrict__ x, __nv_bfloat16 *__restrict__ x_lo)
{
    const int i = blockIdx.x*blockDim.x + threadIdx.x;
    if (i >= n_pad) return;
    float f[16];
    #pragma unroll
    for (int j = 0; j < 16; ++j) f[j] = 0.0f;
    if (i < n) feature_row(radius[i], length[i], rpd[i], lpd[i], drho[i], q[i], flag[i], f);
    save_features(f, x, x_lo, i);
}

// Points that come as runs sharing a parameter set: run r covers the points
// starts[r] <= i < starts[r + 1] (starts[0] = 0), its row of `table` is (radius,
// length, radius pd, length pd, contrast, flag, inside the domain).
__device__ __forceinline__ int run_of(const int *__restrict__ starts, int runs, int i)
{
    int lo = 0, hi = runs;                 // starts[lo] <= i < starts[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (starts[mid] <= i) lo = mid; else hi = mid;
    }
    return lo;
}

constexpr int RUN_COLS = 7;
// The features of such points, without the seven columns of n doubles in between
// (56 bytes a point written and read again, by eight launches).
__global__ void __launch_bounds__(128)
features_runs(int n, int n_pad, int runs, const int *__restrict__ starts,
              const double *__restrict__ table, const double *__restrict__ q,
              __nv_bfloat16 *__restrict__ x, __nv_bfloat16 *__restrict__ x_lo)
{
    const int i = blockIdx.x*blockDim.x + threadIdx.x;
    if (i >= n_pad) return;
    float f[16];
    #pragma unroll
    for (int j = 0; j < 16; ++j) f[j] = 0.0f;
    if (i < n) {
        const double *row = table + (size_t)RUN_COLS*run_of(starts, runs, i);
        feature_row(row[0], row[1], row[2], row[3], row[4], q[i], row[5], f);
    }
    save_features(f, x, x_lo, i);
}

// I = exp(out y_std + y_mean + 2 log|contrast|) of every point, and whether the
// network is trusted there: inside the domain, q inside its range and the gate's
// prediction at most thr (gate null: nowhere).  Every operation rounds on its own.
__global__ void __launch_bounds__(256)
finish_runs(int n, int runs, const int *__restrict__ starts, const double *__restrict__ table,
            const double *__restrict__ q, const float *__restrict__ out,
            const float *__restrict__ gate, double y_std, double y_mean, double g_std,
            double g_mean, double thr, double q_lo, double q_hi, double *__restrict__ I,
            uint8_t *__restrict__ accept)
{
    const int i = blockIdx.x*blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double *row = table + (size_t)RUN_COLS*run_of(starts, runs, i);
    const double y = __dadd_rn(__dmul_rn((double)out[i], y_std), y_mean);
    I[i] = exp(__dadd_rn(y, __dmul_rn(2.0, log(fabs(row[4])))));
    bool ok = row[6] > 0.5 && q[i] >= q_lo && q[i] <= q_hi;
    if (ok) ok = gate != nullptr
                 && __dadd_rn(__dmul_rn((double)gate[i], g_std), g_mean) <= thr;
    accept[i] = ok ? 1 : 0;
}

inline char *errbuf()
{
    static thread_local char buf[256] = "";
    return buf;
}

inline int32_t status(const char *what)
{
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        std::snprintf(errbuf(), 256, "%s: %s", what, cudaGetErrorString(e));
        return -3;
    }
    return 0;
}

// ---------------------------------------------------------------- inference --
// mlp_infer: the forward pass without the training planes, as a persistent,
// pipelined kernel.  One CTA per SM walks 128-row tiles; a producer warp
// streams the 24 weight chunks of every tile (layers 1-3, 8 chunks of
// 256 x 32) through a 4-stage shared-memory ring with bulk copies (TMA
// engine) that complete on mbarriers, running ahead into the next layer and
// tile while the eight consumer warps do the epilogues; one consumer thread
// issues the MMAs and frees each stage with tcgen05.commit.  The weights
// come pre-arranged (mlp_pack) so every chunk is one contiguous 16 KB copy
// that lands in the canonical K-major layout.  The arithmetic is that of
// mlp_forward (same compensated activations, bias, SiLU, output dot).
constexpr int KCI = 32;                          // K per streamed chunk
constexpr int CHUNK_BYTES = HID*KCI*2;           // 16 KB
constexpr int CHUNKS_PER_LAYER = HID/KCI;        // 8
constexpr int CHUNKS_PER_TILE = 3*CHUNKS_PER_LAYER;
constexpr int STAGES = 4;
constexpr int W0_BYTES = HID*NIN*2;              // 8 KB
constexpr int IMG_BYTES = W0_BYTES + CHUNKS_PER_TILE*CHUNK_BYTES;
constexpr int X_BYTES = TM*NIN*2;                // 4 KB
constexpr int INF_CONSUMERS = 256;               // 8 warps
constexpr int INF_THREADS = INF_CONSUMERS + 32;  // + producer warp
constexpr int INF_SMEM = 2*ACT_BYTES + STAGES*CHUNK_BYTES + W0_BYTES + 2*X_BYTES;

// The batch of a captured training step: rows idx[n] of a data set of `rows` rows,
// and the schedule to advance (see schedule_step).  idx null: none.
struct Batch {
    const int64_t *idx;
    long long rows;
    const __nv_bfloat16 *x_all, *xlo_all;
    const float *y_all;
    __nv_bfloat16 *x, *x_lo;      // where the batch goes
    float *y;
    int *counters;
    float *sched;                 // sched[3] != 0: a row was outside, nothing is updated any more
    int *refused;                 // the same for the host (its memory)
    int total, warmup;
    float lr0, b1, b2;
};

// The data set's row of batch row r, or -1 outside the data set.  Such a step may
// not train: its loss is undefined and adam_pack leaves everything as it is, in
// this step and all that follow with this schedule.
__device__ __forceinline__ long long batch_row(const Batch &batch, int r, int *err)
{
    const long long src = batch.idx[r];
    if (src >= 0 && src < batch.rows) return src;
    atomicExch(err, 5);
    batch.sched[3] = 1.0f;
    *(volatile int *)batch.refused = 1;
    return -1;
}

struct InferParams {
    const uint8_t *img;           // packed weights (mlp_pack)
    const float *b[4];
    const float *w_out;
    const float *b_out;
    __nv_bfloat16 *z_save;        // optional [4][n_pad x 256] pre-activations (training)
    __nv_bfloat16 *h_save;        // optional [4][n_pad x 256] activations (training)
    // training step (tiled planes): targets, Huber threshold, the loss gradient
    // [n_pad], and [2][4 n_tiles] sums over 32 rows of the loss and of dout
    const float *y;
    float delta;
    float *dout, *row_sums;
    Batch batch;                  // mlp_halves: instead of x, x_lo and y
};

// W_l [out][in] bf16 -> the chunk image: W0 as one 256 x 16 canonical tile,
// then for l = 1..3 and c = 0..7 the 256 x 32 canonical tile of columns
// [32c, 32c + 32).
__global__ void mlp_pack(const __nv_bfloat16 *__restrict__ w0, const __nv_bfloat16 *__restrict__ w1,
                         const __nv_bfloat16 *__restrict__ w2, const __nv_bfloat16 *__restrict__ w3,
                         uint8_t *__restrict__ img)
{
    constexpr int G0 = HID*(NIN/8);                 // 16-byte groups of W0
    constexpr int GL = HID*(HID/8);                 // of one hidden layer
    for (int i = blockIdx.x*blockDim.x + threadIdx.x; i < G0 + 3*GL; i += gridDim.x*blockDim.x) {
        if (i < G0) {
            const int r = i/(NIN/8), k = 8*(i % (NIN/8));
            *reinterpret_cast<uint4 *>(img + tc::kmajor_offset<HID>(r, k)) =
                *reinterpret_cast<const uint4 *>(w0 + r*NIN + k);
            continue;
        }
        const int j = i - G0, l = j/GL, rem = j % GL;
        const int r = rem/(HID/8), k = 8*(rem % (HID/8));
        const __nv_bfloat16 *w = l == 0 ? w1 : (l == 1 ? w2 : w3);
        const int c = k/KCI;
        uint8_t *dst = img + W0_BYTES + (size_t)(l*CHUNKS_PER_LAYER + c)*CHUNK_BYTES
                     + tc::kmajor_offset<HID>(r, k - c*KCI);
        *reinterpret_cast<uint4 *>(dst) = *reinterpret_cast<const uint4 *>(w + r*HID + k);
    }
}

// The 24 chunks of three 256 x 256 matrices without W0 (layers a, b, c in
// consumption order): the transposed weights W3^T, W2^T, W1^T that the
// pipelined backward streams.
__global__ void mlp_pack_layers(const __nv_bfloat16 *__restrict__ wa,
                                const __nv_bfloat16 *__restrict__ wb,
                                const __nv_bfloat16 *__restrict__ wc, uint8_t *__restrict__ img)
{
    constexpr int GL = HID*(HID/8);
    for (int j = blockIdx.x*blockDim.x + threadIdx.x; j < 3*GL; j += gridDim.x*blockDim.x) {
        const int l = j/GL, rem = j % GL;
        const int r = rem/(HID/8), k = 8*(rem % (HID/8));
        const __nv_bfloat16 *w = l == 0 ? wa : (l == 1 ? wb : wc);
        const int c = k/KCI;
        uint8_t *dst = img + (size_t)(l*CHUNKS_PER_LAYER + c)*CHUNK_BYTES
                     + tc::kmajor_offset<HID>(r, k - c*KCI);
        *reinterpret_cast<uint4 *>(dst) = *reinterpret_cast<const uint4 *>(w + r*HID + k);
    }
}

__global__ void __launch_bounds__(INF_THREADS, 1)
mlp_infer(int n, int n_tiles, const __nv_bfloat16 *__restrict__ x,
          const __nv_bfloat16 *__restrict__ x_lo, InferParams prm, float *__restrict__ out,
          int *__restrict__ err)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t *act = smem;
    uint8_t *act_lo = smem + ACT_BYTES;
    uint8_t *ring = smem + 2*ACT_BYTES;
    uint8_t *w0 = ring + STAGES*CHUNK_BYTES;
    uint8_t *xs = w0 + W0_BYTES;
    uint8_t *xs_lo = xs + X_BYTES;
    __shared__ __align__(8) uint64_t full[STAGES], empty[STAGES], acc_bar, w0_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ float dot_half[TM];
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int my_tiles = blockIdx.x < n_tiles ? (n_tiles - 1 - blockIdx.x)/gridDim.x + 1 : 0;

    if (warp == 0) {
        tc::tmem_alloc(&tmem_slot, HID);
        tc::tmem_relinquish();
    }
    if (t == 0) {
        for (int s = 0; s < STAGES; ++s) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], 1);
        }
        tc::mbar_init(&acc_bar, 1);
        tc::mbar_init(&w0_bar, 1);
        tc::mbar_fence_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_slot;

    if (warp == INF_CONSUMERS/32) {
        // ---- producer: one lane issues every bulk copy ----
        if (lane == 0) {
            bool ok = true;
            tc::mbar_arrive_expect_tx(&w0_bar, W0_BYTES);
            tc::bulk_load(w0, prm.img, W0_BYTES, &w0_bar);
            const int total = my_tiles*CHUNKS_PER_TILE;
            int i = 0;
            for (; i < total; ++i) {
                const int s = i % STAGES, use = i/STAGES;
                if (use > 0 && !tc::mbar_wait(&empty[s], (uint32_t)((use - 1) & 1))) {
                    ok = false;
                    break;
                }
                tc::mbar_arrive_expect_tx(&full[s], CHUNK_BYTES);
                tc::bulk_load(ring + s*CHUNK_BYTES,
                              prm.img + W0_BYTES + (size_t)(i % CHUNKS_PER_TILE)*CHUNK_BYTES,
                              CHUNK_BYTES, &full[s]);
            }
            // every issued copy has landed before the CTA may exit
            for (int j = (i > STAGES ? i - STAGES : 0); j < i; ++j)
                ok = tc::mbar_wait(&full[j % STAGES], (uint32_t)((j/STAGES) & 1)) && ok;
            ok = tc::mbar_wait(&w0_bar, 0u) && ok;
            if (!ok) atomicExch(err, 2);
        }
    } else {
        // ---- consumers ----
        bool ok = true;
        uint32_t acc_phase = 0;
        int chunk = 0;                                  // used by t == 0 only
        const int quad = warp & 3, half = warp >> 2;
        const int row = 32*quad + lane;                 // TMEM lane = tile row
        const uint32_t lane_base = (uint32_t)(32*quad) << 16;
        const size_t plane = (size_t)n_tiles*TM*HID;
        constexpr uint32_t idesc = tc::idesc_bf16(TM, HID);
        if (t == 0) ok = tc::mbar_wait(&w0_bar, 0u);
        ok = tc::bar_and(1, INF_CONSUMERS, ok);
        for (int k = 0; k < my_tiles && ok; ++k) {
            const int row0 = (blockIdx.x + k*gridDim.x)*TM;
            {
                const int r = t >> 1, c = (t & 1)*8;
                const size_t g = (size_t)(row0 + r)*NIN + c;
                *reinterpret_cast<uint4 *>(xs + tc::kmajor_offset<TM>(r, c)) =
                    *reinterpret_cast<const uint4 *>(x + g);
                *reinterpret_cast<uint4 *>(xs_lo + tc::kmajor_offset<TM>(r, c)) =
                    *reinterpret_cast<const uint4 *>(x_lo + g);
            }
            tc::fence_async_smem();
            tc::fence_before_sync();
            ok = tc::bar_and(1, INF_CONSUMERS, ok);
            tc::fence_after_sync();
            if (!ok) break;
            if (t == 0) {
                const uint64_t bdesc = tc::kmajor_desc<HID>(tc::smem_u32(w0), 0);
                tc::mma_bf16(tmem, tc::kmajor_desc<TM>(tc::smem_u32(xs), 0), bdesc, idesc, 0u);
                tc::mma_bf16(tmem, tc::kmajor_desc<TM>(tc::smem_u32(xs_lo), 0), bdesc, idesc, 1u);
                tc::mma_commit(&acc_bar);
            }
            for (int l = 0; l < 4; ++l) {
                if (l > 0 && t == 0) {
                    const uint32_t a_hi = tc::smem_u32(act), a_lo = tc::smem_u32(act_lo);
                    for (int c = 0; c < CHUNKS_PER_LAYER; ++c, ++chunk) {
                        const int s = chunk % STAGES;
                        if (!tc::mbar_wait(&full[s], (uint32_t)((chunk/STAGES) & 1))) {
                            ok = false;
                            break;
                        }
                        tc::fence_after_sync();
                        const uint32_t b_addr = tc::smem_u32(ring + s*CHUNK_BYTES);
                        #pragma unroll
                        for (int st = 0; st < KCI/16; ++st) {
                            const uint64_t bdesc = tc::kmajor_desc<HID>(b_addr, st);
                            const int as = c*(KCI/16) + st;
                            tc::mma_bf16(tmem, tc::kmajor_desc<TM>(a_hi, as), bdesc, idesc,
                                         (c > 0 || st > 0) ? 1u : 0u);
                            tc::mma_bf16(tmem, tc::kmajor_desc<TM>(a_lo, as), bdesc, idesc, 1u);
                        }
                        tc::mma_commit(&empty[s]);
                    }
                    tc::mma_commit(&acc_bar);
                }
                const bool done = tc::mbar_wait(&acc_bar, acc_phase);
                acc_phase ^= 1u;
                tc::fence_after_sync();
                ok = tc::bar_and(1, INF_CONSUMERS, ok && done);
                if (!ok) break;
                // epilogue: this thread's row, columns [128 half, 128 half + 128),
                // 32 columns per TMEM wait (two loads in flight), each group of
                // 16 processed in column order as before
                const float *bias = prm.b[l];
                float dot = 0.0f;
                #pragma unroll 1
                for (int c32 = 128*half; c32 < 128*half + 128; c32 += 32) {
                    uint32_t r32[2][16];
                    tc::tmem_ld16(tmem + lane_base + (uint32_t)c32, r32[0]);
                    tc::tmem_ld16(tmem + lane_base + (uint32_t)(c32 + 16), r32[1]);
                    tc::tmem_wait_ld();
                    #pragma unroll
                    for (int g = 0; g < 2; ++g) {
                        const int c0 = c32 + 16*g;
                        float z[16], h[16];
                        #pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            z[j] = __uint_as_float(r32[g][j]) + bias[c0 + j];
                            h[j] = silu(z[j]);
                        }
                        if (prm.z_save != nullptr) {
                            const size_t at = (size_t)l*plane + (size_t)(row0 + row)*HID + c0;
                            save16(prm.z_save + at, z);
                            save16(prm.h_save + at, h);
                        }
                        if (l == 3) {
                            #pragma unroll
                            for (int j = 0; j < 16; ++j)
                                dot = fmaf(h[j], prm.w_out[c0 + j], dot);
                        } else {
                            store16_split(act, act_lo, row, c0, h);
                        }
                    }
                }
                if (l == 3) {
                    if (half == 1) dot_half[row] = dot;
                    tc::bar_sync(2, INF_CONSUMERS);
                    if (half == 0 && row0 + row < n) out[row0 + row] = dot + dot_half[row] + *prm.b_out;
                }
                tc::fence_async_smem();
                tc::fence_before_sync();
                ok = tc::bar_and(1, INF_CONSUMERS, ok);
                tc::fence_after_sync();
                if (!ok) break;
            }
        }
        if (!ok && t == 0) atomicExch(err, 1);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, HID);
}

// -------------------------------------------------------- training planes --
// The pre-activations z, the activations h and the gradients dZ of a
// training step live in tiled planes [4 layers][n_tiles][32 groups][128 rows][8]
// bf16: the 128 x 256 tile of a CTA is one 64 KB image, the 8 columns of a group
// 16 contiguous bytes per row.  A warp whose lanes hold consecutive rows reads
// and writes 512 contiguous bytes (of row-major planes 32 separate 16-byte
// pieces: the forward of 8192 rows took 50 us with them and takes 28), and the
// image is at the same time the canonical MN-major operand of dW = dZ^T H, whose
// K dimension is the rows, so nothing is transposed on the way.
constexpr int TILE_ELEMS = TM*HID;
constexpr int GROUP_ELEMS = TM*8;

// Element of a tiled plane: tile `tile` of layer `l`, column group kg, row.
__device__ __forceinline__ size_t tiled_at(int l, int n_tiles, int tile, int kg, int row)
{
    return ((size_t)l*n_tiles + tile)*TILE_ELEMS + (size_t)kg*GROUP_ELEMS + 8*row;
}

// ------------------------------------------------------- paired arithmetic --
// Two FP32 lanes in one register pair: each half rounded to nearest.
__device__ __forceinline__ uint64_t f2_pack(float a, float b)
{
    uint64_t v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
    return v;
}
__device__ __forceinline__ void f2_unpack(uint64_t v, float &a, float &b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// silu of two pre-activations (see silu())
__device__ __forceinline__ uint64_t silu2(uint64_t z)
{
    const uint64_t hz = f2_mul(z, f2_pack(0.5f, 0.5f));
    float x0, x1, t0, t1;
    f2_unpack(hz, x0, x1);
    asm("tanh.approx.f32 %0, %1;" : "=f"(t0) : "f"(x0));
    asm("tanh.approx.f32 %0, %1;" : "=f"(t1) : "f"(x1));
    return f2_fma(hz, f2_pack(t0, t1), hz);
}
// two accumulator columns plus bias
__device__ __forceinline__ uint64_t bias2(uint32_t a0, uint32_t a1, uint64_t bias)
{
    return f2_add(f2_pack(__uint_as_float(a0), __uint_as_float(a1)), bias);
}
__device__ __forceinline__ uint32_t pack2(uint64_t v)
{
    float x, y;
    f2_unpack(v, x, y);
    return pack2(x, y);
}

// 8 columns of a row, from the accumulators r[at ..]: silu, then the hi and lo
// halves (one 16-byte unit each), and the pre-activations if they are wanted
template <bool Z = false, int N>
__device__ __forceinline__ void silu_columns(const uint32_t (&r)[N], int at, const float *bias,
                                             uint4 &hi, uint4 &lo, uint4 *zq = nullptr)
{
    const ulonglong2 *b2 = reinterpret_cast<const ulonglong2 *>(bias + at);
    const uint64_t minus1 = f2_pack(-1.0f, -1.0f);
    uint32_t *hp = &hi.x, *lp = &lo.x;
    #pragma unroll
    for (int e = 0; e < 2; ++e) {
        const ulonglong2 b = b2[e];
        #pragma unroll
        for (int q = 0; q < 2; ++q) {
            const uint64_t z = bias2(r[at + 4*e + 2*q], r[at + 4*e + 2*q + 1], q ? b.y : b.x);
            const uint64_t h = silu2(z);
            const uint32_t u = pack2(h);
            hp[2*e + q] = u;
            lp[2*e + q] = pack2(f2_fma(f2_pack(bf_lo(u), bf_hi(u)), minus1, h));
            if (Z) (&zq->x)[2*e + q] = pack2(z);
        }
    }
}

// dot + sum over 8 columns of silu(acc + bias) wo, in column order
__device__ __forceinline__ float dot8(const uint32_t (&r)[8], const float *bias, const float *wo,
                                      float dot)
{
    const ulonglong2 *b2 = reinterpret_cast<const ulonglong2 *>(bias);
    const float4 *w4 = reinterpret_cast<const float4 *>(wo);
    #pragma unroll
    for (int e = 0; e < 2; ++e) {
        const ulonglong2 b = b2[e];
        const float4 w = w4[e];
        float h0, h1, h2, h3;
        f2_unpack(silu2(bias2(r[4*e], r[4*e + 1], b.x)), h0, h1);
        f2_unpack(silu2(bias2(r[4*e + 2], r[4*e + 3], b.y)), h2, h3);
        dot = fmaf(h0, w.x, dot);
        dot = fmaf(h1, w.y, dot);
        dot = fmaf(h2, w.z, dot);
        dot = fmaf(h3, w.w, dot);
    }
    return dot;
}

// ------------------------------------------------------------------ serve --
// mlp_serve: the forward pass (inference, or training with the z/h planes)
// with the tensor core and the epilogue busy at the same time.  Arithmetic per element as mlp_infer
// (bias, SiLU, the compensated hi/lo split rounded to nearest), so the
// hidden activations are bitwise those of mlp_infer; the output dot sums
// the 256 columns in another order (four partial sums per row).
//
// Roles, 20 warps per CTA (one CTA per SM, persistent over 128-row tiles):
//   warps 0-15  epilogue.  Warp w reads the TMEM lanes of its quadrant
//               (rows 32(w%4) .. +31) and the 16 columns at 16(w/4) of every 64,
//               all of them before the first is used (which frees the
//               accumulator); 64 by 64 columns: bias + SiLU + split into the
//               activation tile, then one arrive per warp on act_ready[64 columns];
//               but for the first and the last it comes behind the arithmetic
//               of the next 64, under which the stores land.  In the last layer the 8 columns at 8(w/4) of every 32.
//   warp 16     lane 0 issues every MMA; all lanes load the next tile's
//               features while the tensor core runs the last layer.  An MMA
//               issue holds its thread for about the tensor core's time for
//               the previous MMA, so this lane does no barrier waits of its
//               own for layers 1-3: it spins on a counter of ready chunks.
//   warp 17     the bulk-copy producer of the weight ring (as mlp_infer).
//   warps 18,   one lane each: count the chunks whose input is written (and whose
//        19     accumulator is free), and those whose weights have landed
//               (release stores), so that neither wait is behind the other.
// Two TMEM accumulators (columns [0, 256) and [256, 512)): layer l of a tile
// accumulates into acc[l & 1], so layer l+1's MMAs start on the first columns of
// its input as soon as the epilogue of layer l has written them.  The activations
// are rewritten in place: the epilogue of layer l starts only after every MMA of
// layer l (the readers of the old activations) has completed.  acc_empty[a] tells
// the MMA warp that all sixteen epilogue warps have finished their TMEM loads of
// acc[a], before the next layer that accumulates there.
//
// Barrier phases (all parity waits, bounded): per tile acc_full[a] and
// acc_empty[a] complete twice (layers a and a + 2), act_ready[c] three times
// (inputs of layers 1-3), dot_bar[quadrant] once; none can run two phases
// ahead of its waiter because each completion needs the waiter's previous
// step (argued at each wait below).
//
// One tile per CTA: 17.5 us (19.0 with one warp waiting for a chunk's three barriers
// in turn, an arrival per 32 columns, and the features loaded 16 bytes at a time).
// Bound by the chain of one tile: 4 x (commit, 16 columns of epilogue, hand-over,
// 8 chunks of MMA at 540-690 cycles).
constexpr int SV_EPI_WARPS = 16;
constexpr int SV_EPI = 32*SV_EPI_WARPS;                    // 512 epilogue threads
constexpr int SV_MMA_WARP = SV_EPI_WARPS;
constexpr int SV_PROD_WARP = SV_EPI_WARPS + 1;
constexpr int SV_ACT_WARP = SV_EPI_WARPS + 2;
constexpr int SV_WEIGHT_WARP = SV_EPI_WARPS + 3;
constexpr int SV_THREADS = SV_EPI + 128;
constexpr int SV_COLS = KCI/(SV_EPI_WARPS/4);              // 8 columns of a chunk per warp
constexpr int SV_PARAMS = 5*HID;                           // b[0..3], w_out (floats)
constexpr int SV_SMEM = 2*ACT_BYTES + STAGES*CHUNK_BYTES + W0_BYTES + 4*X_BYTES + 4*SV_PARAMS;
constexpr int SV_UNITS = HID/64;                           // 64 columns per hand-over
static_assert(SV_COLS == 8, "the epilogue moves one 16-byte unit per row and chunk");

// Bounded wait by every lane of a warp on one mbarrier phase; the warp agrees
// on the outcome.  (Polling by lane 0 alone with a shuffle of the outcome was
// measured slower here.)
__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity)
{
    return __all_sync(0xffffffffu, tc::mbar_wait(bar, parity)) != 0;
}
// The same for a barrier that both CTAs of a pair arrive on, or their MMAs complete.
__device__ __forceinline__ bool warp_wait_cluster(uint64_t *bar, uint32_t parity)
{
    return __all_sync(0xffffffffu, tc::mbar_wait_cluster(bar, parity)) != 0;
}

// z = acc + bias and h = silu(z) for 8 columns, accumulators r[at ..].
template <int N>
__device__ __forceinline__ void sv_silu8(const uint32_t (&r)[N], int at, const float *bias,
                                         float (&z)[8], float (&h)[8])
{
    const float4 b0 = *reinterpret_cast<const float4 *>(bias + at);
    const float4 b1 = *reinterpret_cast<const float4 *>(bias + at + 4);
    const float bb[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
    #pragma unroll
    for (int j = 0; j < 8; ++j) {
        z[j] = __uint_as_float(r[at + j]) + bb[j];
        h[j] = silu(z[j]);
    }
}

// hi = bf16(h), lo = bf16(h - hi) of 8 columns, one 16-byte unit each
__device__ __forceinline__ void split8(const float (&h)[8], uint4 &hi, uint4 &lo)
{
    uint32_t *hp = &hi.x, *lp = &lo.x;
    #pragma unroll
    for (int e = 0; e < 4; ++e) {
        const uint32_t u = pack2(h[2*e], h[2*e + 1]);
        hp[e] = u;
        lp[e] = pack2(h[2*e] - bf_lo(u), h[2*e + 1] - bf_hi(u));
    }
}

// 8 floats as bf16 (round to nearest) in one 16-byte store
__device__ __forceinline__ void save8(__nv_bfloat16 *dst, const float (&v)[8])
{
    uint4 u;
    u.x = pack2(v[0], v[1]);
    u.y = pack2(v[2], v[3]);
    u.z = pack2(v[4], v[5]);
    u.w = pack2(v[6], v[7]);
    *reinterpret_cast<uint4 *>(dst) = u;
}

// An MMA lane's view of a count of ready units: covers(n) waits until n are ready
// (bounded), reading the count only when the last value does not cover n.
struct ReadyCount {
    const uint32_t *at;
    uint32_t known = 0;
    __device__ explicit ReadyCount(const uint32_t *p) : at(p) {}
    __device__ __forceinline__ bool covers(uint32_t n)
    {
        if (known < n) known = tc::spin_acquire_until(at, n);
        return known >= n;
    }
};
// The same of two counts, each kept by a warp of its own: chunks whose input is
// written (x) and chunks whose weights have landed (y).
struct ReadyCounts {
    const uint2 *at;
    uint32_t known = 0;
    __device__ explicit ReadyCounts(const uint2 *p) : at(p) {}
    __device__ __forceinline__ bool covers(uint32_t n)
    {
        for (uint32_t i = 0; i < tc::WAIT_LIMIT && known < n; ++i) {
            const uint2 v = tc::ld_acquire_shared2(at);
            known = min(v.x, v.y);
        }
        return known >= n;
    }
};

// PLANES: none (inference), row-major z/h planes, or a training step's tiled
// planes with the loss gradient of every row.
enum { PLANES_NONE, PLANES_ROWS, PLANES_TILED };
template <int PLANES>
__global__ void __launch_bounds__(SV_THREADS, 1)
mlp_serve(int n, int n_tiles, const __nv_bfloat16 *x, const __nv_bfloat16 *x_lo, InferParams prm, float *__restrict__ out,
          int *__restrict__ err)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t *act = smem;
    uint8_t *act_lo = smem + ACT_BYTES;
    uint8_t *ring = smem + 2*ACT_BYTES;
    uint8_t *w0 = ring + STAGES*CHUNK_BYTES;
    uint8_t *xs = w0 + W0_BYTES;                  // [2 buffers][hi, lo] x X_BYTES
    float *par = reinterpret_cast<float *>(xs + 4*X_BYTES);
    __shared__ __align__(8) uint64_t full[STAGES], empty[STAGES], act_ready[SV_UNITS];
    __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2], dot_bar[4], w0_bar, drain;
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(8) uint2 ready_seq;
    __shared__ float dot_part[3][TM];
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int my_tiles = blockIdx.x < n_tiles ? (n_tiles - 1 - blockIdx.x)/gridDim.x + 1 : 0;

    if (warp == 0) {
        tc::tmem_alloc(&tmem_slot, 2*HID);
        tc::tmem_relinquish();
    }
    if (t == 0) {
        for (int s = 0; s < STAGES; ++s) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], 1);
        }
        for (int c = 0; c < SV_UNITS; ++c) tc::mbar_init(&act_ready[c], SV_EPI_WARPS);
        for (int a = 0; a < 2; ++a) {
            tc::mbar_init(&acc_full[a], 1);
            tc::mbar_init(&acc_empty[a], SV_EPI_WARPS);
        }
        for (int q = 0; q < 4; ++q) tc::mbar_init(&dot_bar[q], SV_EPI_WARPS/4 - 1);
        tc::mbar_init(&w0_bar, 1);
        tc::mbar_init(&drain, 1);
        ready_seq = make_uint2(0u, 0u);
        tc::mbar_fence_init();
    }
    tc::dependents_launch();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    tc::dependency_wait();
    const uint32_t tmem = tmem_slot;

    if (warp == SV_PROD_WARP) {
        // ---- producer: the weight chunks of every tile, in MMA order ----
        if (lane == 0) {
            bool ok = true;
            tc::mbar_arrive_expect_tx(&w0_bar, W0_BYTES);
            tc::bulk_load(w0, prm.img, W0_BYTES, &w0_bar);
            const int total = my_tiles*CHUNKS_PER_TILE;
            int i = 0;
            for (; i < total; ++i) {
                const int s = i % STAGES, use = i/STAGES;
                if (use > 0 && !tc::mbar_wait(&empty[s], (uint32_t)((use - 1) & 1))) {
                    ok = false;
                    break;
                }
                tc::mbar_arrive_expect_tx(&full[s], CHUNK_BYTES);
                tc::bulk_load(ring + s*CHUNK_BYTES,
                              prm.img + W0_BYTES + (size_t)(i % CHUNKS_PER_TILE)*CHUNK_BYTES,
                              CHUNK_BYTES, &full[s]);
            }
            for (int j = (i > STAGES ? i - STAGES : 0); j < i; ++j)
                ok = tc::mbar_wait(&full[j % STAGES], (uint32_t)((j/STAGES) & 1)) && ok;
            ok = tc::mbar_wait(&w0_bar, 0u) && ok;
            if (!ok) atomicExch(err, 2);
        }
    } else if (warp == SV_ACT_WARP) {
        // ---- inputs: chunks of layers 1-3 whose accumulator is free and whose
        // activations are written, in MMA order ----
        if (lane == 0) {
            bool ok = true;
            uint32_t chunk = 0;
            for (int k = 0; k < my_tiles && ok; ++k) {
                for (int l = 1; l < 4 && ok; ++l) {
                    // previous reader of acc[l & 1]: layer 3 of tile k-1 for l = 1
                    // (completion 2k-1), layer l-2 of this tile for l = 2, 3
                    // (completion 2k); the next completion needs this layer's
                    // MMAs, which wait for what is published here
                    if ((l >= 2 || k > 0)
                        && !(ok = tc::mbar_wait(&acc_empty[l & 1], l >= 2 ? 0u : 1u)))
                        break;
                    for (int q = 0; q < SV_UNITS; ++q) {
                        // 64 columns of this layer's input: completion 3k + l - 1
                        if (!(ok = tc::mbar_wait(&act_ready[q], (uint32_t)((3*k + l - 1) & 1)))) break;
                        chunk += CHUNKS_PER_LAYER/SV_UNITS;
                        tc::st_release_shared(&ready_seq.x, chunk);
                    }
                }
            }
            if (!ok) atomicExch(err, 4);
        }
        __syncwarp();
    } else if (warp == SV_WEIGHT_WARP) {
        // ---- weights: chunks that have landed ----
        if (lane == 0) {
            bool ok = true;
            const uint32_t total = (uint32_t)(my_tiles*CHUNKS_PER_TILE);
            for (uint32_t i = 0; i < total && ok; ++i)
                if ((ok = tc::mbar_wait(&full[i % STAGES], (i/STAGES) & 1u)))
                    tc::st_release_shared(&ready_seq.y, i + 1);
            if (!ok) atomicExch(err, 4);
        }
        __syncwarp();
    } else if (warp == SV_MMA_WARP) {
        // ---- MMA issue (lane 0) and feature loads (all lanes) ----
        constexpr uint32_t idesc = tc::idesc_bf16(TM, HID);
        const uint32_t a_hi = tc::smem_u32(act), a_lo = tc::smem_u32(act_lo);
        auto load_x = [&](int k) {
            uint8_t *xb = xs + (k & 1)*2*X_BYTES;
            const int row0 = (blockIdx.x + k*gridDim.x)*TM;
            uint4 hi[2*TM/32], lo[2*TM/32];          // every load in flight at once
            #pragma unroll
            for (int j = 0; j < 2*TM/32; ++j) {
                const int i = lane + 32*j;
                const size_t g = (size_t)(row0 + (i >> 1))*NIN + (i & 1)*8;
                hi[j] = *reinterpret_cast<const uint4 *>(x + g);
                lo[j] = *reinterpret_cast<const uint4 *>(x_lo + g);
            }
            #pragma unroll
            for (int j = 0; j < 2*TM/32; ++j) {
                const int i = lane + 32*j;
                const uint32_t at = tc::kmajor_offset<TM>(i >> 1, (i & 1)*8);
                *reinterpret_cast<uint4 *>(xb + at) = hi[j];
                *reinterpret_cast<uint4 *>(xb + X_BYTES + at) = lo[j];
            }
            tc::fence_async_smem();
            __syncwarp();
        };
        bool ok = true;
        int chunk = 0;
        ReadyCounts count(&ready_seq);
        if (my_tiles > 0) load_x(0);
        ok = warp_wait(&w0_bar, 0u);
        for (int k = 0; k < my_tiles && ok; ++k) {
            // layer 0 into acc[0]; its previous reader is the epilogue of
            // layer 2 of tile k-1 (acc_empty[0] completion 2k-1, odd), which
            // cannot complete again before this MMA is issued
            if (k > 0 && !(ok = warp_wait(&acc_empty[0], 1u))) break;
            tc::fence_after_sync();
            if (lane == 0) {
                const uint32_t xb = tc::smem_u32(xs + (k & 1)*2*X_BYTES);
                const uint64_t bdesc = tc::kmajor_desc<HID>(tc::smem_u32(w0), 0);
                tc::mma_bf16(tmem, tc::kmajor_desc<TM>(xb, 0), bdesc, idesc, 0u);
                tc::mma_bf16(tmem, tc::kmajor_desc<TM>(xb + X_BYTES, 0), bdesc, idesc, 1u);
                tc::mma_commit(&acc_full[0]);
                // layers 1-3: each chunk as soon as both counts cover
                // it.  An MMA issue holds this thread about as long as the
                // tensor core takes for the previous one, so nothing else
                // runs on this thread between chunks.
                for (int l = 1; l < 4 && ok; ++l) {
                    const uint32_t d = tmem + (uint32_t)(HID*(l & 1));
                    for (int c = 0; c < CHUNKS_PER_LAYER; ++c, ++chunk) {
                        if (!(ok = count.covers((uint32_t)(chunk + 1)))) break;
                        tc::fence_after_sync();
                        const int s = chunk % STAGES;
                        const uint32_t b_addr = tc::smem_u32(ring + s*CHUNK_BYTES);
                        #pragma unroll
                        for (int st = 0; st < KCI/16; ++st) {
                            const uint64_t bdesc = tc::kmajor_desc<HID>(b_addr, st);
                            const int as = c*(KCI/16) + st;
                            tc::mma_bf16(d, tc::kmajor_desc<TM>(a_hi, as), bdesc, idesc,
                                         (c > 0 || st > 0) ? 1u : 0u);
                            tc::mma_bf16(d, tc::kmajor_desc<TM>(a_lo, as), bdesc, idesc, 1u);
                        }
                        tc::mma_commit(&empty[s]);
                    }
                    if (ok) tc::mma_commit(&acc_full[l & 1]);
                }
            }
            ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
            chunk = __shfl_sync(0xffffffffu, chunk, 0);
            // the features of the next tile go to the other buffer, last
            // read by layer 0 of tile k-1, complete since layer 1's inputs
            // of tile k-1 were produced from its result
            if (ok && k + 1 < my_tiles) load_x(k + 1);
        }
        // every MMA issued has completed before TMEM is released
        if (lane == 0) {
            tc::mma_commit(&drain);
            ok = tc::mbar_wait(&drain, 0u) && ok;
            if (!ok) atomicExch(err, 3);
        }
        __syncwarp();
    } else {
        // ---- epilogue warps ----
        for (int i = t; i < SV_PARAMS; i += SV_EPI)
            par[i] = i < 4*HID ? prm.b[i/HID][i % HID] : prm.w_out[i - 4*HID];
        tc::bar_sync(1, SV_EPI);
        const float b_out = *prm.b_out;
        const int quad = warp & 3, slot = warp >> 2;
        const int row = 32*quad + lane;
        const int cs = SV_COLS*slot;
        const size_t plane = (size_t)n_tiles*TM*HID;
        const uint32_t lane_base = (uint32_t)(32*quad) << 16;
        bool ok = true;
        for (int k = 0; k < my_tiles && ok; ++k) {
            const int row0 = (blockIdx.x + k*gridDim.x)*TM;
            for (int l = 0; l < 4; ++l) {
                const int a = l & 1;
                // acc_full[a]: completion 2k + (l >> 1)
                if (!(ok = warp_wait(&acc_full[a], (uint32_t)(l >> 1))))
                    break;
                tc::fence_after_sync();
                float dot = 0.0f;
                // 8 columns of a plane of this layer, for this row
                auto plane_at = [&](int col) {
                    return PLANES == PLANES_TILED ? tiled_at(l, n_tiles, row0/TM, col/8, row)
                                                  : (size_t)l*plane + (size_t)(row0 + row)*HID + col;
                };
                if (l < 3) {
                    // 16 columns of every 64
                    const uint32_t acc = tmem + lane_base + (uint32_t)(HID*a + 16*slot);
                    const float *bias = par + l*HID + 16*slot;
                    uint32_t r[SV_UNITS][16];
                    #pragma unroll
                    for (int q = 0; q < SV_UNITS; ++q) tc::tmem_ld16(acc + (uint32_t)(64*q), r[q]);
                    tc::tmem_wait_ld();
                    #pragma unroll
                    for (int q = 0; q < SV_UNITS; ++q) tc::tmem_tie16(r[q]);
                    tc::fence_before_sync();
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive(&acc_empty[a]);
                    #pragma unroll
                    for (int q = 0; q < SV_UNITS; ++q) {
                        uint4 hi[2], lo[2];
                        #pragma unroll
                        for (int g = 0; g < 2; ++g) {
                            if (PLANES == PLANES_NONE) {
                                silu_columns(r[q], 8*g, bias + 64*q, hi[g], lo[g]);
                            } else {
                                float z[8], h[8];
                                sv_silu8(r[q], 8*g, bias + 64*q, z, h);
                                split8(h, hi[g], lo[g]);
                                const size_t at = plane_at(64*q + 16*slot + 8*g);
                                save8(prm.z_save + at, z);
                                *reinterpret_cast<uint4 *>(prm.h_save + at) = hi[g];
                            }
                            // the stores of the 64 columns before have had time to land
                            if (g == 0 && q > 1) {
                                tc::fence_async_smem();
                                __syncwarp();
                                if (lane == 0) tc::mbar_arrive(&act_ready[q - 1]);
                            }
                        }
                        #pragma unroll
                        for (int g = 0; g < 2; ++g) {
                            const uint32_t off = tc::kmajor_offset<TM>(row, 64*q + 16*slot + 8*g);
                            *reinterpret_cast<uint4 *>(act + off) = hi[g];
                            *reinterpret_cast<uint4 *>(act_lo + off) = lo[g];
                        }
                        // the tensor core is waiting for the first and the last
                        if (q == 0 || q == SV_UNITS - 1) {
                            tc::fence_async_smem();
                            __syncwarp();
                            if (lane == 0) tc::mbar_arrive(&act_ready[q]);
                        }
                    }
                } else {
                    // the output dot: 8 columns of every 32
                    const uint32_t acc = tmem + lane_base + (uint32_t)(HID*a + cs);
                    const float *bias = par + 3*HID + cs, *wo = par + 4*HID + cs;
                    uint32_t r[CHUNKS_PER_LAYER][8];
                    #pragma unroll
                    for (int c = 0; c < CHUNKS_PER_LAYER; ++c) tc::tmem_ld8(acc + (uint32_t)(KCI*c), r[c]);
                    #pragma unroll
                    for (int c = 0; c < CHUNKS_PER_LAYER; ++c) tc::tmem_wait_ld8(r[c]);
                    tc::fence_before_sync();
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive(&acc_empty[a]);
                    #pragma unroll
                    for (int c = 0; c < CHUNKS_PER_LAYER; ++c) {
                        if (PLANES == PLANES_NONE) {
                            dot = dot8(r[c], bias + KCI*c, wo + KCI*c, dot);
                        } else {
                            float z[8], h[8];
                            sv_silu8(r[c], 0, bias + KCI*c, z, h);
                            const size_t at = plane_at(KCI*c + cs);
                            save8(prm.z_save + at, z);
                            save8(prm.h_save + at, h);
                            #pragma unroll
                            for (int e = 0; e < 8; ++e) dot = fmaf(h[e], wo[KCI*c + e], dot);
                        }
                    }
                }
                if (l == 3) {
                    // four partial sums per row; slot 0 adds them.  Slots
                    // 1-3 write dot_part again only in the next tile's last
                    // layer, which needs slot 0's activations of that tile.
                    if (slot > 0) {
                        dot_part[slot - 1][row] = dot;
                        __syncwarp();
                        if (lane == 0) tc::mbar_arrive(&dot_bar[quad]);
                    } else {
                        if (!(ok = warp_wait(&dot_bar[quad], (uint32_t)(k & 1))))
                            break;
                        const bool valid = row0 + row < n;
                        const float o = ((dot + dot_part[0][row]) + dot_part[1][row])
                                        + dot_part[2][row] + b_out;
                        if (valid) out[row0 + row] = o;
                        if (PLANES == PLANES_TILED) {
                            float g, loss;
                            loss_of(valid ? o - prm.y[row0 + row] : 0.0f, prm.delta, g, loss);
                            g = valid ? g/(float)n : 0.0f;
                            prm.dout[row0 + row] = g;
                            #pragma unroll
                            for (int o2 = 16; o2 > 0; o2 >>= 1) {
                                g += __shfl_xor_sync(0xffffffffu, g, o2);
                                loss += __shfl_xor_sync(0xffffffffu, loss, o2);
                            }
                            if (lane == 0) {
                                float *sums = prm.row_sums + 4*(row0/TM) + quad;
                                sums[0] = loss;
                                sums[4*n_tiles] = g;
                            }
                        }
                    }
                }
            }
        }
        if (!ok && lane == 0) atomicExch(err, 1);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, 2*HID);
}

#include "mlp_train.cuh"
#include "mlp_pairs.cuh"
#include "mlp_halves.cuh"

// ---------------------------------------------------------------- backward --
// mlp_backward_p: the backward pass through the three 256 x 256 layers as a
// persistent, pipelined kernel with the structure of mlp_infer: a producer
// warp streams the 24 chunks of W3^T, W2^T, W1^T (packed by
// mlp_pack_layers) through the 4-stage ring, one consumer thread issues the
// MMAs (A = dZ_l in shared memory, B = W_l^T), eight consumer warps run the
// epilogues dZ_{l-1} = (dZ_l W_l) * silu'(z_{l-1}), reading z from the saved
// plane and writing dZ to its plane and, for the next layer, to shared
// memory.  The arithmetic is that of mlp_backward.
constexpr int BWDP_SMEM = ACT_BYTES + STAGES*CHUNK_BYTES;
constexpr int WT_IMG_BYTES = CHUNKS_PER_TILE*CHUNK_BYTES;

__global__ void __launch_bounds__(INF_THREADS, 1)
mlp_backward_p(int n, int n_tiles, const uint8_t *__restrict__ img_t,
               const float *__restrict__ w_out, const float *__restrict__ dout,
               const __nv_bfloat16 *__restrict__ z_save, __nv_bfloat16 *__restrict__ dz_save,
               int *__restrict__ err)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t *act = smem;
    uint8_t *ring = smem + ACT_BYTES;
    __shared__ __align__(8) uint64_t full[STAGES], empty[STAGES], acc_bar;
    __shared__ uint32_t tmem_slot;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int my_tiles = blockIdx.x < n_tiles ? (n_tiles - 1 - blockIdx.x)/gridDim.x + 1 : 0;

    if (warp == 0) {
        tc::tmem_alloc(&tmem_slot, HID);
        tc::tmem_relinquish();
    }
    if (t == 0) {
        for (int s = 0; s < STAGES; ++s) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], 1);
        }
        tc::mbar_init(&acc_bar, 1);
        tc::mbar_fence_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_slot;

    if (warp == INF_CONSUMERS/32) {
        if (lane == 0) {
            bool ok = true;
            const int total = my_tiles*CHUNKS_PER_TILE;
            int i = 0;
            for (; i < total; ++i) {
                const int s = i % STAGES, use = i/STAGES;
                if (use > 0 && !tc::mbar_wait(&empty[s], (uint32_t)((use - 1) & 1))) {
                    ok = false;
                    break;
                }
                tc::mbar_arrive_expect_tx(&full[s], CHUNK_BYTES);
                tc::bulk_load(ring + s*CHUNK_BYTES,
                              img_t + (size_t)(i % CHUNKS_PER_TILE)*CHUNK_BYTES,
                              CHUNK_BYTES, &full[s]);
            }
            for (int j = (i > STAGES ? i - STAGES : 0); j < i; ++j)
                ok = tc::mbar_wait(&full[j % STAGES], (uint32_t)((j/STAGES) & 1)) && ok;
            if (!ok) atomicExch(err, 2);
        }
    } else {
        bool ok = true;
        uint32_t acc_phase = 0;
        int chunk = 0;                                  // used by t == 0 only
        const int quad = warp & 3, half = warp >> 2;
        const int row = 32*quad + lane;
        const uint32_t lane_base = (uint32_t)(32*quad) << 16;
        const size_t plane = (size_t)n_tiles*TM*HID;
        constexpr uint32_t idesc = tc::idesc_bf16(TM, HID);
        for (int k = 0; k < my_tiles && ok; ++k) {
            const int row0 = (blockIdx.x + k*gridDim.x)*TM;
            const size_t grow = (size_t)(row0 + row);
            {
                // dZ3 = dout * w_out * silu'(z3)
                const float d = row0 + row < n ? dout[row0 + row] : 0.0f;
                #pragma unroll 1
                for (int c0 = 128*half; c0 < 128*half + 128; c0 += 16) {
                    float z[16], g[16];
                    load16(z_save + 3*plane + grow*HID + c0, z);
                    #pragma unroll
                    for (int j = 0; j < 16; ++j) g[j] = d*w_out[c0 + j]*dsilu(z[j]);
                    store16(act, row, c0, g);
                    save16(dz_save + 3*plane + grow*HID + c0, g);
                }
            }
            tc::fence_async_smem();
            tc::fence_before_sync();
            ok = tc::bar_and(1, INF_CONSUMERS, ok);
            tc::fence_after_sync();
            if (!ok) break;
            for (int l = 3; l >= 1; --l) {
                if (t == 0) {
                    const uint32_t a_addr = tc::smem_u32(act);
                    for (int c = 0; c < CHUNKS_PER_LAYER; ++c, ++chunk) {
                        const int s = chunk % STAGES;
                        if (!tc::mbar_wait(&full[s], (uint32_t)((chunk/STAGES) & 1))) {
                            ok = false;
                            break;
                        }
                        tc::fence_after_sync();
                        const uint32_t b_addr = tc::smem_u32(ring + s*CHUNK_BYTES);
                        #pragma unroll
                        for (int st = 0; st < KCI/16; ++st) {
                            tc::mma_bf16(tmem, tc::kmajor_desc<TM>(a_addr, c*(KCI/16) + st),
                                         tc::kmajor_desc<HID>(b_addr, st), idesc,
                                         (c > 0 || st > 0) ? 1u : 0u);
                        }
                        tc::mma_commit(&empty[s]);
                    }
                    tc::mma_commit(&acc_bar);
                }
                const bool done = tc::mbar_wait(&acc_bar, acc_phase);
                acc_phase ^= 1u;
                tc::fence_after_sync();
                ok = tc::bar_and(1, INF_CONSUMERS, ok && done);
                if (!ok) break;
                const __nv_bfloat16 *zrow = z_save + (l - 1)*plane + grow*HID;
                __nv_bfloat16 *drow = dz_save + (l - 1)*plane + grow*HID;
                #pragma unroll 1
                for (int c0 = 128*half; c0 < 128*half + 128; c0 += 16) {
                    uint32_t r16[16];
                    tc::tmem_ld16(tmem + lane_base + (uint32_t)c0, r16);
                    tc::tmem_wait_ld();
                    float z[16], g[16];
                    load16(zrow + c0, z);
                    #pragma unroll
                    for (int j = 0; j < 16; ++j) g[j] = __uint_as_float(r16[j])*dsilu(z[j]);
                    if (l > 1) store16(act, row, c0, g);
                    save16(drow + c0, g);
                }
                tc::fence_async_smem();
                tc::fence_before_sync();
                ok = tc::bar_and(1, INF_CONSUMERS, ok);
                tc::fence_after_sync();
                if (!ok) break;
            }
        }
        if (!ok && t == 0) atomicExch(err, 1);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, HID);
}

}  // namespace mlp

using namespace mlp;

// A kernel lets its dependents in before it has allocated its tensor memory, so a
// dependent that allocates some must not come to the same SM: it would wait there for
// the kernel, which would wait for the memory.  No two of these fit one SM's shared memory.
constexpr int SM_SHARED = 227*1024;
constexpr int LEAST_TMEM_SMEM = BT_SMEM < WG_SMEM ? BT_SMEM : WG_SMEM;
static_assert(LEAST_TMEM_SMEM <= SV_SMEM && LEAST_TMEM_SMEM <= HV_SMEM
              && 2*LEAST_TMEM_SMEM > SM_SHARED, "two kernels with tensor memory on one SM");

// A launch whose CTAs may be placed while the kernels before it on the stream still
// run; the kernel waits for them by itself (tc::dependency_wait).  Hides the
// launch and the set-up of each kernel of a training step behind the one before:
// a captured step of 8192 rows in five launches 67.0 us without, 65.5 with it; the
// gradients of 3001 rows 62.5 and 56.5.
template <typename... P, typename... A>
static cudaError_t launch_dependent(void (*kernel)(P...), dim3 grid, unsigned threads, size_t bytes,
                                    cudaStream_t stream, A... args)
{
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

extern "C" {

// see Batch
struct sasb200_mlp_batch {
    const int64_t *idx;
    int64_t rows;
    const void *x_all, *x_lo_all;
    const float *y_all;
    int32_t *counters;
    float *sched;
    int32_t *refused;
    int32_t total, warmup;
    float lr0, b1, b2;
};

// the operands of sasb200_mlp_train_pass
struct sasb200_mlp_pass {
    int32_t n, n_pad, splits;
    float delta;
    const void *x, *x_lo;
    const float *y;
    const void *img, *img_t;
    const float *b[4];
    const float *w_out, *b_out;
    float *out, *dout, *row_sums;
    void *z, *h, *dz;
    float *dw[4];
    float *db, *dw_out, *loss, *db_out;
    const sasb200_mlp_batch *batch;
    int32_t *err;
    int32_t sums;
    int32_t sum_sizes[16], sum_splits[16];
    const float *sum_parts[16];
    float *sum_outs[16];
};

const char *sasb200_mlp_last_error(void) { return errbuf(); }

// Pack the bf16 weights [out][in] into the chunk image mlp_infer streams
// (IMG_BYTES = 8 KB + 24 x 16 KB).
int32_t sasb200_mlp_pack(const void *w0, const void *w1, const void *w2, const void *w3,
                         void *img, void *stream)
{
    errbuf()[0] = 0;
    if (!w0 || !w1 || !w2 || !w3 || !img)
        return (std::snprintf(errbuf(), 256, "bad arguments"), -1);
    mlp_pack<<<96, 256, 0, (cudaStream_t)stream>>>(
        static_cast<const __nv_bfloat16 *>(w0), static_cast<const __nv_bfloat16 *>(w1),
        static_cast<const __nv_bfloat16 *>(w2), static_cast<const __nv_bfloat16 *>(w3),
        static_cast<uint8_t *>(img));
    return status("mlp_pack");
}

int32_t sasb200_mlp_image_bytes(void) { return IMG_BYTES; }

// Pack W3^T, W2^T, W1^T (bf16 [in][out]) into the chunk image the pipelined
// backward streams (sasb200_mlp_image_t_bytes() = 24 x 16 KB).
int32_t sasb200_mlp_pack_t(const void *wt1, const void *wt2, const void *wt3, void *img_t,
                           void *stream)
{
    errbuf()[0] = 0;
    if (!wt1 || !wt2 || !wt3 || !img_t)
        return (std::snprintf(errbuf(), 256, "bad arguments"), -1);
    mlp_pack_layers<<<96, 256, 0, (cudaStream_t)stream>>>(
        static_cast<const __nv_bfloat16 *>(wt3), static_cast<const __nv_bfloat16 *>(wt2),
        static_cast<const __nv_bfloat16 *>(wt1), static_cast<uint8_t *>(img_t));
    return status("mlp_pack_t");
}

int32_t sasb200_mlp_image_t_bytes(void) { return WT_IMG_BYTES; }

// Backward through the hidden layers, pipelined: dZ planes [4][n_pad x 256]
// from dout[n] and the saved pre-activations; same results as
// sasb200_mlp_backward.
int32_t sasb200_mlp_backward_p(int32_t n, int32_t n_pad, const void *img_t, const float *w_out,
                               const float *dout, const void *z_save, void *dz_save,
                               int32_t *err, int32_t blocks, void *stream)
{
    errbuf()[0] = 0;
    if (n < 0 || n_pad % TM || n > n_pad || !img_t || !w_out || !dout || !z_save || !dz_save
        || !err || blocks < 0)
        return (std::snprintf(errbuf(), 256, "bad arguments"), -1);
    if (reinterpret_cast<uintptr_t>(img_t) % 16)
        return (std::snprintf(errbuf(), 256, "weight image must be 16-byte aligned"), -1);
    if (n_pad == 0) return 0;
    const int n_tiles = n_pad/TM;
    if (blocks == 0) {
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        blocks = sms > 0 ? sms : 1;
    }
    if (blocks > n_tiles) blocks = n_tiles;
    cudaFuncSetAttribute(mlp_backward_p, cudaFuncAttributeMaxDynamicSharedMemorySize, BWDP_SMEM);
    mlp_backward_p<<<blocks, INF_THREADS, BWDP_SMEM, (cudaStream_t)stream>>>(
        n, n_tiles, static_cast<const uint8_t *>(img_t), w_out, dout,
        static_cast<const __nv_bfloat16 *>(z_save), static_cast<__nv_bfloat16 *>(dz_save), err);
    return status("mlp_backward_p");
}

// Forward pass: out[n] for x, x_lo [n_pad x 16] (n_pad a multiple of 128)
// with the packed weights, and, when z_save/h_save are given, the
// pre-activations and activations of all four layers ([4][n_pad x 256] bf16
// each) for training; persistent grid of at most `blocks` CTAs (0 = one per
// SM).  err receives 1 or 2 if a pipeline wait ran out.
int32_t sasb200_mlp_infer(int32_t n, int32_t n_pad, const void *x, const void *x_lo,
                          const void *img, const float *const *b, const float *w_out,
                          const float *b_out, float *out, void *z_save, void *h_save,
                          int32_t *err, int32_t blocks, void *stream)
{
    errbuf()[0] = 0;
    if (n < 0 || n_pad % TM || n > n_pad || !x || !x_lo || !img || !b || !w_out || !b_out
        || !out || !err || blocks < 0)
        return (std::snprintf(errbuf(), 256, "bad arguments"), -1);
    if (reinterpret_cast<uintptr_t>(img) % 16)
        return (std::snprintf(errbuf(), 256, "weight image must be 16-byte aligned"), -1);
    if (n_pad == 0) return 0;
    InferParams prm = {};
    prm.img = static_cast<const uint8_t *>(img);
    for (int l = 0; l < 4; ++l) prm.b[l] = b[l];
    prm.w_out = w_out;
    prm.b_out = b_out;
    if ((z_save == nullptr) != (h_save == nullptr))
        return (std::snprintf(errbuf(), 256, "z_save and h_save go together"), -1);
    prm.z_save = static_cast<__nv_bfloat16 *>(z_save);
    prm.h_save = static_cast<__nv_bfloat16 *>(h_save);
    const int n_tiles = n_pad/TM;
    if (blocks == 0) {
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        blocks = sms > 0 ? sms : 1;
    }
    if (blocks > n_tiles) blocks = n_tiles;
    cudaFuncSetAttribute(mlp_infer, cudaFuncAttributeMaxDynamicSharedMemorySize, INF_SMEM);
    mlp_infer<<<blocks, INF_THREADS, INF_SMEM, (cudaStream_t)stream>>>(
        n, n_tiles, static_cast<const __nv_bfloat16 *>(x),
        static_cast<const __nv_bfloat16 *>(x_lo), prm, out, err);
    return status("mlp_infer");
}

// out[n] for x, x_lo [n_pad x 16] with the packed weights through the
// overlapped kernels (mlp_serve; where no planes are wanted, mlp_halves for few
// tiles and mlp_serve_pairs where a CTA has several: the same values), and, when
// z_save/h_save are given, the pre-activations and activations of all four layers
// ([4][n_pad x 256] bf16 each, those of mlp_infer) for training; grid of at most
// `blocks` CTAs (0 = one per SM).  err receives 1, 2, 3 or 4 if a pipeline wait ran
// out.
int32_t sasb200_mlp_serve(int32_t n, int32_t n_pad, const void *x, const void *x_lo,
                          const void *img, const float *const *b, const float *w_out,
                          const float *b_out, float *out, void *z_save, void *h_save,
                          int32_t *err, int32_t blocks, void *stream)
{
    errbuf()[0] = 0;
    if (n < 0 || n_pad % TM || n > n_pad || !x || !x_lo || !img || !b || !w_out || !b_out
        || !out || !err || blocks < 0)
        return (std::snprintf(errbuf(), 256, "bad arguments"), -1);
    if (reinterpret_cast<uintptr_t>(img) % 16)
        return (std::snprintf(errbuf(), 256, "weight image must be 16-byte aligned"), -1);
    for (int l = 0; l < 4; ++l)
        if (!b[l] || reinterpret_cast<uintptr_t>(b[l]) % 4)
            return (std::snprintf(errbuf(), 256, "bad bias pointer"), -1);
    if (n_pad == 0) return 0;
    InferParams prm = {};
    prm.img = static_cast<const uint8_t *>(img);
    for (int l = 0; l < 4; ++l) prm.b[l] = b[l];
    prm.w_out = w_out;
    prm.b_out = b_out;
    if ((z_save == nullptr) != (h_save == nullptr))
        return (std::snprintf(errbuf(), 256, "z_save and h_save go together"), -1);
    prm.z_save = static_cast<__nv_bfloat16 *>(z_save);
    prm.h_save = static_cast<__nv_bfloat16 *>(h_save);
    const int n_tiles = n_pad/TM;
    if (blocks == 0) {
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        blocks = sms > 0 ? sms : 1;
    }
    const auto *xp = static_cast<const __nv_bfloat16 *>(x);
    const auto *xlp = static_cast<const __nv_bfloat16 *>(x_lo);
    // two CTAs per tile where all may run at once (74 tiles: 13.4 us, 18.0 with one);
    // beyond, the second round would cost more than the halves save
    CUtensorMap map;
    if (!z_save && n_tiles <= blocks/2 && hv_map(map, img, IMG_BYTES/(8*HV_RUN))) {
        const auto kernel = mlp_halves<false>;
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, HV_SMEM);
        kernel<<<2*n_tiles, SP_THREADS, HV_SMEM, (cudaStream_t)stream>>>(n, n_tiles, xp, xlp, map, map,
                                                                         prm, out, nullptr, err);
        return status("mlp_serve");
    }
    if (blocks > n_tiles) blocks = n_tiles;
    // by pairs of CTAs, two tiles in flight, where a CTA has several tiles
    const bool in_pairs = !z_save && blocks > 1 && n_tiles > SP_TILES*blocks;
    if (in_pairs) blocks &= ~1;
    const auto kernel = z_save ? mlp_serve<PLANES_ROWS>
                               : (in_pairs ? mlp_serve_pairs : mlp_serve<PLANES_NONE>);
    const int bytes = in_pairs ? SP_SMEM : SV_SMEM, threads = in_pairs ? SP_THREADS : SV_THREADS;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    kernel<<<blocks, threads, bytes, (cudaStream_t)stream>>>(n, n_tiles, xp, xlp, prm, out, err);
    return status("mlp_serve");
}

// The forward and the backward of a gradient pass: out[n] as sasb200_mlp_serve, the
// tiled z and h planes, dout[n_pad] of the mean Huber loss (threshold delta; squared
// error for delta <= 0) against y[n], 0 on padding, row_sums[2][n_pad/32]: the loss
// and dout summed over 32 rows each; and the dZ planes.  With a batch, x, x_lo and y
// receive its rows of the data set first (a row outside it: see batch_row) and the
// schedule advances as by sasb200_lr_schedule.
static int32_t forward_backward(const sasb200_mlp_pass &p, cudaStream_t st)
{
    const int n = p.n, n_pad = p.n_pad;
    if (n < 0 || n_pad < 0 || n_pad % TM || n > n_pad || !p.x || !p.x_lo || !p.img || !p.img_t
        || !p.w_out || !p.b_out || !p.y || !p.out || !p.dout || !p.row_sums || !p.z || !p.h || !p.dz
        || !p.err)
        return (std::snprintf(errbuf(), 256, "bad arguments"), -1);
    if ((reinterpret_cast<uintptr_t>(p.img) | reinterpret_cast<uintptr_t>(p.img_t)
         | reinterpret_cast<uintptr_t>(p.w_out)) % 16)
        return (std::snprintf(errbuf(), 256, "weights must be 16-byte aligned"), -1);
    InferParams prm = {};
    prm.img = static_cast<const uint8_t *>(p.img);
    for (int l = 0; l < 4; ++l) {
        if (!p.b[l]) return (std::snprintf(errbuf(), 256, "bad bias pointer"), -1);
        prm.b[l] = p.b[l];
    }
    const auto *xp = static_cast<const __nv_bfloat16 *>(p.x);
    const auto *xlp = static_cast<const __nv_bfloat16 *>(p.x_lo);
    if (const sasb200_mlp_batch *batch = p.batch) {
        if (!batch->idx || batch->rows < 0 || !batch->x_all || !batch->x_lo_all || !batch->y_all
            || !batch->counters || !batch->sched || !batch->refused || batch->total <= 0 || batch->warmup <= 0
            || n <= 0)
            return (std::snprintf(errbuf(), 256, "bad batch"), -1);
        if ((reinterpret_cast<uintptr_t>(batch->x_all) | reinterpret_cast<uintptr_t>(batch->x_lo_all)
             | reinterpret_cast<uintptr_t>(p.x) | reinterpret_cast<uintptr_t>(p.x_lo)) % 16)
            return (std::snprintf(errbuf(), 256, "features must be 16-byte aligned"), -1);
        prm.batch = {batch->idx, batch->rows, static_cast<const __nv_bfloat16 *>(batch->x_all),
                     static_cast<const __nv_bfloat16 *>(batch->x_lo_all), batch->y_all,
                     const_cast<__nv_bfloat16 *>(xp), const_cast<__nv_bfloat16 *>(xlp),
                     const_cast<float *>(p.y), batch->counters, batch->sched, batch->refused,
                     batch->total, batch->warmup, batch->lr0, batch->b1, batch->b2};
    }
    if (n_pad == 0) return 0;
    prm.w_out = p.w_out;
    prm.b_out = p.b_out;
    prm.z_save = static_cast<__nv_bfloat16 *>(p.z);
    prm.h_save = static_cast<__nv_bfloat16 *>(p.h);
    prm.y = p.y;
    prm.delta = p.delta;
    prm.dout = p.dout;
    prm.row_sums = p.row_sums;
    auto *dz = static_cast<__nv_bfloat16 *>(p.dz);
    const int n_tiles = n_pad/TM;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // two CTAs per tile where all may run at once (see sasb200_mlp_serve)
    CUtensorMap map, map_t;
    if (n_tiles <= sms/2 && hv_map(map, p.img, IMG_BYTES/(8*HV_RUN))
        && hv_map(map_t, p.img_t, WT_IMG_BYTES/(8*HV_RUN))) {
        const auto kernel = mlp_halves<true>;
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, HV_SMEM);
        launch_dependent(kernel, dim3(2*n_tiles), SP_THREADS, HV_SMEM, st, n, n_tiles, xp, xlp, map,
                         map_t, prm, p.out, dz, p.err);
        return status("mlp_halves");
    }
    if (p.batch)
        launch_dependent(gather_batch, dim3((unsigned)((4ll*n + 255)/256)), 256, 0, st, n, prm.batch,
                         p.err);
    const dim3 blocks(n_tiles < sms || sms <= 0 ? n_tiles : sms);
    const auto forward = mlp_serve<PLANES_TILED>;
    cudaFuncSetAttribute(forward, cudaFuncAttributeMaxDynamicSharedMemorySize, SV_SMEM);
    launch_dependent(forward, blocks, SV_THREADS, SV_SMEM, st, n, n_tiles, xp, xlp, prm, p.out, p.err);
    cudaFuncSetAttribute(mlp_backward_t, cudaFuncAttributeMaxDynamicSharedMemorySize, BT_SMEM);
    launch_dependent(mlp_backward_t, blocks, SV_THREADS, BT_SMEM, st, n_tiles,
                     static_cast<const uint8_t *>(p.img_t), p.w_out, p.dout, prm.z_save, dz, p.err);
    return status("mlp_backward_t");
}

// Every gradient of a training step from its planes: dw[0..3] [splits][256 x (16
// or 256)], db [4][splits][256] and dw_out [splits][256] as partial sums over
// splits of the rows; the mean loss over n rows and db_out as scalars.  refused: null,
// or nonzero there for an undefined loss.
static int32_t weight_grads(int32_t n, int32_t n_pad, int32_t splits, const void *x,
                            const void *h, const void *dz, const float *dout,
                            const float *row_sums, float *const *dw, float *db,
                            float *dw_out, float *loss, float *db_out, const float *refused,
                            int32_t *err, void *stream)
{
    errbuf()[0] = 0;
    if (n < 0 || n > n_pad || n_pad <= 0 || n_pad % TM || splits <= 0 || splits > 4096 || !x || !h
        || !dz || !dout || !row_sums || !dw || !db || !dw_out || !loss || !db_out || !err)
        return (std::snprintf(errbuf(), 256, "bad arguments"), -1);
    if ((reinterpret_cast<uintptr_t>(h) | reinterpret_cast<uintptr_t>(dz)
         | reinterpret_cast<uintptr_t>(x)) % 16)
        return (std::snprintf(errbuf(), 256, "planes must be 16-byte aligned"), -1);
    WeightGrads prm;
    prm.x = static_cast<const __nv_bfloat16 *>(x);
    prm.h = static_cast<const __nv_bfloat16 *>(h);
    prm.dz = static_cast<const __nv_bfloat16 *>(dz);
    prm.dout = dout;
    prm.row_sums = row_sums;
    for (int l = 0; l < 4; ++l) {
        if (!dw[l] || reinterpret_cast<uintptr_t>(dw[l]) % 32)
            return (std::snprintf(errbuf(), 256, "bad gradient pointer"), -1);
        prm.dw[l] = dw[l];
    }
    prm.db = db;
    prm.dw_out = dw_out;
    prm.loss = loss;
    prm.db_out = db_out;
    prm.n = (float)n;
    prm.refused = refused;
    // the tensor core's sums lose about half an ulp of the sum per step of 16 rows,
    // always towards zero, so a chain is no longer than those of a batch split 32
    // ways, and 256 rows at most; chains are added in FP32
    const auto kernel = n_pad <= 2048 ? mlp_weight_grads<1>
                      : n_pad <= 6144 ? mlp_weight_grads<2> : mlp_weight_grads<4>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, WG_SMEM);
    launch_dependent(kernel, dim3((WG_BIG + 2)*splits), WG_THREADS, WG_SMEM, (cudaStream_t)stream,
                     n_pad/TM, splits, prm, err);
    return status("mlp_weight_grads");
}

// Adam for the whole network (host arrays of 10 device pointers, in the order
// W0..W3, b0..b3, w_out, b_out; splits partial gradients each) refreshing the
// bf16 weights w[4], their transposes wt[4] and both weight images; lr and the
// bias corrections from sched when it is not NULL (nothing is updated where sched[3] is
// set), else lr and step (>= 1).
int32_t sasb200_adam_pack(const float *const *grads, const int32_t *splits, float *const *p,
                          float *const *m, float *const *v, void *const *w, void *const *wt,
                          void *img, void *img_t, const float *sched, float lr, int32_t step,
                          float b1, float b2, float eps, void *stream)
{
    errbuf()[0] = 0;
    if (!grads || !splits || !p || !m || !v || !w || !wt || !img || !img_t || (!sched && step < 1))
        return (std::snprintf(errbuf(), 256, "bad arguments"), -1);
    AdamPack A;
    uintptr_t bits = reinterpret_cast<uintptr_t>(img) | reinterpret_cast<uintptr_t>(img_t);
    for (int k = 0; k < 10; ++k) {
        if (!grads[k] || splits[k] <= 0 || !p[k] || !m[k] || !v[k])
            return (std::snprintf(errbuf(), 256, "bad tensor"), -1);
        A.grad[k] = grads[k];
        A.splits[k] = splits[k];
        A.p[k] = p[k];
        A.m[k] = m[k];
        A.v[k] = v[k];
        if (k < 4) {
            if (!w[k] || !wt[k]) return (std::snprintf(errbuf(), 256, "bad tensor"), -1);
            A.w[k] = static_cast<__nv_bfloat16 *>(w[k]);
            A.wt[k] = static_cast<__nv_bfloat16 *>(wt[k]);
            bits |= reinterpret_cast<uintptr_t>(grads[k]) | reinterpret_cast<uintptr_t>(p[k])
                  | reinterpret_cast<uintptr_t>(m[k]) | reinterpret_cast<uintptr_t>(v[k])
                  | reinterpret_cast<uintptr_t>(w[k]) | reinterpret_cast<uintptr_t>(wt[k]);
        }
    }
    if (bits % 16) return (std::snprintf(errbuf(), 256, "tensors must be 16-byte aligned"), -1);
    A.img = static_cast<uint8_t *>(img);
    A.img_t = static_cast<uint8_t *>(img_t);
    A.sched = sched;
    A.lr = lr;
    A.bc1 = sched ? 0.0f : 1.0f - powf(b1, (float)step);
    A.bc2 = sched ? 0.0f : 1.0f - powf(b2, (float)step);
    A.b1 = b1;
    A.b2 = b2;
    A.eps = eps;
    launch_dependent(adam_pack, dim3(AP_BLOCKS), 256, 0, (cudaStream_t)stream, A);
    return status("adam_pack");
}

// outs[k][i] = sum over s < splits[k] of parts[k][s*sizes[k] + i] for n (<= 16)
// tensors (host arrays of device pointers).
static int32_t sum_partials_of(int32_t n, const int32_t *sizes, const int32_t *splits,
                               const float *const *parts, float *const *outs, void *stream)
{
    errbuf()[0] = 0;
    if (n <= 0 || n > SUM_TENSORS || !sizes || !splits || !parts || !outs)
        return (std::snprintf(errbuf(), 256, "bad arguments"), -1);
    SumTensors T = {};
    int most = 0;
    for (int k = 0; k < n; ++k) {
        if (sizes[k] <= 0 || splits[k] <= 0 || !parts[k] || !outs[k])
            return (std::snprintf(errbuf(), 256, "bad tensor"), -1);
        T.size[k] = sizes[k];
        T.splits[k] = splits[k];
        T.part[k] = parts[k];
        T.out[k] = outs[k];
        most = sizes[k] > most ? sizes[k] : most;
    }
    launch_dependent(sum_partials, dim3((most + 255)/256, n), 256, 0, (cudaStream_t)stream, T);
    return status("sum_partials");
}

// Loss and gradients of one batch: the forward and the backward, the weight
// gradients, then `sums` tensors added over the splits into their places.
// One call, as the four cost a caller as long as the kernels take.
int32_t sasb200_mlp_train_pass(const sasb200_mlp_pass *p, void *stream)
{
    errbuf()[0] = 0;
    if (!p || p->sums < 0 || p->sums > SUM_TENSORS)
        return (std::snprintf(errbuf(), 256, "bad arguments"), -1);
    int32_t rc = forward_backward(*p, (cudaStream_t)stream);
    if (rc == 0)
        rc = weight_grads(p->n, p->n_pad, p->splits, p->x, p->h, p->dz, p->dout, p->row_sums, p->dw,
                          p->db, p->dw_out, p->loss, p->db_out,
                          p->batch ? p->batch->sched + 3 : nullptr, p->err, stream);
    if (rc == 0 && p->sums > 0)
        rc = sum_partials_of(p->sums, p->sum_sizes, p->sum_splits, p->sum_parts, p->sum_outs, stream);
    return rc;
}

// out[n] (and z/h planes [4][n_pad x 256] when non-null) for x[n_pad x 16];
// n_pad a multiple of 128.
int32_t sasb200_mlp_forward(int32_t n, int32_t n_pad, const void *x, const void *x_lo,
                            const void *const *w,
                            const float *const *b, const float *w_out, const float *b_out, float *out,
                            void *z_save, void *h_save, int32_t *err, void *stream)
{
    errbuf()[0] = 0;
    if (n < 0 || n_pad % TM || n > n_pad || !x || !x_lo || !w || !b || !w_out || !b_out || !out
        || !err)
        return (std::snprintf(errbuf(), 256, "bad arguments"), -1);
    if ((z_save == nullptr) != (h_save == nullptr))
        return (std::snprintf(errbuf(), 256, "z_save and h_save go together"), -1);
    if (n_pad == 0) return 0;
    Weights wts;
    for (int l = 0; l < 4; ++l) {
        wts.w[l] = static_cast<const __nv_bfloat16 *>(w[l]);
        wts.b[l] = b[l];
    }
    wts.w_out = w_out;
    wts.b_out = b_out;
    cudaFuncSetAttribute(mlp_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, FWD_SMEM);
    mlp_forward<<<n_pad/TM, THREADS, FWD_SMEM, (cudaStream_t)stream>>>(
        n, static_cast<const __nv_bfloat16 *>(x), static_cast<const __nv_bfloat16 *>(x_lo), wts, out,
        static_cast<__nv_bfloat16 *>(z_save), static_cast<__nv_bfloat16 *>(h_save), err);
    return status("mlp_forward");
}

int32_t sasb200_mlp_backward(int32_t n, int32_t n_pad, const void *const *wt, const float *w_out,
                             const float *dout, const void *z_save, void *dz_save,
                             int32_t *err, void *stream)
{
    errbuf()[0] = 0;
    if (n < 0 || n_pad % TM || n > n_pad || !wt || !w_out || !dout || !z_save || !dz_save || !err)
        return (std::snprintf(errbuf(), 256, "bad arguments"), -1);
    if (n_pad == 0) return 0;
    WeightsT wts;
    for (int l = 0; l < 4; ++l) wts.wt[l] = static_cast<const __nv_bfloat16 *>(wt[l]);
    wts.w_out = w_out;
    cudaFuncSetAttribute(mlp_backward, cudaFuncAttributeMaxDynamicSharedMemorySize, BWD_SMEM);
    mlp_backward<<<n_pad/TM, THREADS, BWD_SMEM, (cudaStream_t)stream>>>(
        n, wts, dout, static_cast<const __nv_bfloat16 *>(z_save),
        static_cast<__nv_bfloat16 *>(dz_save), err);
    return status("mlp_backward");
}

int32_t sasb200_loss_grad(int32_t n, int32_t n_pad, const float *out, const float *y, float delta,
                          float *dout, float *loss, void *stream)
{
    if (n < 0 || n > n_pad || !out || !y || !dout || !loss) return -1;
    if (!n_pad) return 0;
    loss_grad<<<(n_pad + 255)/256, 256, 0, (cudaStream_t)stream>>>(n, n_pad, out, y, delta,
                                                                   dout, loss);
    return status("loss_grad");
}

int32_t sasb200_adam(int32_t size, int32_t splits, const float *grad, float *p, float *m, float *v,
                     float lr, float b1, float b2, float eps, int32_t step, void *w, void *wt,
                     int32_t rows, int32_t cols, void *stream)
{
    if (size <= 0 || splits <= 0 || !grad || !p || !m || !v || step < 1) return -1;
    if (wt && rows*cols != size) return -1;
    const float bc1 = 1.0f - powf(b1, (float)step), bc2 = 1.0f - powf(b2, (float)step);
    adam_step<<<(size + 255)/256, 256, 0, (cudaStream_t)stream>>>(
        size, splits, grad, p, m, v, lr, b1, b2, eps, bc1, bc2,
        static_cast<__nv_bfloat16 *>(w), static_cast<__nv_bfloat16 *>(wt), rows, cols);
    return status("adam_step");
}

int32_t sasb200_col_sums(int32_t rows, int32_t cols, const void *M, const float *v, float *part,
                         float *out, void *stream)
{
    if (rows < 0 || cols <= 0 || !M || !part || !out) return -1;
    const int nparts = rows > 0 ? (rows + CS_ROWS - 1)/CS_ROWS : 0;
    if (nparts)
        col_sum_partial<<<dim3(nparts, (cols + 255)/256), 256, 0, (cudaStream_t)stream>>>(
            rows, cols, static_cast<const __nv_bfloat16 *>(M), v, part);
    col_sum_final<<<(cols + 7)/8, 256, 0, (cudaStream_t)stream>>>(nparts, cols, part, out);
    return status("col_sums");
}

int32_t sasb200_col_sum_parts(int32_t rows)
{
    return rows > 0 ? (rows + CS_ROWS - 1)/CS_ROWS : 0;
}

int32_t sasb200_lr_schedule(int32_t *counters, float *sched, int32_t total, int32_t warmup,
                            float lr0, float b1, float b2, void *stream)
{
    if (!counters || !sched || total <= 0 || warmup <= 0) return -1;
    lr_schedule<<<1, 32, 0, (cudaStream_t)stream>>>(counters, sched, total, warmup, lr0, b1, b2);
    return status("lr_schedule");
}

int32_t sasb200_mlp_features(int32_t n, int32_t n_pad, const double *radius, const double *length,
                             const double *rpd, const double *lpd, const double *drho,
                             const double *q, const double *flag, void *x, void *x_lo,
                             void *stream)
{
    if (n < 0 || n > n_pad || !x || !x_lo) return -1;
    if (!n_pad) return 0;
    features<<<(n_pad + 127)/128, 128, 0, (cudaStream_t)stream>>>(
        n, n_pad, radius, length, rpd, lpd, drho, q, flag, static_cast<__nv_bfloat16 *>(x),
        static_cast<__nv_bfloat16 *>(x_lo));
    return status("features");
}

// Features of n points in runs of equal parameters: run r covers starts[r] <= i <
// starts[r + 1] (starts[0] = 0; the last run ends at n), table[runs x 7] = (radius,
// length, radius pd, length pd, contrast, flag, inside).
int32_t sasb200_features_runs(int32_t n, int32_t n_pad, int32_t runs, const int32_t *starts,
                              const double *table, const double *q, void *x, void *x_lo,
                              void *stream)
{
    errbuf()[0] = 0;
    if (n <= 0 || n > n_pad || runs <= 0 || runs > n || !starts || !table || !q || !x || !x_lo)
        return (std::snprintf(errbuf(), 256, "bad arguments"), -1);
    features_runs<<<(n_pad + 127)/128, 128, 0, (cudaStream_t)stream>>>(
        n, n_pad, runs, starts, table, q, static_cast<__nv_bfloat16 *>(x),
        static_cast<__nv_bfloat16 *>(x_lo));
    return status("features_runs");
}

// I[n] and accept[n] from the networks' outputs at those points; gate may be
// NULL (nothing accepted).
int32_t sasb200_finish_runs(int32_t n, int32_t runs, const int32_t *starts, const double *table,
                            const double *q, const float *out, const float *gate, double y_std,
                            double y_mean, double g_std, double g_mean, double thr, double q_lo,
                            double q_hi, double *I, uint8_t *accept, void *stream)
{
    errbuf()[0] = 0;
    if (n <= 0 || runs <= 0 || runs > n || !starts || !table || !q || !out || !I || !accept)
        return (std::snprintf(errbuf(), 256, "bad arguments"), -1);
    finish_runs<<<(n + 255)/256, 256, 0, (cudaStream_t)stream>>>(
        n, runs, starts, table, q, out, gate, y_std, y_mean, g_std, g_mean, thr, q_lo, q_hi, I,
        accept);
    return status("finish_runs");
}

}  // extern "C"
