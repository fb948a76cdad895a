// mlp_halves: serving, or the forward and the backward of a training step, of few
// tiles, each tile on two SMs.  Included by mlp.cu.
//
// With one tile per SM (mlp_serve, mlp_backward_t) a small batch takes the chain of
// one tile, a layer's MMAs, its epilogue and the hand-overs between them, four
// times, on as many SMs as there are tiles.  Here a cluster of two CTAs takes a
// tile (cta_group::2, M = 128): each holds 64 of its rows, their activations and
// accumulators, and half of the weights, so that an SM has half of the epilogue and
// of the weight bytes, and nothing but barrier counts crosses between the two.
//   Accumulators.  A CTA's 64 rows lie in TMEM lanes 0-63 with the outputs of CTA
// 0's weights and again in lanes 64-127 with those of CTA 1's, in 128 TMEM columns.
// CTA 0 has outputs 0-31 of each 64, CTA 1 the others, so that all warps work on
// the 64 inputs of the next layer that its MMAs need first.  (With outputs 0-127 and
// 128-255 the second 64 came 900 cycles after the first: 14.1 us for 8 tiles.)
// Layer l accumulates in acc[l & 1].  (The MMAs of layer l + 2 need inputs that were
// computed from layer l + 1, whose MMAs needed every warp's part of layer l: all
// its loads of acc[l & 1] are done by then.)
//   Roles of each CTA:
//   warps 0-15  epilogue: warp w, the lanes of quadrant w % 4, the 8 columns at
//               8 (w/4) of each 32 of its lanes; an arrive per warp for each 64 of
//               the layer (a chunk of the next layer's inputs).
//   warp 16     the TMEM allocation; CTA 0, lane 0: issues the MMAs, a chunk as soon
//               as its barrier says that inputs and weights are there.
//   warp 17     producer of this CTA's half of the weights, a box copy per chunk.
//   warp 18     layer 0's weights.  CTA 1: passes on to CTA 0 that its weights have
//               landed.
//   warp 19     the features.
// A cluster has one tile and every barrier one phase: all waits are for parity 0,
// bounded.  CTA 1's arrivals in CTA 0 release what they stand for, as in
// mlp_serve_pairs.  Both CTAs meet before either exits.
//
// Training goes on in the same launch: the rows of a CTA have their loss gradient
// when their output is known, so dZ3 forms from the z that the warps still hold, and
// the transposed weights follow the others through the ring.  In a captured step the
// features are gathered here and the schedule advances.  A step of 8192 rows with
// launches of their own for the backward 50.5 us and for the gathering 51.5, in one
// 47.1; 48.7 with hand-overs that release what they stand for (mbar_arrive_cta).
//
// Every value is that of the kernels of one tile per SM, bit for bit.  Bound by the
// chain of a tile still: an MMA of a pair takes 103 cycles here (32 of them a layer),
// an epilogue 700 cycles until its first hand-over, 170 from there to the MMAs.
// Serving 8 tiles 16.6 us with one SM each, 12.1 with two; 64 tiles 16.9 and 13.2.
#pragma once

constexpr int HV_RELAY_WARP = SV_EPI_WARPS + 2;
constexpr int HV_ROWS = TM/2;                      // rows of a CTA
constexpr int HV_CHUNKS = 3*SP_CHUNKS;             // of 64 inputs: layers 1-3, then W3, W2,
                                                   // W1 transposed
constexpr int HV_ACT = ACT_BYTES/2;
constexpr int HV_X = X_BYTES/2;
constexpr int HV_ACC = HID/2;                      // TMEM columns of an accumulator
constexpr int HV_STAGES = 8;                       // of the ring: two layers of weights
constexpr int HV_SMEM = 2*HV_ACT + HV_STAGES*SP_HALF + W0_BYTES/2 + 2*HV_X + 4*SV_PARAMS;
// Arrivals of a chunk in CTA 0: its inputs, by the warps of both CTAs, and its
// weights, by both producers (with the bytes) -- one barrier, because each that the
// MMA thread looks at costs it 100 cycles.  In CTA 1 its own weights.
constexpr int HV_ARRIVALS = 2*SV_EPI_WARPS + 2;
constexpr int HV_RUN = 32*16;                      // 32 outputs of 8 inputs

// A weight image as [groups of 8 inputs][4][2][32 outputs x 8 inputs]: a CTA's half of
// a chunk is 8 groups x 4 runs of 512 bytes, one copy of a box.  (As 32 copies of a
// run each, 55 cycles apart, a chunk took 1750 cycles.)  False where the driver does
// not take it.
static bool hv_map(CUtensorMap &map, const void *img, int groups)
{
    using Encode = decltype(&cuTensorMapEncodeTiled);
    static const Encode encode = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult found;
        const cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000,
                                                               cudaEnableDefault, &found);
        return e == cudaSuccess && found == cudaDriverEntryPointSuccess ? (Encode)f : nullptr;
    }();
    if (!encode) return false;
    const cuuint64_t dims[4] = {HV_RUN/2, 2, 4, (cuuint64_t)groups};
    const cuuint64_t strides[3] = {HV_RUN, 2*HV_RUN, 8*HV_RUN};
    const cuuint32_t box[4] = {HV_RUN/2, 1, 4, SP_K/8}, steps[4] = {1, 1, 1, 1};
    return encode(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void *>(img), dims, strides,
                  box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE)
           == CUDA_SUCCESS;
}

// This CTA's half of weight chunk i (64 inputs), whose first group is `group`.
__device__ __forceinline__ void hv_load_chunk(uint8_t *to, const CUtensorMap &map, int group, int rank,
                                              uint64_t *bar)
{
    tc::mbar_arrive_expect_tx(bar, SP_HALF);
    tc::box_load4(to, &map, 0, rank, 0, group, bar);
}

// Bounded wait without suspending, for the thread that the tensor core waits for.
__device__ __forceinline__ bool hv_spin(uint64_t *bar)
{
    for (uint32_t i = 0; i < tc::WAIT_LIMIT; ++i)
        if (tc::mbar_test_relaxed(bar, 0u)) {
            tc::cluster_acquire();
            return true;
        }
    return false;
}

// CTA 1: passes on to CTA 0 that its weights have landed (whole warp).
__device__ __forceinline__ bool hv_relay(int lane, int chunks, uint64_t *ready)
{
    for (int c = 0; c < chunks; ++c) {
        if (!warp_wait(&ready[c], 0u)) return false;
        if (lane == 0) tc::mbar_arrive_cta(&ready[c], 0);
    }
    return true;
}

// Both CTAs are here (whole CTA).  Relaxed: every arrival that one sends the other
// has been waited for there, and no data passes.
__device__ __forceinline__ void hv_leave_together()
{
    tc::fence_before_sync();
    __syncthreads();
    tc::cluster_arrive_relaxed();
    tc::cluster_wait();
}

// TRAIN: with the tiled planes, the loss gradient and the backward.
template <bool TRAIN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(SP_THREADS, 1)
mlp_halves(int n, int n_tiles, const __nv_bfloat16 *x, const __nv_bfloat16 *x_lo, const __grid_constant__ CUtensorMap img,
           const __grid_constant__ CUtensorMap img_t, InferParams prm, float *__restrict__ out,
           __nv_bfloat16 *__restrict__ dz_save, int *__restrict__ err)
{
    constexpr int CHUNKS = TRAIN ? 2*HV_CHUNKS : HV_CHUNKS, LAYERS = TRAIN ? 7 : 4;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t *act = smem;
    uint8_t *act_lo = smem + HV_ACT;
    uint8_t *ring = smem + 2*HV_ACT;
    uint8_t *w0 = ring + HV_STAGES*SP_HALF;
    uint8_t *xs = w0 + W0_BYTES/2;                // [hi, lo] x HV_X
    float *par = reinterpret_cast<float *>(xs + 2*HV_X);
    __shared__ __align__(8) uint64_t ready[CHUNKS], acc_full[LAYERS];
    __shared__ __align__(8) uint64_t stage_free[SP_CHUNKS];
    __shared__ __align__(8) uint64_t other_half[2][4], dot_bar[2], dout_bar[2], x_ready, drain;
    __shared__ uint32_t tmem_slot;
    __shared__ float dot_part[3][HV_ROWS], dout_s[HV_ROWS];
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int rank = (int)tc::cluster_rank(), tile = blockIdx.x >> 1;
    const int row0 = tile*TM + rank*HV_ROWS;

    if (t == 0) {
        for (int c = 0; c < CHUNKS; ++c) tc::mbar_init(&ready[c], rank == 0 ? HV_ARRIVALS : 1);
        for (int l = 0; l < LAYERS; ++l) tc::mbar_init(&acc_full[l], 1);
        for (int c = 0; c < SP_CHUNKS; ++c) tc::mbar_init(&stage_free[c], 1);
        for (int q = 0; q < 2; ++q) {
            for (int s = 0; s < 4; ++s) tc::mbar_init(&other_half[q][s], 1);
            tc::mbar_init(&dot_bar[q], SV_EPI_WARPS/4 - 1);
            tc::mbar_init(&dout_bar[q], 1);
        }
        tc::mbar_init(&x_ready, 4);
        tc::mbar_init(&drain, 1);
        tc::mbar_fence_init();
    }
    tc::dependents_launch();
    __syncthreads();
    // the accumulators and what reaches the other CTA come after cluster_wait
    if (warp == SV_MMA_WARP) {
        tc::tmem_alloc2(&tmem_slot, 2*HID);
        tc::fence_before_sync();
        tc::bar_arrive(1, SV_EPI + 32);
    }
    tc::cluster_arrive_relaxed();
    tc::dependency_wait();
    auto arrive0 = [&](uint64_t *bar) {
        if (rank == 0) tc::mbar_arrive(bar);
        else tc::mbar_arrive_cta(bar, 0);
    };

    if (warp == SV_PROD_WARP) {
        bool ok = true;
        constexpr int first = W0_BYTES/(8*HV_RUN);
        if (lane == 0) {
            for (int c = 0; c < HV_STAGES; ++c)
                hv_load_chunk(ring + c*SP_HALF, img, first + c*(SP_K/8), rank, &ready[c]);
        }
        __syncwarp();
        tc::cluster_wait();
        if (lane == 0) {
            int issued = HV_STAGES;
            // layer 3's take the places of layer 1's chunk by chunk, the later ones
            // those of the layer two before
            for (; issued < CHUNKS; ++issued) {
                const int c = issued - HV_STAGES;
                if (!(ok = tc::mbar_wait_cluster(
                          c < SP_CHUNKS ? &stage_free[c] : &acc_full[1 + c/SP_CHUNKS], 0u)))
                    break;
                const bool back = issued >= HV_CHUNKS;
                hv_load_chunk(ring + (issued % HV_STAGES)*SP_HALF, back ? img_t : img,
                              back ? (issued - HV_CHUNKS)*(SP_K/8) : first + issued*(SP_K/8), rank,
                              &ready[issued]);
            }
            // every issued copy has landed before the CTA may exit
            for (int c = 0; c < issued; ++c) ok = tc::mbar_wait(&ready[c], 0u) && ok;
            if (!ok) atomicExch(err, 2);
        }
        __syncwarp();
    } else if (warp == HV_RELAY_WARP) {
        // layer 0's weights of this CTA
        constexpr int N = W0_BYTES/2/(32*16);
        uint4 v[N];
        #pragma unroll
        for (int j = 0; j < N; ++j)
            v[j] = *reinterpret_cast<const uint4 *>(prm.img + (2*j + rank)*HV_RUN + 16*lane);
        #pragma unroll
        for (int j = 0; j < N; ++j) *reinterpret_cast<uint4 *>(w0 + j*HV_RUN + 16*lane) = v[j];
        tc::fence_async_smem();
        __syncwarp();
        tc::cluster_wait();
        if (lane == 0) arrive0(&x_ready);
        if (TRAIN && prm.batch.idx && blockIdx.x == 0 && lane == 0)
            schedule_step(prm.batch.counters, prm.batch.sched, prm.batch.total, prm.batch.warmup,
                          prm.batch.lr0, prm.batch.b1, prm.batch.b2);
        __syncwarp();
        if (rank != 0 && !hv_relay(lane, CHUNKS, ready) && lane == 0) atomicExch(err, 4);
        __syncwarp();
    } else if (warp == SP_X_WARP) {
        uint4 v[4], w[4];
        #pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int u = lane + 32*j;
            const size_t g = (size_t)(row0 + (u >> 1))*NIN + (u & 1)*8;
            if (TRAIN && prm.batch.idx) {
                const int r = row0 + (u >> 1);
                const long long src = r < n ? batch_row(prm.batch, r, err) : -1;
                v[j] = w[j] = make_uint4(0, 0, 0, 0);
                if (src >= 0) {
                    v[j] = *reinterpret_cast<const uint4 *>(prm.batch.x_all + src*NIN + (u & 1)*8);
                    w[j] = *reinterpret_cast<const uint4 *>(prm.batch.xlo_all + src*NIN + (u & 1)*8);
                }
            } else {
                v[j] = *reinterpret_cast<const uint4 *>(x + g);
                w[j] = *reinterpret_cast<const uint4 *>(x_lo + g);
            }
        }
        #pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int u = lane + 32*j;
            const uint32_t at = tc::kmajor_offset<HV_ROWS>(u >> 1, (u & 1)*8);
            *reinterpret_cast<uint4 *>(xs + at) = v[j];
            *reinterpret_cast<uint4 *>(xs + HV_X + at) = w[j];
        }
        tc::fence_async_smem();
        __syncwarp();
        tc::cluster_wait();
        if (lane == 0) arrive0(&x_ready);
        __syncwarp();
        // the batch's features, for the weight gradients
        if (TRAIN && prm.batch.idx) {
            #pragma unroll
            for (int j = 0; j < 4; ++j) {
                const size_t g = (size_t)row0*NIN + (lane + 32*j)*8;
                *reinterpret_cast<uint4 *>(prm.batch.x + g) = v[j];
                *reinterpret_cast<uint4 *>(prm.batch.x_lo + g) = w[j];
            }
        }
    } else if (warp == SV_MMA_WARP) {
        tc::cluster_wait();
        tc::fence_after_sync();
        const uint32_t tmem = tmem_slot;
        if (lane == 0 && rank == 0) {
            constexpr uint32_t idesc = tc::idesc_bf16(TM, HID);
            const uint32_t a_hi = tc::smem_u32(act), a_lo = tc::smem_u32(act_lo);
            const uint32_t xb = tc::smem_u32(xs);
            bool ok = hv_spin(&x_ready);
            if (ok) {
                tc::fence_after_sync();
                const uint64_t bdesc = tc::kmajor_desc<HID/2>(tc::smem_u32(w0), 0);
                tc::mma_bf16_pair(tmem, tc::kmajor_desc<HV_ROWS>(xb, 0), bdesc, idesc, 0u);
                tc::mma_bf16_pair(tmem, tc::kmajor_desc<HV_ROWS>(xb + HV_X, 0), bdesc, idesc, 1u);
                tc::mma_commit_pair(&acc_full[0]);
            }
            for (int i = 0; i < HV_CHUNKS && ok; ++i) {
                const int l = 1 + i/SP_CHUNKS, c = i % SP_CHUNKS;
                if (!(ok = hv_spin(&ready[i]))) break;
                tc::fence_after_sync();
                const uint32_t d = tmem + (uint32_t)(HV_ACC*(l & 1));
                const uint32_t b_addr = tc::smem_u32(ring + (i % HV_STAGES)*SP_HALF);
                #pragma unroll
                for (int st = 0; st < SP_K/16; ++st) {
                    const uint64_t bdesc = tc::kmajor_desc<HID/2>(b_addr, st);
                    const int as = c*(SP_K/16) + st;
                    tc::mma_bf16_pair(d, tc::kmajor_desc<HV_ROWS>(a_hi, as), bdesc, idesc,
                                      (c > 0 || st > 0) ? 1u : 0u);
                    tc::mma_bf16_pair(d, tc::kmajor_desc<HV_ROWS>(a_lo, as), bdesc, idesc, 1u);
                }
                if (c == SP_CHUNKS - 1) tc::mma_commit_pair(&acc_full[l]);
                if (l == 1) tc::mma_commit_pair(&stage_free[c]);
            }
            // the backward: dZ3 W3, dZ2 W2, dZ1 W1 into acc[0], acc[1], acc[0]
            for (int i = HV_CHUNKS; i < CHUNKS && ok; ++i) {
                const int s = i/SP_CHUNKS - 3, c = i % SP_CHUNKS;
                if (!(ok = hv_spin(&ready[i]))) break;
                tc::fence_after_sync();
                const uint32_t d = tmem + (uint32_t)(HV_ACC*(s & 1));
                const uint32_t b_addr = tc::smem_u32(ring + (i % HV_STAGES)*SP_HALF);
                #pragma unroll
                for (int st = 0; st < SP_K/16; ++st)
                    tc::mma_bf16_pair(d, tc::kmajor_desc<HV_ROWS>(a_hi, c*(SP_K/16) + st),
                                      tc::kmajor_desc<HID/2>(b_addr, st), idesc,
                                      (c > 0 || st > 0) ? 1u : 0u);
                if (c == SP_CHUNKS - 1) tc::mma_commit_pair(&acc_full[4 + s]);
            }
            // every MMA issued has completed before TMEM is released
            tc::mma_commit_pair(&drain);
            ok = tc::mbar_wait_cluster(&drain, 0u) && ok;
            if (!ok) atomicExch(err, 3);
        } else if (lane == 0) {
            if (!tc::mbar_wait_cluster(&drain, 0u)) atomicExch(err, 3);
        }
        __syncwarp();
    } else {
        // ---- epilogue warps ----
        for (int i = t; i < SV_PARAMS; i += SV_EPI)
            par[i] = i < 4*HID ? prm.b[i/HID][i % HID] : prm.w_out[i - 4*HID];
        tc::bar_sync(1, SV_EPI + 32);                  // the parameters, and tmem_slot
        tc::fence_after_sync();
        tc::cluster_wait();
        const float b_out = *prm.b_out;
        const int quad = warp & 3, slot = warp >> 2;
        const int q2 = quad & 1, half = quad >> 1;     // 32 rows, 32 columns of each 64
        const int row = 32*q2 + lane, trow = rank*HV_ROWS + row;
        const int col0 = 32*half + 8*slot;
        const uint32_t lane_base = tmem_slot + ((uint32_t)(32*quad) << 16) + (uint32_t)(8*slot);
        // the target of this row, for the warps that form the output
        float target = 0.0f;
        if (TRAIN && half == 0 && slot == 0) {
            if (prm.batch.idx) {
                const long long src = row0 + row < n ? batch_row(prm.batch, row0 + row, err) : -1;
                if (src >= 0) target = prm.batch.y_all[src];
                if (row0 + row < n) prm.batch.y[row0 + row] = target;
            } else if (row0 + row < n) {
                target = prm.y[row0 + row];
            }
        }
        // z and h of this thread's columns, stored when all are handed over (each with
        // its chunk: 0.4 us more)
        auto save_planes = [&](int l, const uint4 (&z)[SP_CHUNKS], const uint4 (&h)[SP_CHUNKS]) {
            #pragma unroll
            for (int c = 0; c < SP_CHUNKS; ++c) {
                const size_t at = tiled_at(l, n_tiles, tile, (col0 + 64*c)/8, trow);
                *reinterpret_cast<uint4 *>(prm.z_save + at) = z[c];
                *reinterpret_cast<uint4 *>(prm.h_save + at) = h[c];
            }
        };
        bool ok = true;
        uint4 zq[SP_CHUNKS];                           // layer 3's z, later the next needed
        #pragma unroll 1
        for (int l = 0; l < 3; ++l) {
            if (!(ok = warp_wait_cluster(&acc_full[l], 0u))) break;
            tc::fence_after_sync();
            const float *bias = par + l*HID + col0;
            uint32_t r[SP_CHUNKS][8];
            #pragma unroll
            for (int c = 0; c < SP_CHUNKS; ++c)
                tc::tmem_ld8(lane_base + (uint32_t)(HV_ACC*(l & 1) + 32*c), r[c]);
            #pragma unroll
            for (int c = 0; c < SP_CHUNKS; ++c) tc::tmem_wait_ld8(r[c]);
            tc::fence_before_sync();
            uint4 hi[SP_CHUNKS], z[SP_CHUNKS];
            #pragma unroll
            for (int c = 0; c < SP_CHUNKS; ++c) {
                uint4 lo;
                silu_columns<TRAIN>(r[c], 0, bias + 64*c, hi[c], lo, &z[c]);
                const uint32_t off = tc::kmajor_offset<HV_ROWS>(row, col0 + 64*c);
                *reinterpret_cast<uint4 *>(act + off) = hi[c];
                *reinterpret_cast<uint4 *>(act_lo + off) = lo;
                tc::fence_async_smem();
                __syncwarp();
                if (lane == 0) arrive0(&ready[SP_CHUNKS*l + c]);
            }
            if (TRAIN) save_planes(l, z, hi);
        }
        if (ok && (ok = warp_wait_cluster(&acc_full[3], 0u))) {
            // the output dot: the 8 columns at 8 (w/4) of every 32, summed in order as
            // in mlp_serve by the warps that hold the first of each pair of 32; the
            // others leave their activations in the place of the inputs' lo halves, all
            // read (the hi halves' place is for dZ)
            tc::fence_after_sync();
            const float *bias = par + 3*HID + col0, *wo = par + 4*HID + 8*slot;
            uint32_t r[SP_CHUNKS][8];
            uint4 hq[SP_CHUNKS];
            float h[SP_CHUNKS][8];
            #pragma unroll
            for (int c = 0; c < SP_CHUNKS; ++c) tc::tmem_ld8(lane_base + (uint32_t)(HV_ACC + 32*c), r[c]);
            #pragma unroll
            for (int c = 0; c < SP_CHUNKS; ++c) tc::tmem_wait_ld8(r[c]);
            tc::fence_before_sync();
            // [slot][chunk][4 columns][row] of 16 bytes
            float4 *over = reinterpret_cast<float4 *>(act_lo) + slot*(2*SP_CHUNKS*HV_ROWS) + row;
            #pragma unroll
            for (int c = 0; c < SP_CHUNKS; ++c) {
                const ulonglong2 *b2 = reinterpret_cast<const ulonglong2 *>(bias + 64*c);
                #pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const ulonglong2 b = b2[e >> 1];
                    const uint64_t z = bias2(r[c][2*e], r[c][2*e + 1], e & 1 ? b.y : b.x);
                    const uint64_t v = silu2(z);
                    f2_unpack(v, h[c][2*e], h[c][2*e + 1]);
                    if (TRAIN) {
                        (&zq[c].x)[e] = pack2(z);
                        (&hq[c].x)[e] = pack2(v);
                    }
                }
                if (half == 1) {
                    over[2*c*HV_ROWS] = make_float4(h[c][0], h[c][1], h[c][2], h[c][3]);
                    over[(2*c + 1)*HV_ROWS] = make_float4(h[c][4], h[c][5], h[c][6], h[c][7]);
                }
            }
            if (half == 1) {
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&other_half[q2][slot]);
            }
            if (TRAIN) save_planes(3, zq, hq);
            float dot = 0.0f;
            if (half == 0 && (ok = warp_wait(&other_half[q2][slot], 0u))) {
                #pragma unroll
                for (int c = 0; c < SP_CHUNKS; ++c) {
                    const float4 o0 = over[2*c*HV_ROWS], o1 = over[(2*c + 1)*HV_ROWS];
                    const float oh[8] = {o0.x, o0.y, o0.z, o0.w, o1.x, o1.y, o1.z, o1.w};
                    #pragma unroll
                    for (int e = 0; e < 8; ++e) dot = fmaf(h[c][e], wo[64*c + e], dot);
                    #pragma unroll
                    for (int e = 0; e < 8; ++e) dot = fmaf(oh[e], wo[64*c + 32 + e], dot);
                }
            }
            if (half == 1) {
                // done
            } else if (slot > 0) {
                dot_part[slot - 1][row] = dot;
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&dot_bar[q2]);
            } else if (ok && (ok = warp_wait(&dot_bar[q2], 0u))) {
                const bool valid = row0 + row < n;
                const float o = ((dot + dot_part[0][row]) + dot_part[1][row])
                                + dot_part[2][row] + b_out;
                if (valid) out[row0 + row] = o;
                if (TRAIN) {
                    float g, loss;
                    loss_of(valid ? o - target : 0.0f, prm.delta, g, loss);
                    g = valid ? g/(float)n : 0.0f;
                    prm.dout[row0 + row] = g;
                    dout_s[row] = g;
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive(&dout_bar[q2]);
                    #pragma unroll
                    for (int o2 = 16; o2 > 0; o2 >>= 1) {
                        g += __shfl_xor_sync(0xffffffffu, g, o2);
                        loss += __shfl_xor_sync(0xffffffffu, loss, o2);
                    }
                    if (lane == 0) {
                        float *sums = prm.row_sums + 4*tile + 2*rank + q2;
                        sums[0] = loss;
                        sums[4*n_tiles] = g;
                    }
                }
            }
        }
        // ---- backward: dZ3 from dout, then the epilogues of W3, W2, W1 ----
        if (TRAIN && ok && (ok = warp_wait(&dout_bar[q2], 0u))) {
            const size_t plane16 = (size_t)n_tiles*TILE_ELEMS/8;       // in 16-byte units
            constexpr int GROUP16 = GROUP_ELEMS/8;
            const size_t at0 = tiled_at(0, n_tiles, tile, col0/8, trow);
            const uint4 *z0 = reinterpret_cast<const uint4 *>(prm.z_save + at0);
            uint4 *dz0 = reinterpret_cast<uint4 *>(dz_save + at0);
            const float d = dout_s[row];
            #pragma unroll 1
            for (int s = -1; s < 3; ++s) {
                const int l = 2 - s;
                uint32_t r[SP_CHUNKS][8];
                if (s >= 0) {
                    if (!(ok = warp_wait_cluster(&acc_full[4 + s], 0u))) break;
                    tc::fence_after_sync();
                    #pragma unroll
                    for (int c = 0; c < SP_CHUNKS; ++c)
                        tc::tmem_ld8(lane_base + (uint32_t)(HV_ACC*(s & 1) + 32*c), r[c]);
                    #pragma unroll
                    for (int c = 0; c < SP_CHUNKS; ++c) tc::tmem_wait_ld8(r[c]);
                    tc::fence_before_sync();
                } else {
                    #pragma unroll
                    for (int c = 0; c < SP_CHUNKS; ++c)
                        #pragma unroll
                        for (int e = 0; e < 8; ++e)
                            r[c][e] = __float_as_uint(d*par[4*HID + col0 + 64*c + e]);
                }
                uint4 o[SP_CHUNKS];
                #pragma unroll
                for (int c = 0; c < SP_CHUNKS; ++c) {
                    const uint32_t zu[4] = {zq[c].x, zq[c].y, zq[c].z, zq[c].w};
                    uint32_t *op = &o[c].x;
                    #pragma unroll
                    for (int e = 0; e < 4; ++e)
                        op[e] = pack2(__uint_as_float(r[c][2*e])*dsilu(bf_lo(zu[e])),
                                      __uint_as_float(r[c][2*e + 1])*dsilu(bf_hi(zu[e])));
                    if (s < 2) {
                        *reinterpret_cast<uint4 *>(
                            act + tc::kmajor_offset<HV_ROWS>(row, col0 + 64*c)) = o[c];
                        tc::fence_async_smem();
                        __syncwarp();
                        if (lane == 0) arrive0(&ready[HV_CHUNKS + SP_CHUNKS*(s + 1) + c]);
                    }
                }
                // the next layer's z (this thread stored it), in use one epilogue from now
                if (s < 2) {
                    #pragma unroll
                    for (int c = 0; c < SP_CHUNKS; ++c)
                        zq[c] = z0[(size_t)(l - 1)*plane16 + 8*c*GROUP16];
                }
                #pragma unroll
                for (int c = 0; c < SP_CHUNKS; ++c) dz0[(size_t)l*plane16 + 8*c*GROUP16] = o[c];
            }
        }
        if (!ok && lane == 0) atomicExch(err, 1);
        __syncwarp();
    }
    hv_leave_together();
    if (warp == SV_MMA_WARP) tc::tmem_dealloc2(tmem_slot, 2*HID);
}
