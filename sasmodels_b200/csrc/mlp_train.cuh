// The training step's kernels after the forward: the backward pass, the weight
// gradients and their reduction.  Included by mlp.cu.
#pragma once

// Sum over the 32 lanes of each of a lane's 8 values in 9 shuffles: halves of
// the set are exchanged while the set shrinks to one value per lane.  Lane L
// returns the sum of value L/4 (every fourth lane's is the one to use).
__device__ __forceinline__ float warp_sum8(float (&v)[8], int lane)
{
    #pragma unroll
    for (int half = 4; half >= 1; half >>= 1) {
        const bool up = (lane & (4*half)) != 0;
        #pragma unroll
        for (int j = 0; j < half; ++j) {
            const float mine = up ? v[j + half] : v[j], other = up ? v[j] : v[j + half];
            v[j] = mine + __shfl_xor_sync(0xffffffffu, other, 4*half);
        }
    }
    float s = v[0];
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    return s;
}

// ---------------------------------------------------------------- backward --
// mlp_backward_t: dZ3 = dout w_out silu'(z3), then dZ(l-1) = (dZl W_l)
// silu'(z(l-1)) for l = 3, 2, 1, from tiled z to tiled dZ planes; the values of
// mlp_backward.  Built as mlp_serve: sixteen epilogue warps (quadrant w % 4, 16
// columns of every 64 at 16(w / 4)), one MMA warp, a bulk-copy producer and the two
// counting warps, two TMEM accumulators, so that the MMAs of the next layer start on the
// first columns while the epilogue works on the last.  For batches of more tiles
// than half the SMs (fewer: mlp_halves).  Bound by the latency of one tile's
// chain: the ring holds a whole layer of weights (fetched while dZ3 forms), and each
// warp loads the z of its eight chunks one layer ahead.  100 tiles: 20.4 us with cold
// caches.
constexpr int BT_STAGES = 8;
constexpr int BT_SMEM = ACT_BYTES + BT_STAGES*CHUNK_BYTES;

__global__ void __launch_bounds__(SV_THREADS, 1)
mlp_backward_t(int n_tiles, const uint8_t *img_t, const float *w_out, const float *dout,
               const __nv_bfloat16 *z_save, __nv_bfloat16 *__restrict__ dz_save, int *__restrict__ err)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t *act = smem;
    uint8_t *ring = smem + ACT_BYTES;
    __shared__ __align__(8) uint64_t full[BT_STAGES], empty[BT_STAGES];
    __shared__ __align__(8) uint64_t act_ready[SV_UNITS], acc_full[2], acc_empty[2], drain;
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(8) uint2 ready_seq;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int my_tiles = blockIdx.x < n_tiles ? (n_tiles - 1 - blockIdx.x)/gridDim.x + 1 : 0;

    if (warp == 0) {
        tc::tmem_alloc(&tmem_slot, 2*HID);
        tc::tmem_relinquish();
    }
    if (t == 0) {
        for (int s = 0; s < BT_STAGES; ++s) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], 1);
        }
        for (int c = 0; c < SV_UNITS; ++c) tc::mbar_init(&act_ready[c], SV_EPI_WARPS);
        for (int a = 0; a < 2; ++a) {
            tc::mbar_init(&acc_full[a], 1);
            tc::mbar_init(&acc_empty[a], SV_EPI_WARPS);
        }
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
        if (lane == 0) {
            bool ok = true;
            const int total = my_tiles*CHUNKS_PER_TILE;
            int i = 0;
            for (; i < total; ++i) {
                const int s = i % BT_STAGES, use = i/BT_STAGES;
                if (use > 0 && !tc::mbar_wait(&empty[s], (uint32_t)((use - 1) & 1))) {
                    ok = false;
                    break;
                }
                tc::mbar_arrive_expect_tx(&full[s], CHUNK_BYTES);
                tc::bulk_load(ring + s*CHUNK_BYTES,
                              img_t + (size_t)(i % CHUNKS_PER_TILE)*CHUNK_BYTES,
                              CHUNK_BYTES, &full[s]);
            }
            for (int j = (i > BT_STAGES ? i - BT_STAGES : 0); j < i; ++j)
                ok = tc::mbar_wait(&full[j % BT_STAGES], (uint32_t)((j/BT_STAGES) & 1)) && ok;
            if (!ok) atomicExch(err, 2);
        }
    } else if (warp == SV_ACT_WARP) {
        // step g = 3 k + s accumulates in acc[g & 1]; its previous reader is the
        // epilogue of step g - 2 (completion (g - 2)/2 of acc_empty), and its input
        // is completion g of act_ready.  No barrier can run two phases ahead: each
        // next completion needs what is published here first.
        if (lane == 0) {
            bool ok = true;
            uint32_t chunk = 0;
            for (int g = 0; g < 3*my_tiles && ok; ++g) {
                if (g >= 2 && !(ok = tc::mbar_wait(&acc_empty[g & 1], (uint32_t)(((g - 2) >> 1) & 1))))
                    break;
                for (int q = 0; q < SV_UNITS; ++q) {
                    if (!(ok = tc::mbar_wait(&act_ready[q], (uint32_t)(g & 1)))) break;
                    chunk += CHUNKS_PER_LAYER/SV_UNITS;
                    tc::st_release_shared(&ready_seq.x, chunk);
                }
            }
            if (!ok) atomicExch(err, 4);
        }
        __syncwarp();
    } else if (warp == SV_WEIGHT_WARP) {
        if (lane == 0) {
            bool ok = true;
            const uint32_t total = (uint32_t)(my_tiles*CHUNKS_PER_TILE);
            for (uint32_t i = 0; i < total && ok; ++i)
                if ((ok = tc::mbar_wait(&full[i % BT_STAGES], (i/BT_STAGES) & 1u)))
                    tc::st_release_shared(&ready_seq.y, i + 1);
            if (!ok) atomicExch(err, 4);
        }
        __syncwarp();
    } else if (warp == SV_MMA_WARP) {
        bool ok = true;
        if (lane == 0) {
            constexpr uint32_t idesc = tc::idesc_bf16(TM, HID);
            const uint32_t a_addr = tc::smem_u32(act);
            int chunk = 0;
            ReadyCounts count(&ready_seq);
            for (int g = 0; g < 3*my_tiles && ok; ++g) {
                const uint32_t d = tmem + (uint32_t)(HID*(g & 1));
                for (int c = 0; c < CHUNKS_PER_LAYER; ++c, ++chunk) {
                    if (!(ok = count.covers((uint32_t)(chunk + 1)))) break;
                    tc::fence_after_sync();
                    const int s = chunk % BT_STAGES;
                    const uint32_t b_addr = tc::smem_u32(ring + s*CHUNK_BYTES);
                    #pragma unroll
                    for (int st = 0; st < KCI/16; ++st)
                        tc::mma_bf16(d, tc::kmajor_desc<TM>(a_addr, c*(KCI/16) + st),
                                     tc::kmajor_desc<HID>(b_addr, st), idesc,
                                     (c > 0 || st > 0) ? 1u : 0u);
                    tc::mma_commit(&empty[s]);
                }
                if (ok) tc::mma_commit(&acc_full[g & 1]);
            }
            // every MMA issued has completed before TMEM is released
            tc::mma_commit(&drain);
            ok = tc::mbar_wait(&drain, 0u) && ok;
            if (!ok) atomicExch(err, 3);
        }
        __syncwarp();
    } else {
        const int quad = warp & 3, slot = warp >> 2;
        const int row = 32*quad + lane;
        const uint32_t lane_base = (uint32_t)(32*quad) << 16;
        bool ok = true;
        for (int k = 0; k < my_tiles && ok; ++k) {
            const int tile = blockIdx.x + k*gridDim.x;
            const float d = dout[tile*TM + row];
            // this thread's 16 columns of every 64: two groups of 8
            const size_t at0 = tiled_at(0, n_tiles, tile, 2*slot, row);
            const uint4 *z0 = reinterpret_cast<const uint4 *>(z_save + at0);
            uint4 *dz0 = reinterpret_cast<uint4 *>(dz_save + at0);
            const size_t plane16 = (size_t)n_tiles*TILE_ELEMS/8;   // a plane in 16-byte units
            constexpr int GROUP16 = GROUP_ELEMS/8;
            uint4 z[SV_UNITS][2];
            #pragma unroll
            for (int q = 0; q < SV_UNITS; ++q) {
                z[q][0] = z0[3*plane16 + 8*q*GROUP16];
                z[q][1] = z0[3*plane16 + (8*q + 1)*GROUP16];
            }
            // s = -1: dZ3 from dout; s = 0, 1, 2: the epilogues of W3, W2, W1
            #pragma unroll 1
            for (int s = -1; s < 3; ++s) {
                const int g = 3*k + s, l = 2 - s, a = g & 1;
                const uint32_t acc = tmem + lane_base + (uint32_t)(HID*a + 16*slot);
                uint32_t ra[16], rb[16];
                if (s >= 0) {
                    if (!(ok = warp_wait(&acc_full[a], (uint32_t)((g >> 1) & 1)))) break;
                    tc::fence_after_sync();
                    tc::tmem_ld16(acc, ra);
                    tc::tmem_wait_ld();
                    tc::tmem_tie16(ra);
                }
                #pragma unroll
                for (int q = 0; q < SV_UNITS; ++q) {
                    const bool more = q + 1 < SV_UNITS;
                    if (s >= 0) {
                        if (more) {
                            tc::tmem_ld16(acc + (uint32_t)(64*(q + 1)), rb);
                        } else {
                            tc::fence_before_sync();
                            __syncwarp();
                            if (lane == 0) tc::mbar_arrive(&acc_empty[a]);
                        }
                    } else {
                        const float4 *wp = reinterpret_cast<const float4 *>(w_out + 64*q + 16*slot);
                        #pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float4 w = wp[e];
                            ra[4*e] = __float_as_uint(d*w.x);
                            ra[4*e + 1] = __float_as_uint(d*w.y);
                            ra[4*e + 2] = __float_as_uint(d*w.z);
                            ra[4*e + 3] = __float_as_uint(d*w.w);
                        }
                    }
                    uint4 o[2];
                    #pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint32_t zu[4] = {z[q][h].x, z[q][h].y, z[q][h].z, z[q][h].w};
                        uint32_t *op = &o[h].x;
                        #pragma unroll
                        for (int e = 0; e < 4; ++e)
                            op[e] = pack2(__uint_as_float(ra[8*h + 2*e])*dsilu(bf_lo(zu[e])),
                                          __uint_as_float(ra[8*h + 2*e + 1])*dsilu(bf_hi(zu[e])));
                        // the stores of the 64 columns before have had time to land
                        if (h == 0 && q > 1 && s < 2) {
                            tc::fence_async_smem();
                            __syncwarp();
                            if (lane == 0) tc::mbar_arrive(&act_ready[q - 1]);
                        }
                    }
                    #pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        if (s < 2) {
                            *reinterpret_cast<uint4 *>(
                                act + tc::kmajor_offset<TM>(row, 64*q + 16*slot + 8*h)) = o[h];
                            // the next layer's z, in use one epilogue from now
                            z[q][h] = z0[(size_t)(l - 1)*plane16 + (8*q + h)*GROUP16];
                        }
                        dz0[(size_t)l*plane16 + (8*q + h)*GROUP16] = o[h];
                    }
                    // the tensor core is waiting for the first and the last
                    if (s < 2 && (q == 0 || !more)) {
                        tc::fence_async_smem();
                        __syncwarp();
                        if (lane == 0) tc::mbar_arrive(&act_ready[q]);
                    }
                    if (s >= 0 && more) {
                        tc::tmem_wait_ld();
                        tc::tmem_tie16(rb);
                        #pragma unroll
                        for (int e = 0; e < 16; ++e) ra[e] = rb[e];
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

// -------------------------------------------------------- weight gradients --
// mlp_weight_grads: every gradient of a step from the tiled planes in one
// launch.  With S splits of the tiles, block b is
//   b < 12 S        layer 1 + (b % 12)/4, M half (b/2) % 2 (columns of dZ), N half
//                   b % 2 (columns of h), split b/12: dW_l += dZ_l^T h_{l-1} over
//                   the split's tiles (M 128, N 128, K 128 per tile); the blocks
//                   of N half 0 also sum their columns of dZ_l (bias gradients);
//   next S blocks   layer 0: all of dZ_0 against the 16 features, and its sums;
//   next S blocks   the output weights, columns of h_3 weighted by dout; block 0
//                   of them also adds the loss and dout sums of the forward.
// The rows are the K dimension of both operands, so the 32 KB halves of the tile
// images are MN-major operands as they lie in memory: each half is one bulk
// copy into a three-stage ring.  An accumulation chain in TMEM is 64 to 256 rows (the
// tensor core's sums round towards zero: with a split's 819 rows in one chain the
// gradients of 8192 rows were off by 8e-7 and are by 2.3e-7, at 131,072 rows 1.4e-5
// and 2.4e-7); eight warps add the chains, which alternate between two buffers, in
// FP32 registers, and the columns from the same stages meanwhile.  Bound by the copies
// (64 KB per 512-cycle tile of MMAs) and, in layer 0, the hand-over of the features.
// 14 S <= 148 blocks are one wave: S = 10.  Partial sums leave per split, added by
// whoever reads them (Adam, sum_partials).  With cold caches 15.7 us for 8192 rows (15.4
// with a split in one chain), 11.7 for 3001.
constexpr int WG_STAGES = 3;
constexpr int WG_HALF = ACT_BYTES/2;                   // 32 KB: 128 columns of a tile
constexpr int WG_STAGE_BYTES = 2*WG_HALF;
constexpr int WG_SUM_WARPS = 8;
constexpr int WG_THREADS = 32*(WG_SUM_WARPS + 2);      // + producer, MMA
constexpr int WG_SMEM = WG_STAGES*(WG_STAGE_BYTES + X_BYTES);
constexpr int WG_BIG = 12;
// Threads by which the registers are bounded (to 96), so that two blocks of adam_pack
// (48 registers, 256 threads) fit beside a block and all are set up when the last
// gradients leave: a quarter of the SM holds 3 warps of one and 4 of the others.  A captured
// step of 8192 rows 48.7 us, with 128 registers 50.7, with up to 168 49.8.
constexpr int WG_BOUND = 576;
constexpr int WG_PART = TM/2;                          // rows by which chains grow
constexpr int WG_ACC = 128;                            // TMEM columns of an accumulator

struct WeightGrads {
    const __nv_bfloat16 *x;          // [n_pad x 16] features (high halves)
    const __nv_bfloat16 *h, *dz;     // tiled planes
    const float *dout;               // [n_pad]
    const float *row_sums;           // [2][4 n_tiles]: loss and dout sums of 32 rows each
    float *dw[4];                    // [S][256 x (16 or 256)]
    float *db;                       // [4][S][256]
    float *dw_out;                   // [S][256]
    float *loss, *db_out;            // scalars
    float n;                         // rows of the mean loss
    const float *refused;            // null, or nonzero there: the loss is undefined
};

// CHAIN: parts of an accumulation chain (1, 2 or 4)
template <int CHAIN>
__global__ void __launch_bounds__(WG_BOUND, 1)
mlp_weight_grads(int n_tiles, int splits, WeightGrads prm, int *__restrict__ err)
{
    constexpr int PARTS = TM/WG_PART;                  // of a tile
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t *xs = smem + WG_STAGES*WG_STAGE_BYTES;
    __shared__ __align__(8) uint64_t full[WG_STAGES], empty[WG_STAGES], x_full[WG_STAGES], done;
    __shared__ __align__(8) uint64_t acc_full[2], acc_free[2];
    __shared__ uint32_t tmem_slot;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int b = blockIdx.x;
    const bool big = b < WG_BIG*splits, first = !big && b < (WG_BIG + 1)*splits;
    const int split = big ? b/WG_BIG : (first ? b - WG_BIG*splits : b - (WG_BIG + 1)*splits);
    const int layer = big ? 1 + (b % WG_BIG)/4 : (first ? 0 : 4);
    const int mh = big ? (b >> 1) & 1 : 0, nh = big ? b & 1 : 0;
    const bool mma = layer < 4, sums = !big || nh == 0;
    const int t0 = (int)((long long)n_tiles*split/splits);
    const int tiles = (int)((long long)n_tiles*(split + 1)/splits) - t0;

    if (warp == 0) {
        tc::tmem_alloc(&tmem_slot, 2*WG_ACC);
        tc::tmem_relinquish();
    }
    if (t == 0) {
        for (int s = 0; s < WG_STAGES; ++s) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], (mma ? 1 : 0) + (sums ? WG_SUM_WARPS : 0));
            tc::mbar_init(&x_full[s], WG_SUM_WARPS);
        }
        for (int a = 0; a < 2; ++a) {
            tc::mbar_init(&acc_full[a], 1);
            tc::mbar_init(&acc_free[a], WG_SUM_WARPS);
        }
        tc::mbar_init(&done, 1);
        tc::mbar_fence_init();
    }
    tc::dependents_launch();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    tc::dependency_wait();
    const uint32_t tmem = tmem_slot;
    bool ok = true;

    if (warp == WG_SUM_WARPS) {
        // ---- producer ----
        if (lane == 0) {
            int i = 0;
            for (; i < tiles; ++i) {
                const int s = i % WG_STAGES, use = i/WG_STAGES;
                if (use > 0 && !(ok = tc::mbar_wait(&empty[s], (uint32_t)((use - 1) & 1)))) break;
                uint8_t *to = smem + s*WG_STAGE_BYTES;
                tc::mbar_arrive_expect_tx(&full[s], 2*WG_HALF);
                const size_t own = (size_t)(t0 + i)*TILE_ELEMS, plane = (size_t)n_tiles*TILE_ELEMS;
                if (big) {
                    tc::bulk_load(to, prm.dz + layer*plane + own + mh*(TILE_ELEMS/2), WG_HALF,
                                  &full[s]);
                    tc::bulk_load(to + WG_HALF, prm.h + (layer - 1)*plane + own + nh*(TILE_ELEMS/2),
                                  WG_HALF, &full[s]);
                } else {
                    tc::bulk_load(to, (first ? prm.dz : prm.h + 3*plane) + own, 2*WG_HALF, &full[s]);
                }
            }
            // every issued copy has landed before the CTA may exit
            for (int j = (i > WG_STAGES ? i - WG_STAGES : 0); j < i; ++j)
                ok = tc::mbar_wait(&full[j % WG_STAGES], (uint32_t)((j/WG_STAGES) & 1)) && ok;
            if (!ok) atomicExch(err, 2);
        }
    } else if (warp == WG_SUM_WARPS + 1) {
        // ---- MMA issue ----
        // Nothing but the first MMA of a tile asks whether it starts a chain: what
        // this thread works out between two MMAs is time without them.
        auto issue = [&](auto is_big) {
            constexpr bool BIG = decltype(is_big)::value;
            constexpr uint32_t idesc = tc::idesc_bf16_mn(TM, BIG ? 128 : NIN);
            for (int i = 0; i < tiles; ++i) {
                const int s = i % WG_STAGES;
                const uint32_t parity = (uint32_t)((i/WG_STAGES) & 1);
                if (!(ok = tc::mbar_wait(&full[s], parity)
                           && (BIG || tc::mbar_wait(&x_full[s], parity))))
                    break;
                tc::fence_after_sync();
                const uint32_t a = tc::smem_u32(smem + s*WG_STAGE_BYTES);
                const uint32_t bm = BIG ? a + WG_HALF : tc::smem_u32(xs + s*X_BYTES);
                #pragma unroll
                for (int k = 0; k < PARTS; ++k) {
                    // the chain, and whether it starts here: its buffer was read
                    // two chains ago (completion u/2 - 1)
                    const int u = CHAIN <= PARTS ? PARTS/CHAIN*i + k/CHAIN : i/(CHAIN/PARTS);
                    const bool starts = k % CHAIN == 0 && (CHAIN <= PARTS || i % (CHAIN/PARTS) == 0);
                    const uint32_t d = tmem + (uint32_t)(WG_ACC*(u & 1));
                    if (starts && u >= 2) {
                        if (!(ok = tc::mbar_wait(&acc_free[u & 1], (uint32_t)((u/2 - 1) & 1)))) break;
                        tc::fence_after_sync();
                    }
                    #pragma unroll
                    for (int st = 0; st < WG_PART/16; ++st) {
                        const int ks = k*(WG_PART/16) + st;
                        const uint64_t bd = tc::mnmajor_desc<TM>(bm, ks);
                        const uint32_t acc = (st > 0 || !starts) ? 1u : 0u;
                        tc::mma_bf16(d, tc::mnmajor_desc<TM>(a, ks), bd, idesc, acc);
                        if (!BIG) tc::mma_bf16(d + WG_ACC/2, tc::mnmajor_desc<TM>(a + WG_HALF, ks), bd,
                                               idesc, acc);
                    }
                    if (CHAIN <= PARTS ? (k + 1) % CHAIN == 0
                                       : k + 1 == PARTS && ((i + 1) % (CHAIN/PARTS) == 0 || i + 1 == tiles))
                        tc::mma_commit(&acc_full[u & 1]);
                }
                if (!ok) break;
                tc::mma_commit(&empty[s]);
            }
        };
        if (lane == 0) {
            if (big) issue(std::true_type());
            else if (mma) issue(std::false_type());
            tc::mma_commit(&done);
            ok = tc::mbar_wait(&done, 0u) && ok;
            if (!ok) atomicExch(err, 3);
        }
        __syncwarp();
    } else {
        // ---- column sums (lane = row (mod 32), a warp 2 or 4 groups of 8 columns)
        // and the sums of the chains: warps 0-3 the first 64 columns of the
        // accumulators, 4-7 the rest, lane = row.  By the kind of block, so that
        // neither keeps the other's registers: what they leave lets the next
        // kernel's blocks in early ----
        auto add_up = [&](auto is_big) {
            constexpr bool BIG = decltype(is_big)::value;
            constexpr int GROUPS = BIG ? 2 : 4, COLUMNS = BIG ? WG_ACC/2 : NIN;
            float acc[GROUPS][8];
            #pragma unroll
            for (int q = 0; q < GROUPS; ++q) {
                #pragma unroll
                for (int e = 0; e < 8; ++e) acc[q][e] = 0.0f;
            }
            const int quad = warp & 3, part = warp >> 2;
            const uint32_t at = tmem + ((uint32_t)(32*quad) << 16) + (uint32_t)(WG_ACC/2*part);
            float g[COLUMNS];
            #pragma unroll
            for (int j = 0; j < COLUMNS; ++j) g[j] = 0.0f;
            // the features of a tile: one 16-byte unit per thread, a tile ahead
            const int xr = t >> 1, xc = (t & 1)*8;
            const uint4 *xsrc = reinterpret_cast<const uint4 *>(prm.x + ((size_t)t0*TM + xr)*NIN + xc);
            uint4 xv = make_uint4(0, 0, 0, 0);
            if (!BIG && first && tiles > 0) xv = *xsrc;
            int u = 0;                                       // chain
            for (int i = 0; i < tiles && ok; ++i) {
                const int s = i % WG_STAGES;
                if (!BIG && first) {
                    if (i >= WG_STAGES
                        && !(ok = warp_wait(&empty[s], (uint32_t)((i/WG_STAGES - 1) & 1))))
                        break;
                    *reinterpret_cast<uint4 *>(xs + s*X_BYTES + tc::kmajor_offset<TM>(xr, xc)) = xv;
                    tc::fence_async_smem();
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive(&x_full[s]);
                    if (i + 1 < tiles) xv = xsrc[(size_t)(i + 1)*(TM*NIN/8)];
                }
                if (sums) {
                    float w[4] = {1.0f, 1.0f, 1.0f, 1.0f};
                    if (!BIG && layer == 4) {
                        #pragma unroll
                        for (int r = 0; r < 4; ++r) w[r] = prm.dout[(t0 + i)*TM + 32*r + lane];
                    }
                    if (!(ok = warp_wait(&full[s], (uint32_t)((i/WG_STAGES) & 1)))) break;
                    const uint8_t *from = smem + s*WG_STAGE_BYTES + warp*GROUPS*(2*GROUP_ELEMS)
                                        + 16*lane;
                    #pragma unroll
                    for (int q = 0; q < GROUPS; ++q) {
                        #pragma unroll
                        for (int r = 0; r < 4; ++r) {
                            const uint4 z = *reinterpret_cast<const uint4 *>(
                                from + q*(2*GROUP_ELEMS) + 512*r);
                            const uint32_t v[4] = {z.x, z.y, z.z, z.w};
                            #pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                acc[q][2*e] = fmaf(bf_lo(v[e]), w[r], acc[q][2*e]);
                                acc[q][2*e + 1] = fmaf(bf_hi(v[e]), w[r], acc[q][2*e + 1]);
                            }
                        }
                    }
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive(&empty[s]);
                }
                if (!mma) continue;
                // the chains that end in this tile
                if (CHAIN > PARTS && (i + 1) % (CHAIN/PARTS) != 0 && i + 1 < tiles) continue;
                #pragma unroll 1
                for (int k = 0; k < (CHAIN < PARTS ? PARTS/CHAIN : 1); ++k, ++u) {
                    if (!(ok = warp_wait(&acc_full[u & 1], (uint32_t)((u/2) & 1)))) break;
                    tc::fence_after_sync();
                    #pragma unroll
                    for (int c0 = 0; c0 < COLUMNS; c0 += 16) {
                        uint32_t r[16];
                        tc::tmem_ld16(at + (uint32_t)(WG_ACC*(u & 1) + c0), r);
                        tc::tmem_wait_ld();
                        tc::tmem_tie16(r);
                        #pragma unroll
                        for (int j = 0; j < 16; ++j) g[c0 + j] += __uint_as_float(r[j]);
                    }
                    tc::fence_before_sync();
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive(&acc_free[u & 1]);
                }
            }
            if (sums) {
                float *to = layer == 4 ? prm.dw_out + (size_t)split*HID
                                       : prm.db + ((size_t)layer*splits + split)*HID + mh*128;
                #pragma unroll
                for (int q = 0; q < GROUPS; ++q) {
                    const float v = warp_sum8(acc[q], lane);
                    if ((lane & 3) == 0) to[8*(warp*GROUPS + q) + (lane >> 2)] = v;
                }
            }
            if (mma) {
                const int m = 32*quad + lane;
                float *crow = prm.dw[layer]
                            + (BIG ? (size_t)split*HID*HID + (size_t)(mh*128 + m)*HID + nh*128 + 64*part
                                   : (size_t)split*HID*NIN + (size_t)(128*part + m)*NIN);
                // a whole 32-byte sector per store (in halves: 0.9 us more per launch)
                #pragma unroll
                for (int j = 0; j < COLUMNS; j += 8)
                    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                                 :: "l"(crow + j), "f"(g[j]), "f"(g[j + 1]), "f"(g[j + 2]),
                                    "f"(g[j + 3]), "f"(g[j + 4]), "f"(g[j + 5]), "f"(g[j + 6]),
                                    "f"(g[j + 7]) : "memory");
            }
        };
        if (big) add_up(std::true_type());
        else add_up(std::false_type());
        if (layer == 4 && split == 0 && warp < 2) {
            // warp 0 the loss, warp 1 the output bias: sums of 4 n_tiles partials
            const float *part = prm.row_sums + (size_t)warp*4*n_tiles;
            double sum = 0.0;
            for (int j = lane; j < 4*n_tiles; j += 32) sum += (double)part[j];
            #pragma unroll
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            float v = (float)(warp == 0 ? sum/(double)prm.n : sum);
            if (warp == 0 && prm.refused && *prm.refused != 0.0f) v = __int_as_float(0x7fffffff);
            if (lane == 0) *(warp == 0 ? prm.loss : prm.db_out) = v;
        }
        if (!ok && lane == 0) atomicExch(err, 1);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, 2*WG_ACC);
}

// out[k][i] = the sum over its splits of part[k][s*size + i], in split order, for
// up to 16 tensors in one launch (blockIdx.y = tensor): a step's gradients as
// one set of plain tensors.  In double precision, so that the sum rounds once.  Bound by
// the bytes of the partials (8 MB, in L2): 6.3 us with cold caches.
constexpr int SUM_TENSORS = 16;
struct SumTensors {
    int size[SUM_TENSORS], splits[SUM_TENSORS];
    const float *part[SUM_TENSORS];
    float *out[SUM_TENSORS];
};

__global__ void __launch_bounds__(256)
sum_partials(SumTensors T)
{
    tc::dependents_launch();
    tc::dependency_wait();
    const int k = blockIdx.y, size = T.size[k], splits = T.splits[k];
    const int i = blockIdx.x*256 + threadIdx.x;
    if (i >= size) return;
    const float *p = T.part[k] + i;
    double v = 0.0;
    #pragma unroll 8
    for (int s = 0; s < splits; ++s) v += (double)p[(size_t)s*size];
    T.out[k][i] = (float)v;
}

// ------------------------------------------------------ batch and schedule --
// The batch of a captured training step for a forward of one tile per SM (that of
// two SMs per tile gathers its own): the batch's rows of the data set (idx, 32 bytes
// of x and of x_lo and one target each) and, by one thread, the schedule.  Bound by
// the random 32-byte reads; 5.6 us with cold caches for 8192 rows, where three
// index_select launches and lr_schedule took 29.  A row outside the data set leaves
// zeros (see batch_row).
__global__ void __launch_bounds__(256)
gather_batch(int n, Batch batch, int *__restrict__ err)
{
    tc::dependents_launch();
    tc::dependency_wait();
    if (blockIdx.x == 0 && threadIdx.x == 0)
        schedule_step(batch.counters, batch.sched, batch.total, batch.warmup, batch.lr0, batch.b1,
                      batch.b2);
    const int i = blockIdx.x*256 + threadIdx.x, row = i >> 2, part = i & 3;
    if (row >= n) return;
    const long long src = batch_row(batch, row, err);
    const bool in = src >= 0;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (in) v = reinterpret_cast<const uint4 *>(part < 2 ? batch.x_all : batch.xlo_all)[2*src + (part & 1)];
    reinterpret_cast<uint4 *>(part < 2 ? batch.x : batch.x_lo)[2*row + (part & 1)] = v;
    if (part == 0) batch.y[row] = in ? batch.y_all[src] : 0.0f;
}

// -------------------------------------------------------------------- Adam --
// adam_pack: the update of every parameter and everything that is kept of the
// weights in bf16 -- W, W^T and the chunk images that the forward and the
// backward stream -- in one launch.  A block owns a 32 x 32 tile of a hidden
// weight, so that the partial gradients, masters and moments are read and
// written in 16-byte units along the rows, and W^T and both images from the
// tile in shared memory as whole 16-byte units too.  Bound by the bytes (8 MB of
// partials, 6 MB of state): 7.1 us with cold caches, where adam_multi and the two
// packing kernels took 14.6.
// Blocks: 64 per hidden layer, 4 for W0 (64 rows each), one per vector.
struct AdamPack {
    const float *grad[10];           // W0..W3, b0..b3, w_out, b_out
    int splits[10];
    float *p[10], *m[10], *v[10];
    __nv_bfloat16 *w[4], *wt[4];
    uint8_t *img, *img_t;
    const float *sched;              // {lr, bc1, bc2, refused}, or null and the values below
    float lr, bc1, bc2, b1, b2, eps;
};
constexpr int AP_TILES = (HID/32)*(HID/32);
constexpr int AP_W0 = 4;
constexpr int AP_BLOCKS = 3*AP_TILES + AP_W0 + 6;
constexpr int AP_LD = 40;            // bf16 per row of the tile: 16-byte units stay aligned

__device__ __forceinline__ float4 adam4(const AdamPack &A, int k, int i, int size, float lr,
                                        float bc1, float bc2)
{
    const float *grad = A.grad[k] + i;
    const int splits = A.splits[k];
    float g[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    #pragma unroll 5
    for (int s = 0; s < splits; ++s) {
        const float4 u = *reinterpret_cast<const float4 *>(grad + (size_t)s*size);
        g[0] += u.x;
        g[1] += u.y;
        g[2] += u.z;
        g[3] += u.w;
    }
    float4 p = *reinterpret_cast<float4 *>(A.p[k] + i), m = *reinterpret_cast<float4 *>(A.m[k] + i),
           v = *reinterpret_cast<float4 *>(A.v[k] + i);
    float *pp = &p.x, *mp = &m.x, *vp = &v.x;
    #pragma unroll
    for (int e = 0; e < 4; ++e) adam_update(g[e], pp[e], mp[e], vp[e], lr, A.b1, A.b2, A.eps, bc1, bc2);
    *reinterpret_cast<float4 *>(A.p[k] + i) = p;
    *reinterpret_cast<float4 *>(A.m[k] + i) = m;
    *reinterpret_cast<float4 *>(A.v[k] + i) = v;
    return p;
}

__global__ void __launch_bounds__(256)
adam_pack(AdamPack A)
{
    __shared__ __align__(16) __nv_bfloat16 tile[32*AP_LD];
    tc::dependents_launch();
    tc::dependency_wait();
    const int t = threadIdx.x, b = blockIdx.x;
    if (A.sched && A.sched[3] != 0.0f) return;           // see batch_row
    const float lr = A.sched ? A.sched[0] : A.lr, bc1 = A.sched ? A.sched[1] : A.bc1,
                bc2 = A.sched ? A.sched[2] : A.bc2;
    if (b < 3*AP_TILES) {
        const int l = 1 + b/AP_TILES, tr = (b % AP_TILES)/(HID/32), tc_ = b % (HID/32);
        const int r = t >> 3, c = 4*(t & 7);
        const int at = (32*tr + r)*HID + 32*tc_ + c;
        const float4 p = adam4(A, l, at, HID*HID, lr, bc1, bc2);
        uint2 h;
        h.x = pack2(p.x, p.y);
        h.y = pack2(p.z, p.w);
        *reinterpret_cast<uint2 *>(A.w[l] + at) = h;
        *reinterpret_cast<uint2 *>(tile + r*AP_LD + c) = h;
        __syncthreads();
        const int j = t & 31, g = (t >> 5) & 3;
        if (t < 128) {
            // row j of the tile, input group g
            *reinterpret_cast<uint4 *>(A.img + W0_BYTES
                                       + (size_t)((l - 1)*CHUNKS_PER_LAYER + tc_)*CHUNK_BYTES
                                       + tc::kmajor_offset<HID>(32*tr + j, 8*g)) =
                *reinterpret_cast<const uint4 *>(tile + j*AP_LD + 8*g);
        } else {
            // column j of the tile, output group g
            uint4 u;
            uint32_t *up = &u.x;
            #pragma unroll
            for (int e = 0; e < 4; ++e) {
                const __nv_bfloat162 two = __halves2bfloat162(tile[(8*g + 2*e)*AP_LD + j],
                                                              tile[(8*g + 2*e + 1)*AP_LD + j]);
                up[e] = *reinterpret_cast<const uint32_t *>(&two);
            }
            *reinterpret_cast<uint4 *>(A.wt[l] + (32*tc_ + j)*HID + 32*tr + 8*g) = u;
            *reinterpret_cast<uint4 *>(A.img_t + (size_t)((3 - l)*CHUNKS_PER_LAYER + tr)*CHUNK_BYTES
                                       + tc::kmajor_offset<HID>(32*tc_ + j, 8*g)) = u;
        }
    } else if (b < 3*AP_TILES + AP_W0) {
        const int r = 64*(b - 3*AP_TILES) + (t >> 2), c = 4*(t & 3);
        const float4 p = adam4(A, 0, r*NIN + c, HID*NIN, lr, bc1, bc2);
        uint2 h;
        h.x = pack2(p.x, p.y);
        h.y = pack2(p.z, p.w);
        *reinterpret_cast<uint2 *>(A.w[0] + r*NIN + c) = h;
        *reinterpret_cast<uint2 *>(A.img + tc::kmajor_offset<HID>(r, c)) = h;
        const float *pp = &p.x;
        #pragma unroll
        for (int e = 0; e < 4; ++e) A.wt[0][(c + e)*HID + r] = __float2bfloat16_rn(pp[e]);
    } else {
        const int k = 4 + b - 3*AP_TILES - AP_W0, size = k < 9 ? HID : 1;
        if (t >= size) return;
        double sum = 0.0;
        for (int s = 0; s < A.splits[k]; ++s) sum += (double)A.grad[k][s*size + t];
        const float g = (float)sum;
        float p = A.p[k][t], m = A.m[k][t], v = A.v[k][t];
        adam_update(g, p, m, v, lr, A.b1, A.b2, A.eps, bc1, bc2);
        A.p[k][t] = p;
        A.m[k][t] = m;
        A.v[k][t] = v;
    }
}
