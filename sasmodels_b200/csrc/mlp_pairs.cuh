// mlp_serve_pairs: inference over many tiles, by pairs of SMs with two tiles in
// flight on each.  Included by mlp.cu.
//
// mlp_serve works on one tile at a time, so that each layer's MMAs wait for the
// last epilogue's chunks and each epilogue for the layer's last MMAs: 28,500
// cycles per tile, where the MMAs take 12,500.  With two tiles in flight and all
// else as there, the shared memory was 91 % busy at 22,400.  Here
//  - a CTA interleaves two tiles, A and B: the MMAs of B's layer run while the
//    epilogue works on A's accumulator, and the reverse.  The activations need
//    room for one tile all the same: chunk c of A's next input (64 columns, hi
//    and lo halves, 32 KB) is written into the place of chunk c of B's current
//    input once the MMAs that read that are done, so that the activation buffer
//    is a ring of chunks in MMA order and one commit per chunk frees its
//    activations and its weights;
//  - two CTAs of a cluster work as one (cta_group::2, M = 256): each holds its
//    own 128 rows of activations and accumulators and half of every weight
//    chunk, which halves the weight bytes that an SM fetches and reads.
//
// Order.  Layers 1-3 of a tile are "steps" of four chunks (64 inputs: 4 K steps,
// both halves); the steps take A and B strictly in turn, B a layer ahead of A:
//     A1 B2' A2 B3' A3 B1 | A1 B2 ...              (' = B's tile before)
// so that a tile's epilogue has the other tile's step to run under, and the
// epilogues follow as  A1 B2' A2 B3' B0 A3 A0 B1.  Layer 0 (16 features, two MMAs)
// of a tile is issued in the middle of the step after its predecessor's last
// layer, when that layer's accumulator has long been read.  The epilogues write
// the steps' inputs in the order in which they are consumed.
//   warps 0-15  epilogue: warp w, rows of quadrant w % 4, the 16 columns at
//               16 (w/4) of every 64, chunk by chunk, so that the first is ready
//               early; all 64 columns leave TMEM first, which frees the
//               accumulator.  In the last layer the 8 columns at 8 (w/4) of every
//               chunk, so that the output dot sums as mlp_serve's does.
//   warp 16     CTA 0, lane 0: issues the MMAs, a "unit" (a chunk, or a layer 0) as
//               soon as the count of ready units covers it.  An issue holds the
//               thread for about the time of the MMA before, so nothing else is
//               waited for here.
//   warp 17     producer of this CTA's half of the weight ring.
//   warp 18     CTA 0: polls the barriers of the current step's units, one per lane,
//               and publishes how many are ready in order.  (Waiting for a chunk's
//               barriers in turn took longer than its MMAs.)  CTA 1: passes on
//               that its weights have landed.
//   warp 19     the features of the next tiles.
// Barriers (parity waits, bounded).  In both CTAs, completed by the MMA's commit:
// chunk_done[c], once per step (frees the chunk's activations and weights),
// acc_full[p], once per layer of a tile in p, x_free[p], once per tile.  In CTA 0,
// arrived on by both: act_ready[c], acc_empty[p], x_ready[p], full (the weights of
// both).  No barrier can run two phases ahead of a waiter, because each next
// completion needs what the waiter does after its wait (the poll keeps what it
// has seen of a step: a chunk's barriers may move on once it is published).  No
// role waits for a later one: the epilogue that writes step s needs the chunks of
// step s - 1 done, whose inputs come from epilogues before it.  Both CTAs meet
// before either exits.
//
// CTA 1's arrivals in CTA 0 stand for its activations, features and weights, which its
// own tensor core reads for an MMA that CTA 0 issues: each writer hands them to the
// async proxy (fence.proxy.async, or a bulk copy's completion), the arrival releases
// them at cluster scope, and who polls the barrier acquires them before the count goes
// on.  Both fences are restricted to shared memory (see mbar_arrive_cta).  An
// accumulator that has been read is handed over as tcgen05.fence asks.
//
// The hidden activations and the output are those of mlp_serve bit for bit (the
// paired FP32 operations round each half as the scalar ones).  4,000,000 rows 3.10
// -> 2.14 ms (1.50 PFLOP/s of MMA, both halves counted: 0.93 of the measured
// BF16 peak), 500,000 rows 411 -> 275 us, 50,021 rows 51.8 -> 38.4 us; without the
// fences of the hand-overs 2.13 ms, 269 and 37.6 us.  Chunks of 32 inputs took 3 % more,
// of 128 14 %.
#pragma once

constexpr int SP_POLL_WARP = SV_EPI_WARPS + 2;
constexpr int SP_X_WARP = SV_EPI_WARPS + 3;
constexpr int SP_THREADS = SV_EPI + 128;
constexpr int SP_K = 64;                           // inputs of a chunk
constexpr int SP_CHUNKS = HID/SP_K;                // of a step, and of the weight ring
constexpr int SP_SIDE = SP_CHUNKS/2;               // chunk before which a layer 0 goes
constexpr int SP_GROUP = HID/2*16;                 // 8 inputs of this CTA's 128 outputs: 2 KB
constexpr int SP_HALF = SP_K/8*SP_GROUP;           // this CTA's weights of a chunk
constexpr int SP_SMEM = 2*ACT_BYTES + SP_CHUNKS*SP_HALF + W0_BYTES/2 + 4*X_BYTES + 4*SV_PARAMS;
// Tiles per CTA up to which mlp_serve is taken: 8 tiles 17.5 us there and 18.9 here,
// 148 tiles 18.6 and 20.2; but 157 tiles on 148 CTAs 35.0 and 32.7.
constexpr int SP_TILES = 1;

// Turn j (from SP_FIRST on) of the epilogues, for `mine` tiles (A the even ones,
// B the odd): accumulator p, layer l and tile i of p; false where there is none.
// The steps are its turns with l > 0.
constexpr int SP_FIRST = -2;
__device__ __forceinline__ bool sp_turn(int j, int mine, int &p, int &l, int &i)
{
    const int q = j & 7, k = j >> 3;               // k = -1 for the first A0
    // A1 B2' A2 B3' B0 A3 A0" B1: accumulator, layer and tile offset + 1
    p = (0x9a >> q) & 1;
    l = (0x4ce9 >> (2*q)) & 3;
    i = k + ((0x6511 >> (2*q)) & 3) - 1;
    return i >= 0 && 2*i + p < mine;
}
// The accumulator of the layer 0 that goes into the step (p, l, i): that of p' 's
// next tile in the step after (p', layer 3), or none (-1).
__device__ __forceinline__ int sp_side(int p, int l, int i, int mine)
{
    if (p == 0 && l == 3 && i > 0 && 2*i + 1 < mine) return 1;       // after B3'
    if (p == 1 && l == 1 && 2*(i + 1) < mine) return 0;              // after A3
    return -1;
}
// One past the last turn: layer 3 of the last tile of A or of B.
__device__ __forceinline__ int sp_turns(int mine)
{
    return max(8*((mine + 1)/2 - 1) + 6, mine > 1 ? 8*(mine/2) + 4 : SP_FIRST);
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(SP_THREADS, 1)
mlp_serve_pairs(int n, int n_tiles, const __nv_bfloat16 *__restrict__ x,
                const __nv_bfloat16 *__restrict__ x_lo, InferParams prm, float *__restrict__ out,
                int *__restrict__ err)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t *act = smem;                          // the chunks' hi halves,
    uint8_t *act_lo = smem + ACT_BYTES;           // their lo halves
    uint8_t *ring = smem + 2*ACT_BYTES;
    uint8_t *w0 = ring + SP_CHUNKS*SP_HALF;
    uint8_t *xs = w0 + W0_BYTES/2;                // [tile of the pair][hi, lo] x X_BYTES
    float *par = reinterpret_cast<float *>(xs + 4*X_BYTES);
    __shared__ __align__(8) uint64_t full[SP_CHUNKS];
    __shared__ __align__(8) uint64_t chunk_done[SP_CHUNKS], act_ready[SP_CHUNKS];
    __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2], dot_bar[2][4], x_ready[2], x_free[2];
    __shared__ __align__(8) uint64_t w0_bar, drain;
    __shared__ uint32_t tmem_slot, ready_seq;
    __shared__ float dot_part[2][3][TM];
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    // double tiles of 256 rows, this CTA's half 128 of them
    const int rank = (int)tc::cluster_rank();
    const int cluster = blockIdx.x >> 1, clusters = gridDim.x >> 1;
    const int doubles = (n_tiles + 1)/2;
    const int mine = cluster < doubles ? (doubles - 1 - cluster)/clusters + 1 : 0;
    const int turns = sp_turns(mine);
    // first row of this CTA's half of double tile i of its cluster
    auto row_of = [&](int i) { return (2*(cluster + i*clusters) + rank)*TM; };

    if (warp == 0) tc::tmem_alloc2(&tmem_slot, 2*HID);
    if (t == 0) {
        // CTA 0's also takes an arrival for CTA 1's weights
        for (int s = 0; s < SP_CHUNKS; ++s) tc::mbar_init(&full[s], 2 - rank);
        ready_seq = 0;
        for (int c = 0; c < SP_CHUNKS; ++c) {
            tc::mbar_init(&chunk_done[c], 1);
            tc::mbar_init(&act_ready[c], 2*SV_EPI_WARPS);
        }
        for (int a = 0; a < 2; ++a) {
            tc::mbar_init(&acc_full[a], 1);
            tc::mbar_init(&acc_empty[a], 2*SV_EPI_WARPS);
            tc::mbar_init(&x_ready[a], 2);
            tc::mbar_init(&x_free[a], 1);
            for (int q = 0; q < 4; ++q) tc::mbar_init(&dot_bar[a][q], SV_EPI_WARPS/4 - 1);
        }
        tc::mbar_init(&w0_bar, 1);
        tc::mbar_init(&drain, 1);
        tc::mbar_fence_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::cluster_sync();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_slot;
    // one arrival on a barrier of CTA 0
    auto arrive0 = [&](uint64_t *bar) {
        if (rank == 0) tc::mbar_arrive(bar);
        else tc::mbar_arrive_cta(bar, 0);
    };

    if (warp == SV_PROD_WARP) {
        // ---- producer: this CTA's half (128 outputs) of the weight chunks of
        // every step, in MMA order; their groups of 8 inputs are 4 KB apart in
        // the image, 2 KB here ----
        if (lane == 0) {
            bool ok = true;
            const uint8_t *img = prm.img + rank*SP_GROUP;
            tc::mbar_arrive_expect_tx(&w0_bar, W0_BYTES/2);
            for (int g = 0; g < NIN/8; ++g)
                tc::bulk_load(w0 + g*SP_GROUP, img + g*2*SP_GROUP, SP_GROUP, &w0_bar);
            int i = 0;
            for (int j = SP_FIRST; j < turns && ok; ++j) {
                int p, l, tile;
                if (!sp_turn(j, mine, p, l, tile) || l == 0) continue;
                // chunk c of a step has stage c, last read by chunk c of the step
                // before
                for (int c = 0; c < SP_CHUNKS; ++c) {
                    if (i > 0 && !(ok = tc::mbar_wait_cluster(&chunk_done[c], (uint32_t)((i - 1) & 1))))
                        break;
                    tc::mbar_arrive_expect_tx(&full[c], SP_HALF);
                    const uint8_t *src = img + W0_BYTES + (size_t)(l - 1)*HID*HID*2
                                       + (size_t)c*(SP_K/8)*2*SP_GROUP;
                    #pragma unroll
                    for (int g = 0; g < SP_K/8; ++g)
                        tc::bulk_load(ring + c*SP_HALF + g*SP_GROUP, src + g*2*SP_GROUP, SP_GROUP,
                                      &full[c]);
                }
                ++i;
            }
            // every issued copy has landed before the CTA may exit
            for (int c = 0; c < SP_CHUNKS && i > 0 && ok; ++c)
                ok = tc::mbar_wait(&full[c], (uint32_t)((i - 1) & 1));
            ok = tc::mbar_wait(&w0_bar, 0u) && ok;
            if (!ok) atomicExch(err, 2);
        }
        __syncwarp();
    } else if (warp == SP_POLL_WARP) {
        bool ok = true;
        if (rank == 0) {
            // ---- poll: the units of every step ----
            // lanes 0.. activations of the chunks, 8.. weights (of both CTAs),
            // 16 the step's accumulator, read by the epilogue of the layer
            // before (completion 4 i + l - 1); 17 and 18 features and accumulator
            // (completion 4 i - 1) of the layer 0 that goes into the step
            uint32_t unit = 0;
            ok = warp_wait(&w0_bar, 0u);
            for (int p = 0; p < 2 && p < mine && ok; ++p) {
                ok = warp_wait_cluster(&x_ready[p], 0u);
                __syncwarp();
                ++unit;
                if (lane == 0 && ok) tc::st_release_shared(&ready_seq, unit);
            }
            int s = 0;
            for (int j = SP_FIRST; j < turns && ok; ++j) {
                int p, l, i;
                if (!sp_turn(j, mine, p, l, i) || l == 0) continue;
                const int z = sp_side(p, l, i, mine);
                const int zi = z == 1 ? i : i + 1;          // the layer 0's tile of z
                uint64_t *bar = lane < 8 ? &act_ready[lane & (SP_CHUNKS - 1)]
                              : lane < 16 ? &full[lane & (SP_CHUNKS - 1)]
                              : lane == 16 ? &acc_empty[p] : lane == 17 ? &x_ready[z & 1]
                              : &acc_empty[z & 1];
                const uint32_t parity = lane < 16 ? (uint32_t)(s & 1)
                                      : lane == 16 ? (uint32_t)((l + 1) & 1)
                                      : lane == 17 ? (uint32_t)(zi & 1) : 1u;
                const int units = SP_CHUNKS + (z >= 0 ? 1 : 0);
                constexpr uint32_t all = (1u << SP_CHUNKS) - 1u;
                const uint32_t need = all | all << 8 | 1u << 16 | (z >= 0 ? 3u << 17 : 0u);
                uint32_t seen = 0;
                int done = 0;
                for (uint32_t n_try = 0; done < units && n_try < tc::WAIT_LIMIT; ++n_try) {
                    const bool on = (need & ~seen & (1u << lane)) != 0;
                    seen |= __ballot_sync(0xffffffffu, on && tc::mbar_test_relaxed(bar, parity));
                    // units in order, the layer 0 in the middle
                    uint32_t r = seen & (seen >> 8) & all;
                    if (z >= 0)
                        r = (r & ((1u << SP_SIDE) - 1u)) | ((r >> SP_SIDE) << (SP_SIDE + 1))
                          | (((seen >> 17) & (seen >> 18) & 1u) << SP_SIDE);
                    const int here = (seen >> 16) & 1u ? __ffs(~r) - 1 : 0;
                    if (here > done) {
                        done = here;
                        tc::cluster_acquire();
                        __syncwarp();
                        if (lane == 0) tc::st_release_shared(&ready_seq, unit + (uint32_t)done);
                    }
                }
                ok = done == units;
                unit += (uint32_t)units;
                ++s;
            }
        } else {
            int s = 0;
            for (int j = SP_FIRST; j < turns && ok; ++j) {
                int p, l, i;
                if (!sp_turn(j, mine, p, l, i) || l == 0) continue;
                for (int c = 0; c < SP_CHUNKS; ++c) {
                    if (!(ok = warp_wait(&full[c], (uint32_t)(s & 1)))) break;
                    if (lane == 0) arrive0(&full[c]);
                }
                ++s;
            }
        }
        if (!ok && lane == 0) atomicExch(err, 4);
    } else if (warp == SP_X_WARP) {
        // features of tile i of p
        auto load_x = [&](int p, int i) {
            uint8_t *xb = xs + p*2*X_BYTES;
            const int row0 = row_of(2*i + p);
            const bool in = row0 < n_tiles*TM;         // the last double tile may be half
            uint4 v[8], w[8];
            #pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int u = lane + 32*j;
                const size_t g = (size_t)(row0 + (u >> 1))*NIN + (u & 1)*8;
                v[j] = w[j] = make_uint4(0, 0, 0, 0);
                if (in) {
                    v[j] = *reinterpret_cast<const uint4 *>(x + g);
                    w[j] = *reinterpret_cast<const uint4 *>(x_lo + g);
                }
            }
            #pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int u = lane + 32*j;
                const uint32_t at = tc::kmajor_offset<TM>(u >> 1, (u & 1)*8);
                *reinterpret_cast<uint4 *>(xb + at) = v[j];
                *reinterpret_cast<uint4 *>(xb + X_BYTES + at) = w[j];
            }
            tc::fence_async_smem();
            __syncwarp();
        };
        bool ok = warp_wait(&w0_bar, 0u);
        for (int i = 0; 2*i < mine && ok; ++i) {
            for (int p = 0; p < 2 && 2*i + p < mine; ++p) {
                // the buffer's last reader, layer 0 of the tile before
                if (i > 0 && !(ok = warp_wait_cluster(&x_free[p], (uint32_t)((i - 1) & 1)))) break;
                load_x(p, i);
                if (lane == 0) arrive0(&x_ready[p]);
            }
        }
        if (!ok && lane == 0) atomicExch(err, 4);
    } else if (warp == SV_MMA_WARP) {
        // ---- MMA issue ----
        if (lane == 0 && rank == 0) {
            constexpr uint32_t idesc = tc::idesc_bf16(2*TM, HID);
            const uint32_t a_hi = tc::smem_u32(act), a_lo = tc::smem_u32(act_lo);
            bool ok = true;
            uint32_t unit = 0;
            ReadyCount count(&ready_seq);
            auto next_unit = [&]() {
                const bool there = count.covers(++unit);
                tc::fence_after_sync();
                return there;
            };
            auto layer0 = [&](int z) {
                const uint32_t dz = tmem + (uint32_t)(HID*z);
                const uint32_t xb = tc::smem_u32(xs + z*2*X_BYTES);
                const uint64_t bdesc = tc::kmajor_desc<HID/2>(tc::smem_u32(w0), 0);
                tc::mma_bf16_pair(dz, tc::kmajor_desc<TM>(xb, 0), bdesc, idesc, 0u);
                tc::mma_bf16_pair(dz, tc::kmajor_desc<TM>(xb + X_BYTES, 0), bdesc, idesc, 1u);
                tc::mma_commit_pair(&x_free[z]);
                tc::mma_commit_pair(&acc_full[z]);
            };
            for (int p = 0; p < 2 && p < mine && ok; ++p)
                if ((ok = next_unit())) layer0(p);
            for (int j = SP_FIRST; j < turns && ok; ++j) {
                int p, l, i;
                if (!sp_turn(j, mine, p, l, i) || l == 0) continue;
                const int z = sp_side(p, l, i, mine);
                const uint32_t d = tmem + (uint32_t)(HID*p);
                for (int c = 0; c < SP_CHUNKS; ++c) {
                    if (c == SP_SIDE && z >= 0) {
                        if (!(ok = next_unit())) break;
                        layer0(z);
                    }
                    if (!(ok = next_unit())) break;
                    const uint32_t b_addr = tc::smem_u32(ring + c*SP_HALF);
                    #pragma unroll
                    for (int st = 0; st < SP_K/16; ++st) {
                        const uint64_t bdesc = tc::kmajor_desc<HID/2>(b_addr, st);
                        const int as = c*(SP_K/16) + st;
                        tc::mma_bf16_pair(d, tc::kmajor_desc<TM>(a_hi, as), bdesc, idesc,
                                          (c > 0 || st > 0) ? 1u : 0u);
                        tc::mma_bf16_pair(d, tc::kmajor_desc<TM>(a_lo, as), bdesc, idesc, 1u);
                    }
                    tc::mma_commit_pair(&chunk_done[c]);
                }
                if (ok) tc::mma_commit_pair(&acc_full[p]);
            }
            // every MMA issued has completed before TMEM is released
            tc::mma_commit_pair(&drain);
            ok = tc::mbar_wait_cluster(&drain, 0u) && ok;
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
        const uint32_t lane_base = tmem + ((uint32_t)(32*quad) << 16);
        bool ok = true;
        int s = 0;                                   // step whose input is being written
        for (int j = SP_FIRST; j < turns && ok; ++j) {
            int p, l, i;
            if (!sp_turn(j, mine, p, l, i)) continue;
            if (!(ok = warp_wait_cluster(&acc_full[p], (uint32_t)(l & 1)))) break;
            tc::fence_after_sync();
            if (l < 3) {
                // 16 columns of every 64
                const float *bias = par + l*HID + 16*slot;
                const uint32_t acc = lane_base + (uint32_t)(HID*p + 16*slot);
                uint32_t r[4][16];
                #pragma unroll
                for (int q = 0; q < 4; ++q) tc::tmem_ld16(acc + (uint32_t)(64*q), r[q]);
                tc::tmem_wait_ld();
                #pragma unroll
                for (int q = 0; q < 4; ++q) tc::tmem_tie16(r[q]);
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) arrive0(&acc_empty[p]);
                // chunk c of step s takes the place of chunk c of step s - 1
                // (completion s - 1); the last one done means that all are
                const uint32_t before = (uint32_t)((s - 1) & 1);
                const bool free_all = s == 0 || tc::mbar_test_relaxed(&chunk_done[SP_CHUNKS - 1], before);
                tc::cluster_acquire();
                #pragma unroll
                for (int q = 0; q < 4; ++q) {
                    constexpr int RU = SP_K/64;
                    const int c = q/RU;
                    uint4 hi[2], lo[2];
                    silu_columns(r[q], 0, bias + 64*q, hi[0], lo[0]);
                    // the stores of the chunk before have had time to land
                    if (q > 0 && q % RU == 0) {
                        tc::fence_async_smem();
                        __syncwarp();
                        if (lane == 0) arrive0(&act_ready[c - 1]);
                    }
                    silu_columns(r[q], 8, bias + 64*q, hi[1], lo[1]);
                    if (q % RU == 0 && !free_all && !tc::mbar_wait_cluster(&chunk_done[c], before)) ok = false;
                    #pragma unroll
                    for (int g = 0; g < 2; ++g) {
                        const uint32_t off = tc::kmajor_offset<TM>(row, 64*q + 16*slot + 8*g);
                        *reinterpret_cast<uint4 *>(act + off) = hi[g];
                        *reinterpret_cast<uint4 *>(act_lo + off) = lo[g];
                    }
                }
                tc::fence_async_smem();
                ok = __all_sync(0xffffffffu, ok) != 0;
                __syncwarp();
                if (lane == 0) arrive0(&act_ready[SP_CHUNKS - 1]);
                if (!ok) break;
                ++s;
            } else {
                const float *bias = par + 3*HID + SV_COLS*slot;
                const float *wo = par + 4*HID + SV_COLS*slot;
                const uint32_t acc = lane_base + (uint32_t)(HID*p + SV_COLS*slot);
                float dot = 0.0f;
                uint32_t r[CHUNKS_PER_LAYER][8];
                #pragma unroll
                for (int c = 0; c < CHUNKS_PER_LAYER; ++c) tc::tmem_ld8(acc + (uint32_t)(KCI*c), r[c]);
                #pragma unroll
                for (int c = 0; c < CHUNKS_PER_LAYER; ++c) tc::tmem_wait_ld8(r[c]);
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) arrive0(&acc_empty[p]);
                #pragma unroll
                for (int c = 0; c < CHUNKS_PER_LAYER; ++c) dot = dot8(r[c], bias + KCI*c, wo + KCI*c, dot);
                // four partial sums per row; slot 0 adds them.  Slots 1-3
                // write dot_part[p] again in the last layer of p's next
                // tile, which needs slot 0's activations of that tile.
                if (slot > 0) {
                    dot_part[p][slot - 1][row] = dot;
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive(&dot_bar[p][quad]);
                } else {
                    if (!(ok = warp_wait(&dot_bar[p][quad], (uint32_t)(i & 1)))) break;
                    const int at = row_of(2*i + p) + row;
                    if (at < n)
                        out[at] = ((dot + dot_part[p][0][row]) + dot_part[p][1][row])
                                  + dot_part[p][2][row] + b_out;
                }
            }
        }
        if (!ok && lane == 0) atomicExch(err, 1);
    }
    // neither CTA leaves while the other may still reach its shared memory
    tc::fence_before_sync();
    __syncthreads();
    tc::cluster_sync();
    if (warp == 0) tc::tmem_dealloc2(tmem, 2*HID);
}
