// Resolution smearing on the GPU, the step that follows the kernel in every
// fit (sasmodels/direct_model.py:345 -> Resolution.apply).
//
//   pinhole_smear       1D pinhole (sasmodels/resolution.py:172-220): each
//                       measured q_i averages the theory over the calculated
//                       points q_calc[j] within [q_i - 2.5 s_i, q_i + 3 s_i],
//                       weighted by the gaussian mass of each point's bin,
//                       erf((e[j+1] - q_i)/(sqrt2 s_i)) - erf((e[j] - q_i)/(sqrt2 s_i)),
//                       normalised by the weights' sum.  The reference builds
//                       the dense n_calc x nq matrix and multiplies; here one
//                       warp per q_i walks only its band (computed on the host
//                       by binary search), forming the weights on the fly: the
//                       work is the band, not the matrix.
//   slit_smear          1D slit (sasmodels/resolution.py:223-395): per q_i
//                       and per step across the slit width, the bins between
//                       |q| and sqrt(q^2 + l^2) found by binary search, the
//                       u-substituted bin widths formed on the fly.
//   pinhole_weights,    the same weights formed once per resolution object, and
//   slit_weights,       their banded product with one curve or many.
//   band_apply(_sets)
//   nllf_sets           the fit objective of every curve of a population
//                       against one data set (bumps_model.py:263-282).
//   pinhole2d_average   2D pinhole (sasmodels/resolution2d.py:162-175): the
//                       weighted average over the nbins oversampling points of
//                       every q, products and sums rounded separately in bin
//                       order, as numpy's axis-0 reduction does.
//
// Both read theory values the model kernel left on the device, so a fit step
// needs no host round trip between the kernel and the smearing.
#include <cstdint>
#include <cstdio>
#include <cuda_runtime.h>

namespace res {

constexpr unsigned FULL = 0xffffffffu;

// band_apply (a warp per q and curve) up to this many (q, curve) pairs, then
// band_apply_sets: 181 q x 61 curves 3.8 against 4.3 us and 400 x 32 4.1 against
// 4.7, but 181 x 100 4.9 against 4.2 and 400 x 61 5.8 against 4.6.
constexpr long long BAND_WARP_LIMIT = 14000;

// nllf_sets (a block per curve) up to this many curves, then nllf_rows: 800
// curves of 1000 points 4.3 against 6.2 us, 1600 of 1000 6.8 against 6.7, 1600
// of 400 4.8 against 3.9, 4096 of 1000 14.3 against 8.6.
constexpr int NLLF_BLOCKS = 1200;
constexpr double SQRT2 = 1.4142135623730951;     // numpy sqrt(2.0), correctly rounded

// One curve per blockIdx.y: theory + y*theory_stride -> out + y*out_stride.
__global__ void __launch_bounds__(256)
pinhole_smear(int nq, const double *__restrict__ q, const double *__restrict__ width,
              const int32_t *__restrict__ lo, const int32_t *__restrict__ hi,
              const double *__restrict__ edges, const double *__restrict__ theory,
              double *__restrict__ out, size_t theory_stride, size_t out_stride)
{
    const int i = (int)((blockIdx.x*(size_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (i >= nq) return;                      // whole warps leave together
    theory += blockIdx.y*theory_stride;
    out += blockIdx.y*out_stride;
    const double qi = q[i];
    const double s = SQRT2*width[i];
    double acc = 0.0, wsum = 0.0;
    for (int j = lo[i] + lane; j < hi[i]; j += 32) {
        const double w = erf((edges[j + 1] - qi)/s) - erf((edges[j] - qi)/s);
        acc += w*theory[j];
        wsum += w;
    }
    #pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        acc += __shfl_xor_sync(FULL, acc, off);
        wsum += __shfl_xor_sync(FULL, wsum, off);
    }
    if (lane == 0) out[i] = acc/wsum;
}

// 8 bytes global -> shared, asynchronously; zeros where !valid (src is not read)
__device__ __forceinline__ void copy8(double *dst, const double *src, bool valid = true)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;"
                 :: "r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(valid ? 8 : 0)
                 : "memory");
}
__device__ __forceinline__ void copy_commit()
{
    asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void copy_wait()
{
    asm volatile("cp.async.wait_group %0;" :: "n"(N) : "memory");
}

// One thread per q, its bins summed in order.  Bound by the bytes of theory,
// whose latency the chain of rounded additions would expose: each thread keeps
// the next 40 bins on their way into its own slots of shared memory (no other
// thread reads them, so there is nothing to synchronise), in groups of 8.
// Blocks of 64 spread an image of any size over the SMs, and 24 KB each lets one
// wave of them hold 256 x 256 q.  256 x 256 q of 60 bins 9.6 us (3.3 TB/s; 16.7
// with the loads inside the chain), of 200 bins 27 (51), 64 x 64 of 200 16.6 (50).
constexpr int P2_THREADS = 64, P2_GROUP = 8, P2_GROUPS = 6;
__global__ void __launch_bounds__(P2_THREADS)
pinhole2d_average(int nq, int nbins, const double *__restrict__ theory,
                  const double *__restrict__ weights, double wsum, double *__restrict__ out)
{
    __shared__ double ring[P2_GROUPS*P2_GROUP*P2_THREADS];
    const int i = (int)(blockIdx.x*(size_t)blockDim.x + threadIdx.x);
    if (i >= nq) return;
    const size_t step = (size_t)nq;
    const double *src = theory + i;                      // bin of the next fetch
    double *slot = ring + threadIdx.x;
    const int full = nbins/P2_GROUP;                     // groups of 8, then the rest
    auto fetch = [&](int g) {
        if (g < full) {
            double *to = slot + (g % P2_GROUPS)*P2_GROUP*P2_THREADS;
            #pragma unroll
            for (int k = 0; k < P2_GROUP; ++k) {
                copy8(to + k*P2_THREADS, src);
                src += step;
            }
        }
        copy_commit();               // one group per call, empty beyond the last
    };
    #pragma unroll
    for (int g = 0; g < P2_GROUPS - 1; ++g) fetch(g);
    double num = -0.0;                                   // -0 + p is p, its sign too
    for (int g = 0; g < full; ++g) {
        fetch(g + P2_GROUPS - 1);
        copy_wait<P2_GROUPS - 1>();
        const double *x = slot + (g % P2_GROUPS)*P2_GROUP*P2_THREADS;
        double p[P2_GROUP];
        #pragma unroll
        for (int k = 0; k < P2_GROUP; ++k)
            p[k] = __dmul_rn(x[k*P2_THREADS], weights[P2_GROUP*g + k]);
        #pragma unroll
        for (int k = 0; k < P2_GROUP; ++k) num = __dadd_rn(num, p[k]);
    }
    for (int b = full*P2_GROUP; b < nbins; ++b, src += step)
        num = __dadd_rn(num, __dmul_rn(*src, weights[b]));
    out[i] = num/wsum;
}

// Binary search: first index in edges[0..n) with edges[k] >= x (or > x
// when strict), the same in every lane.
__device__ __forceinline__ int lower_edge(const double *edges, int n, double x, bool strict)
{
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        const bool before = strict ? edges[mid] <= x : edges[mid] < x;
        if (before) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// u(e) of the slit integral (sasmodels/resolution.py:387-395): e^2 - q^2
// inside [|q|, sqrt(q^2 + l^2)], 0 below, (limit^2 - q^2) above.  Each
// product and difference is rounded on its own (no contraction into an
// FMA): sqrt(u) near the lower limit amplifies the last bit of u.
__device__ __forceinline__ double sq_diff(double a, double b)
{
    return __dsub_rn(__dmul_rn(a, a), __dmul_rn(b, b));
}

__device__ __forceinline__ double slit_u(double e, double qk, double limit)
{
    if (e < fabs(qk)) return 0.0;
    if (e > limit) return sq_diff(limit, qk);
    return sq_diff(e, qk);
}

__global__ void __launch_bounds__(256)
slit_smear(int nq, int n_calc, const double *__restrict__ q, const double *__restrict__ width,
           const double *__restrict__ length, int n_length, const double *__restrict__ q_calc,
           const double *__restrict__ edges, const double *__restrict__ theory,
           double *__restrict__ out)
{
    const int i = (int)((blockIdx.x*(size_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (i >= nq) return;
    const double qi = q[i], wi = width[i], li = length[i];
    double acc = 0.0;
    if (wi == 0.0 && li == 0.0) {
        // perfect resolution: the theory at q_calc == q
        for (int j = lane; j < n_calc; j += 32)
            if (q_calc[j] == qi) acc += theory[j];
    } else {
        const int kmax = wi == 0.0 ? 0 : n_length;
        for (int k = -kmax; k <= kmax; ++k) {
            const double qk = kmax ? qi + (k*wi)/n_length : qi;
            const double limit = sqrt(__dadd_rn(__dmul_rn(qk, qk), __dmul_rn(li, li)));
            // bins whose u changes: from the last edge below |qk| to the
            // first edge above the limit
            const int a = max(lower_edge(edges, n_calc + 1, fabs(qk), false) - 1, 0);
            const int b = min(lower_edge(edges, n_calc + 1, limit, true), n_calc);
            for (int j = a + lane; j < b; j += 32) {
                const double w = __dsub_rn(sqrt(slit_u(edges[j + 1], qk, limit)),
                                           sqrt(slit_u(edges[j], qk, limit)))/li;
                acc += w*theory[j];
            }
        }
        acc /= (double)(2*kmax + 1);
    }
    #pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(FULL, acc, off);
    if (lane == 0) out[i] = acc;
}

// ------------------------------------------------- banded weights (plans) --
// A resolution object is applied to new theory curves at every step of a fit
// while its weights never change, so they are formed once (pinhole_weights,
// slit_weights) and each application is a banded product.  Weights of q i:
// w[off[i] + j - lo[i]] for the calculated points lo[i] <= j < hi[i], divided
// by norm[i] after the sum.  A weight of -0.0 marks a point that is not part of
// the sum, whatever the theory there (the steps across a wide slit with a short
// length leave such points between them); no sum forms one by itself.
constexpr long long NO_WEIGHT = 0x8000000000000000ll;        // the bits of -0.0

// One warp per q: the bin masses of pinhole_smear and their sum, in its order.
__global__ void __launch_bounds__(256)
pinhole_weights(int nq, const double *__restrict__ q, const double *__restrict__ width,
                const int32_t *__restrict__ lo, const int32_t *__restrict__ hi,
                const int64_t *__restrict__ off, const double *__restrict__ edges,
                double *__restrict__ w, double *__restrict__ norm)
{
    const int i = (int)((blockIdx.x*(size_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (i >= nq) return;
    const double qi = q[i];
    const double s = SQRT2*width[i];
    double *wi = w + off[i];
    const int a = lo[i], b = hi[i];
    double wsum = 0.0;
    for (int j = a + lane; j < b; j += 32) {
        const double m = erf((edges[j + 1] - qi)/s) - erf((edges[j] - qi)/s);
        wi[j - a] = m;
        wsum += m;
    }
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) wsum += __shfl_xor_sync(FULL, wsum, o);
    if (lane == 0) norm[i] = wsum;
}

// One block per q (bound by the square roots: 61 per edge of the band, 199 us
// per application of 251 q when slit_smear forms them, now once per plan and
// 3 us per application), the steps across the slit (qk and its upper limit) in
// shared memory.  A warp takes 31 bins at a time: lane L forms sqrt(u) at edge
// L of the group and gets the next edge's from lane L + 1, so each (edge,
// step) costs one square root instead of slit_smear's two and its two binary
// searches per step.  A step that does not reach a bin (see slit_smear's searches)
// has equal u at both of its edges and adds 0.
constexpr int SLIT_BATCH = 128;
__global__ void __launch_bounds__(256)
slit_weights(const double *__restrict__ q, const double *__restrict__ width,
             const double *__restrict__ length, int n_length, const double *__restrict__ q_calc,
             const double *__restrict__ edges, const int32_t *__restrict__ lo,
             const int32_t *__restrict__ hi, const int64_t *__restrict__ off,
             double *__restrict__ w, double *__restrict__ norm)
{
    __shared__ double sq[SLIT_BATCH], sl[SLIT_BATCH];
    const int i = blockIdx.x, t = threadIdx.x;
    const int warp = t >> 5, lane = t & 31, warps = (int)blockDim.x >> 5;
    const double qi = q[i], wi = width[i], li = length[i];
    const int a = lo[i], b = hi[i];
    double *out = w + off[i];
    if (wi == 0.0 && li == 0.0) {
        // perfect resolution: the theory at q_calc == q
        if (t == 0) norm[i] = 1.0;
        for (int j = a + t; j < b; j += (int)blockDim.x)
            out[j - a] = q_calc[j] == qi ? 1.0 : __longlong_as_double(NO_WEIGHT);
        return;
    }
    const int kmax = wi == 0.0 ? 0 : n_length;
    const int steps = 2*kmax + 1;
    if (t == 0) norm[i] = (double)steps;
    for (int k0 = 0; k0 < steps; k0 += SLIT_BATCH) {
        const int nk = min(SLIT_BATCH, steps - k0);
        __syncthreads();
        for (int k = t; k < nk; k += (int)blockDim.x) {
            const double qk = kmax ? qi + ((k0 + k - kmax)*wi)/n_length : qi;
            sq[k] = qk;
            sl[k] = sqrt(__dadd_rn(__dmul_rn(qk, qk), __dmul_rn(li, li)));
        }
        __syncthreads();
        for (int j0 = a + 31*warp; j0 < b; j0 += 31*warps) {
            const double edge = edges[min(j0 + lane, b)];
            const double above = __shfl_down_sync(FULL, edge, 1);
            double acc = 0.0;
            bool reached = false;
            #pragma unroll 4
            for (int k = 0; k < nk; ++k) {
                const double r = sqrt(slit_u(edge, sq[k], sl[k]));
                acc += __dsub_rn(__shfl_down_sync(FULL, r, 1), r);
                reached = reached || (above >= fabs(sq[k]) && edge <= sl[k]);
            }
            const int j = j0 + lane;
            if (lane < 31 && j < b) {
                const double part = reached ? acc/li : __longlong_as_double(NO_WEIGHT);
                out[j - a] = k0 == 0 ? part : out[j - a] + part;
            }
        }
    }
}

// One warp per (q, curve): bound by latency and the two streams of doubles;
// taken for one curve and for few (see sasb200_band_apply).  order: the place of each
// q in the output (null: its own).
__global__ void __launch_bounds__(128)
band_apply(int nq, const int32_t *__restrict__ order, const int32_t *__restrict__ lo, const int32_t *__restrict__ hi,
           const int64_t *__restrict__ off, const double *__restrict__ w,
           const double *__restrict__ norm, const double *__restrict__ theory,
           size_t theory_stride, double *__restrict__ out, size_t out_stride)
{
    const int i = (int)((blockIdx.x*(size_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (i >= nq) return;
    const int a = lo[i], n = hi[i] - a;
    const double *wi = w + off[i], *th = theory + blockIdx.y*theory_stride + a;
    double acc = 0.0;
    #pragma unroll 4
    for (int j = lane; j < n; j += 32) {
        const double m = wi[j], x = th[j];
        if (__double_as_longlong(m) != NO_WEIGHT) acc += m*x;
    }
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(FULL, acc, o);
    if (lane == 0) out[blockIdx.y*out_stride + (order ? order[i] : i)] = acc/norm[i];
}

// x/d from r = 1/d, correctly rounded, by one correction of x r with its residual
// (Markstein 1990), which rounds as the division does.  That wants a residual
// without rounding of its own: the division itself where the numerator or the
// quotient is so small that the residual's last bits fall below the smallest number,
// where the quotient is infinite, and for divisors that sr_of refuses (r = 0).
__device__ __forceinline__ double sr_of(double d)
{
    return fabs(d) > 1e-290 && fabs(d) < 1e290 ? 1.0/d : 0.0;
}
__device__ __forceinline__ double quotient(double x, double d, double r)
{
    const double q = x*r;
    const bool normal = fabs(x) > 1e-290 && fabs(q) > 1e-290 && fabs(q) <= 1.7e308;
    return r != 0.0 && normal ? fma(fma(-q, d, x), r, q) : x/d;
}

// c = a b + c on the FP64 tensor pipe: a 16 x 4 (row-major), b 4 x 8, c 16 x 8, as
// fused multiply-adds in the order of the 4 points.  Lane L holds rows L/4 and
// L/4 + 8: of a the column L % 4, of c the columns 2 (L % 4) and the next; of b
// row L % 4 and column L/4.
__device__ __forceinline__ void mma_f64(double (&c)[4], double a0, double a1, double b)
{
    asm volatile("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5}, {%6},"
                 " {%0, %1, %2, %3};"
                 : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3]) : "d"(a0), "d"(a1), "d"(b));
}

// Many curves: a block takes 32 q and 32 curves, a warp 16 q and 16 curves as two
// tiles of the FP64 tensor pipe, which has the rate of the plain one but takes a
// third of the shared-memory reads and few instructions.  The points of the 32
// bands pass through shared memory 16 at a time, the next 16 on their way
// meanwhile.  Sums over 16 points are added to the totals, which keeps the
// rounding error below that of one long sum.  A warp runs over the union of its
// 16 bands, 4 points at a time, with weight 0 outside each; a sum that this leaves
// infinite or undefined is formed again over its own band alone, so that such a
// theory value reaches only the q that see it.
//   Bound by latency: a band is 60 points, four chunks, so that a block is mostly
// its start and the waits between chunks; six blocks per SM hide that best.
// 4096 curves of 1000 q, 5 % width: 35 us (17 at the FP64 rate); 46 with
// multiply-adds (8 q and 64 curves per warp), 38 with 32 curves per warp (four
// blocks), 35-41 with blocks that go on to further curves, 37 with three stages,
// 39 with chunks of 32.  200 curves of 181 q: 4.3 us, 6.2 with multiply-adds.
constexpr int BQ = 32, BQW = 16, BJ = 16, BS = 32, BSW = 16, BWARPS = 4, BTHREADS = 32*BWARPS;
constexpr int BR = BTHREADS/BJ;              // rows staged at once
constexpr int B_LD = BJ + 4;                 // a fragment's 4 points x 8 rows hit all banks

__global__ void __launch_bounds__(BTHREADS, 6)
band_apply_sets(int n_sets, int nq, const int32_t *__restrict__ order,
                const int32_t *__restrict__ lo,
                const int32_t *__restrict__ hi, const int64_t *__restrict__ off,
                const double *__restrict__ w, const double *__restrict__ norm,
                const double *__restrict__ theory, size_t theory_stride,
                double *__restrict__ out, size_t out_stride)
{
    constexpr int TH = 2*BS*B_LD, OUT = BS*(BQ + 1);
    __shared__ double th[TH > OUT ? TH : OUT];       // [2][curve][point]
    __shared__ double ws[2*BQ*B_LD];                 // [2][q][point]
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int q0 = blockIdx.x*BQ, s0 = blockIdx.y*BS;
    const int wq = BQW*(warp & 1), wc = BSW*(warp >> 1);     // this warp's q and curves
    const int qs = q0 + lane;
    const int my_lo = qs < nq ? lo[qs] : 0x7fffffff, my_hi = qs < nq ? hi[qs] : 0;
    const int jmin = __reduce_min_sync(FULL, my_lo), jmax = __reduce_max_sync(FULL, my_hi);
    const int chunks = jmax > jmin ? (jmax - jmin + BJ - 1)/BJ : 0;
    // the union of this warp's bands
    const bool mine = lane/BQW == (warp & 1);
    const int ulo = __reduce_min_sync(FULL, mine ? my_lo : 0x7fffffff);
    const int uhi = __reduce_max_sync(FULL, mine ? my_hi : 0);
    // staging: thread t copies point t % 16 of a chunk, of four curves and of four q
    const int js = t & (BJ - 1), rs = t/BJ;
    const double *tsrc = theory + (size_t)min(s0 + rs, n_sets - 1)*theory_stride + jmin + js;
    const int t_rows = n_sets - s0 - rs;
    int wlo[BQ/BR], whi[BQ/BR];
    const double *wsrc[BQ/BR];
    #pragma unroll
    for (int r = 0; r < BQ/BR; ++r) {
        const int iq = q0 + rs + BR*r;
        wlo[r] = iq < nq ? lo[iq] : 0;
        whi[r] = iq < nq ? hi[iq] : 0;
        wsrc[r] = w + (iq < nq ? off[iq] : 0) - wlo[r];
    }
    auto stage = [&](int c) {
        const int j = jmin + c*BJ + js;
        double *tb = th + (c & 1)*BS*B_LD + rs*B_LD + js;
        double *wb = ws + (c & 1)*BQ*B_LD + rs*B_LD + js;
        const double *src = tsrc + c*BJ;
        if (n_sets - s0 >= BS && jmin + (c + 1)*BJ <= jmax) {
            #pragma unroll
            for (int r = 0; r < BS/BR; ++r) {
                copy8(tb + BR*r*B_LD, src, true);
                src += BR*theory_stride;
            }
        } else {
            #pragma unroll
            for (int r = 0; r < BS/BR; ++r) {
                const bool ok = BR*r < t_rows && j < jmax;
                copy8(tb + BR*r*B_LD, ok ? src : theory, ok);
                src += BR*theory_stride;
            }
        }
        #pragma unroll
        for (int r = 0; r < BQ/BR; ++r) {
            const bool ok = j >= wlo[r] && j < whi[r];
            copy8(wb + BR*r*B_LD, ok ? wsrc[r] + j : w, ok);
        }
        copy_commit();
    };
    constexpr int NT = BSW/8;                        // tiles of 16 q x 8 curves
    double acc[NT][4];
    #pragma unroll
    for (int n = 0; n < NT; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.0;
    if (chunks > 0) stage(0);
    for (int c = 0; c < chunks; ++c) {
        if (c + 1 < chunks) {
            stage(c + 1);
            copy_wait<1>();
        } else {
            copy_wait<0>();
        }
        __syncthreads();
        const int jc = jmin + c*BJ;
        const int first = ulo - jc, last = uhi - jc;
        if (first < BJ && last > 0) {
            const double *wb = ws + (c & 1)*BQ*B_LD + (wq + lane/4)*B_LD + lane % 4;
            const double *tb = th + (c & 1)*BS*B_LD + (wc + lane/4)*B_LD + lane % 4;
            double part[NT][4];
            #pragma unroll
            for (int n = 0; n < NT; ++n) part[n][0] = part[n][1] = part[n][2] = part[n][3] = 0.0;
            #pragma unroll
            for (int k = 0; k < BJ; k += 4) {
                if (k + 4 <= first || k >= last) continue;
                const double a0 = wb[k], a1 = wb[8*B_LD + k];
                #pragma unroll
                for (int n = 0; n < NT; ++n) mma_f64(part[n], a0, a1, tb[8*n*B_LD + k]);
            }
            #pragma unroll
            for (int n = 0; n < NT; ++n)
                #pragma unroll
                for (int e = 0; e < 4; ++e) acc[n][e] += part[n][e];
        }
        __syncthreads();
    }
    // through shared memory, so that rows of 32 q leave together
    #pragma unroll
    for (int n = 0; n < NT; ++n)
        #pragma unroll
        for (int e = 0; e < 4; ++e)
            th[(wc + 8*n + 2*(lane % 4) + (e & 1))*(BQ + 1) + wq + lane/4 + 8*(e >> 1)] = acc[n][e];
    __syncthreads();
    if (qs < nq) {
        const double d = norm[qs], r = sr_of(d);
        const int64_t o = off[qs];
        const int at = order ? order[qs] : qs;
        for (int k = warp; k < BS && s0 + k < n_sets; k += BWARPS) {
            double v = th[k*(BQ + 1) + lane];
            if (!isfinite(v)) {
                v = 0.0;
                const double *src = theory + (s0 + k)*theory_stride;
                for (int j = my_lo; j < my_hi; ++j) v = fma(w[o + (j - my_lo)], src[j], v);
            }
            out[(s0 + k)*out_stride + at] = quotient(v, d, r);
        }
    }
}

// Negative log-likelihood of each curve against one data set
// (bumps_model.py:263-282): 0.5 sum_i ((theory_i - y_i)/dy_i)^2, one block
// per curve, a fixed-order tree over its points.
__global__ void __launch_bounds__(256)
nllf_sets(int nq, const double *__restrict__ theory, size_t theory_stride,
          const double *__restrict__ y, const double *__restrict__ dy, double *__restrict__ out)
{
    const double *th = theory + blockIdx.x*theory_stride;
    double acc = 0.0;
    for (int i = threadIdx.x; i < nq; i += 256) {
        const double r = (th[i] - y[i])/dy[i];
        acc += r*r;
    }
    __shared__ double red[256];
    red[threadIdx.x] = acc;
    for (int s = 128; s > 0; s >>= 1) {
        __syncthreads();
        if ((int)threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    }
    if (threadIdx.x == 0) out[blockIdx.x] = 0.5*red[0];
}

// The same for many curves: a warp per curve, eight curves per block sharing y,
// dy and 1/dy of 256 points in shared memory, so the block divides once per
// point instead of once per (curve, point); each lane's 8 theory values are on
// their way meanwhile.
constexpr int NL_POINTS = 256, NL_CURVES = 8;
__global__ void __launch_bounds__(32*NL_CURVES)
nllf_rows(int n_sets, int nq, const double *__restrict__ theory, size_t theory_stride,
          const double *__restrict__ y, const double *__restrict__ dy, double *__restrict__ out)
{
    __shared__ double sy[NL_POINTS], sd[NL_POINTS], sr[NL_POINTS];
    const int t = threadIdx.x, lane = t & 31;
    const int s = blockIdx.x*NL_CURVES + (t >> 5);
    const double *th = theory + (size_t)min(s, n_sets - 1)*theory_stride;
    double acc = 0.0;
    for (int i0 = 0; i0 < nq; i0 += NL_POINTS) {
        const int n = min(NL_POINTS, nq - i0);
        // this lane's points of the curve, on their way while y and dy are staged
        double x[NL_POINTS/32];
        #pragma unroll
        for (int k = 0; k < NL_POINTS/32; ++k)
            x[k] = 32*k + lane < n ? th[i0 + 32*k + lane] : 0.0;
        __syncthreads();
        for (int i = t; i < n; i += 32*NL_CURVES) {
            const double d = dy[i0 + i];
            sy[i] = y[i0 + i];
            sd[i] = d;
            sr[i] = sr_of(d);
        }
        __syncthreads();
        #pragma unroll
        for (int k = 0; k < NL_POINTS/32; ++k) {
            const int i = 32*k + lane;
            if (i < n) {
                const double z = quotient(x[k] - sy[i], sd[i], sr[i]);
                acc += z*z;
            }
        }
    }
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(FULL, acc, o);
    if (lane == 0 && s < n_sets) out[s] = 0.5*acc;
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

}  // namespace res

extern "C" {

const char *sasb200_resolution_last_error(void) { return res::errbuf(); }

// out[nq] = smeared theory; lo/hi: band [lo_i, hi_i) of calculated points of
// each q (0 <= lo_i <= hi_i <= n_calc); edges[n_calc + 1]; theory[n_calc].
int32_t sasb200_pinhole_smear(int32_t nq, int32_t n_calc, const double *q, const double *width,
                              const int32_t *lo, const int32_t *hi, const double *edges,
                              const double *theory, double *out, void *stream)
{
    res::errbuf()[0] = 0;
    if (nq < 0 || n_calc < 0 || (nq > 0 && (!q || !width || !lo || !hi || !edges || !theory
                                            || !out)))
        return (std::snprintf(res::errbuf(), 256, "bad arguments"), -1);
    if (nq == 0) return 0;
    const int threads = 256;
    const long long warps = nq;
    const unsigned blocks = (unsigned)((warps*32 + threads - 1)/threads);
    res::pinhole_smear<<<blocks, threads, 0, (cudaStream_t)stream>>>(nq, q, width, lo, hi,
                                                                      edges, theory, out, 0, 0);
    return res::status("pinhole_smear");
}

// The same smearing for n_sets curves at once (a fit population sharing one
// data set): theory[s*theory_stride + j], out[s*out_stride + i].
int32_t sasb200_pinhole_smear_sets(int32_t n_sets, int32_t nq, int32_t n_calc, const double *q,
                                   const double *width, const int32_t *lo, const int32_t *hi,
                                   const double *edges, const double *theory,
                                   int64_t theory_stride, double *out, int64_t out_stride,
                                   void *stream)
{
    res::errbuf()[0] = 0;
    if (n_sets < 0 || n_sets > 65535 || nq < 0 || n_calc < 0 || theory_stride < n_calc
        || out_stride < nq || (nq > 0 && n_sets > 0 && (!q || !width || !lo || !hi || !edges
                                                          || !theory || !out)))
        return (std::snprintf(res::errbuf(), 256, "bad arguments"), -1);
    if (nq == 0 || n_sets == 0) return 0;
    const int threads = 256;
    const dim3 grid((unsigned)(((long long)nq*32 + threads - 1)/threads), (unsigned)n_sets);
    res::pinhole_smear<<<grid, threads, 0, (cudaStream_t)stream>>>(
        nq, q, width, lo, hi, edges, theory, out, (size_t)theory_stride, (size_t)out_stride);
    return res::status("pinhole_smear_sets");
}

// The weights of a pinhole resolution for sasb200_band_apply: w[off[i] .. off[i]
// + hi[i] - lo[i]) and norm[nq], from the arrays of sasb200_pinhole_smear.
int32_t sasb200_pinhole_weights(int32_t nq, const double *q, const double *width,
                                const int32_t *lo, const int32_t *hi, const int64_t *off,
                                const double *edges, double *w, double *norm, void *stream)
{
    res::errbuf()[0] = 0;
    if (nq < 0 || (nq > 0 && (!q || !width || !lo || !hi || !off || !edges || !w || !norm)))
        return (std::snprintf(res::errbuf(), 256, "bad arguments"), -1);
    if (nq == 0) return 0;
    const unsigned blocks = (unsigned)(((long long)nq*32 + 255)/256);
    res::pinhole_weights<<<blocks, 256, 0, (cudaStream_t)stream>>>(nq, q, width, lo, hi, off,
                                                                    edges, w, norm);
    return res::status("pinhole_weights");
}

// The weights of a slit resolution for sasb200_band_apply; lo/hi: the bins
// that any step across the slit reaches.
int32_t sasb200_slit_weights(int32_t nq, const double *q, const double *width,
                             const double *length, int32_t n_length, const double *q_calc,
                             const double *edges, const int32_t *lo, const int32_t *hi,
                             const int64_t *off, double *w, double *norm, void *stream)
{
    res::errbuf()[0] = 0;
    if (nq < 0 || n_length < 1 || (nq > 0 && (!q || !width || !length || !q_calc || !edges || !lo
                                               || !hi || !off || !w || !norm)))
        return (std::snprintf(res::errbuf(), 256, "bad arguments"), -1);
    if (nq == 0) return 0;
    res::slit_weights<<<nq, 256, 0, (cudaStream_t)stream>>>(q, width, length, n_length, q_calc,
                                                             edges, lo, hi, off, w, norm);
    return res::status("slit_weights");
}

// out[s*out_stride + i] = sum_j w[off[i] + j - lo[i]] theory[s*theory_stride + j]/norm[i]
// over lo[i] <= j < hi[i], for n_sets curves; to out[s*out_stride + order[i]] where order is
// not NULL.  Neighbouring i should have neighbouring bands: a block of many curves
// reads all points between the first and the last of its 32 (1000 curves and q of 20,000
// points, 1 % width: 82 us in order of q, 2064 in any).
int32_t sasb200_band_apply_ordered(int32_t n_sets, int32_t nq, int32_t n_calc,
                                   const int32_t *order, const int32_t *lo, const int32_t *hi,
                                   const int64_t *off, const double *w, const double *norm,
                                   const double *theory, int64_t theory_stride, double *out,
                                   int64_t out_stride, void *stream)
{
    res::errbuf()[0] = 0;
    if (n_sets < 0 || n_sets > 65535 || nq < 0 || n_calc < 0 || theory_stride < n_calc
        || out_stride < nq || (nq > 0 && n_sets > 0 && (!lo || !hi || !off || !w || !norm
                                                          || !theory || !out)))
        return (std::snprintf(res::errbuf(), 256, "bad arguments"), -1);
    if (nq == 0 || n_sets == 0) return 0;
    cudaStream_t st = (cudaStream_t)stream;
    const size_t ts = (size_t)theory_stride, os = (size_t)out_stride;
    const unsigned qb = (unsigned)((nq + res::BQ - 1)/res::BQ);
    if ((long long)nq*n_sets <= res::BAND_WARP_LIMIT) {
        const dim3 grid((unsigned)((nq + 3)/4), (unsigned)n_sets);
        res::band_apply<<<grid, 128, 0, st>>>(nq, order, lo, hi, off, w, norm, theory, ts, out, os);
    } else {
        const dim3 grid(qb, (unsigned)((n_sets + res::BS - 1)/res::BS));
        res::band_apply_sets<<<grid, res::BTHREADS, 0, st>>>(n_sets, nq, order, lo, hi, off, w, norm,
                                                             theory, ts, out, os);
    }
    return res::status("band_apply");
}

int32_t sasb200_band_apply(int32_t n_sets, int32_t nq, int32_t n_calc, const int32_t *lo,
                           const int32_t *hi, const int64_t *off, const double *w,
                           const double *norm, const double *theory, int64_t theory_stride,
                           double *out, int64_t out_stride, void *stream)
{
    return sasb200_band_apply_ordered(n_sets, nq, n_calc, nullptr, lo, hi, off, w, norm, theory,
                                      theory_stride, out, out_stride, stream);
}

// out[s] = 0.5 sum_i ((theory[s*theory_stride + i] - y[i])/dy[i])^2.
int32_t sasb200_nllf_sets(int32_t n_sets, int32_t nq, const double *theory,
                          int64_t theory_stride, const double *y, const double *dy,
                          double *out, void *stream)
{
    res::errbuf()[0] = 0;
    if (n_sets < 0 || nq < 0 || theory_stride < nq
        || (n_sets > 0 && (!theory || !y || !dy || !out)))
        return (std::snprintf(res::errbuf(), 256, "bad arguments"), -1);
    if (n_sets == 0) return 0;
    if (n_sets > res::NLLF_BLOCKS)
        res::nllf_rows<<<(n_sets + res::NL_CURVES - 1)/res::NL_CURVES, 32*res::NL_CURVES, 0,
                         (cudaStream_t)stream>>>(n_sets, nq, theory, (size_t)theory_stride, y, dy,
                                                 out);
    else
        res::nllf_sets<<<n_sets, 256, 0, (cudaStream_t)stream>>>(nq, theory,
                                                                  (size_t)theory_stride, y, dy,
                                                                  out);
    return res::status("nllf_sets");
}

// Slit smearing: out[i] = sum_j W[i, j] theory[j] with the slit weights of
// sasmodels/resolution.py:223-395 (length only, or width and length with
// 2 n_length + 1 steps across the width); q_calc[n_calc] sorted, edges
// [n_calc + 1].  A nonzero width with a zero length is refused on the host,
// as by the reference.
int32_t sasb200_slit_smear(int32_t nq, int32_t n_calc, const double *q, const double *width,
                           const double *length, int32_t n_length, const double *q_calc,
                           const double *edges, const double *theory, double *out,
                           void *stream)
{
    res::errbuf()[0] = 0;
    if (nq < 0 || n_calc < 0 || n_length < 1 || (nq > 0 && (!q || !width || !length || !q_calc
                                                             || !edges || !theory || !out)))
        return (std::snprintf(res::errbuf(), 256, "bad arguments"), -1);
    if (nq == 0) return 0;
    const int threads = 256;
    const unsigned blocks = (unsigned)(((long long)nq*32 + threads - 1)/threads);
    res::slit_smear<<<blocks, threads, 0, (cudaStream_t)stream>>>(
        nq, n_calc, q, width, length, n_length, q_calc, edges, theory, out);
    return res::status("slit_smear");
}

// out[nq] = sum_b weights[b] theory[b*nq + i] / wsum, bins in order.
int32_t sasb200_pinhole2d_average(int32_t nq, int32_t nbins, const double *theory,
                                  const double *weights, double wsum, double *out, void *stream)
{
    res::errbuf()[0] = 0;
    if (nq < 0 || nbins < 1 || (nq > 0 && (!theory || !weights || !out)))
        return (std::snprintf(res::errbuf(), 256, "bad arguments"), -1);
    if (nq == 0) return 0;
    res::pinhole2d_average<<<(nq + res::P2_THREADS - 1)/res::P2_THREADS, res::P2_THREADS, 0,
                             (cudaStream_t)stream>>>(nq, nbins, theory, weights, wsum, out);
    return res::status("pinhole2d_average");
}

}  // extern "C"
