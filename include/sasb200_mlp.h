/*
 * sasb200_mlp.h -- C-ABI of libsasb200_mlp.so (the learned I(q) surrogate)
 * and of libsasb200_peaks.so (the pipe-throughput probes used as roofline
 * denominators).
 *
 * No counterpart in the reference: sasmodels has no learned surrogate and
 * no throughput probes.  The network is 16 (7 used) -> 4 x 256 SiLU -> 1
 * with BF16 operands, compensated (hi + lo) BF16 activations and FP32
 * accumulation in tensor memory (tcgen05).  All pointers are device
 * pointers; bf16 tensors are passed as void*.  Every function returns 0 on
 * success, -1 for a bad argument, -3 for a CUDA launch error;
 * sasb200_mlp_last_error() describes the last failure on the calling host
 * thread.  Kernels with pipeline waits write a nonzero value to *err when a
 * bounded wait runs out (the kernel then unwinds instead of hanging).
 * n_pad is n rounded up to a multiple of 128 (one tile of rows).
 */
#ifndef SASB200_MLP_H
#define SASB200_MLP_H

#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

const char *sasb200_mlp_last_error(void);

/* features: the compensated BF16 pair x + x_lo [n_pad x 16] from float64
 * per-point inputs (radius, length, radius pd, length pd, contrast, q,
 * orientation flag); rows >= n are zero. */
int32_t sasb200_mlp_features(int32_t n, int32_t n_pad, const double *radius,
                             const double *length, const double *rpd, const double *lpd,
                             const double *drho, const double *q, const double *flag,
                             void *x, void *x_lo, void *stream);

/* the same for n points in runs that share a parameter set: run r covers starts[r] <=
 * i < starts[r + 1] (starts[0] = 0, the last run ends at n), table[runs x 7] =
 * (radius, length, radius pd, length pd, contrast, flag, inside the domain); and, from
 * the networks' outputs there, I = exp(out y_std + y_mean + 2 log|contrast|) and
 * accept (inside, q in [q_lo, q_hi] and gate g_std + g_mean <= thr; gate NULL: 0). */
int32_t sasb200_features_runs(int32_t n, int32_t n_pad, int32_t runs, const int32_t *starts,
                              const double *table, const double *q, void *x, void *x_lo,
                              void *stream);
int32_t sasb200_finish_runs(int32_t n, int32_t runs, const int32_t *starts, const double *table,
                            const double *q, const float *out, const float *gate, double y_std,
                            double y_mean, double g_std, double g_mean, double thr, double q_lo,
                            double q_hi, double *I, uint8_t *accept, void *stream);

/* pipelined forward: the weights packed once by sasb200_mlp_pack into an
 * image of sasb200_mlp_image_bytes() bytes (16-byte aligned); out[n], and
 * for training the z/h planes [4][n_pad x 256] bf16 (both NULL for
 * inference); persistent grid of at most `blocks` CTAs (0 = one per SM). */
int32_t sasb200_mlp_image_bytes(void);
int32_t sasb200_mlp_pack(const void *w0, const void *w1, const void *w2, const void *w3,
                         void *img, void *stream);
int32_t sasb200_mlp_infer(int32_t n, int32_t n_pad, const void *x, const void *x_lo,
                          const void *img, const float *const *b, const float *w_out,
                          const float *b_out, float *out, void *z_save, void *h_save,
                          int32_t *err, int32_t blocks, void *stream);

/* the same forward through the overlapped kernels (a dedicated MMA warp, layer
 * l+1's MMAs running under layer l's epilogue chunk by chunk), same image and
 * arguments: two SMs per tile of 128 rows while 2 n_pad/128 CTAs may run at
 * once, then a tile per SM, then pairs of SMs with two tiles each in flight;
 * with planes always a tile per SM.  The values do not depend on the choice.
 * Hidden activations and the z/h planes bitwise those of sasb200_mlp_infer; out
 * differs only by the order of the output dot's sums.  *err receives 1, 2, 3 or
 * 4 if a pipeline wait ran out. */
int32_t sasb200_mlp_serve(int32_t n, int32_t n_pad, const void *x, const void *x_lo,
                          const void *img, const float *const *b, const float *w_out,
                          const float *b_out, float *out, void *z_save, void *h_save,
                          int32_t *err, int32_t blocks, void *stream);

/* pipelined backward (training): W3^T, W2^T, W1^T packed once per weight
 * update by sasb200_mlp_pack_t into sasb200_mlp_image_t_bytes() bytes; dZ
 * planes [4][n_pad x 256] bf16 from dout and the saved pre-activations. */
int32_t sasb200_mlp_image_t_bytes(void);
int32_t sasb200_mlp_pack_t(const void *wt1, const void *wt2, const void *wt3, void *img_t,
                           void *stream);
int32_t sasb200_mlp_backward_p(int32_t n, int32_t n_pad, const void *img_t, const float *w_out,
                               const float *dout, const void *z_save, void *dz_save,
                               int32_t *err, int32_t blocks, void *stream);

/* training: forward with saved pre-activations and activations
 * (z_save, h_save: [4][n_pad x 256] bf16 each, or both NULL), backward
 * through the hidden layers (wt: transposed bf16 weights),
 * Huber loss gradient, Adam (also refreshing the bf16
 * copies w and, if non-NULL, the transposed wt). */
int32_t sasb200_mlp_forward(int32_t n, int32_t n_pad, const void *x, const void *x_lo,
                            const void *const *w, const float *const *b, const float *w_out,
                            const float *b_out, float *out, void *z_save, void *h_save,
                            int32_t *err, void *stream);
int32_t sasb200_mlp_backward(int32_t n, int32_t n_pad, const void *const *wt,
                             const float *w_out, const float *dout, const void *z_save,
                             void *dz_save, int32_t *err, void *stream);
int32_t sasb200_loss_grad(int32_t n, int32_t n_pad, const float *out, const float *y,
                          float delta, float *dout, float *loss, void *stream);
int32_t sasb200_adam(int32_t size, int32_t splits, const float *grad, float *p, float *m,
                     float *v, float lr, float b1, float b2, float eps, int32_t step, void *w,
                     void *wt, int32_t rows, int32_t cols, void *stream);

/* Loss and gradients of one batch, on tiled planes [4 layers][n_pad/128 tiles][32
 * groups][128 rows][8] bf16 (group g holds columns 8g .. 8g + 7): the forward
 * (out[n], z, h) with the loss gradient dout[n_pad] of the mean Huber loss (delta
 * <= 0: squared error) against y[n] and row_sums[2][n_pad/32] (loss and dout
 * summed over 32 rows each); the backward (dz); every gradient as partial sums
 * over splits of the rows (dw[l]: [splits][256 x (16 or 256)], 32-byte aligned,
 * db: [4][splits][256], dw_out: [splits][256]), the mean loss and db_out as
 * scalars; then, for k < sums (at most 16), sum_outs[k][i] = sum of
 * sum_parts[k][s*sum_sizes[k] + i] over s < sum_splits[k].
 *
 * A captured step takes a batch (else NULL): x, x_lo and y then receive the rows
 * idx[n] of the data set (x_all, x_lo_all [rows x 16] bf16, y_all[rows]) first,
 * and the schedule advances as by sasb200_lr_schedule.  An index outside the set
 * leaves zeros, *err = 5, sched[3] = 1 (sched has four floats, the last 0 before the
 * first step), *refused = 1 (memory that the host reads, page-locked) and an undefined
 * loss; see sasb200_adam_pack. */
typedef struct sasb200_mlp_batch {
    const int64_t *idx;
    int64_t rows;
    const void *x_all, *x_lo_all;
    const float *y_all;
    int32_t *counters;
    float *sched;
    int32_t *refused;
    int32_t total, warmup;
    float lr0, b1, b2;
} sasb200_mlp_batch;
typedef struct sasb200_mlp_pass {
    int32_t n, n_pad, splits;
    float delta;
    const void *x, *x_lo;
    const float *y;
    const void *img, *img_t;       /* sasb200_mlp_pack, sasb200_mlp_pack_t */
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
} sasb200_mlp_pass;
int32_t sasb200_mlp_train_pass(const sasb200_mlp_pass *pass, void *stream);

/* Adam for the whole network in one launch (host arrays of 10 device pointers:
 * W0..W3, b0..b3, w_out, b_out, with splits[k] partial gradients each) with the
 * bf16 weights w[4], transposes wt[4] and both weight images; lr and the bias
 * corrections from sched (sasb200_lr_schedule), or from lr and step when it is
 * NULL.  Where the fourth float of sched is not 0, nothing is updated. */
int32_t sasb200_adam_pack(const float *const *grads, const int32_t *splits, float *const *p,
                          float *const *m, float *const *v, void *const *w, void *const *wt,
                          void *img, void *img_t, const float *sched, float lr, int32_t step,
                          float b1, float b2, float eps, void *stream);

/* the learning rate and Adam bias corrections of a training step, on the
 * device: counters = {schedule step s, Adam step count t} (int32), sched =
 * {lr, 1 - b1^t, 1 - b2^t} with lr = lr0 min(1, (s + 1)/warmup)
 * (1 + cos(pi s/total))/2, then s and t advance by one.  A CUDA graph of a
 * whole training step replays with these. */
int32_t sasb200_lr_schedule(int32_t *counters, float *sched, int32_t total, int32_t warmup,
                            float lr0, float b1, float b2, void *stream);

/* out[c] = sum over r of M[r][c] (times v[r] when v is non-NULL) for a
 * row-major bf16 [rows x cols] matrix, in a fixed order: partial sums of
 * 64-row blocks into part (sasb200_col_sum_parts(rows) x cols floats), then
 * each column's partials combined in a fixed order (one warp per column). */
int32_t sasb200_col_sums(int32_t rows, int32_t cols, const void *M, const float *v, float *part,
                         float *out, void *stream);
int32_t sasb200_col_sum_parts(int32_t rows);

/* libsasb200_peaks.so: dependent-chain throughput probes (FP64 FMA, FP32
 * FMA, MUFU sine) whose measured rates are the roofline peaks of the
 * FP64 and FP32-compensated kernels. */
int32_t sasb200_probe_fp64_fma(double *out, int32_t blocks, int32_t iters, void *stream);
int32_t sasb200_probe_fp32_fma(float *out, int32_t blocks, int32_t iters, void *stream);
int32_t sasb200_probe_mufu_sin(float *out, int32_t blocks, int32_t iters, void *stream);
int32_t sasb200_probe_threads_per_block(void);
int32_t sasb200_probe_chains(void);

#ifdef __cplusplus
}
#endif

#endif /* SASB200_MLP_H */
