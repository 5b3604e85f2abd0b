// Launchers shared by the likelihood translation units (pmatrix.cu).
#pragma once
#include "pgpu_internal.cuh"

// Eigendecomposition of n_models reversible S x S rate matrices (device
// buffers).  status_dev[m] receives 0 or a PGPU_ERR_* code per model.
pgpu_status pgpu_launch_eig(pgpu_ctx *ctx, const double *Q_dev, const double *pi_dev, int S,
                            int n_models, double *U_dev, double *lam_dev, double *Ui_dev,
                            int *status_dev);

// P[b][r] = U diag(exp(lambda * rates[r] * t[b])) Ui for n_br branch lengths
// of one model; FP64 into P_dev and/or FP32 into P32_dev (either may be
// null).  With allow_q, t == -1 yields Q (MlModel.compose's special case).
// If status_dev is given and non-zero the matrices are not built and the
// context's error word records the model failure.  p32_mode selects the FP32
// copy: P, P - I (formed in FP64 before rounding, which keeps the small
// entries of short branches at full relative precision), or P as (hi, lo)
// float pairs in the pair form's row-pair layout.
enum P32Mode {
  P32_PLAIN = 0,          // fl32(P)
  P32_MINUS_I = 1,        // fl32(P - I)
  // (hi, lo) float pairs of a 4 x 4 P, rows taken two at a time for packed
  // float2 arithmetic: float4 k = 4 (i / 2) + j of a block holds
  // {hi P[i][j], hi P[i+1][j], lo P[i][j], lo P[i+1][j]} for even i
  P32_PAIRS_ROWS4 = 4
};
pgpu_status pgpu_launch_compose(pgpu_ctx *ctx, const double *U_dev, const double *lam_dev,
                                const double *Ui_dev, int S, const double *t_dev, int n_br,
                                const double *rates_dev, int R, double *P_dev, float *P32_dev,
                                bool allow_q, const int *status_dev = nullptr,
                                int p32_mode = P32_PLAIN);

// Tip rows tab[t][r][c][i] = (P(t, r) code_tab[c])[i] for the n_tips branches
// above the tips (t_dev holds their lengths), in FP64, stored as float
// (form 0), double (form 2), or for S = 4 float pairs with the elements two at a time, {h0, h1, l0, l1}, {h2, h3,
// l2, l3} per code (form 3, the pair form's packed layout).
pgpu_status pgpu_launch_tip_table(pgpu_ctx *ctx, const double *U_dev, const double *lam_dev,
                                  const double *Ui_dev, int S, const double *t_dev, int n_tips,
                                  const double *rates_dev, int R, const double *code_tab_dev,
                                  int n_codes, void *out_dev, int form, const int *status_dev);

// The setup of a pruning call over 4 states in one launch (dna_setup_kernel):
// the P matrices of the 2 n_tips - 2 branches and the tips' rows, rate
// classes interleaved, for the form `precision` (32: P - I, 48: float pairs,
// 64: double), model m at P_stride and rows_stride bytes.  Clears done_dev[m]
// and row_flag_dev[m][n_flags].
pgpu_status pgpu_launch_dna_setup(pgpu_ctx *ctx, const double *U_dev, const double *lam_dev,
                                  const double *Ui_dev, int n_models, const double *t_dev, int n_tips,
                                  const double *rates_dev, int R, int RT, const double *code_tab_dev,
                                  int n_codes, int precision, void *P_dev, size_t P_stride, void *rows_dev,
                                  size_t rows_stride, const int *status_dev, unsigned *done_dev,
                                  int *row_flag_dev, int n_flags);

// Eigen system of one reversible 4 x 4 rate matrix on the host; 0 or a
// PGPU_ERR_* status as the GPU solver gives.
int pgpu_host_eig4(const double *Q, const double *pi, double *U, double *lam, double *Ui);
