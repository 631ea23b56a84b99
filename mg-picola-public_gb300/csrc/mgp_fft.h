/* Launch arguments of the power-of-two transform kernels (mgp_fft.cuh), one
 * translation unit per mesh size, and their table. */
#ifndef MGP_FFT_H
#define MGP_FFT_H

#include "mgp_internal.h"

enum { MGP_X_NONE = 0, MGP_X_INV, MGP_X_FORCE, MGP_X_IC };
enum { MGP_Z_R2C = 0, MGP_Z_C2R, MGP_Z_SCREEN, MGP_Z_SOURCE };

/* x pass; strides between boxes in complex values */
typedef struct {
  const float2 *in;
  float2 *spec;      /* FWD: the spectrum */
  const float2 *add; /* X_FORCE, mg_kind 1 and 2: delta(k) */
  float2 *o[3];
  long long bs_in, bs_spec, bs_add, bs_o;
  int nbox;
  const float2 *tw;  /* W_N^m, m = 0..N-1 */
  int filter_kind, filter;  /* mg_kfilter's */
  float kR1, norm;
  const float *gauss;       /* Gaussian smoothing factor per stored index, or NULL */
  int mg_kind;
  float cfac, coupling, mass2;
  const mgp_box_scalars *bs;
  int kc;
  int neg; /* X_FORCE: wave number -N/2 at the Nyquist index (the IC's convention), else +N/2 */
} mgp_fft_x;

/* strides between boxes in complex values */
typedef struct {
  const float2 *in;
  float2 *out[3];
  long long bs_in, bs_out[3];
  int nout, ypow[3], zpow[3];
} mgp_fft_ytask;

typedef struct {
  mgp_fft_ytask task[3];
  int ntask, nbox;
  const float2 *tw;
  int kc, neg;
} mgp_fft_y;

/* z rows; strides between grids in float2 */
typedef struct {
  const float2 *in;             /* real (Z_R2C) or spectra */
  const float2 *grad[6];        /* Z_SOURCE: the gradient spectra of a box, bs_in to the next */
  float2 *out;                  /* spectra */
  float2 *real;                 /* real rows written */
  const float2 *rho;            /* Z_SCREEN: the density */
  long long rows;               /* of all grids */
  long long bs_in, bs_out, bs_real;
  const float2 *tw, *ztw;
  int kc;
  int density;
  float phicrit, coupling, pref, base;
  const mgp_box_scalars *scalars;
} mgp_fft_z;

typedef struct {
  int (*x)(int fwd, int epi, const mgp_fft_x &a, int sms, cudaStream_t st);
  int (*y)(int dir, int gen, const mgp_fft_y &a, int sms, cudaStream_t st);
  int (*z)(int mode, const mgp_fft_z &a, int sms, cudaStream_t st);
  int radix[3];      /* of the row passes */
} mgp_fft_ops;

const mgp_fft_ops *mgp_fft_ops_64(void);
const mgp_fft_ops *mgp_fft_ops_128(void);
const mgp_fft_ops *mgp_fft_ops_256(void);
const mgp_fft_ops *mgp_fft_ops_512(void);
const mgp_fft_ops *mgp_fft_ops_1024(void);

#endif
