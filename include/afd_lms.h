/*
 * afd_lms.h - LMS impulse-response estimation on the GPU.
 *
 * Replaces EstimateIr of anc_field_py/ancutil.py:24-37, the reference's
 * identification of an impulse response from a source signal x and a
 * receiver recording d (examples/ie224-noise.py:61,90, dsp.py:48,
 * identification.py:36,54): `epochs` passes of sample-serial LMS with step
 * size mu over the first min(nx, nd) samples, the delay line cleared at the
 * start of each pass and the weights kept, all in FP64. The GPU evaluates
 * the same recursion in blocks of 512 samples (exact up to the order of
 * floating-point additions).
 */
#ifndef AFD_LMS_H
#define AFD_LMS_H

#include <stdint.h>

#include "afd.h"

#ifdef __cplusplus
extern "C" {
#endif

/* w[taps] (host) = the estimate; x, d host arrays. The reference's default
 * is epochs = 16. Returns AFD_OK or AFD_ERR_*. Calls may run on several threads.
 * Device memory of a call (1.1 MB per 512 samples, about 1 GB at most beside the
 * signals) stays with the library for the next one, 1 GB a device at most, until
 * another allocation of this process needs it or afd_lms_release. */
int afd_lms_estimate(const double* x, int64_t nx, const double* d, int64_t nd, int32_t taps, double mu,
                     int32_t epochs, int32_t device, double* w);
/* Gives the device memory kept for later calls back to the device (for other
 * processes, say); calls in progress keep theirs. */
int afd_lms_release(int32_t device);
const char* afd_lms_last_error(void);

#ifdef __cplusplus
}
#endif

#endif
