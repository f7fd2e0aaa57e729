// lines3.cuh -- FP32 transforms with the rounding of the three-radix plans.
//
// press_stag_array on real(8) host arrays of an FP32-storage context returns FP32-accurate
// numbers in a type that resolves far more.  Another factorisation of the transforms is as
// exact (5.2e-7 against 5.3e-7 from 64 bits) but rounds differently, 3e-7 to 6e-7 of the
// field, which a caller who compares or restarts real(8) results sees; and the two-pass
// kernels gain that call nothing, its host copies being an order longer than its kernels.
// So it keeps the three-radix plans of fft2.cuh with one scalar instruction per component,
// whose results stay what they were to the bit.
#pragma once
#include "lines.cuh"

namespace obl {

// Rows: OP_FWD (real rows -> half spectra, x-Nyquist zeroed) or OP_INV (half spectra -> real
// rows; pad_mode is not served).  twF / twB: the three-radix tables of n (ROLE_FWD, ROLE_BWD).
cudaError_t launch_rows3(int op, int n, const RowArgs<float> &a, cudaStream_t s);
// Complex columns: OP_FWD (zero_nyq honoured) or OP_INV; kmul multiplies the input of OP_INV
// by i*ktab[column] (1) or i*ktab[row] (2).
cudaError_t launch_cols3(int op, int n, const ColArgs<float> &a, int kmul, cudaStream_t s);

} // namespace obl
