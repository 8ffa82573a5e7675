// Phases of the row operators (rows_op.cu, rows_op_mma.cu), as indices into the 8N roots of unity exp(2 pi i j / 8N).
#pragma once

namespace adrt {

// column c of the output: the conjugate of D_c = z_k^(c/2) is applied
template <int n> __device__ __forceinline__ int op_phase_out(int k, int c) { return (2 * k * c) & ((8 << n) - 1); }
// entry c of the input: D_c (G), or the conjugate of beta_c = z_k^((2c - N + 1)/4) (BP, c the slope)
template <int n> __device__ __forceinline__ int op_phase_in(int k, int c, bool bp) {
    return (bp ? -k * (2 * c - (1 << n) + 1) : 2 * k * c) & ((8 << n) - 1);
}

}  // namespace adrt
