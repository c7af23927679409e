// Run-time-radix pass kernel, inverse direction.
#include "gl_kern_generic_impl.cuh"

void gl_launch_generic_inv(const gl_pass_args &args, dim3 grid, cudaStream_t stream, bool pdl) {
  gl_launch_generic<true>(args, grid, stream, pdl);
}

const void *gl_generic_kernel_inv() { return (const void *)gl_generic_kernel<true>; }
