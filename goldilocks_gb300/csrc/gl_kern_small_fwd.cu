// Four-lane pass kernels of fixed radices for the sizes with a factor 3, 5 or
// 17 that plans of up to 2^16 points and interleaved columns reach with the
// run-time-radix kernel (forward).  They run in its place (same radices, same four
// lanes): its 256 threads hold 32 groups at 120 points, and its switch over the
// radices takes more registers.  Measured on GB300 (us): 15 360 points 19.0 ->
// 9.4, 64 transforms of 61 440 116 -> 48.6, 1 000 of 255 16.8 -> 6.6.
#include "gl_kernels_impl.cuh"

static const gl_kernel_entry k_entries[] = {
    GL_ENTRY3M(17, 4, 1, 4, 68, 8, false),   GL_ENTRY3M(16, 5, 1, 4, 64, 8, false),
    GL_ENTRY3M(16, 6, 1, 4, 64, 8, false),   GL_ENTRY3M(15, 8, 1, 4, 64, 8, false),
    GL_ENTRY3M(17, 8, 1, 4, 68, 8, false),   GL_ENTRY3M(16, 10, 1, 4, 64, 8, false),
    GL_ENTRY3M(16, 12, 1, 4, 64, 8, false),  GL_ENTRY3M(17, 12, 1, 4, 68, 8, false),
    GL_ENTRY3M(16, 15, 1, 4, 64, 8, false),  GL_ENTRY3M(17, 15, 1, 4, 68, 8, false),
    GL_ENTRY3M(17, 15, 2, 4, 136, 4, false), GL_ENTRY3M(17, 16, 3, 4, 272, 3, false),
    GL_ENTRY3M(16, 15, 4, 4, 256, 4, false), GL_ENTRY3M(17, 15, 4, 4, 272, 3, false),
};

const gl_kernel_entry *gl_kernels_small_fwd(size_t *count) {
  *count = sizeof(k_entries) / sizeof(k_entries[0]);
  return k_entries;
}
