// Four-lane pass kernels for the pass sizes with a factor 3 or 5 that the default splits of the
// lengths 3, 5, 15 x 2^k reach, compiled instead of the run-time-radix kernel
// (forward).  A unit of its own so that the pass kernels compile in parallel.
#include "gl_kernels_impl.cuh"

static const gl_kernel_entry k_entries[] = {
    GL_ENTRY3T(16, 16, 6, 4, 1024, 192, 4, false, 3),
    GL_ENTRY3T(16, 16, 10, 4, 1024, 320, 2, false),
    // 680 column tiles (8 355 840 points) ran 1 % slower in the second form,
    // 1 024 row tiles (12 582 912) 5 % faster.
    GL_ENTRY3T(16, 16, 12, 4, 1024, 384, 2, false, 5),
    GL_ENTRY3(16, 16, 15, 4, 1024, false),
    GL_ENTRY3T(16, 16, 5, 4, 1024, 160, 5, false, 4),
    GL_ENTRY3T(16, 15, 8, 4, 1024, 256, 3, false),
    // 320..768 points (lengths up to about 2^19): 256 threads for few tiles.
    // Rows of 512 x m, 16 transforms (13 tiles per SM), second form: m = 768
    // 1.13, 640 1.11, 480 1.15, 384 1.20, 320 1.26 times as fast; 4 transforms
    // (3.4 per SM): 1.10, 1.05, 0.81, 0.78, 1.23, so the line lies at 3 or 8.
    GL_ENTRY3T(16, 16, 3, 4, 256, 192, 5, false, 3),
    GL_ENTRY3T(16, 10, 4, 4, 256, 160, 6, false, 3),
    GL_ENTRY3T(16, 15, 2, 4, 256, 128, 8, false, 8),
    GL_ENTRY3T(16, 8, 3, 4, 256, 96, 10, false, 8),
    GL_ENTRY3T(16, 10, 2, 4, 256, 128, 8, false, 3),
};

const gl_kernel_entry *gl_kernels_mixed35_fwd(size_t *count) {
  *count = sizeof(k_entries) / sizeof(k_entries[0]);
  return k_entries;
}
