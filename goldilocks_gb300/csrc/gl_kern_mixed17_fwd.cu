// Four-lane pass kernels for the pass sizes with a factor 17 that the default splits of the
// lengths 17, 51, 85, 255 x 2^k reach, compiled instead of the run-time-radix kernel
// (forward).  A unit of its own so that the pass kernels compile in parallel.
#include "gl_kernels_impl.cuh"

static const gl_kernel_entry k_entries[] = {
    GL_ENTRY3(16, 15, 17, 4, 1024, false),
    GL_ENTRY3T(16, 8, 17, 4, 1024, 272, 3, false, 3),
    GL_ENTRY3T(8, 15, 17, 4, 1024, 272, 3, false, 4),
    GL_ENTRY3T(16, 10, 17, 4, 1024, 384, 2, false),
    GL_ENTRY3T(16, 12, 17, 4, 1024, 416, 2, false),
    // Up to 1632 points: 512 threads for few tiles.
    GL_ENTRY3T(16, 5, 17, 4, 512, 192, 4, false, 3),
    GL_ENTRY3M(16, 6, 17, 4, 512, 2, false),
    GL_ENTRY3T(16, 4, 17, 4, 512, 272, 3, false),
    // 272..680 points (lengths up to about 2^19).  Second form, rows of
    // 512 x m, 16 and 4 transforms (13 and 3.4 tiles per SM): m = 680 1.08 and
    // 0.93, 544 1.11 and 0.88, 408 1.13 and 1.07, 340 1.18 and 0.95 times as
    // fast.  (1632 points gained nothing: 1.00 and 0.93.)
    // 68 threads: the 68 groups of round 1 in one walk (64 threads took two;
    // 139 264 points 14.3 -> 13.0 us).
    GL_ENTRY3M(16, 17, 1, 4, 68, 8, false),
    GL_ENTRY3T(16, 17, 2, 4, 256, 144, 6, false, 8),
    GL_ENTRY3T(8, 5, 17, 4, 256, 192, 5, false, 8),
    GL_ENTRY3T(8, 3, 17, 4, 256, 208, 4, false, 3),
    GL_ENTRY3T(17, 10, 2, 4, 256, 136, 6, false, 8),
};

const gl_kernel_entry *gl_kernels_mixed17_fwd(size_t *count) {
  *count = sizeof(k_entries) / sizeof(k_entries[0]);
  return k_entries;
}
