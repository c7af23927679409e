// Four-step column/row pass kernels of 1024 and 2048 points with two lanes per
// 256-thread CTA and four CTAs per SM (forward): the schedules nearest sqrt(n),
// for launches of up to two four-lane tiles per SM.  More tiles take the
// four-lane kernels in 512 threads (measured at gl_contiguous_pass).
#include "gl_kernels_impl.cuh"

static const gl_kernel_entry k_entries[] = {
    GL_ENTRY3M(16, 16, 8, 2, 256, 4, false),
    GL_ENTRY3M(16, 8, 8, 2, 256, 4, false),
};

const gl_kernel_entry *gl_kernels_pass2_fwd(size_t *count) {
  *count = sizeof(k_entries) / sizeof(k_entries[0]);
  return k_entries;
}

// Passes up to 512 points over interleaved columns (C > 1): 8-32 adjacent
// columns per CTA read 64-256-byte row pieces and fill a 256-512-thread CTA.
static const gl_kernel_entry k_col_entries[] = {
    GL_ENTRY3C(8, 8, 8, 8, 512, 2, false),
    GL_ENTRY3C(16, 16, 1, 16, 256, 4, false),
    GL_ENTRY3C(16, 8, 1, 32, 256, 4, false),
    GL_ENTRY3C(8, 8, 1, 32, 256, 4, false),
};

// 1024 and 2048 points in eight lanes: with the entries above, the passes that
// read or write host memory (64-byte pieces) and three-pass columns.
static const gl_kernel_entry k_wide_entries[] = {
    GL_ENTRY3M(16, 8, 8, 8, 512, 2, false),
    GL_ENTRY3M(16, 16, 8, 8, 1024, 1, false),
};

const gl_kernel_entry *gl_kernels_wide_fwd(size_t *count) {
  *count = sizeof(k_wide_entries) / sizeof(k_wide_entries[0]);
  return k_wide_entries;
}

const gl_kernel_entry *gl_kernels_cols_fwd(size_t *count) {
  *count = sizeof(k_col_entries) / sizeof(k_col_entries[0]);
  return k_col_entries;
}
