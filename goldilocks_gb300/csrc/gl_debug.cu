// Device-side checks of the field primitives (gl_field.cuh): one kernel that
// applies a primitive elementwise, so that tests can compare the inline-PTX
// arithmetic with exact integer arithmetic on adversarial inputs (words at
// and above p, all-ones words), which random transform inputs almost never
// produce.  No counterpart in the reference.
#include <cuda_runtime.h>

#include "../../include/goldilocks_gpu.h"
#include "gl_internal.h"

namespace {

__device__ uint64_t apply(int op, uint64_t a, uint64_t b) {
  switch (op) {
    case GL_FOP_ADD: return gl_add(a, b);
    case GL_FOP_SUB: return gl_sub(a, b);
    case GL_FOP_CANON: return gl_canon(a);
    case GL_FOP_MONT_MUL: return gl_mont_mul(a, b);
    case GL_FOP_MUL: return gl_mul(a, b);
    default: break;
  }
  switch (op - GL_FOP_SHL) {
    case 12: return gl_shl<12>(a);
    case 24: return gl_shl<24>(a);
    case 32: return gl_shl<32>(a);
    case 36: return gl_shl<36>(a);
    case 48: return gl_shl<48>(a);
    case 64: return gl_shl<64>(a);
    case 72: return gl_shl<72>(a);
    case 84: return gl_shl<84>(a);
    case 96: return gl_shl<96>(a);
    case 108: return gl_shl<108>(a);
    case 144: return gl_shl<144>(a);
    default: return 0;
  }
}

// The codelets' three-limb operations (GL_FOP_LAZY), compiled shifts.
#define GL_LAZY_SHIFTS(X) X(3) X(12) X(24) X(30) X(32) X(36) X(48) X(60) X(63) X(64) X(72) X(84) X(93)

__device__ uint64_t apply_lazy(int op, uint64_t a, uint64_t b) {
  const gl_l3 x = {(uint32_t)a, (uint32_t)(a >> 32), (uint32_t)(b >> 32)};
  const gl_l3 y = {(uint32_t)b, (uint32_t)(b >> 32), (uint32_t)a};
  gl_l3 r = {0, 0, 0};
  switch (op / 2) {
    case 0: r = gl_ladd(x, y); break;
    case 1: r = gl_lsub(x, y); break;
    case 2: r = gl_ladd(a, b); break;
    case 3: r = gl_lsub(a, b); break;
    case 4: r = gl_lbias<12345>(x); break;
    case 5: r = gl_lnegb<12345>(x); break;
    case 6: r = gl_lnorm(x); break;
    case 7: r = gl_l3_of(gl_lfold(x)); break;
#define GL_LAZY_CASE(K) case 8 + K: r = gl_lshl<K>(x); break;
    GL_LAZY_SHIFTS(GL_LAZY_CASE)
#undef GL_LAZY_CASE
    default: break;
  }
  return op % 2 ? r.x2 : (uint64_t)r.x1 << 32 | r.x0;
}

__global__ void lazy_op_kernel(int op, const uint64_t *a, const uint64_t *b, uint64_t *out, uint64_t n) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    out[i] = apply_lazy(op, a[i], b[i]);
}

bool known_lazy_op(int op) {
  if (op < 0) return false;
#define GL_LAZY_KNOWN(K) || op / 2 == 8 + K
  return op / 2 < 8 GL_LAZY_SHIFTS(GL_LAZY_KNOWN);
#undef GL_LAZY_KNOWN
}

__global__ void field_op_kernel(int op, const uint64_t *a, const uint64_t *b, uint64_t *out, uint64_t n) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    out[i] = apply(op, a[i], b ? b[i] : 0);
}

bool known_op(int op) {
  if (op >= GL_FOP_ADD && op <= GL_FOP_MUL && op != 2) return true;
  const int k = op - GL_FOP_SHL;
  return k == 12 || k == 24 || k == 32 || k == 36 || k == 48 || k == 64 || k == 72 || k == 84 || k == 96 ||
         k == 108 || k == 144;
}

}  // namespace

extern "C" int gl_debug_field_op(int op, const uint64_t *a, const uint64_t *b, uint64_t *out, uint64_t n,
                                 void *stream) {
  const int lazy = op - GL_FOP_LAZY;
  if (!(known_op(op) || (known_lazy_op(lazy) && (b || !n))) || (n && (!a || !out))) return GL_ERR_INVALID;
  if (n == 0) return GL_OK;
  const unsigned blocks = (unsigned)((n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096);
  if (lazy >= 0) {
    lazy_op_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>(lazy, a, b, out, n);
    return gl_cuda_status(cudaGetLastError());
  }
  field_op_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>(op, a, b, out, n);
  return gl_cuda_status(cudaGetLastError());
}
