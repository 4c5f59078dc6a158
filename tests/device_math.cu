// Test harness: the arithmetic of bc_mech.cuh in its device forms, for
// tests/test_device_math_gpu.py.  Not part of the library.
#include "../braincell_gb300/csrc/bc_mech.cuh"

namespace {
enum { kRcp = 0, kExp2_256, kLn, kDiv, kOverExprel, kOver1pExp, kDivSum };

__global__ void apply_f64(int fn, const double* x, int n, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = fn == kRcp ? bc::srcp(x[i]) : fn == kExp2_256 ? bc::exp2_256(x[i]) : bc::ln_pos(x[i]);
}
__global__ void apply_f32(int fn, const float* a, const float* b, int n, float* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  switch (fn) {
    case kDiv: out[i] = bc::adiv(a[i], b[i]); break;
    case kDivSum: out[i] = bc::adiv_sum(a[i], b[i]); break;
    case kOverExprel: out[i] = bc::over_exprel(a[i], b[i]); break;
    default: out[i] = bc::over_1pexp(a[i], b[i]);
  }
}

template <typename T>
struct Buf {
  T* p = nullptr;
  cudaError_t e;
  explicit Buf(int n) { e = cudaMalloc(reinterpret_cast<void**>(&p), size_t(n) * sizeof(T)); }
  ~Buf() { cudaFree(p); }
};
}  // namespace

// Host arrays of n values; returns the CUDA error code.
extern "C" int bc_test_device_f64(int fn, const double* x, int n, double* out) {
  Buf<double> dx(n), dy(n);
  if (dx.e || dy.e) return int(dx.e ? dx.e : dy.e);
  cudaError_t e = cudaMemcpy(dx.p, x, size_t(n) * 8, cudaMemcpyHostToDevice);
  if (e) return int(e);
  apply_f64<<<(n + 255) / 256, 256>>>(fn, dx.p, n, dy.p);
  e = cudaGetLastError();
  if (e) return int(e);
  return int(cudaMemcpy(out, dy.p, size_t(n) * 8, cudaMemcpyDeviceToHost));
}
extern "C" int bc_test_device_f32(int fn, const float* a, const float* b, int n, float* out) {
  Buf<float> da(n), db(n), dy(n);
  if (da.e || db.e || dy.e) return int(cudaErrorMemoryAllocation);
  cudaError_t e = cudaMemcpy(da.p, a, size_t(n) * 4, cudaMemcpyHostToDevice);
  if (!e) e = cudaMemcpy(db.p, b, size_t(n) * 4, cudaMemcpyHostToDevice);
  if (e) return int(e);
  apply_f32<<<(n + 255) / 256, 256>>>(fn, da.p, db.p, n, dy.p);
  e = cudaGetLastError();
  if (e) return int(e);
  return int(cudaMemcpy(out, dy.p, size_t(n) * 4, cudaMemcpyDeviceToHost));
}
