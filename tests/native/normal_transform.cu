// The division and square root of the normal transform (g4s_device.cuh) against the intrinsics,
// for every float s of the polar method's range.
#include "g4s_device.cuh"

namespace {

// out[0..2]: values of s where the quotient in log s, -2 log(s) / s, or its square root differ
// in any bit; out[3]: the values of s looked at.
__global__ void k_sweep(unsigned first, unsigned last, unsigned long long *out) {
  unsigned long long bad[3] = {0, 0, 0}, seen = 0;
  for (unsigned long long b = first + blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; b < last;
       b += (unsigned long long)gridDim.x * blockDim.x) {
    const float s = __uint_as_float((unsigned)b);
    unsigned mb = ((unsigned)b & 0x7FFFFFu) | 0x3F800000u;
    if (mb > 0x3FB504F3u) mb -= 0x00800000u;
    const float m = __uint_as_float(mb);
    const float num = __fsub_rn(m, 1.0f), den = __fadd_rn(m, 1.0f);
    bad[0] += __float_as_uint(g4s::div_near(num, den)) != __float_as_uint(__fdiv_rn(num, den));
    const float l = __fmul_rn(-2.0f, g4s::log_pos(s)), q = __fdiv_rn(l, s);
    bad[1] += __float_as_uint(g4s::div_near(l, s)) != __float_as_uint(q);
    bad[2] += __float_as_uint(g4s::sqrt_near(q)) != __float_as_uint(__fsqrt_rn(q));
    ++seen;
  }
  for (int k = 0; k < 3; ++k)
    if (bad[k]) atomicAdd(out + k, bad[k]);
  atomicAdd(out + 3, seen);
}

}  // namespace

extern "C" int sweep_normal_transform(unsigned first, unsigned last, unsigned long long *h_out) {
  unsigned long long *out = nullptr;
  cudaError_t e = cudaMalloc((void **)&out, 4 * sizeof(*out));
  if (e == cudaSuccess) e = cudaMemset(out, 0, 4 * sizeof(*out));
  if (e == cudaSuccess) {
    k_sweep<<<1024, 256>>>(first, last, out);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(h_out, out, 4 * sizeof(*out), cudaMemcpyDeviceToHost);
  cudaFree(out);
  return (int)e;
}
