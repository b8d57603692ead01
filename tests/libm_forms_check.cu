// tests/libm_forms_check.cu -- on the device: the branch-free forms of ww3-gpu_b200/csrc/libm_dev.cuh and
// srce_point.cuh against the general functions and IEEE division (libm_device_check.cu holds those to
// glibc), where the reciprocal's seed is rcp.approx and not the host's division. Unary forms take all
// float bit patterns of their range, the others seeded pairs drawn over their range. Prints a line per form:
// name, arguments inside the range, mismatches.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>

#include "../ww3-gpu_b200/csrc/srce_point.cuh"

namespace {

using namespace wwb;

enum Form { kDivCore, kDivBy, kAtan2, kPowMid, kExpNeg, kExpQ, kLogQ, kPowCore, kSincos, kForms };
const char* const kNames[kForms] = {"div_core", "div_by", "atan2f_core", "powf_mid", "expf_neg",
                                    "expf_q",   "logf_q", "powf_core",   "sincosf_core"};

__device__ uint64_t mix(uint64_t i) {
  uint64_t h = (i + 1) * 0x9E3779B97F4A7C15ULL;
  h ^= h >> 29;
  h *= 0xBF58476D1CE4E5B9ULL;
  h ^= h >> 32;
  return h;
}
__device__ bool diff(float a, float b) {
  return dm::asuint(a) != dm::asuint(b) && !(a != a && b != b);
}
/// Sign and mantissa of `bits`, exponent field lo + e % n.
__device__ float spread(uint32_t bits, uint32_t e, uint32_t lo, uint32_t n) {
  return dm::asfloat((bits & 0x807fffffu) | (lo + e % n) << 23);
}

/// 0: not in the form's range, 1: equal, 2: different.
__device__ int check(int form, uint64_t i) {
  const uint64_t h = mix(i), g = mix(h);
  const uint32_t u = static_cast<uint32_t>(h), v = static_cast<uint32_t>(h >> 32);
  const uint32_t e = static_cast<uint32_t>(g), d = static_cast<uint32_t>(g >> 32);
  const float any = dm::asfloat(static_cast<uint32_t>(i));
  switch (form) {
    case kDivCore: {
      float b = spread(v, d, 67, 121);
      if (i % 4 == 0) b = dm::asfloat((dm::asuint(b) | 0x7fffffu) - (e >> 28));  // mantissas next to all ones
      const float a = i % 8 == 1 ? spread(u & 0x80000007u, e, 67, 121) : spread(u, e, 67, 121);
      if (!dm::div_ok(a, b)) return 0;
      return diff(dm::div_core(a, b), a / b) ? 2 : 1;
    }
    case kDivBy: {
      const float a = i % 16 == 0 ? 0.0f : dm::asfloat(u), b = ::fabsf(spread(v, d, 107, 40));
      if (dm::asuint(a) == 0x80000000u) return 0;  // -0 gives +0
      return diff(pt::div_by(a, b, 1.0f / b), a / b) ? 2 : 1;
    }
    case kAtan2: {
      const float y = spread(u, e, 67, 121), x = dm::asfloat((v & 0x807fffffu) |
          ((dm::asuint(y) >> 23 & 0xff) + d % 49 - 24) << 23);
      if (!dm::atan2f_ok(y, x)) return 0;
      bool bad = false;
      const float r = dm::atan2f_core(y, x, &bad);
      if (bad) return 0;
      return diff(r, dm::atan2f(y, x)) ? 2 : 1;
    }
    case kPowMid: {
      const float x = spread(u & 0x7fffffffu, e, 120, 8), y = static_cast<float>(v) * 0x1p-32f * 16.0f;
      if (!(x < 2.0f && y > 0.0f && y < 16.0f)) return 0;
      return diff(dm::powf_mid(x, y), dm::powf(x, y)) ? 2 : 1;
    }
    case kExpNeg: return any < 0.0f ? (diff(dm::expf_neg(any), dm::expf(any)) ? 2 : 1) : 0;
    case kExpQ: return diff(dm::expf_q(any), dm::expf(any)) ? 2 : 1;
    case kLogQ: return diff(dm::logf_q(any), dm::logf(any)) ? 2 : 1;
    case kPowCore: return dm::normal_pos(any) ? (diff(dm::powf_core(any, 0.25f), dm::powf(any, 0.25f)) ? 2 : 1) : 0;
    default: {
      if (!(any > -120.0f && any < 120.0f)) return 0;
      float s, c, s2, c2;
      dm::sincosf(any, &s, &c);
      dm::sincosf_core(any, &s2, &c2);
      return diff(s, s2) || diff(c, c2) ? 2 : 1;
    }
  }
}

__global__ void run(int form, uint64_t n, unsigned long long* out) {
  unsigned long long seen = 0, bad = 0;
  for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    const int r = check(form, i);
    seen += r != 0;
    bad += r == 2;
  }
  atomicAdd(out, seen);
  atomicAdd(out + 1, bad);
}

}  // namespace

int main() {
  unsigned long long* d = nullptr;
  if (cudaMalloc(&d, 2 * sizeof *d) != cudaSuccess) return 3;
  for (int form = 0; form < kForms; ++form) {
    unsigned long long h[2] = {};
    cudaMemset(d, 0, sizeof h);
    run<<<148 * 8, 256>>>(form, form < kExpNeg ? 1ULL << 30 : 1ULL << 32, d);
    if (cudaMemcpy(h, d, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) {
      std::fprintf(stderr, "CUDA error: %s\n", cudaGetErrorString(cudaGetLastError()));
      return 3;
    }
    std::printf("%s %llu %llu\n", kNames[form], h[0], h[1]);
  }
  cudaFree(d);
  return 0;
}
