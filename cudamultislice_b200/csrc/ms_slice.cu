// ms_slice.cu -- routing of the fused slice passes by line length and plan
// variant (kernels in ms_slice_impl.cuh, one translation unit per length).
#include "ms_slice_impl.cuh"
#include "ms_unit.h"

namespace ms {

namespace {
template <class F>
cudaError_t by_length(int n, F&& f) {
  switch (n) {
    case 64: return f(std::integral_constant<int, 64>());
    case 128: return f(std::integral_constant<int, 128>());
    case 256: return f(std::integral_constant<int, 256>());
    case 512: return f(std::integral_constant<int, 512>());
    case 1024: return f(std::integral_constant<int, 1024>());
    case 2048: return f(std::integral_constant<int, 2048>());
    case 4096: return f(std::integral_constant<int, 4096>());
    default: return cudaErrorInvalidValue;
  }
}
bool supported_length(int n) { return n >= 64 && n <= 4096 && (n & (n - 1)) == 0; }
}  // namespace

bool fused_supported(int nx, int ny) { return supported_length(nx) && supported_length(ny); }

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link to
// the driver library), looked up once.
bool wave_tensor_map(CUtensorMap* m, const float2* base, int nx, int ny, int cb) {
  using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static Encode encode = []() -> Encode {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return nullptr;
    return reinterpret_cast<Encode>(fn);
  }();
  if (!encode || ((uintptr_t)base & 15) || nx <= 0 || ny <= 0 || ((size_t)nx * sizeof(float2)) % 16 ||
      (2 * cb * (int)sizeof(float)) % 16 || ny % kTmaRows)
    return false;
  // the wave as floats: 2 nx per row, ny rows; boxes of 2 cb floats x 256 rows
  const cuuint64_t dims[2] = {(cuuint64_t)2 * nx, (cuuint64_t)ny};
  const cuuint64_t strides[1] = {(cuuint64_t)nx * sizeof(float2)};
  const cuuint32_t box[2] = {(cuuint32_t)(2 * cb), (cuuint32_t)kTmaRows};
  const cuuint32_t elem[2] = {1, 1};
  return encode(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float2*>(base), dims, strides, box, elem,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

void band_limit_thresholds(float kmax, float* k2_lt, float* k2_le) {
  auto first = [](float m, bool strict) {
    // smallest x >= 0 with sqrtf(x) >= m (strict: > m); sqrtf is monotone
    auto pass = [&](float x) { return strict ? std::sqrt(x) > m : std::sqrt(x) >= m; };
    float x = (float)((double)m * (double)m);
    while (x > 0.0f && pass(std::nextafter(x, 0.0f))) x = std::nextafter(x, 0.0f);
    while (!pass(x)) x = std::nextafter(x, INFINITY);
    return x;
  };
  *k2_lt = first(kmax, false);
  *k2_le = first(kmax, true);
}

float2 unit_fp32(double c, double s) {
  float2 u;
  unit_fp32(c, s, &u.x, &u.y);
  return u;
}

void unit_roots(int n, float2* out) {
  const long double twopi = 6.283185307179586476925286766559L;
  for (int m = 0; m < n; ++m) {
    const long double a = twopi * (long double)m / (long double)n;
    out[m] = unit_fp32((double)std::cos(a), (double)(-std::sin(a)));
  }
}

int plan_variants() { return kPlanVariants; }

// Measured per line length and batch of square grids, us per launch (B200, the
// passes of the slice loop, 300 launches back to back; 4, 12, 16, 32 and 64
// instances of up to 512 points, 4, 16 and 64 of 1024, 4 and 8 or 16 above):
//                  chosen                            the next
//   rows  128      5: 2.2 2.4 3.3 3.4, 0: 4.5        2: 2.2 2.3 3.2 3.4, 5: 5.1
//         256      5: 3.9, 0: 4.6 4.6, 3: 7.6 11.9   2: 3.9, 5: 5.2, 1: 5.6, 0: 7.6 12.9
//         512      0: 5.4 13.6 16.5 29.9 58.1        1: 5.6, 5: 13.9, 4: 16.5 31.3 60.4
//         1024     0: 17.8 61.2 246                  4: 19.3 67.1 258
//         2048     4: 72.5 141                       1: 77.0 153
//         4096     4: 302                            0: 326
//   rows, tc, 128  5: 2.3 2.2 3.3 3.4, 0: 4.1        1: 2.2 3.8 3.9 4.0, 4: 4.9
//         256      4: 3.0, 0: 4.3 4.3 7.1 11.6       1: 2.9 4.0 4.9 8.0 14.4
//         512      0: 5.8 9.9 12.2 21.0 40.1         3: 5.3, 1: 13.5 15.8 29.6 57.6
//         1024     0: 16.7 56.0 221                  3: 18.9 62.5 254
//         2048     0: 74.1 140                       1: 76.8 149
//         4096     1: 324                            4: 338
//   columns 128    5: 2.5 3.6 3.9 4.0 4.4            2: 2.5 3.7 4.0 4.0 4.4
//         256      5: 4.6 4.8 4.9, 3: 5.3 9.8        3: 4.0, 4: 4.5 5.0, 0: 5.5 10.0
//         512      3: 6.0, 0: 9.7 9.7 18.7 36.0      5: 6.2, 4: 10.3 12.1 21.2 40.5
//         1024     0: 11.2 38.4 172                  3: 15.8 54.4 230
//         2048     0: 54.1 117                       4: 58.5 126
//         4096     0: 254                            3: 305
// One instance (at most 512 points: bound by the launches, chosen by whole slices):
// 1024 rows 0 5.9, columns 3 7.2; 2048 4 20.5, 3 18.6; 4096 4 79.7, 3 60.6.
// Timing them on each handle's first use instead took 2-5 ms, and at one
// instance, where a launch takes as long as the kernel, picked at random.
int pass_plan(int n, long long lines, bool columns, bool tc) {
  const long long eff = lines / n;  // instances of a square grid
  const int b = eff < 2 ? 0 : eff < 8 ? 1 : eff < 20 ? 2 : eff < 48 ? 3 : 4;
  static const signed char kRow[7][5] = {{5, 5, 5, 5, 5}, {5, 5, 5, 5, 0}, {5, 5, 0, 3, 3}, {5, 0, 0, 0, 0},
                                         {0, 0, 0, 0, 0}, {4, 4, 4, 4, 4}, {4, 4, 4, 4, 4}};
  static const signed char kRowTc[7][5] = {{5, 5, 5, 5, 5}, {5, 5, 5, 5, 0}, {5, 4, 0, 0, 0}, {5, 0, 0, 0, 0},
                                           {0, 0, 0, 0, 0}, {0, 0, 0, 0, 0}, {1, 1, 1, 1, 1}};
  static const signed char kCol[7][5] = {{5, 5, 5, 5, 5}, {5, 5, 5, 5, 5}, {5, 5, 5, 3, 3}, {5, 3, 0, 0, 0},
                                         {3, 0, 0, 0, 0}, {3, 0, 0, 0, 0}, {3, 0, 0, 0, 0}};
  int i = 0;
  while ((64 << i) < n && i < 6) ++i;
  return columns ? kCol[i][b] : tc ? kRowTc[i][b] : kRow[i][b];
}

int make_twiddles(int n, int variant, const float2* roots, float2* host_out) {
  int size = 0;
  by_length(n, [&](auto c) {
    size = twiddles_n<decltype(c)::value>(variant, roots, host_out);
    return cudaSuccess;
  });
  return size;
}

cudaError_t launch_pass_a(const PassAArgs& a, int variant, int flags, int batch, cudaStream_t s) {
  return by_length(a.nx, [&](auto c) { return dispatch_a_n<decltype(c)::value>(a, variant, flags, batch, s); });
}

cudaError_t launch_pass_b(const PassBArgs& a, int variant, int mode, int batch, cudaStream_t s) {
  return by_length(a.ny, [&](auto c) { return dispatch_b_n<decltype(c)::value>(a, variant, mode, batch, s); });
}

}  // namespace ms
