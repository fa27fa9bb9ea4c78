// cg_steric.cu -- steric clash energy of bead pairs on the device.
//
// The detailed chromatin model with sterics (DetailedChromatinWithSterics,
// chromo/polymers.pyx:2738-2938) adds, for every pair of beads closer than
// the excluded distance e (twice the bead radius), V0 ((e/d)^12 - 2 (e/d)^6 + 1).
// The reference keeps an N x N distance matrix and refreshes the rows of the
// moved beads each move (get_delta_distances); here distances are computed on
// the fly from the resident positions, in tiles of kRows rows (beads, or the
// moved beads: the O(m N) update of one move) against chunks of columns, and
// the tiles' partial sums are added in a fixed order, so the results are
// deterministic.
//
// Nearly every pair is further apart than e, and FP64 runs at 1/64 of the FP32
// rate here, so a pair is first tested in FP32 (seven instructions); only pairs
// within e and a margin above the test's error take the FP64 distance and
// energy.  Every pair in FP64 with its square root, and the 10,000 row sums
// added by one thread, took 2.57 ms for a 10,000-bead chain (with one segment's
// change 2.75 ms, now 0.17 ms).
#include <cuda_runtime.h>

#include <algorithm>

#include "cg_kernels.h"

namespace cg {

constexpr int kRows = 32;       // rows of a tile
constexpr int kStericThr = 256; // threads of a tile: one column each

__device__ __forceinline__ double clash_energy(double d, double e, double V0) {
  if (!(d < e)) return 0.0;
  const double f = e / d, f2 = f * f, f6 = f2 * f2 * f2;
  return V0 * (f6 * f6 - 2 * f6 + 1);
}

__device__ __forceinline__ double dist3(const double a[3], const double b[3]) {
  const double x = a[0] - b[0], y = a[1] - b[1], z = a[2] - b[2];
  return sqrt(x * x + y * y + z * z);
}

// Offset of a position from the tile's origin, rounded to FP32.  Pairs closer
// than e have both offsets within L + e (L: the largest row offset), where the
// rounding is below 2^-23 (L + e).
__device__ __forceinline__ float3 offset_of(const V4<float>& p, const V4<float>& o) {
  return make_float3(p.x - o.x, p.y - o.y, p.z - o.z);
}
__device__ __forceinline__ float3 offset_of(const V4<double>& p, const V4<double>& o) {
  return make_float3((float)(p.x - o.x), (float)(p.y - o.y), (float)(p.z - o.z));
}
template <typename Pos>
__device__ __forceinline__ float3 offset_of(const double* t, const V4<Pos>& o) {
  return make_float3((float)(t[0] - (double)o.x), (float)(t[1] - (double)o.y), (float)(t[2] - (double)o.z));
}
__device__ __forceinline__ float dist2(const float3& a, const float3& b) {
  const float x = a.x - b.x, y = a.y - b.y, z = a.z - b.z;
  return x * x + y * y + z * z;
}

__device__ __forceinline__ double tile_total(double v, double* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0;
  if (threadIdx.x == 0)
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += sh[w];
  return t;  // valid in thread 0
}

// Rows [kRows blockIdx.x, ...) against columns [blockIdx.y chunk, ...): the
// pairs i < j of the resident chain, or with trial != null (positions of the
// beads [ind0, indf), m x 3) the change of the pairs of the moved beads, those
// of two moved beads counted once (j < i).  parts: one sum per tile, by row
// tile and chunk.
template <typename Pos>
__global__ void __launch_bounds__(kStericThr)
    steric_tile_kernel(KArgs a, int rep, long long n_rows, long long ind0, long long indf, long long chunk,
                       const double* trial, double e, double V0, double* parts) {
  __shared__ float3 cur[kRows], tri[kRows];
  __shared__ float far_sh;
  __shared__ double sh[kStericThr / 32];
  const RepDev& rd = a.reps[rep];
  const V4<Pos>* r4 = reinterpret_cast<const V4<Pos>*>(a.r4) + rd.bead_off;
  const long long N = rd.n_beads;
  const long long first = trial ? ind0 : 0;  // bead of row 0
  const long long k0 = (long long)blockIdx.x * kRows;
  const int rows = (int)(n_rows - k0 < kRows ? n_rows - k0 : kRows);
  const long long c0 = (long long)blockIdx.y * chunk, c1 = c0 + chunk < N ? c0 + chunk : N;
  double part = 0;
  if (trial || c1 > k0 + 1) {  // a chunk below the diagonal has no pair
    const V4<Pos> org = r4[first + k0];
    if (threadIdx.x < 32) {
      float far = 0;
      if ((int)threadIdx.x < rows) {
        const long long i = first + k0 + threadIdx.x;
        const float3 c = offset_of(r4[i], org), t = trial ? offset_of(trial + 3 * (i - ind0), org) : c;
        cur[threadIdx.x] = c;
        tri[threadIdx.x] = t;
        far = fmaxf(fmaxf(fabsf(c.x), fmaxf(fabsf(c.y), fabsf(c.z))), fmaxf(fabsf(t.x), fmaxf(fabsf(t.y), fabsf(t.z))));
      }
      for (int o = 16; o > 0; o >>= 1) far = fmaxf(far, __shfl_xor_sync(kFull, far, o));
      if (threadIdx.x == 0) far_sh = far;
    }
    __syncthreads();
    const float ef = (float)e;
    const float reach = ef + 4e-6f * (ef + 2.0f * far_sh) + 1e-30f;
    // beyond FP32's squares every pair takes the FP64 distance (NaN: no d2 is >= thr)
    const float thr = reach < 1e18f ? reach * reach * 1.00001f : __int_as_float(0x7FFFFFFF);
    for (long long j = c0 + threadIdx.x; j < c1; j += kStericThr) {
      const float3 cj = offset_of(r4[j], org);
      const bool moved = trial && j >= ind0 && j < indf;
      const float3 tj = moved ? offset_of(trial + 3 * (j - ind0), org) : cj;
      for (int k = 0; k < rows; k++) {
        const long long i = first + k0 + k;
        bool near = !(dist2(cur[k], cj) >= thr);
        if (trial) near = (near || !(dist2(tri[k], tj) >= thr)) && !(moved && j >= i);
        else near = near && j > i;
        if (near) {
          double ri[3], rj[3];
          ld3(r4, i, ri);
          ld3(r4, j, rj);
          const double before = clash_energy(dist3(ri, rj), e, V0);
          if (trial) {
            const double* ti = trial + 3 * (i - ind0);
            const double t0[3] = {ti[0], ti[1], ti[2]};
            if (moved)
              for (int q = 0; q < 3; q++) rj[q] = trial[3 * (j - ind0) + q];
            part += clash_energy(dist3(t0, rj), e, V0) - before;
          } else {
            part += before;
          }
        }
      }
    }
  }
  const double t = tile_total(part, sh);
  if (threadIdx.x == 0) parts[(long long)blockIdx.x * gridDim.y + blockIdx.y] = t;
}

// out[0] = the tiles' sums, added in a fixed order by one CTA.
__global__ void __launch_bounds__(kStericThr) steric_sum_kernel(const double* parts, long long n, double* out) {
  __shared__ double sh[kStericThr / 32];
  double s = 0;
  for (long long k = threadIdx.x; k < n; k += kStericThr) s += parts[k];
  const double t = tile_total(s, sh);
  if (threadIdx.x == 0) out[0] = t;
}

}  // namespace cg

// parts holds at least n_beads doubles: at most 32 chunks of columns.
void cg_launch_steric(const cg::KArgs& a, bool fp64, int rep, long long n_beads, long long n_rows, long long ind0,
                      long long indf, const double* trial, double e, double V0, double* parts, double* out,
                      cudaStream_t s) {
  const long long tiles = (n_rows + cg::kRows - 1) / cg::kRows;
  const long long chunk =
      std::max<long long>(1024, ((n_beads + 31) / 32 + cg::kStericThr - 1) / cg::kStericThr * cg::kStericThr);
  const long long chunks = (n_beads + chunk - 1) / chunk;
  const dim3 grid((unsigned)tiles, (unsigned)chunks);
  if (fp64)
    cg::steric_tile_kernel<double><<<grid, cg::kStericThr, 0, s>>>(a, rep, n_rows, ind0, indf, chunk, trial, e, V0,
                                                                   parts);
  else
    cg::steric_tile_kernel<float><<<grid, cg::kStericThr, 0, s>>>(a, rep, n_rows, ind0, indf, chunk, trial, e, V0,
                                                                  parts);
  cg::steric_sum_kernel<<<1, cg::kStericThr, 0, s>>>(parts, tiles * chunks, out);
}
