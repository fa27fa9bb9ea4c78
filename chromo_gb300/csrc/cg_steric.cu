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
// change 2.75 ms); tested one by one and summed where they are met 112 us (184
// us), with the near pairs listed per tile 51 us (86 us).
#include <cuda_runtime.h>

#include "cg_kernels.h"
#include "cg_steric_tiles.h"

namespace cg {

constexpr int kRows = CG_STERIC_ROWS;          // rows of a tile
constexpr int kStericThr = CG_STERIC_THREADS;  // threads of a tile
constexpr int kGroup = 8;       // rows between two tests
constexpr int kList = 1024;     // near pairs a CTA lists (5 bits of row, 10 of column)
static_assert(kRows == 32 && kRows % kGroup == 0, "a bit per row, groups of whole rows");

// The pair energy from the squared distance: the powers of (e / d)^2, one quotient of
// squares (e2 = e^2; 0 where squares leave FP64's range, with the square root).  The
// roundings of the root and of e / d count twelvefold in (e / d)^12, those of the
// squares and their quotient sixfold: the error is 0.7 of that of pow(e / d, 12), at
// half the FP64 operations.
__device__ __forceinline__ double clash_energy(double d2, double e, double e2, double V0) {
  double f2;
  if (!is_zero64(e2)) {
    if (!(d2 < e2)) return 0.0;
    f2 = e2 / d2;
  } else {
    const double d = sqrt(d2);
    if (!(d < e)) return 0.0;
    const double f = e / d;
    f2 = f * f;
  }
  const double f6 = f2 * f2 * f2;
  return V0 * (f6 * f6 - 2 * f6 + 1);
}

__device__ __forceinline__ double square3(const double a[3], const double b[3]) {
  const double x = a[0] - b[0], y = a[1] - b[1], z = a[2] - b[2];
  return x * x + y * y + z * z;
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
__device__ __forceinline__ float dist2(const float4& a, const float3& b) {
  const float x = a.x - b.x, y = a.y - b.y, z = a.z - b.z;
  return __fmaf_rn(z, z, __fmaf_rn(y, y, x * x));
}

// Sum over the CTA, valid in thread 0.  Most threads, and warps, hold zero: their
// FP64 additions (~60 cycles of the pipe each) are left out.
__device__ __forceinline__ double tile_total(double v, double* sh) {
  if (__any_sync(kFull, !is_zero64(v)))
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0;
  if (threadIdx.x == 0)
    #pragma unroll 1
    for (int w = 0; w < (int)(blockDim.x >> 5); w++)
      if (!is_zero64(sh[w])) t += sh[w];
  return t;
}

// The FP64 term of beads i (a row) and j.
template <typename Pos, bool TRIAL>
static __device__ __noinline__ double pair_term(const V4<Pos>* r4, long long i, long long j, long long ind0,
                                                long long indf, const double* trial, double e, double e2, double V0) {
  double ri[3], rj[3];
  ld3(r4, i, ri);
  ld3(r4, j, rj);
  const double before = clash_energy(square3(ri, rj), e, e2, V0);
  if (!TRIAL) return before;
  const double* ti = trial + 3 * (i - ind0);
  const double t0[3] = {ti[0], ti[1], ti[2]};
  if (j >= ind0 && j < indf)
    for (int q = 0; q < 3; q++) rj[q] = trial[3 * (j - ind0) + q];
  return clash_energy(square3(t0, rj), e, e2, V0) - before;
}

// Rows [height blockIdx.x, ...) (at most kRows) against columns [blockIdx.y chunk, ...): the
// pairs i < j of the resident chain, or (TRIAL) with positions `trial` of the
// beads [ind0, indf) (m x 3) the change of the pairs of the moved beads, those of
// two moved beads counted once (j < i).  parts: one sum per tile, by row tile and
// chunk.  A thread holds COLS columns and takes the smallest squared distance of
// kGroup rows before it branches, so that a pair costs seven FP32 instructions
// and a quarter of a shared load; the near pairs are listed, and their FP64 terms
// taken on consecutive threads (near pairs of a chain lie along the diagonal: row
// by row, one lane at a time, a tile's took 70 k cycles).
template <typename Pos, bool TRIAL, int COLS>
__global__ void __launch_bounds__(kStericThr)
    steric_tile_kernel(KArgs a, int rep, long long n_rows, long long ind0, long long indf, long long chunk,
                       int height, const double* trial, double e, double e2, double V0, double* parts) {
  __shared__ float4 cur[kRows], tri[TRIAL ? kRows : 1];
  __shared__ float far_sh;
  __shared__ int found[kStericThr / 32];
  __shared__ unsigned short list[kList];
  __shared__ double sh[kStericThr / 32];
  const RepDev& rd = a.reps[rep];
  const V4<Pos>* r4 = reinterpret_cast<const V4<Pos>*>(a.r4) + rd.bead_off;
  const long long N = rd.n_beads;
  const int lane = (int)(threadIdx.x & 31u), warp = (int)(threadIdx.x >> 5);
  const long long k0 = (long long)blockIdx.x * height, row0 = (TRIAL ? ind0 : 0) + k0;  // bead of row 0
  const int rows = (int)(n_rows - k0 < height ? n_rows - k0 : height);
  long long c0 = (long long)blockIdx.y * chunk;
  const long long c1 = c0 + chunk < N ? c0 + chunk : N;
  if (!TRIAL && c0 < k0 + 1) c0 = k0 + 1;  // pairs above the diagonal
  if (c0 >= c1) {  // a chunk below the diagonal
    if (threadIdx.x == 0) parts[(long long)blockIdx.x * gridDim.y + blockIdx.y] = 0.0;
    return;
  }
  double part = 0;
  {
    const float inf = __int_as_float(0x7F800000);
    const V4<Pos> org = r4[row0];
    if (threadIdx.x < 32) {
      float far = 0;
      // rows past the last are nowhere near (inf - inf drops out of the minimum)
      float3 c = make_float3(inf, inf, inf), t = c;
      if ((int)threadIdx.x < rows) {
        const long long i = row0 + threadIdx.x;
        c = offset_of(r4[i], org);
        t = TRIAL ? offset_of(trial + 3 * (i - ind0), org) : c;
        far = fmaxf(fmaxf(fabsf(c.x), fmaxf(fabsf(c.y), fabsf(c.z))), fmaxf(fabsf(t.x), fmaxf(fabsf(t.y), fabsf(t.z))));
      }
      cur[threadIdx.x] = make_float4(c.x, c.y, c.z, 0.0f);
      if (TRIAL) tri[threadIdx.x] = make_float4(t.x, t.y, t.z, 0.0f);
      for (int o = 16; o > 0; o >>= 1) far = fmaxf(far, __shfl_xor_sync(kFull, far, o));
      if (threadIdx.x == 0) far_sh = far;
    }
    __syncthreads();
    const float ef = (float)e;
    const float reach = ef + 4e-6f * (ef + 2.0f * far_sh) + 1e-30f;
    // beyond FP32's squares, and where they lose bits below its normal numbers, every
    // pair takes the FP64 distance (NaN: no d2 is >= thr)
    const bool all = !(reach > 1e-18f && reach < 1e18f);
    const float thr = all ? __int_as_float(0x7FFFFFFF) : reach * reach * 1.00001f;
    #pragma unroll 1
    for (long long jb = c0; jb < c1; jb += COLS * kStericThr) {
      const long long j0 = jb + threadIdx.x;
      float3 cj[COLS], tj[COLS];
      bool moved[COLS];
#pragma unroll
      for (int u = 0; u < COLS; u++) {
        const long long j = j0 + u * kStericThr;
        cj[u] = j < c1 ? offset_of(r4[j], org) : make_float3(inf, inf, inf);
        moved[u] = TRIAL && j >= ind0 && j < indf && j < c1;
        tj[u] = moved[u] ? offset_of(trial + 3 * (j - ind0), org) : cj[u];
      }
      unsigned hit[COLS];
#pragma unroll
      for (int u = 0; u < COLS; u++) hit[u] = 0;
      #pragma unroll 1
      for (int g = 0; g < rows; g += kGroup) {
        float low[COLS];
#pragma unroll
        for (int u = 0; u < COLS; u++) low[u] = inf;
#pragma unroll
        for (int q = 0; q < kGroup; q++) {
          const float4 c = cur[g + q];
#pragma unroll
          for (int u = 0; u < COLS; u++) low[u] = fminf(low[u], dist2(c, cj[u]));
          if (TRIAL) {
            const float4 t = tri[g + q];
#pragma unroll
            for (int u = 0; u < COLS; u++) low[u] = fminf(low[u], dist2(t, tj[u]));
          }
        }
#pragma unroll
        for (int u = 0; u < COLS; u++) {
          const long long j = j0 + u * kStericThr;
          if (!(all || low[u] < thr) || j >= c1) continue;
          #pragma unroll 1
          for (int k = g; k < g + kGroup && k < rows; k++) {
            const long long i = row0 + k;
            bool near = !(dist2(cur[k], cj[u]) >= thr);
            if (TRIAL) near = (near || !(dist2(tri[k], tj[u]) >= thr)) && !(moved[u] && j >= i);
            else near = near && j > i;
            if (near) hit[u] |= 1u << k;
          }
        }
      }
      // the marked pairs, in thread order, as a list of the CTA: their FP64 terms on
      // consecutive threads
      int cnt = 0;
#pragma unroll
      for (int u = 0; u < COLS; u++) cnt += __popc(hit[u]);
      int at = cnt;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kFull, at, o);
        if (lane >= o) at += y;
      }
      if (lane == 31) found[warp] = at;
      __syncthreads();
      at -= cnt;
      int total = 0;
      for (int w = 0; w < kStericThr / 32; w++) {
        if (w < warp) at += found[w];
        total += found[w];
      }
      const bool listed = total <= kList;
      #pragma unroll 1
      while (cnt > 0) {
        int u = 0;
        unsigned h = 0;
#pragma unroll
        for (int v = COLS - 1; v >= 0; v--)
          if (hit[v]) { u = v; h = hit[v]; }
        const int k = __ffs((int)h) - 1;
#pragma unroll
        for (int v = 0; v < COLS; v++)
          if (v == u) hit[v] &= hit[v] - 1;
        cnt--;
        if (listed) list[at++] = (unsigned short)((u * kStericThr + (int)threadIdx.x) << 5 | k);
        else part += pair_term<Pos, TRIAL>(r4, row0 + k, j0 + u * kStericThr, ind0, indf, trial, e, e2, V0);
      }
      __syncthreads();
      if (listed)
        #pragma unroll 1
        for (int q = threadIdx.x; q < total; q += kStericThr)
          part += pair_term<Pos, TRIAL>(r4, row0 + (list[q] & 31), jb + (list[q] >> 5), ind0, indf, trial, e, e2, V0);
      __syncthreads();  // the list is read
    }
  }
  const double t = tile_total(part, sh);
  if (threadIdx.x == 0) parts[(long long)blockIdx.x * gridDim.y + blockIdx.y] = t;
}

// out[0] = the tiles' sums, added in a fixed order by one CTA.
__global__ void __launch_bounds__(kStericThr) steric_sum_kernel(const double* parts, long long n, double* out) {
  __shared__ double sh[kStericThr / 32];
  double s = 0;
  for (long long k = threadIdx.x; k < n; k += kStericThr) {
    const double p = parts[k];
    if (!is_zero64(p)) s += p;
  }
  const double t = tile_total(s, sh);
  if (threadIdx.x == 0) out[0] = t;
}

}  // namespace cg

// parts holds at least n_beads + 32 doubles (the split: cg_steric_tiles.h).
template <typename Pos>
static void launch_tiles(const cg::KArgs& a, dim3 grid, int rep, long long n_rows, long long ind0, long long indf,
                         long long chunk, int height, const double* trial, double e, double V0, double* parts,
                         cudaStream_t s) {
  const double e2 = e > 1e-150 && e < 1e150 ? e * e : 0.0;
  auto run = [&](auto kernel) {
    kernel<<<grid, cg::kStericThr, 0, s>>>(a, rep, n_rows, ind0, indf, chunk, height, trial, e, e2, V0, parts);
  };
  const bool one = chunk == cg::kStericThr;
  if (trial) run(one ? cg::steric_tile_kernel<Pos, true, 1> : cg::steric_tile_kernel<Pos, true, 4>);
  else run(one ? cg::steric_tile_kernel<Pos, false, 1> : cg::steric_tile_kernel<Pos, false, 4>);
}
void cg_launch_steric(const cg::KArgs& a, bool fp64, int rep, long long n_beads, long long n_rows, long long ind0,
                      long long indf, const double* trial, double e, double V0, double* parts, double* out,
                      int n_sm, cudaStream_t s) {
  int height;
  const long long chunk = cg_steric_split(n_beads, n_rows, n_sm, &height);
  const long long tiles = (n_rows + height - 1) / height;
  const long long chunks = (n_beads + chunk - 1) / chunk;
  const dim3 grid((unsigned)tiles, (unsigned)chunks);
  if (fp64) launch_tiles<double>(a, grid, rep, n_rows, ind0, indf, chunk, height, trial, e, V0, parts, s);
  else launch_tiles<float>(a, grid, rep, n_rows, ind0, indf, chunk, height, trial, e, V0, parts, s);
  if (cudaPeekAtLastError() != cudaSuccess) return;  // the caller reports it; no sums to add
  cg::steric_sum_kernel<<<1, cg::kStericThr, 0, s>>>(parts, tiles * chunks, out);
}
