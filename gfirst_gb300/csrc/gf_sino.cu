// gf_sino.cu -- sinogram-domain kernels: the subset-local (radial-major,
// padded-row) layouts the projectors use, the data/projection ratio, the
// normalization mask and the VLOR count/split.
//
// Elements of a subset-layout array are indexed by
//   (angle-in-subset tl, radial bin r, padded row p): (tl*NRAD + r)*PS + p,
// with one array holding every subset back to back when it is static.
#include <cub/device/device_radix_sort.cuh>

#include "gf_kernels.h"

namespace gf {

__device__ __forceinline__ size_t file_lor(const DevGeom& g, int seg, int plane, int theta, int r) {
  const DevSeg& sg = g.seg[seg];
  return ((size_t)(plane - sg.zmin) + sg.acc) * ((size_t)g.nrad * g.nang) + (size_t)theta * g.nrad + r;
}

// rowmap entries: (seg, plane) for real rows; (seg, -1 - edge) for pad rows,
// edge 0 = before the block, 1 = after; (-1, -1) past PP.
__device__ __forceinline__ bool resolve_row(const DevGeom& g, int2 m, int* seg, int* plane) {
  if (m.x < 0) return false;
  *seg = m.x;
  if (m.y >= 0) {
    *plane = m.y;
    return true;
  }
  if (m.x != 0) return false;  // oblique pad row: sentinel
  *plane = (m.y == -1) ? 0 : g.nzs - 1;
  return true;
}

// Rank of angle theta in the all-subset layout: subsets are stored in order,
// subset s = theta % nsub holding angles s, s + nsub, ...; the first
// nang % nsub subsets hold one angle more than the others.
__device__ __forceinline__ int angle_rank(const DevGeom& g, int theta) {
  const int s = theta % g.nsub, l = theta / g.nsub;
  const int q = g.nang / g.nsub, rem = g.nang % g.nsub;
  return s * q + min(s, rem) + l;
}

// The static subset layouts are a transpose of the file layout: for one
// angle, file element (plane, radial) goes to (radial, padded row).  A block
// moves a tile of 32 radial bins x 32 padded rows through shared memory, so
// both the file reads (along radial bins) and the layout writes (along rows)
// are whole 128-byte lines.

// (data*RES, max(bg*RES, 0)) for every subset, from the parsed file
// (2*NDATA floats: prompts then background).  GFIRST.cu:224-226, 423.
// Pad rows hold (0, 0).
__global__ void __launch_bounds__(256) build_dbg_kernel(const DevGeom g, const int2* __restrict__ rowmap,
                                                        const float* __restrict__ sino2, float2* __restrict__ dbg,
                                                        size_t ndata) {
  __shared__ float2 tile[32][33];
  const int r0 = blockIdx.x * 32, p0 = blockIdx.y * 32, theta = blockIdx.z;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const float res = (float)g.res;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int p = p0 + ty + 8 * k, r = r0 + tx;
    float2 v = make_float2(0.f, 0.f);
    if (p < g.PS && r < g.nrad) {
      const int2 m = rowmap[p];
      if (m.x >= 0 && m.y >= 0) {
        const size_t lor = file_lor(g, m.x, m.y, theta, r);
        const float bg = __fmul_rn(res, sino2[ndata + lor]);
        v = make_float2(__fmul_rn(res, sino2[lor]), ((double)bg < 0.) ? 0.f : bg);
      }
    }
    tile[ty + 8 * k][tx] = v;
  }
  __syncthreads();
  const size_t base = (size_t)angle_rank(g, theta) * g.nrad;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int r = r0 + ty + 8 * k, p = p0 + tx;
    if (r < g.nrad && p < g.PS) dbg[(base + r) * g.PS + p] = tile[tx][ty + 8 * k];
  }
}

cudaError_t launch_build_dbg(const DevGeom& g, const int2* rowmap, const float* sino2, float2* dbg,
                             cudaStream_t st) {
  const size_t ndata = (size_t)g.P * g.nang * g.nrad;
  const dim3 grid((g.nrad + 31) / 32, (g.PS + 31) / 32, g.nang);
  build_dbg_kernel<<<grid, dim3(32, 8), 0, st>>>(g, rowmap, sino2, dbg, ndata);
  return cudaGetLastError();
}

// Normalization mask per subset element, GFIRST.cu:447, 453-458: 1 where
// proj_blank > 0.01 and blank > 0.01, else -1000; oblique pad rows -1000,
// segment 0's pad rows repeat its first/last plane.
__global__ void __launch_bounds__(256) build_cal_kernel(const DevGeom g, const int2* __restrict__ rowmap,
                                                        const float* __restrict__ proj_ref,
                                                        const float* __restrict__ norm, float* __restrict__ cal) {
  __shared__ float tile[32][33];
  const int r0 = blockIdx.x * 32, p0 = blockIdx.y * 32, theta = blockIdx.z;
  const int tx = threadIdx.x, ty = threadIdx.y;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int p = p0 + ty + 8 * k, r = r0 + tx;
    float v = -1000.f;
    int seg, plane;
    if (p < g.PS && r < g.nrad && resolve_row(g, rowmap[p], &seg, &plane)) {
      const size_t lor = file_lor(g, seg, plane, theta, r);
      v = ((double)proj_ref[lor] > 0.01 && (double)norm[lor] > 0.01) ? 1.0f : -1000.f;
    }
    tile[ty + 8 * k][tx] = v;
  }
  __syncthreads();
  const size_t base = (size_t)angle_rank(g, theta) * g.nrad;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int r = r0 + ty + 8 * k, p = p0 + tx;
    if (r < g.nrad && p < g.PS) cal[(base + r) * g.PS + p] = tile[tx][ty + 8 * k];
  }
}

cudaError_t launch_build_cal(const DevGeom& g, const int2* rowmap, const float* proj_ref, const float* norm,
                             float* cal, cudaStream_t st) {
  const dim3 grid((g.nrad + 31) / 32, (g.PS + 31) / 32, g.nang);
  build_cal_kernel<<<grid, dim3(32, 8), 0, st>>>(g, rowmap, proj_ref, norm, cal);
  return cudaGetLastError();
}

// One word of mask bits per (angle row, radial bin, 32 padded rows), lane =
// row, and the dirty bits: segments with a masked plane in this word.  at: the
// (angle row, radial bin) index.
__device__ __forceinline__ void put_mask_word(const DevGeom& g, const int2* __restrict__ rowmap, size_t at, int p0,
                                              int lane, bool bit, unsigned* mask, unsigned* dirty) {
  const unsigned word = __ballot_sync(0xffffffffu, bit);
  if (lane == 0) mask[at * (g.PS >> 5) + (p0 >> 5)] = word;
  const int2 m = p0 + lane < g.PS ? rowmap[p0 + lane] : make_int2(-1, -1);
  const int nsw = (g.nseg + 31) >> 5;
  const bool real = m.x >= 0 && m.y >= 0;
  unsigned pend = __ballot_sync(0xffffffffu, real && !bit);
  while (pend) {  // one atomic per segment in the word
    const int seg = __shfl_sync(0xffffffffu, m.x, __ffs(pend) - 1);
    if (lane == 0) atomicOr(dirty + at * nsw + (seg >> 5), 1u << (seg & 31));
    pend &= ~__ballot_sync(0xffffffffu, real && m.x == seg);
  }
}

// Normalization mask bits, GFIRST.cu:447, 453-458: 1 where proj_blank > 0.01
// and blank > 0.01; oblique pad rows 0, segment 0's pad rows repeat its
// first/last plane.
__global__ void __launch_bounds__(256) build_mask_kernel(const DevGeom g, const int2* __restrict__ rowmap,
                                                         const float* __restrict__ proj_ref,
                                                         const float* __restrict__ norm, unsigned* mask,
                                                         unsigned* dirty) {
  __shared__ unsigned char tile[32][36];
  const int r0 = blockIdx.x * 32, p0 = blockIdx.y * 32, theta = blockIdx.z;
  const int tx = threadIdx.x, ty = threadIdx.y;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int p = p0 + ty + 8 * k, r = r0 + tx;
    bool v = false;
    int seg, plane;
    if (p < g.PS && r < g.nrad && resolve_row(g, rowmap[p], &seg, &plane)) {
      const size_t lor = file_lor(g, seg, plane, theta, r);
      v = (double)proj_ref[lor] > 0.01 && (double)norm[lor] > 0.01;
    }
    tile[ty + 8 * k][tx] = v;
  }
  __syncthreads();
  const size_t base = (size_t)angle_rank(g, theta) * g.nrad;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int r = r0 + ty + 8 * k;
    if (r < g.nrad) put_mask_word(g, rowmap, base + r, p0, tx, tile[tx][ty + 8 * k] != 0, mask, dirty);
  }
}

cudaError_t launch_build_mask(const DevGeom& g, const int2* rowmap, const float* proj_ref, const float* norm,
                              unsigned* mask, unsigned* dirty, cudaStream_t st) {
  const dim3 grid((g.nrad + 31) / 32, g.PS / 32, g.nang);
  build_mask_kernel<<<grid, dim3(32, 8), 0, st>>>(g, rowmap, proj_ref, norm, mask, dirty);
  return cudaGetLastError();
}

__device__ __forceinline__ float ratio_rule(float proj, float data, float bg) {
  // GFIRST.cu:423-429
  if ((double)bg < 0.) bg = 0.f;
  const float s = __fadd_rn(proj, bg);
  return (s >= 0.01f) ? __fdiv_rn(data, s) : -1000.f;
}

// One subset from the file layout (gf_back_project), moved in 32x32 tiles as
// above; pad rows of oblique segments hold the gap value.  PAIRS: (ratio, mask)
// pairs, where *general is set (null: always); else ratios, mask bits, dirty
// bits and *general = 1 where a mask value is neither 1 nor -1000.
template <bool PAIRS>
__global__ void __launch_bounds__(256) ratio_from_file_kernel(const DevGeom g, const int2* __restrict__ rowmap,
                                                              int subset, const float* __restrict__ corr,
                                                              const float* __restrict__ calib, void* out,
                                                              unsigned* mask, unsigned* dirty, int* general) {
  if (PAIRS && general && !*general) return;
  __shared__ float tc[32][33], tm[32][33];
  const int r0 = blockIdx.x * 32, p0 = blockIdx.y * 32, tl = blockIdx.z;
  const int theta = subset_angle(g, subset, tl);
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int r = min(r0 + tx, g.nrad - 1);
  // the rows' planes first, then their data: two waits instead of two a row
  int pl[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int p = p0 + ty + 8 * k;
    pl[k] = row_plane(p, rowmap[p], g.nzs);
  }
  float c[4], m[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const size_t lor = (size_t)pl[k] * ((size_t)g.nrad * g.nang) + (size_t)theta * g.nrad + r;
    c[k] = pl[k] >= 0 ? corr[lor] : -1000.f;
    m[k] = pl[k] >= 0 ? calib[lor] : -1000.f;
  }
  bool other = false;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    tc[ty + 8 * k][tx] = c[k];
    tm[ty + 8 * k][tx] = m[k];
    other |= !(m[k] == 1.f || m[k] == -1000.f);
  }
  if (PAIRS) {
    __syncthreads();
  } else if (__syncthreads_or(other)) {
    // the tiles will not run: one store a block and no bits (gf_back_project of 21
    // angles x 1293 planes of other values all over: 724 us; 745 with both)
    if (tx == 0 && ty == 0) *general = 1;
    return;
  }
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int r = r0 + ty + 8 * k;
    if (r < g.nrad) {
      const size_t at = (size_t)tl * g.nrad + r;
      const float c = tc[tx][ty + 8 * k], m = tm[tx][ty + 8 * k];
      if (PAIRS) {
        static_cast<float2*>(out)[at * g.PS + p0 + tx] = make_float2(c, m);
      } else {
        static_cast<float*>(out)[at * g.PS + p0 + tx] = c;
        put_mask_word(g, rowmap, at, p0, tx, m == 1.f, mask, dirty);
      }
    }
  }
}

cudaError_t launch_ratio_from_file(const DevGeom& g, const int2* rowmap, int subset, int na, const float* corr,
                                   const float* calib, float* out, unsigned* mask, unsigned* dirty, int* general,
                                   cudaStream_t st) {
  const dim3 grid((g.nrad + 31) / 32, g.PS / 32, na);
  ratio_from_file_kernel<false><<<grid, dim3(32, 8), 0, st>>>(g, rowmap, subset, corr, calib, out, mask, dirty, general);
  return cudaGetLastError();
}

cudaError_t launch_pairs_from_file(const DevGeom& g, const int2* rowmap, int subset, int na, const float* corr,
                                   const float* calib, float2* out, const int* general, cudaStream_t st) {
  const dim3 grid((g.nrad + 31) / 32, g.PS / 32, na);
  ratio_from_file_kernel<true><<<grid, dim3(32, 8), 0, st>>>(g, rowmap, subset, corr, calib, out, nullptr, nullptr,
                                                             const_cast<int*>(general));
  return cudaGetLastError();
}

// Ratio for the VLOR triples (GFIRST.cu:415-430 with val_dato = datos_v*RES,
// GFIRST.cu:397, 421) of one subset, as ratios or, with cal, (ratio, mask)
// pairs; projection and data come in 32x32 tiles as above.  Bound: HBM latency
// and bytes.  One element a thread, with both file arrays read along rows (a
// sector per element), took 36 us at 21 angles x 147 bins x 1293 planes, tiles 29.
template <int STORE, bool PAIRS>
__global__ void __launch_bounds__(256) ratio_gather_kernel(const DevGeom g, const int2* __restrict__ rowmap, int subset,
                                                           const float* __restrict__ proj_full,
                                                           const float* __restrict__ datos_v,
                                                           const float2* __restrict__ dbg_t,
                                                           const float* __restrict__ cal, void* __restrict__ out) {
  __shared__ float tp[32][33], td[32][33];
  const int r0 = blockIdx.x * 32, p0 = blockIdx.y * 32, tl = blockIdx.z;
  const int theta = subset_angle(g, subset, tl);
  const int tx = threadIdx.x, ty = threadIdx.y;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int p = p0 + ty + 8 * k, r = r0 + tx;
    float proj = 0.f, data = 0.f;
    int seg, plane;
    if (r < g.nrad && resolve_row(g, rowmap[p], &seg, &plane)) {
      const size_t lor = file_lor(g, seg, plane, theta, r);
      proj = proj_full[lor];
      data = datos_v[lor];
    }
    tp[ty + 8 * k][tx] = proj;
    td[ty + 8 * k][tx] = data;
  }
  __syncthreads();
  const int p = p0 + tx;
  const int2 m = rowmap[p];
  int seg, plane;
  const bool row = resolve_row(g, m, &seg, &plane);
  // the edge row's own element for segment 0's pad rows
  const int prow = (m.y >= 0) ? p : (m.y == -1 ? p + 1 : p - 1);
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int r = r0 + ty + 8 * k;
    if (r >= g.nrad) break;
    const size_t at = ((size_t)tl * g.nrad + r) * g.PS;
    float v = -1000.f, mask = -1000.f;
    if (row) {
      v = ratio_rule(tp[tx][ty + 8 * k], __fmul_rn(td[tx][ty + 8 * k], (float)g.res), dbg_t[at + prow].y);
      if (PAIRS) mask = cal[at + prow];
    }
    if constexpr (PAIRS) {
      using P = typename PairT<STORE>::type;
      static_cast<P*>(out)[at + p] = pair_from<P>(make_float2(v, mask));
    } else {
      using T = typename ElemT<STORE>::type;
      static_cast<T*>(out)[at + p] = elem_from<T>(v);
    }
  }
}

cudaError_t launch_ratio_gather(const DevGeom& g, const int2* rowmap, int subset, int na, const float* proj_full,
                                const float* datos_v, const float2* dbg_t, const float* cal, void* out, int storage,
                                cudaStream_t st) {
  const dim3 grid((g.nrad + 31) / 32, g.PS / 32, na), block(32, 8);
  switch (storage * 2 + (cal ? 1 : 0)) {
#define GF_RG(S, P) \
  case S * 2 + P: ratio_gather_kernel<S, P><<<grid, block, 0, st>>>(g, rowmap, subset, proj_full, datos_v, dbg_t, cal, out); break;
    GF_RG(0, 0) GF_RG(0, 1) GF_RG(1, 0) GF_RG(1, 1) GF_RG(2, 0) GF_RG(2, 1)
#undef GF_RG
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

// File-layout ratio over one subset's bins (operator entry point).
__global__ void ratio_file_kernel(const DevGeom g, int subset, const float* __restrict__ proj,
                                  const float* __restrict__ data, const float* __restrict__ bg,
                                  float* __restrict__ corr, size_t n) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int theta = (int)((i / g.nrad) % g.nang);
  if (theta % g.nsub != subset) return;
  corr[i] = ratio_rule(proj[i], data[i], bg[i]);
}

cudaError_t launch_ratio_file(const DevGeom& g, int subset, const float* proj, const float* data, const float* bg,
                              float* corr, cudaStream_t st) {
  const size_t n = (size_t)g.P * g.nang * g.nrad;
  ratio_file_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(g, subset, proj, data, bg, corr, n);
  return cudaGetLastError();
}

__global__ void norm_mask_kernel(const float* __restrict__ pb, const float* __restrict__ b, float* __restrict__ c,
                                 size_t n) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  c[i] = ((double)pb[i] > 0.01 && (double)b[i] > 0.01) ? 1.0f : -1000.f;
}

// *flag = 1 when a and b differ anywhere in their n floats (bitwise); *flag
// must hold 0 before.
__global__ void differs_kernel(const float* __restrict__ a, const float* __restrict__ b, size_t n, int* flag) {
  int d = 0;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    d |= __float_as_int(a[i]) ^ __float_as_int(b[i]);
  if (__any_sync(0xffffffffu, d != 0) && (threadIdx.x & 31) == 0) atomicExch(flag, 1);
}

cudaError_t launch_differs(const float* a, const float* b, size_t n, int* flag, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(flag, 0, sizeof(int), st);
  if (e != cudaSuccess) return e;
  differs_kernel<<<1216, 256, 0, st>>>(a, b, n, flag);
  return cudaGetLastError();
}

cudaError_t launch_norm_mask(const DevGeom& g, const float* proj_blank, const float* blank, float* calib,
                             cudaStream_t st) {
  const size_t n = (size_t)g.P * g.nang * g.nrad;
  norm_mask_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(proj_blank, blank, calib, n);
  return cudaGetLastError();
}

// ---- VLOR, GFIRST.cu:229-247, 373-389 --------------------------------------
__device__ __forceinline__ bool vlor_bins(const int32_t* ev, long long e, long long ndata, long long* i1,
                                          long long* i2) {
  *i1 = (long long)ev[2 * e] - 1;
  *i2 = (long long)ev[2 * e + 1] - 1;
  return !(*i1 <= 0 || *i2 <= 0 || *i1 >= ndata || *i2 >= ndata);
}

__global__ void vlor_count_kernel(const int32_t* __restrict__ ev, long long nev, long long ndata, float* cnt) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nev) return;
  long long i1, i2;
  if (!vlor_bins(ev, e, ndata, &i1, &i2)) return;
  atomicAdd(cnt + i1, 1.0f);
  atomicAdd(cnt + i2, 1.0f);
}

cudaError_t launch_vlor_count(const DevGeom& g, const int32_t* ev, long long nev, float* cnt, cudaStream_t st) {
  if (nev <= 0) return cudaSuccess;
  const long long ndata = (long long)g.P * g.nang * g.nrad;
  vlor_count_kernel<<<(unsigned)((nev + 255) / 256), 256, 0, st>>>(ev, nev, ndata, cnt);
  return cudaGetLastError();
}

// BLANKT[i] = datos_t[i]/float(RES*cnt) where cnt > 0.01 (datos_t = RES*file).
__global__ void blankt_kernel(const float* __restrict__ cnt, const float* __restrict__ t, float res, float* bl,
                              size_t n) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float val = cnt[i];
  bl[i] = ((double)val > 0.01) ? __fdiv_rn(__fmul_rn(res, t[i]), __fmul_rn(res, val)) : 0.f;
}

cudaError_t launch_blankt(const DevGeom& g, const float* cnt, const float* tsino_raw, float* blankt,
                          cudaStream_t st) {
  const size_t n = (size_t)g.P * g.nang * g.nrad;
  blankt_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(cnt, tsino_raw, (float)g.res, blankt, n);
  return cudaGetLastError();
}

// ---- VLOR split in the reference's order ------------------------------------
// The reference adds each event's two shares to their bins in file order
// (GFIRST.cu:373-389), so a bin's sum is its shares added in event order.
// One 64-bit key per event end, (bin << 32) | (2*event + end), sorted once,
// puts each bin's shares in that order; the split then sums each bin's run
// sequentially: the same additions in the same order, without atomics.
constexpr long long kVlorEventBins = 10 << 20;  // vlor_by_event
constexpr unsigned long long kNoKey = ~0ull;  // an end of a rejected event

__global__ void vlor_keys_kernel(const int32_t* __restrict__ ev, long long nev, long long ndata,
                                 unsigned long long* keys) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nev) return;
  long long i1, i2;
  const bool ok = vlor_bins(ev, e, ndata, &i1, &i2);
  keys[2 * e] = ok ? ((unsigned long long)i1 << 32) | (unsigned long long)(2 * e) : kNoKey;
  keys[2 * e + 1] = ok ? ((unsigned long long)i2 << 32) | (unsigned long long)(2 * e + 1) : kNoKey;
}

size_t vlor_sort_temp_bytes(long long nev) {
  size_t bytes = 0;
  cub::DeviceRadixSort::SortKeys(nullptr, bytes, (const unsigned long long*)nullptr,
                                 (unsigned long long*)nullptr, (int)(2 * nev), 0, 64);
  return bytes;
}

cudaError_t launch_vlor_sort(const DevGeom& g, const int32_t* ev, long long nev, unsigned long long* keys_tmp,
                             unsigned long long* keys, void* temp, size_t temp_bytes, cudaStream_t st) {
  if (nev <= 0) return cudaSuccess;
  if (nev >= (1ll << 30)) return cudaErrorInvalidValue;  // 2*event + end must fit 32 bits, counts an int
  const long long ndata = (long long)g.P * g.nang * g.nrad;
  vlor_keys_kernel<<<(unsigned)((nev + 255) / 256), 256, 0, st>>>(ev, nev, ndata, keys_tmp);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return cub::DeviceRadixSort::SortKeys(temp, temp_bytes, keys_tmp, keys, (int)(2 * nev), 0, 64, st);
}

// Two forms.  By event: one pass over the events for both shares of each, which
// reads projection and weight of two random bins, one over the sorted ends that
// adds them up.  By end: both passes walk the sorted ends, so the two file-sized
// arrays are read in address order; what is random stays in an array of 16 bytes an
// event, and an end's share is worked out where it is added.  By event where both
// arrays lie in L2.  gf_vlor_split (sort included) of 1 M / 3 M events, by event and
// by end, us, by the bins: 402, 472 / 989, 1215 at 6 K; 286, 292 / 655, 707 at 0.8 M;
// 297, 291 / 632, 665 at 7 M; 310, 300 / 653, 668 at 11 M; 319, 306 / 685, 671 at 15 M;
// 355, 338 / 775, 713 at 32 M; the same within 2 % up to 300 K events.
bool vlor_by_event(const DevGeom& g) { return (long long)g.P * g.nang * g.nrad <= kVlorEventBins; }

// The share of one end of an event, from projection and weight of its two ends.
__device__ __forceinline__ float vlor_share(float s1, float s2, float b1, float b2, bool second) {
  const float valor = __fadd_rn(b1, b2);
  const float s = __fadd_rn(s1, s2);
  const float s_inv = (s > 0.01f) ? (float)__drcp_rn((double)s) : 0.f;
  return __fmul_rn(__fmul_rn(second ? s2 : s1, s_inv), valor);
}

// by event, pass 1: share[2e + end]
__global__ void __launch_bounds__(256) vlor_shares_kernel(const int32_t* __restrict__ ev, long long nev, long long ndata,
                                                          const float* __restrict__ proj, const float* __restrict__ bl,
                                                          float2* __restrict__ share) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nev) return;
  long long i1, i2;
  if (!vlor_bins(ev, e, ndata, &i1, &i2)) return;  // its keys are kNoKey: never read
  const float s1 = proj[i1], s2 = proj[i2], b1 = bl[i1], b2 = bl[i2];
  share[e] = make_float2(vlor_share(s1, s2, b1, b2, false), vlor_share(s1, s2, b1, b2, true));
}

// by end, pass 1: projection and weight of each end's bin, ends[2e + end]
__global__ void __launch_bounds__(256) vlor_ends_kernel(const unsigned long long* __restrict__ keys, long long n,
                                                        const float* __restrict__ proj, const float* __restrict__ bl,
                                                        float2* __restrict__ ends) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const unsigned long long k = keys[i];
  if (k == kNoKey) return;
  ends[k & 0xffffffffull] = make_float2(proj[k >> 32], bl[k >> 32]);
}

// pass 2: the first end of each bin adds the bin's shares in event order.  SHARES:
// vals holds them (by event), else its events' float4 (by end).
template <bool SHARES>
__global__ void __launch_bounds__(256) vlor_split_sorted_kernel(const unsigned long long* __restrict__ keys,
                                                                long long n, const void* __restrict__ vals,
                                                                float* out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  unsigned long long k = keys[i];
  if (k == kNoKey) return;
  const unsigned long long bin = k >> 32;
  if (i > 0 && (keys[i - 1] >> 32) == bin) return;  // not the first share of its bin
  float sum = out[bin];  // the shares are added to out, as the reference adds them to SINOG_VLOR
  for (long long j = i;;) {
    const unsigned long long at = k & 0xffffffffull;
    if (SHARES) {
      sum = __fadd_rn(sum, static_cast<const float*>(vals)[at]);
    } else {
      const float4 e = static_cast<const float4*>(vals)[at >> 1];  // (projection, weight) of its two ends
      sum = __fadd_rn(sum, vlor_share(e.x, e.z, e.y, e.w, at & 1));
    }
    if (++j >= n) break;
    k = keys[j];
    if ((k >> 32) != bin) break;
  }
  out[bin] = sum;
}

cudaError_t launch_vlor_split_sorted(const DevGeom& g, const unsigned long long* keys, long long nev,
                                     const int32_t* ev, const float* proj, const float* blankt, float2* vals,
                                     float* out, cudaStream_t st) {
  if (nev <= 0) return cudaSuccess;
  const long long n = 2 * nev;
  const unsigned nb = (unsigned)((n + 255) / 256);
  if (vlor_by_event(g))
    vlor_shares_kernel<<<(unsigned)((nev + 255) / 256), 256, 0, st>>>(ev, nev, (long long)g.P * g.nang * g.nrad, proj,
                                                                      blankt, vals);
  else
    vlor_ends_kernel<<<nb, 256, 0, st>>>(keys, n, proj, blankt, vals);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (vlor_by_event(g))
    vlor_split_sorted_kernel<true><<<nb, 256, 0, st>>>(keys, n, vals, out);
  else
    vlor_split_sorted_kernel<false><<<nb, 256, 0, st>>>(keys, n, vals, out);
  return cudaGetLastError();
}

// ---- VLOR events given as LOR endpoints -----------------------------------
// One LOR (x1,y1,z1,x2,y2,z2 in mm; x/y about the axis, z about the axial
// centre) -> 0-based sinogram bin, or -1.  Inverse of gf_bin_endpoints.
__device__ long long lor_bin(const DevGeom& g, const float* e, float vx, float hs, float pi_ref) {
  const float dx = e[3] - e[0], dy = e[4] - e[1], dzm = e[5] - e[2];
  const float L = sqrtf(dx * dx + dy * dy);
  if (!(L > 0.f)) return -1;
  float ux = dx / L, uy = dy / L, sgn = 1.f;
  // direction (sin t, -cos t) with t in (0, pi]
  float th = atan2f(ux, -uy);
  if (th <= 0.f) {
    th += pi_ref;
    sgn = -sgn;
  }
  int t = __float2int_rn((pi_ref - th) * (float)g.nang / pi_ref);
  if (t >= g.nang) {
    t -= g.nang;
    sgn = -sgn;
  }
  if (t < 0) t += g.nang;
  const float2 sc = g.trig[t];  // (sin, cos)
  ux = sgn * (dx / L);
  uy = sgn * (dy / L);
  const float x0mm = e[0] * sc.y + e[1] * sc.x;
  const int ird = __float2int_rn(x0mm / (vx * g.fx_fp) + g.radm);
  if (ird < 0 || ird >= g.nrad) return -1;
  const float slope = sgn * dzm / L * vx / hs;  // slices per voxel step along the ray
  int best = -1;
  float bd = 3.0e38f;
  for (int s = 0; s < g.nseg; s++) {
    const float d = fabsf(g.seg[s].dz - slope);
    if (d < bd) {
      bd = d;
      best = s;
    }
  }
  const DevSeg sg = g.seg[best];
  const float cx = x0mm * sc.y, cy = x0mm * sc.x;
  const float lam1 = ((e[0] - cx) * ux + (e[1] - cy) * uy) / vx;
  const float z0 = e[2] / hs + 0.5f * (float)g.nzs - lam1 * sg.dz;  // texel z at the closest point
  const int iz0 = __float2int_rn(z0 - 0.5f);
  if (iz0 < sg.zmin || iz0 >= g.nzs - sg.zmin) return -1;
  return ((long long)(iz0 - sg.zmin) + sg.acc) * ((long long)g.nrad * g.nang) + (long long)t * g.nrad + ird;
}

__global__ void vlor_endpoints_kernel(const DevGeom g, const float* __restrict__ lors, long long n, float vx, float hs,
                                      float pi_ref, int32_t* __restrict__ ev) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int k = 0; k < 2; k++) {
    const long long b = lor_bin(g, lors + 12 * i + 6 * k, vx, hs, pi_ref);
    ev[2 * i + k] = (int32_t)(b + 1);  // 1-based; 0 = rejected, as the reference rejects i <= 0
  }
}

cudaError_t launch_vlor_endpoints(const DevGeom& g, const float* lors, long long n, float vx, float hs, int32_t* ev,
                                  cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  vlor_endpoints_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(g, lors, n, vx, hs, 3.1415926f, ev);
  return cudaGetLastError();
}

}  // namespace gf
