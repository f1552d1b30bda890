// gf_fp.cu -- forward projector with the fused data/projection ratio.
//
// Reference: FORWPROJ_K (GFIRST_GPU_Kernels.cu:40-102), one launch per
// (segment, angle) view with a blocking copy and a host scatter per launch
// (GFIRST.cu:346-365), then the ratio loop of GFIRST.cu:413-430.
//
// GB300 design.  One CTA owns one angle and NB (1 or 4) neighbouring radial
// bins: every ray of an (angle, bin) pair, across all segments and planes, is
// parallel and shares the in-plane sample positions (x, y) of each step lambda;
// only z differs.  So the CTA
//  (1) resamples the image once per step onto a z column per bin, B[lambda][z]
//      = bilinear_xy(image[z], x(lambda), y(lambda)), reading the four z-fast
//      image columns around (x, y) with coalesced vector loads (image in L2);
//  (2) sums every ray from shared memory: ray (segment, plane iz0) at step
//      lambda needs B[lambda] at z = iz0 + lambda*dz, a 1-D interpolation whose
//      integer offset and fraction are the same for all planes of a segment, so
//      a thread walks a run of R consecutive planes with R+1 shared loads (of
//      NB floats) and R interpolations per step, two bins at a time as packed
//      FP32 operations;
//  (3) passes the projections through shared memory into plane order, applies
//      the ratio and writes the radial-major layout the back projector reads
//      in whole lines.
// Work per ray-sample is 1/NB shared loads and one 1-D interpolation instead of
// eight texel reads; the image and data stream from HBM once.
//
// Bound: shared-memory wavefronts, a half of them conflicts between the
// segments whose runs share a warp (NB = 1: 2.06 wavefronts per load; NB = 4,
// where a load is served by quarter warps: 1.4).  128x128x159 voxels, 53
// segments, 10 angles with the ratio 268 -> 250 us by resampling four slices a
// thread and reading the data in whole lines, 241 with 40 registers; 15 segments,
// 21 angles 279 -> 221; the whole sinogram of 168 angles x 1293 planes 1934 -> 1263
// (four bins); 64x64x32 voxels, 16 angles 36 -> 29.  Two bins a CTA (264, 222 with
// the ratio) lost to either side of it.
#include <algorithm>

#include "gf_kernels.h"

namespace gf {

namespace {

// The values of NB neighbouring radial bins at one sample or plane.
template <int NB>
struct alignas(4 * NB) Bins {
  float v[NB];
};

// acc += a + w*(b - a), the sample's interpolation then the sum, each operation
// rounded on its own; two bins at a time as packed operations (sm_100+ f32x2).
template <int NB>
__device__ __forceinline__ void add_sample(Bins<NB>& acc, const Bins<NB>& a, const Bins<NB>& b, float w) {
  if constexpr (NB == 1) {
    acc.v[0] += lerp_rn(a.v[0], b.v[0], w);
  } else {
#pragma unroll
    for (int i = 0; i < NB; i += 2) {
      const float2 a2 = make_float2(a.v[i], a.v[i + 1]);
      float2 d;
      asm("{\n\t.reg .b64 ra, rb, rc;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
          "sub.rn.f32x2 rc, rb, ra;\n\tmov.b64 {%0, %1}, rc;\n\t}"
          : "=f"(d.x), "=f"(d.y)
          : "f"(a2.x), "f"(a2.y), "f"(b.v[i]), "f"(b.v[i + 1]));
      const float2 s = __fadd2_rn(make_float2(acc.v[i], acc.v[i + 1]), __ffma2_rn(make_float2(w, w), d, a2));
      acc.v[i] = s.x;
      acc.v[i + 1] = s.y;
    }
  }
}

// NB consecutive floats from global memory (aligned to their size).
template <int NB>
__device__ __forceinline__ Bins<NB> ldg_bins(const float* p) {
  Bins<NB> r;
  static_assert(NB == 2 || NB == 4, "a vector load");
  if constexpr (NB == 2) {
    const float2 v = __ldg(reinterpret_cast<const float2*>(p));
    r.v[0] = v.x;
    r.v[1] = v.y;
  } else {
    const float4 v = __ldg(reinterpret_cast<const float4*>(p));
    r.v[0] = v.x;
    r.v[1] = v.y;
    r.v[2] = v.z;
    r.v[3] = v.w;
  }
  return r;
}

}  // namespace

// PAIRS: the ratio output is (ratio, mask) pairs.
template <int R, int NB, bool RATIO, bool FULL, int STORE, bool PAIRS>
__device__ __forceinline__ void project(const FpArgs& a) {
  using V = Bins<NB>;
  constexpr int ZV = NB == 1 ? 4 : 2;  // slices resampled by a thread at a time
  extern __shared__ __align__(16) unsigned char smraw[];
  const int lc = a.lc, cw = a.cw;
  V* col = reinterpret_cast<V*>(smraw);                       // [lc][cw]
  int4* offs = reinterpret_cast<int4*>(col + (size_t)lc * cw);  // [lc][NB]; cw is a multiple of 4
  float2* wts = reinterpret_cast<float2*>(offs + lc * NB);    // [lc][NB]

  const DevGeom& g = a.g;
  const FpFrame& F = a.fr[blockIdx.z];
  const int ird = blockIdx.x * NB, tl = blockIdx.y;
  // a frame with fewer angles in its subset than the launch's largest: its
  // surplus blocks march no rays and write nothing (an early return here
  // costs the kernel 13 registers)
  const bool active = tl < F.na;
  const int lam_end = active ? g.lam1 : g.lam0 - 1;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int theta = subset_angle(F.subset, F.nsub, active ? tl : 0);
  const float2 sc = g.trig[theta];
  const float sn = sc.x, cs = sc.y;
  const float dx = sn, dy = -cs;
  const int RES = g.res, NZS = g.nzs, NZP = g.nzp;

  int4 run = make_int4(-1, 0, 0, 0);
  if (tid < a.nruns) run = a.runs[tid];
  float dz = 0.f;
  int zbase = 0;
  if (run.x >= 0) {
    dz = g.seg[run.x].dz;
    zbase = a.padl + run.y;
  }
  V acc[R];
#pragma unroll
  for (int j = 0; j < R; j++)
#pragma unroll
    for (int b = 0; b < NB; b++) acc[j].v[b] = 0.f;

  const int npad = cw - NZS;
  for (int lb = g.lam0; lb <= lam_end; lb += lc) {
    const int nl = min(lc, g.lam1 - lb + 1);
    for (int e = tid; e < nl * NB; e += nt) {
      const int l = e / NB, b = e - l * NB;
      // GFIRST_GPU_Kernels.cu:79-87 (fac = RES/NPT = 1 makes dx = sin, dy = -cos exactly);
      // a bin past the last one repeats it
      const float x0 = __fmul_rn(g.fx_fp, __fsub_rn((float)min(ird + b, g.nrad - 1), g.radm));
      const float xc = __fadd_rn(__fadd_rn(g.resm, __fmul_rn(x0, cs)), 0.5f);
      const float yc = __fadd_rn(__fadd_rn(g.resm, __fmul_rn(x0, sn)), 0.5f);
      const float fl = (float)(lb + l);
      const float x = __fadd_rn(xc, __fmul_rn(fl, dx));
      const float y = __fadd_rn(yc, __fmul_rn(fl, dy));
      const float xb = __fsub_rn(x, 0.5f), yb = __fsub_rn(y, 0.5f);
      const float fx = floorf(xb), fy = floorf(yb);
      const int i = (int)fx, j = (int)fy;
      const int i0 = clampi(i, 0, RES - 1), i1 = clampi(i + 1, 0, RES - 1);
      const int j0 = clampi(j, 0, RES - 1), j1 = clampi(j + 1, 0, RES - 1);
      offs[e] = make_int4((j0 * RES + i0) * NZP, (j0 * RES + i1) * NZP, (j1 * RES + i0) * NZP, (j1 * RES + i1) * NZP);
      wts[e] = make_float2(__fsub_rn(xb, fx), __fsub_rn(yb, fy));
    }
    __syncthreads();
    // ZV slices a thread: one 4 ZV-byte load per corner column
    const int nzq = NZP / ZV;
    for (int idx = tid; idx < nl * nzq; idx += nt) {
      const int l = (int)(((float)idx + 0.5f) * a.inv_nzq[ZV == 4]), z = (idx - l * nzq) * ZV;
      V c[ZV];
#pragma unroll
      for (int b = 0; b < NB; b++) {
        const int4 o = offs[l * NB + b];
        const float2 w = wts[l * NB + b];
        const Bins<ZV> v00 = ldg_bins<ZV>(F.img + (o.x + z)), v10 = ldg_bins<ZV>(F.img + (o.y + z));
        const Bins<ZV> v01 = ldg_bins<ZV>(F.img + (o.z + z)), v11 = ldg_bins<ZV>(F.img + (o.w + z));
#pragma unroll
        for (int k = 0; k < ZV; k++)
          c[k].v[b] = lerp_rn(lerp_rn(v00.v[k], v10.v[k], w.x), lerp_rn(v01.v[k], v11.v[k], w.x), w.y);
      }
      V* to = col + l * cw + a.padl + z;
      if (z + ZV <= NZS) {
        if constexpr (NB * ZV <= 4) {
          Bins<NB * ZV> q;
#pragma unroll
          for (int k = 0; k < ZV; k++)
#pragma unroll
            for (int b = 0; b < NB; b++) q.v[k * NB + b] = c[k].v[b];
          *reinterpret_cast<Bins<NB * ZV>*>(to) = q;
        } else {
#pragma unroll
          for (int k = 0; k < ZV; k++) to[k] = c[k];
        }
      } else {
#pragma unroll
        for (int k = 0; k < ZV; k++)
          if (z + k < NZS) to[k] = c[k];
      }
    }
    __syncthreads();
    if (npad > 0) {
      for (int l = tid >> 5; l < nl; l += nt >> 5) {
        V* c = col + l * cw;
        const V lo = c[a.padl], hi = c[a.padl + NZS - 1];
        for (int p = tid & 31; p < npad; p += 32) {
          if (p < a.padl) c[p] = lo;
          else c[NZS + p] = hi;
        }
      }
      __syncthreads();
    }
    if (run.x >= 0) {
      for (int l = 0; l < nl; l++) {
        const float t = __fmul_rn((float)(lb + l), dz);
        const float mf = floorf(t);
        const float f = __fsub_rn(t, mf);
        const V* c = col + l * cw + zbase + (int)mf;
        V va = c[0];
#pragma unroll
        for (int j = 0; j < R; j++) {
          const V vb = c[j + 1];
          add_sample(acc[j], va, vb, f);
          va = vb;
        }
      }
    }
    __syncthreads();
  }

  if (!active) return;  // whole block
  DevSeg sg{};
  if (run.x >= 0) sg = g.seg[run.x];
  const int plane = sg.acc + (run.y - sg.zmin);  // of the run's first ray
  if constexpr (FULL) {
    if (run.x < 0) return;
    const size_t step = (size_t)g.nrad * g.nang;
    float* to = F.proj_full + (size_t)plane * step + (size_t)theta * g.nrad + ird;
#pragma unroll
    for (int j = 0; j < R; j++) {
      if (j < run.z) {
#pragma unroll
        for (int b = 0; b < NB; b++)
          if (NB == 1 || ird + b < g.nrad) to[(size_t)j * step + b] = acc[j].v[b];
      }
    }
  }
  if constexpr (RATIO) {
    // the projections in plane order through shared memory, so that the data
    // are read and the ratios written in whole lines
    static_assert(NB == 1, "ratios are of one bin a CTA");
    float* buf = reinterpret_cast<float*>(smraw);
    if (run.x >= 0) {
#pragma unroll
      for (int j = 0; j < R; j++)
        if (j < run.z) buf[plane + j] = acc[j].v[0];
    }
    __syncthreads();
    const size_t base = ((size_t)tl * g.nrad + ird) * g.PS;
    // U rows of a thread at a time: their planes, then their data loads, are in
    // flight together (row by row, 62x62x63 voxels and 53 segments took 52 us, now 37)
    constexpr int U = 4;
    for (int p0 = tid; p0 < g.PP; p0 += U * nt) {
      int pl[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int p = p0 + u * nt;
        pl[u] = p < g.PP ? row_plane(p, a.rowmap[p], NZS) : -1;
      }
      float2 db[U];
      float cal[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        // pad rows: segment 0's repeat its first and last plane, the others are gaps
        const int p = p0 + u * nt, row = p == 0 ? 1 : (p == NZS + 1 ? NZS : p);
        db[u] = pl[u] >= 0 ? F.dbg[base + row] : make_float2(0.f, 0.f);
        cal[u] = PAIRS && pl[u] >= 0 ? F.cal[base + row] : -1000.f;
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int p = p0 + u * nt;
        if (p >= g.PP) break;
        const float s = __fadd_rn(pl[u] >= 0 ? buf[pl[u]] : 0.f, db[u].y);
        const float corr = pl[u] >= 0 && s >= 0.01f ? __fdiv_rn(db[u].x, s) : -1000.f;
        if constexpr (PAIRS) {
          using P = typename PairT<STORE>::type;
          static_cast<P*>(F.corr)[base + p] = pair_from<P>(make_float2(corr, cal[u]));
        } else {
          using T = typename ElemT<STORE>::type;
          static_cast<T*>(F.corr)[base + p] = elem_from<T>(corr);
        }
      }
    }
  }
}

template <int R, int NB, bool RATIO, bool FULL, int STORE, bool PAIRS>
__global__ void __launch_bounds__(512, R == 9 && NB == 1 ? 2 : 1) fp_kernel(const FpArgs a) {
  project<R, NB, RATIO, FULL, STORE, PAIRS>(a);
}

// The same for CTAs of 288 threads and more: at 56 to 60 registers two or three fit
// an SM, at 40 (16 to 20 bytes spilled) three to five.  One bin, 40 registers over
// the other: 0.98 at 256 threads with the ratio, 1.01 without, 0.92 to 0.98 above
// (1.02 at 480 without), 1.01 to 1.15 below 224.
template <int R>
constexpr int fp_wide_regs = 40;

template <int R, bool RATIO, bool FULL, int STORE, bool PAIRS>
__global__ void __launch_bounds__(512) __maxnreg__(fp_wide_regs<R>) fp_wide_kernel(const FpArgs a) {
  project<R, 1, RATIO, FULL, STORE, PAIRS>(a);
}

template <int R, int NB, bool RATIO, bool FULL, int STORE, bool PAIRS>
static cudaError_t launch_fp_n(FpArgs a, const FpSchedule& s, int na, cudaStream_t st) {
  auto k = fp_kernel<R, NB, RATIO, FULL, STORE, PAIRS>;
  if constexpr (R == 9 && NB == 1)
    if (s.nthreads >= 288) k = fp_wide_kernel<R, RATIO, FULL, STORE, PAIRS>;
  if (NB > 1) a.lc = (s.lc + 1) / 2;  // as many bytes as one bin's steps twice: 43 KB at the default 32 steps and 168 floats a column
  size_t smem = (size_t)a.lc * a.cw * sizeof(Bins<NB>) + (size_t)a.lc * NB * (sizeof(int4) + sizeof(float2));
  if (RATIO) smem = std::max(smem, (size_t)a.g.P * sizeof(float));
  a.inv_nzq[0] = 2.f / (float)a.g.nzp;
  a.inv_nzq[1] = 4.f / (float)a.g.nzp;
  cudaError_t e = allow_max_smem(k);
  if (e != cudaSuccess) return e;
  dim3 grid((a.g.nrad + NB - 1) / NB, na, a.nfr > 1 ? a.nfr : 1);
  k<<<grid, s.nthreads, smem, st>>>(a);
  return cudaGetLastError();
}

template <int R, bool RATIO, bool FULL, int STORE, bool PAIRS>
static cudaError_t launch_fp_t(const FpArgs& a, const FpSchedule& s, cudaStream_t st) {
  int na = 0;
  for (int f = 0; f < (a.nfr > 1 ? a.nfr : 1); f++) na = a.fr[f].na > na ? a.fr[f].na : na;
  if constexpr (R == 9 && !RATIO)
    if (fp_bins(s, a.g.nseg, a.g.nrad, na * (a.nfr > 1 ? a.nfr : 1)) == 4)
      return launch_fp_n<R, 4, RATIO, FULL, STORE, PAIRS>(a, s, na, st);
  return launch_fp_n<R, 1, RATIO, FULL, STORE, PAIRS>(a, s, na, st);
}

template <int R, bool PAIRS>
static cudaError_t launch_fp_p(const FpArgs& a, const FpSchedule& s, cudaStream_t st) {
  switch (a.storage) {
    case 0: return launch_fp_t<R, true, false, 0, PAIRS>(a, s, st);
    case 1: return launch_fp_t<R, true, false, 1, PAIRS>(a, s, st);
    case 2: return launch_fp_t<R, true, false, 2, PAIRS>(a, s, st);
    default: return cudaErrorInvalidValue;
  }
}

template <int R>
static cudaError_t launch_fp_r(const FpArgs& a, const FpSchedule& s, cudaStream_t st) {
  if (!a.fr[0].corr) return launch_fp_t<R, false, true, 0, false>(a, s, st);
  return a.fr[0].cal ? launch_fp_p<R, true>(a, s, st) : launch_fp_p<R, false>(a, s, st);
}

cudaError_t launch_fp(const FpArgs& a, const FpSchedule& s, cudaStream_t st) {
  if (a.nfr < 0 || a.nfr > kMaxFrames) return cudaErrorInvalidValue;
  // every frame of a launch has the outputs of frame 0 (one kernel variant)
  for (int f = 0; f < (a.nfr > 1 ? a.nfr : 1); f++) {
    const FpFrame& F = a.fr[f];
    if (!F.img || (!F.corr && !F.proj_full)) return cudaErrorInvalidValue;
    if (!F.corr != !a.fr[0].corr || !F.proj_full != !a.fr[0].proj_full) return cudaErrorInvalidValue;
    if (F.corr && (!F.dbg || !F.cal != !a.fr[0].cal)) return cudaErrorInvalidValue;
    // the subset's angles: subset + l*nsub for l < na, all inside [0, nang)
    if (F.nsub < 1 || F.subset < 0 || F.subset >= F.nsub || F.na < 1 ||
        F.na != (a.g.nang - F.subset + F.nsub - 1) / F.nsub)
      return cudaErrorInvalidValue;
  }
  if (a.fr[0].corr && a.fr[0].proj_full) return cudaErrorInvalidValue;  // one output or the other
  switch (s.R) {
    case 9: return launch_fp_r<9>(a, s, st);
    case 17: return launch_fp_r<17>(a, s, st);
    case 25: return launch_fp_r<25>(a, s, st);
    case 33: return launch_fp_r<33>(a, s, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace gf
