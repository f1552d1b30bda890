// gf_bp_tile.cu -- voxel-driven back projector over column tiles.
//
// Reference: BACKWPROJ_K (GFIRST_GPU_Kernels.cu:109-164), one launch per
// (segment, angle) view; the same sums as gf_bp.cu, with the reference's
// operations in its order and rounding.
//
// GB300 design.  A warp owns a tile of 4x8 neighbouring image columns, one per
// lane, and a run of ZR consecutive slices; each lane keeps its run's (NUMER,
// DENOM) sums in registers for the whole subset, so the volumes (or, in a
// reconstruction, their update ratio) are written once per sub-iteration.  The
// warps of a CTA hold neighbouring tiles of the same run, so they have work at
// the same views.  At one view the CTA's columns touch a few radial bins (23
// for 16x16 columns) and the run reaches a few rows of each, so per view
// (segments outer, angles inner, the reference's order):
//  (1) one warp copies those rows into shared memory (cp.async, one group of
//      views ahead);
//  (2) every lane walks its run: ZR + 1 rows of two bins, each row
//      interpolated radially once, each voxel axially between two of them.
//
// Masks.  The normalization mask is 1 or -1000 and known before the
// reconstruction starts, so it is not interpolated sample by sample: four
// unmasked corners give exactly 1, and a masked corner gives a negative value
// (the sample is skipped) unless it weighs less than 1/1001.  A view whose
// segment has no masked row in the CTA's bins needs no mask at all; other
// views read one bit per row.  Samples with a masked corner of a tiny weight
// are evaluated one by one with the reference's expression.
//
// Bound: instruction issue (76 % of peak while SMs are busy, 463 M warp
// instructions at the preclinical subset against 777 M for one warp per
// column; data-pipe wavefronts 53 % of peak, DRAM 1 %).  Per voxel and lane
// a run costs 2 (ZR + 1) / ZR four-byte loads; the lanes of a 4x8 tile at a
// bin stride of 4 words modulo 8 conflict about 1.2-fold (16x2 tiles 1.6, 32x1
// 2.1).  Preclinical subset (128x128x159 voxels, 53 segments, 10 angles),
// FP32: 523 us per launch against 1120 us for one warp per column in the
// per-view form, 638 against 1280 us per voxel (704 with each voxel's fraction
// computed); FP16 ratios 561 against 998 us (the conversions).  With 2 % random
// gaps, per voxel, FP32 at the reference geometry: 4.32 ms for a full
// projection against 6.12 (4.64 with tiny weights looked for in every lane).
// Measured on the way: four-warp CTAs 594 us (twice the
// copies), the warps of a CTA along z instead of across columns 785 us (the
// end runs wait for the middle ones), the lanes' weights from a table in
// shared memory instead of recomputed 550 us, groups of half as many views
// 640 us (barriers).
#include <type_traits>

#include "gf_kernels.h"

namespace gf {

namespace {

constexpr unsigned kAll = 0xffffffffu;
// A masked corner weighing more than this makes the interpolated mask
// negative: 1 - 1001 w < 0 for w > 1/1001, with room for rounding.
constexpr float kTinyWeight = 0.0012f;

__device__ __forceinline__ float elem(float v) { return v; }
__device__ __forceinline__ float elem(__half v) { return __half2float(v); }
__device__ __forceinline__ float elem(__nv_bfloat16 v) { return __bfloat162float(v); }

__device__ __forceinline__ void cp_async16(unsigned s, const void* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(g));
}
__device__ __forceinline__ void cp_async4(void* s, const void* g) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(s)), "l"(g));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// a + w*(b - a) on two pairs, each element rounded as the scalar operations
__device__ __forceinline__ float2 lerp2(float2 a, float2 b, float2 w) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rc;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
      "sub.rn.f32x2 rc, rb, ra;\n\tmov.b64 {%0, %1}, rc;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return __ffma2_rn(w, d, a);
}

// A sample whose interpolated mask is 1: counted unless the ratio is negative
// (a gap zeroes both, GFIRST_GPU_Kernels.cu:157).  Predicated additions: as
// branches they cost three more instructions a voxel.
__device__ __forceinline__ void count_sample(float& num, float& den, float v) {
  asm("{\n\t.reg .pred p;\n\tsetp.geu.f32 p, %2, 0f00000000;\n\t@p add.rn.f32 %0, %0, %2;\n\t"
      "@p add.rn.f32 %1, %1, 0f3F800000;\n\t}"
      : "+f"(num), "+f"(den)
      : "f"(v));
}
// The same where `bit` is set in `ok`.
__device__ __forceinline__ void count_sample(float& num, float& den, float v, unsigned ok, unsigned bit) {
  asm("{\n\t.reg .pred p, q;\n\t.reg .b32 t;\n\tand.b32 t, %3, %4;\n\tsetp.ne.u32 q, t, 0;\n\t"
      "setp.geu.and.f32 p, %2, 0f00000000, q;\n\t@p add.rn.f32 %0, %0, %2;\n\t@p add.rn.f32 %1, %1, 0f3F800000;\n\t}"
      : "+f"(num), "+f"(den)
      : "f"(v), "r"(ok), "r"(bit));
}

// bits lo..hi-1 (0 <= lo, hi <= 31)
__device__ __forceinline__ unsigned bits(int lo, int hi) {
  return hi > lo ? ((1u << hi) - 1u) & ~((1u << lo) - 1u) : 0u;
}

// A staged view: what its lanes share (three 16-byte words), then the mask
// words of its bins where a bin has masked rows, then the rows.
//  [0] 1 + the first bin (0: no voxel in range) | row offsets from the pad row for which a
//      whole run needs no mask (0: none) | 1 if the pad rows are gaps | rows
//      with the pad rows
//  [1] fz | z0 - (zmin - 1) | element of row 0 of the first bin | angle
//  [2] mask bit of row 0 (0: no masked rows) | row 0 in the sinogram | zmin | -
constexpr int kHeadBytes = 48;

// A column at one angle (GFIRST_GPU_Kernels.cu:136-146): its two radial bins
// (clamped), their weight, and yrot.
struct Radial {
  int i0, i1;
  float al, yrot;
};
__device__ __forceinline__ Radial radial_of(const DevGeom& g, float xv, float yv, float sn, float cs) {
  Radial p;
  const float xrot = __fadd_rn(__fmul_rn(xv, cs), __fmul_rn(yv, sn));
  p.yrot = __fadd_rn(__fmul_rn(-xv, sn), __fmul_rn(yv, cs));
  const float x = __fadd_rn(__fadd_rn(g.radm, __fmul_rn(xrot, g.fx_bp)), 0.5f);
  const float xb = __fsub_rn(x, 0.5f);
  const float fl = floorf(xb);
  const int i = (int)fl;
  p.i0 = clampi(i, 0, g.nrad - 1);
  p.i1 = clampi(i + 1, 0, g.nrad - 1);
  p.al = __fsub_rn(xb, fl);
  return p;
}

}  // namespace

// FAST: the per-view axial form (gf_set_bp_form).
template <int ZR, class T, bool FAST>
__global__ void __launch_bounds__(256) bp_tile_kernel(const BpArgs a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  constexpr int VE = 16 / (int)sizeof(T);  // elements of one 16-byte copy
  constexpr int PADF = bp_pad_front(ZR, (int)sizeof(T));
  if (a.general && *a.general) return;  // gf_bp.cu interpolates such masks
  const DevGeom& g = a.g;
  const BpFrame& F = a.fr[blockIdx.z];
  const T* __restrict__ corr = static_cast<const T*>(F.in);
  const int nw = blockDim.x >> 5, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rs = a.rs, mw = a.mw;
  // per angle: first bin, bins, extremes of yrot over the CTA's columns; sin,
  // cos, and the segments (up to 64) with a masked row in those bins
  int4* angles = reinterpret_cast<int4*>(smraw);
  unsigned char* slots = smraw + 32 * a.na;

  // The CTA's columns are 2 warp tiles wide in y, nw / 2 in x; its run of
  // slices is the blockIdx.y-th from the middle of the image outwards (the
  // middle runs see the most views and start first).
  const int cx = kTileX * (nw >> 1), cy = kTileY * 2;
  const int ncx = (g.res + cx - 1) / cx;
  const int cx0 = (blockIdx.x % ncx) * cx, cy0 = (blockIdx.x / ncx) * cy;
  const int mid = (int)gridDim.y >> 1, by = blockIdx.y;
  const int z0 = ((int)gridDim.y - 1 - mid + ((by & 1) ? (by + 1) >> 1 : -(by >> 1))) * ZR;
  const int nv = min(ZR, g.nzs - z0);  // slices of the run inside the image
  // this lane's column (a tile that reaches past the image repeats its last columns)
  const int ix = cx0 + (w >> 1) * kTileX + lane % kTileX, iy = cy0 + (w & 1) * kTileY + lane / kTileX;
  const bool mine = ix < g.res && iy < g.res;
  // a warp whose whole tile is past the image only stages
  const bool inside = cx0 + (w >> 1) * kTileX < g.res && cy0 + (w & 1) * kTileY < g.res;
  const float xv = __fsub_rn((float)min(ix, g.res - 1), g.resm), yv = __fsub_rn((float)min(iy, g.res - 1), g.resm);
  // a corner of the CTA's columns: every coordinate is monotone in x and in y,
  // rounding included, so its extremes over the columns are at the corners
  const float xc = __fsub_rn((float)min((lane & 1) ? cx0 + cx - 1 : cx0, g.res - 1), g.resm);
  const float yc = __fsub_rn((float)min((lane & 2) ? cy0 + cy - 1 : cy0, g.res - 1), g.resm);

  for (int tl = w; tl < a.na; tl += nw) {
    const float2 sc = g.trig[subset_angle(g, a.subset, tl)];
    const Radial c = radial_of(g, xc, yc, sc.x, sc.y);
    const int bmin = __reduce_min_sync(kAll, c.i0), nb = __reduce_max_sync(kAll, c.i1) - bmin + 1;
    float lo = fminf(c.yrot, __shfl_xor_sync(kAll, c.yrot, 1)), hi = fmaxf(c.yrot, __shfl_xor_sync(kAll, c.yrot, 1));
    lo = fminf(lo, __shfl_xor_sync(kAll, lo, 2));
    hi = fmaxf(hi, __shfl_xor_sync(kAll, hi, 2));
    unsigned d0 = 0, d1 = 0;
    for (int b = lane; b < nb; b += 32) {
      const unsigned* d = F.dirty + (size_t)(tl * g.nrad + bmin + b) * a.nsw;
      d0 |= d[0];
      if (a.nsw > 1) d1 |= d[1];
    }
    d0 = __reduce_or_sync(kAll, d0);
    d1 = __reduce_or_sync(kAll, d1);
    if (lane == 0) {
      angles[2 * tl] = make_int4(bmin, nb, __float_as_int(lo), __float_as_int(hi));
      angles[2 * tl + 1] = make_int4(__float_as_int(sc.x), __float_as_int(sc.y), (int)d0, (int)d1);
    }
  }
  __syncthreads();
  // Stages view (s, tl) into a slot.
  auto stage = [&](int s, int tl, unsigned char* slot) {
    const DevSeg sg = g.seg[s];
    const int4 e = angles[2 * tl], e2 = angles[2 * tl + 1];
    const int k0 = (int)floorf(__fmul_rn(__int_as_float(e.z), sg.fz)), k1 = (int)floorf(__fmul_rn(__int_as_float(e.w), sg.fz));
    const int kmin = min(k0, k1) - (sg.zmin - 1), kmax = max(k0, k1) - (sg.zmin - 1);
    const int bmin = e.x, nb = e.y, nrow = sg.nplanes + 2, pad = s == 0 ? 0 : 1;
    const int ra = max(0, z0 + kmin), rb = min(nrow - 1, z0 + ZR + kmax + 1);
    const bool active = z0 + kmax + nv - 1 >= 0 && z0 + kmin <= nrow - 2;
    int4* h = reinterpret_cast<int4*>(slot);
    if (!active) {
      if (lane == 0) h[0] = make_int4(0, 0, 0, 0);
      return;
    }
    const int base = (sg.blk + ra) & ~(VE - 1);
    const int nvec = (sg.blk + rb - base) / VE + 1;
    // lanes along a bin's rows; narrow views take several bins at a time
    const int sh = nvec > 16 ? 5 : (nvec > 8 ? 4 : 3);
    const int b0 = lane >> sh, v0 = lane & ((1 << sh) - 1), db = 32 >> sh;
    const char* src = reinterpret_cast<const char*>(corr + (size_t)(tl * g.nrad + bmin) * g.PS + base);
    const unsigned dst = (unsigned)__cvta_generic_to_shared(slot) + a.rows_at + PADF * (unsigned)sizeof(T);
    for (int v = v0; v < nvec; v += 1 << sh) {
      const char* p = src + (unsigned)(b0 * g.PS) * (unsigned)sizeof(T) + 16u * v;
      unsigned d = dst + (unsigned)(b0 * rs) * (unsigned)sizeof(T) + 16u * v;
#pragma unroll 1
      for (int b = b0; b < nb; b += db) {
        cp_async16(d, p);
        p += (unsigned)(db * g.PS) * (unsigned)sizeof(T);
        d += (unsigned)(db * rs) * (unsigned)sizeof(T);
      }
    }
    bool dirty;
    if (s < 64) {
      dirty = ((s < 32 ? e2.z : e2.w) >> (s & 31)) & 1;
    } else {
      unsigned dw = 0;
      for (int b = lane; b < nb; b += 32) dw |= F.dirty[(size_t)(tl * g.nrad + bmin + b) * a.nsw + (s >> 5)];
      dirty = __any_sync(kAll, (dw >> (s & 31)) & 1u);
    }
    int mbit = 0;
    if (dirty) {
      // mask words of the staged rows, at words 1..n of a bin
      const int wb = ((sg.blk + ra) >> 5) - 1, n = ((sg.blk + rb) >> 5) - wb;
      mbit = sg.blk - 32 * wb;
      unsigned* mbits = reinterpret_cast<unsigned*>(slot + kHeadBytes);
      for (int b = lane; b < nb; b += 32)
        for (int q = 1; q <= n; q++)
          cp_async4(mbits + b * mw + q, F.mask + (size_t)(tl * g.nrad + bmin + b) * (g.PS >> 5) + (wb + q));
    }
    if (lane == 0) {
      h[0] = make_int4(1 + bmin, dirty ? 0 : max(0, nrow - 2 * pad - nv), pad, nrow);
      h[1] = make_int4(__float_as_int(sg.fz), z0 - (sg.zmin - 1), sg.blk - base + PADF, tl);
      h[2] = make_int4(mbit, sg.blk, sg.zmin, dirty ? 1 : 0);
    }
  };

  float num[ZR], den[ZR];
#pragma unroll
  for (int i = 0; i < ZR; i++) num[i] = den[i] = 0.f;

  auto view = [&](const unsigned char* slot) {
    const int4 h = reinterpret_cast<const int4*>(slot)[0];
    if (!h.x) return;
    const int4 h1 = reinterpret_cast<const int4*>(slot)[1];
    const int4 e2 = angles[2 * h1.w + 1];
    const Radial c = radial_of(g, xv, yv, __int_as_float(e2.x), __int_as_float(e2.y));
    const float al = c.al;
    const float t = __fmul_rn(c.yrot, __int_as_float(h1.x)), ft = floorf(t);  // t = yrot*fz
    const int j0 = (int)ft + h1.y;  // row of the run's first voxel: voxel z lies between rows z + k and z + k + 1
    const int pad = h.z, nrow = h.w;

    // Rows j0 + i of the lane's two bins.
    const int ba = c.i0 - (h.x - 1), bb = c.i1 - (h.x - 1);
    const T* rows = reinterpret_cast<const T*>(slot + a.rows_at) + h1.z + j0;
    const T *pa = rows + ba * rs, *pb = rows + bb * rs;
    auto ra = [&](int i) { return elem(pa[i]); };
    auto rb = [&](int i) { return elem(pb[i]); };
    auto radial = [&](int i) { return lerp_rn(ra(i), rb(i), al); };

    // Axial fractions.  Per voxel: z = float(iz) + yrot*fz + 0.5f
    // (GFIRST_GPU_Kernels.cu:148) with each sum rounded; its floor is that of
    // iz + t unless the sums round up to the next integer, which takes a
    // fraction of t within their rounding of 1 (|z| < 512: 5e-5).
    const float be = __fsub_rn(t, ft);
    const bool edge = !FAST && be > 0.9999f;  // such a lane: every voxel is evaluated on its own
    auto frac = [&](int i) {
      const float fiz = (float)(z0 + i);
      const float zb = __fsub_rn(__fadd_rn(__fadd_rn(fiz, t), 0.5f), 0.5f);
      return __fsub_rn(zb, fiz + ft);
    };
    // Those sums round the fraction of t to the spacing of floats at n = iz +
    // floor(t), as long as n and n + 1 lie in one power-of-two interval: where
    // the whole run does, its first voxel's fraction is every voxel's (five
    // additions a voxel less in most runs).
    const int n0 = z0 + (int)ft;
    const float bf = FAST ? be : frac(0);
    const bool flat = FAST || __all_sync(kAll, n0 > 0 && __clz(n0) == __clz(n0 + ZR));

    // every voxel of every lane between two rows of the segment, no dead bin
    auto interior = [&](auto one) {
      float S[ZR + 1];
      const float2 al2 = make_float2(al, al);
#pragma unroll
      for (int i = 0; i < ZR; i += 2) {
        const float2 v = lerp2(make_float2(ra(i), ra(i + 1)), make_float2(rb(i), rb(i + 1)), al2);
        S[i] = v.x;
        S[i + 1] = v.y;
      }
      S[ZR] = radial(ZR);
      int sign = 0;
#pragma unroll
      for (int i = 0; i < ZR; i++) {
        S[i] = lerp_rn(S[i], S[i + 1], one ? bf : frac(i));
        sign |= __float_as_int(S[i]);
      }
      if (!__any_sync(kAll, sign < 0)) {
#pragma unroll
        for (int i = 0; i < ZR; i += 2) {
          const float2 n = __fadd2_rn(make_float2(num[i], num[i + 1]), make_float2(S[i], S[i + 1]));
          const float2 d = __fadd2_rn(make_float2(den[i], den[i + 1]), make_float2(1.f, 1.f));
          num[i] = n.x;
          num[i + 1] = n.y;
          den[i] = d.x;
          den[i + 1] = d.y;
        }
      } else {
#pragma unroll
        for (int i = 0; i < ZR; i++) count_sample(num[i], den[i], S[i]);
      }
    };
    if (__all_sync(kAll, (unsigned)(j0 - pad) < (unsigned)h.y && !edge)) {
      if (flat)
        interior(std::true_type());
      else
        interior(std::false_type());
      return;
    }

    const int4 h2 = reinterpret_cast<const int4*>(slot)[2];
    const int first = max(0, -j0), last = min(nv, nrow - 1 - j0);
    const bool has = last > first;  // this lane has voxels in the range
    if (!has) pa = pb = reinterpret_cast<const T*>(slot + a.rows_at);  // and reads the slot's first rows otherwise
    const unsigned range = bits(first, max(last, 0));
    // Mask bits of rows j0 + i, i = 0..31, of the two bins.
    unsigned ma, mb;
    if (h2.w) {
      const unsigned* mbits = reinterpret_cast<const unsigned*>(slot + kHeadBytes);
      const int q = has ? h2.x + j0 : 0;
      const unsigned *qa = mbits + ba * mw + (q >> 5), *qb = mbits + bb * mw + (q >> 5);
      ma = __funnelshift_r(qa[0], qa[1], q & 31);
      mb = __funnelshift_r(qb[0], qb[1], q & 31);
    } else {
      ma = mb = bits(clampi(pad - j0, 0, 31), clampi(nrow - pad - j0, 0, 31));
    }
    const unsigned m = ma & mb;
    const unsigned ok = edge ? 0u : m & (m >> 1) & range;  // four unmasked corners
    // The mask can only be positive with a masked corner where every masked
    // corner weighs next to nothing; those voxels (and the edge lanes') are
    // evaluated one by one.  Per voxel, the fractions are within 5e-5 of be.
    // Most warps have no lane with both such a weight and a masked row.
    const float wa = 1.f - al, wl = 1.f - be;
    const bool tiny = ok != range && (fminf(wa, al) * fminf(wl, be) <= kTinyWeight || edge);
    // The lanes' ranges differ by little: most runs at an edge have stretches
    // that no lane needs.
    constexpr int ZG = 4;
    static_assert(ZR % ZG == 0, "whole stretches");
    const unsigned some = __reduce_or_sync(kAll, ok);
    auto masked = [&](auto one) {
#pragma unroll
      for (int i0 = 0; i0 < ZR; i0 += ZG) {
        if (!(some & (((1u << ZG) - 1u) << i0))) continue;  // whole warp
        float S = radial(i0);
#pragma unroll
        for (int i = i0; i < i0 + ZG; i++) {
          const float Sn = radial(i + 1);
          const float v = lerp_rn(S, Sn, one ? bf : frac(i));
          S = Sn;
          count_sample(num[i], den[i], v, ok, 1u << i);
        }
      }
    };
    if (flat)
      masked(std::true_type());
    else
      masked(std::false_type());
    if (!__any_sync(kAll, tiny)) return;
    auto unless = [](float wgt) { return wgt <= kTinyWeight ? kAll : 0u; };
    unsigned cand = (ma | unless(wa * wl)) & ((ma >> 1) | unless(wa * be)) & (mb | unless(al * wl)) &
                    ((mb >> 1) | unless(al * be)) & range & ~ok;
    if (edge) cand = has ? bits(0, last) : 0u;
    const unsigned any = __reduce_or_sync(kAll, cand);
    if (any) {
      const float zlo = (float)h2.z, zhi = (float)(g.nzs - h2.z);
#pragma unroll
      for (int i = 0; i < ZR; i++) {
        if (!(any & (1u << i))) continue;  // whole warp
        if (!(cand & (1u << i))) continue;
        int d = i;
        float b = be;
        bool in = true;
        if constexpr (!FAST) {
          const float fiz = (float)(z0 + i);
          const float z = __fadd_rn(__fadd_rn(fiz, t), 0.5f), zb = __fsub_rn(z, 0.5f), fz = floorf(zb);
          b = __fsub_rn(zb, fz);
          d = (int)fz - h2.z + 1 - j0;  // i, or i + 1 where the sum rounded up
          in = z >= zlo && z < zhi && d + j0 >= 0;
        }
        if (!in) continue;
        const float a0 = (ma >> d & 1u) ? 1.f : -1000.f, b0 = (mb >> d & 1u) ? 1.f : -1000.f;
        const float a1 = (ma >> (d + 1) & 1u) ? 1.f : -1000.f, b1 = (mb >> (d + 1) & 1u) ? 1.f : -1000.f;
        const float vc = lerp_rn(lerp_rn(a0, b0, al), lerp_rn(a1, b1, al), b);
        const float vr = lerp_rn(radial(d), radial(d + 1), b);
        if (!(vc < 0.f || vr < 0.f)) {
          num[i] = __fadd_rn(num[i], vr);
          den[i] = __fadd_rn(den[i], vc);
        }
      }
    }
  };

  // Views in order, a group of one per warp at a time: while the CTA works on
  // one group, the warps stage the next into the other half of the slots.
  const int nviews = g.nseg * a.na;
  auto slot_of = [&](int buf, int u) { return slots + (size_t)(buf * nw + u) * a.slot_bytes; };
  int s = w / a.na, tl = w - s * a.na;  // the view this warp stages next: every nw-th
  if (w < nviews) stage(s, tl, slot_of(0, w));
  cp_async_commit();
  int buf = 0;
  for (int v0 = 0; v0 < nviews; v0 += nw) {
    cp_async_wait_all();
    __syncthreads();  // the group is staged, and every warp is done with the other half
    tl += nw;
    while (tl >= a.na) {
      tl -= a.na;
      s++;
    }
    if (v0 + nw + w < nviews) stage(s, tl, slot_of(buf ^ 1, w));
    cp_async_commit();
    const int n = min(nw, nviews - v0);
    if (inside)
      for (int u = 0; u < n; u++) view(slot_of(buf, u));
    buf ^= 1;
  }

  // The run's sums, or with `ratio` the update ratio of the two alone in
  // NUMER's buffer; padding slices 0, or 1 (the ratio of zero sums).
  if (!mine) return;
  const size_t cb = ((size_t)iy * g.res + ix) * g.nzp;
#pragma unroll
  for (int i = 0; i < ZR; i += 4) {
    if (z0 + i >= g.nzp) break;
    float n4[4], d4[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const bool in = i + q < nv;
      n4[q] = a.ratio ? (in ? update_ratio(num[i + q], den[i + q]) : 1.f) : (in ? num[i + q] : 0.f);
      d4[q] = in ? den[i + q] : 0.f;
    }
    *reinterpret_cast<float4*>(F.numer + cb + z0 + i) = make_float4(n4[0], n4[1], n4[2], n4[3]);
    if (!a.ratio) *reinterpret_cast<float4*>(F.denom + cb + z0 + i) = make_float4(d4[0], d4[1], d4[2], d4[3]);
  }
  if (z0 + ZR >= g.nzs)
    for (int z = z0 + ZR; z < g.nzp; z++) {
      F.numer[cb + z] = a.ratio ? 1.f : 0.f;
      if (!a.ratio) F.denom[cb + z] = 0.f;
    }
}

template <int ZR, class T>
static cudaError_t launch_tiles_t(const BpArgs& a, int warps, cudaStream_t st) {
  auto k = a.fast ? bp_tile_kernel<ZR, T, true> : bp_tile_kernel<ZR, T, false>;
  const size_t smem = (size_t)32 * a.na + (size_t)2 * warps * a.slot_bytes;
  if (smem > 48 * 1024) {
    cudaError_t e = allow_max_smem(k);
    if (e != cudaSuccess) return e;
  }
  const int cx = kTileX * (warps / 2), cy = kTileY * 2;
  const dim3 grid(((a.g.res + cx - 1) / cx) * ((a.g.res + cy - 1) / cy), (a.g.nzs + ZR - 1) / ZR, a.nfr);
  k<<<grid, warps * 32, smem, st>>>(a);
  return cudaGetLastError();
}

template <int ZR>
static cudaError_t launch_tiles_z(const BpArgs& a, int warps, cudaStream_t st) {
  switch (a.storage) {
    case 0: return launch_tiles_t<ZR, float>(a, warps, st);
    case 1: return launch_tiles_t<ZR, __half>(a, warps, st);
    case 2: return launch_tiles_t<ZR, __nv_bfloat16>(a, warps, st);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_bp_tiles(const BpArgs& in, const BpTile& tile, cudaStream_t st) {
  BpArgs a = in;
  a.nsw = (a.g.nseg + 31) / 32;
  a.rs = tile.rs;
  a.mw = tile.mw;
  a.rows_at = tile.rows_at;
  a.slot_bytes = tile.slot_bytes;
  switch (tile.zr) {
    case kTileRun: return launch_tiles_z<kTileRun>(a, tile.warps, st);
    case kShortRun: return launch_tiles_z<kShortRun>(a, tile.warps, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace gf
