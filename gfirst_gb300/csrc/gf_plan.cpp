// gf_plan.cpp -- geometry tables.  Every float constant is computed with the
// expression (and the float/double promotions) of the reference kernel it
// comes from, so the device code sees the reference's values.
#include "gf_plan.h"

#include <algorithm>
#include <cmath>
#include <cstdlib>

namespace gf {

static const float PI_REF = 3.1415926f;  // GFIRST.h:1

static int seg_idz(int s) { return ((s + 1) / 2) * (1 - (s % 2) * 2); }
static int seg_zmin(const Geom& g, int idz) {
  return idz == 0 ? 0 : (std::abs(idz) - 1) * g.span + (g.span / 2 + 1);
}

static bool tiles_pay(const Plan& p);

bool make_plan(const Geom& g, int nsub, Plan* out, std::string* err) {
  auto fail = [&](const char* m) {
    if (err) *err = m;
    return false;
  };
  if (g.res < 8 || g.res > 1024) return fail("res must be in [8, 1024]");
  if (g.nzs < 5 || g.nzs > 1024) return fail("nzs must be in [5, 1024]");
  if (g.nrad < 2 || g.nrad > 4096) return fail("nrad must be in [2, 4096]");
  if (g.nang < 1 || g.nang > 4096) return fail("nang must be in [1, 4096]");
  if (g.span < 1 || g.nseg < 1 || g.nseg > 1023) return fail("span and nseg must be positive (nseg < 1024)");
  if (!(g.pitch > 0.f) || !(g.diam > 0.f) || !(g.fov > 0.f)) return fail("pitch, diam and fov must be positive");
  if (nsub < 1 || nsub > g.nang) return fail("nsubsets must be in [1, nang]");
  Plan p;
  p.g = g;
  p.nsub = nsub;
  p.NZP = (g.nzs + 31) / 32 * 32;
  int acc = 0;
  const float vx = g.fov / (float)g.res;
  for (int s = 0; s < g.nseg; s++) {
    Seg sg{};
    sg.idz = seg_idz(s);
    sg.zmin = seg_zmin(g, sg.idz);
    sg.nplanes = g.nzs - 2 * sg.zmin;
    if (sg.nplanes <= 0) return fail("a segment has no planes (nzs - 2*zmin <= 0)");
    sg.acc = acc;
    sg.blk = acc + 2 * s;
    int sgn = sg.idz == 0 ? 0 : sg.idz / std::abs(sg.idz);
    // dz = (FOV/NPT)*float(idz_signo*zmin)/(0.5f*DIAM_DET)    (float)
    sg.dz = ((g.fov / (float)g.res) * (float)(sgn * sg.zmin)) / (0.5f * g.diam);
    // fz = (dx)*float(idz_signo*zmin)/(DIAM_DET/2.0)          (float product, double division)
    sg.fz = (float)((double)(vx * (float)(sgn * sg.zmin)) / ((double)g.diam / 2.0));
    acc += sg.nplanes;
    p.seg.push_back(sg);
  }
  p.P = acc;
  p.PP = acc + 2 * g.nseg;
  p.PS = (p.PP + 31) / 32 * 32;
  p.ndata = (int64_t)p.P * g.nang * g.nrad;
  p.nvox = (int64_t)g.res * g.res * g.nzs;
  p.nvoxp = (int64_t)g.res * g.res * p.NZP;
  if (p.ndata >= ((int64_t)1 << 31)) return fail("NDATA must fit in int32 (the reference's VLOR bins are int32)");
  p.sinv.resize(g.nang);
  p.cosv.resize(g.nang);
  for (int t = 0; t < g.nang; t++) {
    float ang = -(float)t / (float)g.nang * PI_REF + PI_REF;
    p.sinv[t] = sinf(ang);
    p.cosv[t] = cosf(ang);
  }
  p.radm = (float)(g.nrad - 1) * 0.5f;
  p.resm = (float)(g.res - 1) * 0.5f;
  p.fx_fp = (0.5f * g.pitch) / vx;
  p.fx_bp = vx / (float)((double)g.pitch / 2.0);
  const float tof_size = (float)g.res / (float)1;
  p.lam0 = (int)floorf((0.0f - 0.5f) * tof_size);
  p.lam1 = (int)floorf((0.0f + 0.5f) * tof_size);
  p.sub_nang.assign(nsub, 0);
  for (int t = 0; t < g.nang; t++) p.sub_nang[t % nsub]++;
  p.sub_off.assign(nsub + 1, 0);
  for (int s = 0; s < nsub; s++) p.sub_off[s + 1] = p.sub_off[s] + p.sub_elems(s);
  p.amax = *std::max_element(p.sub_nang.begin(), p.sub_nang.end());
  p.tiles = tiles_pay(p);
  *out = std::move(p);
  return true;
}

size_t FpSchedule::smem_bytes() const {
  return (size_t)lc * cw * sizeof(float) + (size_t)lc * (4 * sizeof(int) + 2 * sizeof(float));
}

bool make_fp_schedule(const Plan& p, int R, int lc, FpSchedule* out) {
  if (lc < 1 || lc > 256 || R < 1) return false;
  FpSchedule f;
  f.R = R;
  f.lc = lc;
  int kmin = 0, kmax = p.g.nzs - 1;
  for (int s = 0; s < p.g.nseg; s++) {
    const Seg& sg = p.seg[s];
    int end = p.g.nzs - sg.zmin;
    for (int p0 = sg.zmin; p0 < end; p0 += R) {
      f.runs.push_back(Run{s, p0, std::min(R, end - p0)});
      for (int lam : {p.lam0, p.lam1}) {
        float t = (float)lam * sg.dz;
        int m = (int)floorf(t);
        kmin = std::min(kmin, p0 + m);
        kmax = std::max(kmax, p0 + m + R);
      }
    }
  }
  f.nthreads = ((int)f.runs.size() + 31) / 32 * 32;
  if (f.nthreads > 512) return false;
  f.padl = (-kmin + 3) / 4 * 4;  // slice 0 of a column on a 16-byte boundary
  f.padr = kmax - (p.g.nzs - 1);
  f.cw = p.g.nzs + f.padr - kmin;
  if (f.smem_bytes() > 200 * 1024) return false;
  f.cw = (f.padl + p.g.nzs + f.padr + 3) / 4 * 4;  // at most 6 floats a step more, 6 KB at 256 steps
  *out = std::move(f);
  return true;
}

// Four bins share the loads' addresses, a quarter of the warp's conflicts and
// packed arithmetic, but make a quarter of the CTAs with twice the registers:
// they pay where those fill the GPU and a quarter warp's threads are of one
// segment.  Four bins' time over one bin's, calls of one context (layout kernel
// included), at 410 sizes, by the threads of the one-bin grid and of a CTA (nt):
//  - below 150 K threads: 0.81 to 1.61, mean 1.20 (64x64x32, 16 angles: 37 / 27 us);
//  - nt up to 64: 0.67 to 1.29, mean 0.90;
//  - nt of 96 to 192 and at least six runs of planes a segment: 0.79 to 1.16, mean
//    0.95 (15 segments, 21 angles: 201 / 228 us, 168 angles: 1263 / 1641); with
//    fewer runs 0.82 to 1.20, mean 1.03;
//  - nt of 224 and 256, two CTAs an SM: below 230 K threads 1.04 to 1.13, above 0.80
//    to 1.17, mean 0.92 (with fewer runs 1.06);
//  - nt of 288 to 384, one CTA of 9 to 12 warps an SM: 0.84 to 1.30, mean 1.06;
//  - nt from 416, one CTA of 13 to 16 warps: below 600 K threads 0.82 to 1.43, mean
//    1.13, above 0.82 to 1.10, mean 0.96 (128x128x159, 53 segments, 10 angles: 273 /
//    273 us, 320 CTAs on 152 SMs; 190 / 247 a call where another context's kernel
//    fills the last wave).
// With the ratio, whose data the fewer warps wait for, it was 0.82 to 1.52, mean
// 1.03, at 110 sizes of 1.2 M to 7 M threads, and 1.06 at eight frames of 96^3 in one
// launch: one bin.
int fp_bins(const FpSchedule& s, int nseg, int nrad, int views) {
  const int nt = s.nthreads;
  const long long threads = (long long)nrad * views * nt;
  const bool pays = threads >= (nt < 224 ? 150000 : nt <= 256 ? 230000 : 600000) && (nt <= 256 || nt >= 416) &&
                    (nt <= 64 || (int)s.runs.size() >= 6 * nseg);
  const size_t smem = (size_t)((s.lc + 1) / 2) * (s.cw + 6) * 4 * sizeof(float);  // columns, offsets and weights
  return s.R == 9 && pays && smem <= 200 * 1024 ? 4 : 1;
}

BpPads bp_fast_pads(const Plan& p) {
  // Mirrors the kernel's choice of lane chunks (all Q of them, or the NCH + 1
  // from the chunk of floor(zmin - t - 1)) and its row index j = iz +
  // floor(t) - (zmin - 1), and takes the extremes of j and j + 1 over every
  // piece of t: the functions change only where t or zmin - t crosses an
  // integer, so each integer is sampled on both sides (a float evaluation in
  // the kernel can fall only into an adjacent piece) and at its midpoint.
  const int Q = p.NZP / 32;
  const double ymax = std::sqrt(2.0) * (double)p.resm + 1.0;
  int lo = 0, hi = 0;
  for (const Seg& sg : p.seg) {
    const int nrow = sg.nplanes + 2;
    const int W = (nrow + 31) / 32 + 1;
    const double tmax = ymax * std::fabs((double)sg.fz) + 1.0;
    for (int m = (int)std::floor(-tmax) - 1; m <= (int)std::ceil(tmax) + 1; m++) {
      for (double t : {m - 1e-3, (double)m, m + 1e-3, m + 0.5}) {
        const int k = (int)std::floor(t) - (sg.zmin - 1);
        int c0 = 0, c1 = Q - 1;
        if (W < Q) {
          const int izlo = std::max((int)std::floor((double)sg.zmin - t - 1.0), 0);
          c0 = std::min(izlo >> 5, Q - W);
          c1 = c0 + W - 1;
        }
        lo = std::max(lo, -(32 * c0 + k));
        hi = std::max(hi, (32 * c1 + 31 + k + 1) - (nrow - 1));
      }
    }
  }
  BpPads b;
  b.pad_lo = lo + 2;
  b.pad_hi = hi + 2;
  b.rbuf = b.pad_lo + (p.g.nzs + 2) + b.pad_hi;
  return b;
}

// The tile shape of a plan, whether or not it is used.
static BpTile tile_shape(const Plan& p, int warps, int elem_bytes, int zr) {
  BpTile t;
  t.warps = warps;
  // Slices of a run: longer runs share the radial interpolation of a row and a
  // view's set-up among more voxels, shorter ones waste less at the ends of a
  // segment and make more CTAs.  12 / 16 slices, us a launch: 535 / 523 (128 x
  // 128 x 159 voxels, 53 segments, 10 angles, per-view form), 701 / 705 (per
  // voxel), 332 / 322 (15 segments, 21 angles), 201 / 226 (96^3).  8 slices:
  // see run_length.
  const int cx = kTileX * (warps / 2), cy = kTileY * 2;
  t.zr = zr;
  // the CTA's columns are at most `diag` voxels apart, and so are their
  // in-plane coordinates rotated to any angle
  const double diag = std::hypot((double)(cx - 1), (double)(cy - 1));
  double fzmax = 0;
  for (const Seg& s : p.seg) fzmax = std::max(fzmax, (double)std::fabs(s.fz));
  // floor(x + d) - floor(x) <= floor(d) + 1; the 2e-3 covers float rounding: with
  // 1024 columns, 4096 bins and slots of at most 10 KB (fx up to 3.6), each of two
  // corners' bins is off by at most 0.5 ulp in two products and their sum (6e-5 fx),
  // in the scaled sum (6e-5) and in the two additions after it (1.2e-4 each): 1.03e-3
  // together; a row (fz up to 12 before the image's slices bound the rows) by less
  const double nbins = std::floor(diag * p.fx_bp + 2e-3) + 3;
  const double spread = std::floor(diag * fzmax + 2e-3) + 1;
  const int ve = 16 / elem_bytes;
  const int nb = (int)std::min((double)p.g.nrad, nbins);  // radial bins and rows of a view at most
  const int rows = (int)std::min((double)(p.g.nzs + 2), (double)t.zr + spread + 2);
  // bins 4 words apart modulo 8 (16-byte copies, few bank conflicts)
  int words = ((rows + 2 * (ve - 1)) * elem_bytes + 3) / 4;
  words += (12 - words % 8) % 8;
  t.rs = words * 4 / elem_bytes;
  t.mw = (rows + 62) / 32 + 2;
  t.rows_at = (48 + 4 * nb * t.mw + 15) / 16 * 16;
  t.slot_bytes = (t.rows_at + (bp_pad_front(t.zr, elem_bytes) + nb * t.rs + t.zr + 2) * elem_bytes + 15) / 16 * 16;
  return t;
}

// Warps of 12-slice runs over the image (its columns in 4x8 tiles), in CTAs of 8.
static long long run_ctas(const Plan& p) {
  return (long long)((p.g.res + kTileX - 1) / kTileX) * ((p.g.res + kTileY - 1) / kTileY) *
         ((p.g.nzs + kTileRun - 1) / kTileRun) / 8;
}

// Tiles where their CTAs fill the SMs with warps that hide a view's latency and
// enough of each CTA is image; elsewhere one warp per column.  Fewer segments are
// fewer views for a CTA's set-up, and need more CTAs; a single segment stays with
// columns.  The masked path is what decides: without masked bins tiles are the
// faster far below the line, with 2 % of the bins masked they are not.
// Back projection and the forward projection that feeds it, tiles against columns,
// FP32, over 390 geometries of 48 to 128 columns, 24 to 159 slices and 1 to 53
// segments: the 102 that run tiles take 0.56 to 0.89 of the columns' time without
// masked bins (mean 0.69 per view, 0.74 per voxel) and 0.73 to 1.07 with 2 % (0.89,
// 0.95).  The second condition is for CTAs that reach far past the image: without it
// 1.12 / 1.20 (per view / per voxel, masked bins) at 69 x 69 x 147 and 25 segments,
// 1.14 / 1.12 at 97 x 97 x 117 and 5, 1.05 / 1.13 at 117 x 117 x 102 and 3, 0.99 /
// 1.13 at 98 x 98 x 86 and 31.  It leaves to columns a few that gain without masked
// bins (97 x 97 x 117: 0.93; 98 x 98 x 86: 0.80), and the first one more (90 x 90 x
// 54, 29 segments: 0.73, 0.97 with; 115 x 115 x 51, 5: 0.76, 0.95), because their
// neighbours lose as much with them (84 x 84 x 54, 15: 1.24 per voxel).  Masks of
// whole bins, planes or diagonal gaps cost less than 2 % at random (96^3: 0.78 to 0.83
// per view, 0.88 to 0.93 per voxel), 10 to 50 % at random more: up to 1.03 and 1.19
// at 96^3, 0.87 and 0.92 at 128 x 128 x 159.
static bool tiles_pay(const Plan& p) {
  const BpTile t = tile_shape(p, 8, 4, kTileRun);  // the largest of its slots
  if (2ll * t.warps * t.slot_bytes + 32ll * p.amax > 160 * 1024) return false;
  const int nseg = p.g.nseg;
  if (nseg < 2 || run_ctas(p) < 245 + 9 * std::max(0, 20 - nseg)) return false;
  constexpr int side = 16;  // columns of an 8-warp CTA, each way
  const long long across = (p.g.res + side - 1) / side, along = (p.g.nzs + kTileRun - 1) / kTileRun;
  const double launched = (double)(across * across * along);
  const double useful = (double)p.g.res * p.g.res * p.g.nzs / (side * side * kTileRun);  // CTAs full of image
  const double share = useful / launched;
  return useful * share * share >= 130 + 40 * std::max(0, 8 - nseg);
}

// Runs of 8 slices while runs of 12 make few CTAs; one image alone, since two
// frames of any plan with tiles have enough.  8 / 12 slices, per view and per
// voxel without masked bins, by run_ctas: 1.01 / 0.93 at 250 (80 x 80 x 110), 0.91 /
// 0.90 at 252 (93 x 93 x 83), 0.97 / 0.90 at 261 (74 x 74 x 130), 0.95 / 0.95 at 276
// (91 x 91 x 90); then mixed, 1.10 at 288 (96^3, whole CTAs and runs), 1.00 / 0.97 at
// 288 (95 x 95 x 85), 1.14 / 0.98 at 295 (104 x 104 x 82), 1.01 / 0.93 at 302 (88 x
// 88 x 111), 0.97 / 0.90 at 330 (107 x 107 x 78); 12 ahead above: 1.18 / 1.05 at 332
// (88 x 88 x 129), 1.20 / 1.01 at 346 (84 x 84 x 140).  The line lies below 96^3.
static int run_length(const Plan& p, int frames) { return run_ctas(p) * frames < 285 ? kShortRun : kTileRun; }

BpTile bp_tile(const Plan& p, int warps, int elem_bytes, int frames) {
  BpTile t = tile_shape(p, warps, elem_bytes, run_length(p, frames));
  if (!bp_uses_tiles(p)) t.zr = 0;
  t.pads = p.pads;
  return t;
}

int fp_default_R(const Plan& p) {
  for (int R : {9, 17, 25, 33}) {
    FpSchedule f;
    if (make_fp_schedule(p, R, 32, &f) && f.nthreads <= 512) return R;
  }
  return 33;
}

}  // namespace gf
