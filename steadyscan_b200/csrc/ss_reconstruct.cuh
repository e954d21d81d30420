// Reconstruction of motion-corrected frames on the GPU: invert_bilinear_sampling of the
// reference's MATLAB driver (steady_scan.m:290-404), for the frames of one set at a time.
//
// Per frame (a template of th x tw pixels, np = th tw, column-major; data pixels of the cropped
// frame at template coordinates x, y of the frame's knots, steady_scan.m:452-453):
//  * constraints (bilinear_map_linear_constraints, :438-499): every data pixel strictly inside the
//    template adds w_c d to wy and w_c w_c' to ww at its four corners (FP64; MATLAB's sparse sums).
//    ww is kept as a forward stencil: per pixel p its diagonal and its entries with p + 1 (S),
//    p + th - 1 (NE), p + th (E), p + th + 1 (SE); the pair (p, q) of a data pixel's corners is
//    always one of these (a pair across a column boundary needs a corner outside the template);
//  * first guess (resample_frame / pushgrid, :562-599): FP32 push-grid z / n. The reference's
//    z(i) = z(i) + v statements do not accumulate repeated indices: for each statement the data
//    pixel with the largest column-major index among those naming a pixel stands (a pass that
//    records it, then a pass in which it alone adds), and the eight statements keep their order;
//  * system (:319-341, calc_interactions :501-523): mask = column sum of ww > 0 and a finite guess;
//    Q = ww + regfac GtG (GtG the adjacent-difference Laplacian, vertical pairs weighted vfac^2,
//    imageadjdiffquadmat :406-436) with the rows and columns of unmasked pixels zeroed; in FP32
//    R = Q(p,p), the neighbour terms Q(p,q) / R for the eight neighbours N NE E SE S SW W NW within
//    the reference's finders' bounds (calc_indices :645-723; the SE finder's strict "< np" drops
//    one real neighbour, reproduced), L = wy(p) / R (0 where not finite);
//  * iteration (:364-389): sweeps over the colours A B C D of the 2 x 2 pattern [A B; C D],
//    x(p) = L(p) - sum_j x(q_j) Rmat_j(p) in FP32 with the eight terms summed in order; every
//    n-th sweep the energy x'Qx - 2 Le x (FP64 quadratic form of the FP32 iterate, FP32 linear
//    term, compared in FP32) stops the frame when it did not decrease, the output being the
//    iterate of the last check that decreased it (zeros if none did); n is the interval the
//    previous frame's sweep count gave (:391).
// Frames run in parallel, once: the iterates do not depend on n, so every sweep of every frame is kept
// as its own iterate (in a ring of slots) with its energy, and the host follows the chain of intervals
// over the energies; a frame sweeps until its stop is known, or the stop of every interval 1..10 is.
// Guessing the intervals and sweeping again from the first wrong guess took seven runs of a 64-frame
// set and a separate copy of every kept iterate (64 frames of 512 x 512: 153 ms a call, 119 of them on
// the device; here 37 and 20).
#pragma once

#include "ss_common.cuh"

namespace ss {

constexpr int kRcStencil = 5;  // diagonal, S, NE, E, SE
constexpr int kRcParts = 64;   // partial-sum CTAs per frame of the energy
constexpr int kRcBatch = 4;    // iterates whose energies are summed by one launch
constexpr int kRcTerms = 9;    // sweep coefficients of a pixel: Rmat[8], L

// Per-frame buffers of a chunk of frames (device pointers; [frame * np + p] unless noted). What the
// sweeps read lies colour by colour, so that a colour's lanes read consecutive floats: quarter plane
// `colour` of rh x cw entries holds pixel (2 i + colour / 2, 2 j + colour % 2) at i + rh j.
struct RcBufs {
  int th, tw, np, hd, wd, nk;  // template size, data frame size, knots per frame
  int rh, cw, nq;   // quarter planes: ceil(th / 2) x ceil(tw / 2) = nq entries
  int frames;       // frames of a slot
  double* wy;       // np
  double* ww;       // kRcStencil planes of np
  float* z;         // np: push-grid sums
  float* cnt;       // np: push-grid weights
  int* last_z;      // np
  int* last_n;      // np
  uint8_t* mask;    // np
  float* coef;      // kRcTerms x 4 quarter planes (before them z, cnt, last_z and last_n)
  float* le;        // np: single(Lfull) of masked pixels, else 0
  float* x;         // [slot][frame] iterates of 4 quarter planes; slot 0 is the first guess
  double* part;     // frames x kRcParts x kRcBatch: energy partial sums (FP64 quadratic, FP32 linear)
  float* part_l;    // frames x kRcParts x kRcBatch
};

__device__ __forceinline__ float* rc_iterate(const RcBufs& b, int slot, int f) {
  return b.x + ((size_t)slot * b.frames + f) * 4 * b.nq;
}
// Place of pixel (r, c) in an iterate.
__device__ __forceinline__ size_t rc_place(const RcBufs& b, int r, int c) {
  return (size_t)((r & 1) * 2 + (c & 1)) * b.nq + (r >> 1) + (size_t)b.rh * (c >> 1);
}

// Template coordinates of data pixel q (column-major in hd x wd) of frame f (steady_scan.m:452-453).
__device__ __forceinline__ void rc_coords(const double* __restrict__ bx, const double* __restrict__ by,
                                          const double* __restrict__ tf, const int* __restrict__ pk,
                                          const double* __restrict__ dxk, const double* __restrict__ dyk, int q,
                                          double& x, double& y) {
  const int k = pk[q] - 1;
  const double f = tf[q], c = 1.0 - f;
  x = bx[q] + dxk[k] * c + dxk[k + 1] * f;
  y = by[q] + dyk[k] * c + dyk[k + 1] * f;
}

template <class DataT>
__global__ void __launch_bounds__(256) k_rc_constraints(RcBufs b, const void* __restrict__ data, int f0, int nf,
                                                        const double* __restrict__ bx, const double* __restrict__ by,
                                                        const double* __restrict__ tf, const int* __restrict__ pk,
                                                        const double* __restrict__ dxk, const double* __restrict__ dyk) {
  const size_t per = (size_t)b.hd * b.wd, total = per * nf;
  const double eps = 2.220446049250313e-16;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
    const int f = (int)(e / per), q = (int)(e - (size_t)f * per);
    double x, y;
    rc_coords(bx, by, tf, pk, dxk + (size_t)(f0 + f) * b.nk, dyk + (size_t)(f0 + f) * b.nk, q, x, y);
    if (!(x > 1 + eps && x < b.tw - eps && y > 1 + eps && y < b.th - eps)) continue;
    const double xi = floor(x), yi = floor(y), xf = x - xi, yf = y - yi;
    const int p0 = (int)yi - 1 + b.th * ((int)xi - 1);  // corner (y, x), 0-based
    const double d = to_double(reinterpret_cast<const DataT*>(data)[(size_t)(f0 + f) * per + q]);
    const double xc = 1 - xf, yc = 1 - yf;
    const double w[4] = {xc * yc, xc * yf, xf * yc, xf * yf};  // (y,x) (y+1,x) (y,x+1) (y+1,x+1)
    const int pc[4] = {p0, p0 + 1, p0 + b.th, p0 + b.th + 1};
    double* wy = b.wy + (size_t)f * b.np;
    double* ww = b.ww + (size_t)f * b.np * kRcStencil;
#pragma unroll
    for (int c = 0; c < 4; c++) {
      atomicAdd(wy + pc[c], w[c] * d);
      atomicAdd(ww + pc[c], w[c] * w[c]);
    }
    const size_t np = b.np;
    atomicAdd(ww + 1 * np + pc[0], w[0] * w[1]);  // (y,x)-(y+1,x): S
    atomicAdd(ww + 1 * np + pc[2], w[2] * w[3]);  // (y,x+1)-(y+1,x+1): S
    atomicAdd(ww + 3 * np + pc[0], w[0] * w[2]);  // E
    atomicAdd(ww + 3 * np + pc[1], w[1] * w[3]);  // E
    atomicAdd(ww + 4 * np + pc[0], w[0] * w[3]);  // SE
    atomicAdd(ww + 2 * np + pc[1], w[1] * w[2]);  // (y+1,x)-(y,x+1): NE
  }
}

// One push-grid statement pair (step s of 4): z at corner offset oz, n at corner offset on; phase 0
// records the last data pixel naming each pixel, phase 1 lets it add.
template <class DataT>
__global__ void __launch_bounds__(256) k_rc_pushgrid(RcBufs b, const void* __restrict__ data, int f0, int nf, int s,
                                                     int phase, const double* __restrict__ bx,
                                                     const double* __restrict__ by, const double* __restrict__ tf,
                                                     const int* __restrict__ pk, const double* __restrict__ dxk,
                                                     const double* __restrict__ dyk) {
  const size_t per = (size_t)b.hd * b.wd, total = per * nf;
  // statement orders (steady_scan.m:589-598): z at (y,x) (y+1,x) (y,x+1) (y+1,x+1); n at
  // (y+1,x) (y,x+1) (y,x) (y+1,x+1); corner c: offset {0, 1, th, th+1}[c]
  const int cz = s, cn = (s == 0) ? 1 : (s == 1) ? 2 : (s == 2) ? 0 : 3;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
    const int f = (int)(e / per), q = (int)(e - (size_t)f * per);
    double x, y;
    rc_coords(bx, by, tf, pk, dxk + (size_t)(f0 + f) * b.nk, dyk + (size_t)(f0 + f) * b.nk, q, x, y);
    if (!(x >= 1 && x < b.tw && y >= 1 && y < b.th)) continue;
    const double xi = floor(x), yi = floor(y), xf = x - xi, yf = y - yi;
    const int p0 = (int)yi - 1 + b.th * ((int)xi - 1);
    const int off[4] = {0, 1, b.th, b.th + 1};
    const double wc[4] = {(1 - xf) * (1 - yf), (1 - xf) * yf, xf * (1 - yf), xf * yf};
    const int tz = p0 + off[cz], tn = p0 + off[cn];
    int* lz = b.last_z + (size_t)f * b.np;
    int* ln = b.last_n + (size_t)f * b.np;
    if (phase == 0) {
      atomicMax(lz + tz, q);
      atomicMax(ln + tn, q);
    } else {
      const float d = (float)to_double(reinterpret_cast<const DataT*>(data)[(size_t)(f0 + f) * per + q]);
      if (lz[tz] == q) b.z[(size_t)f * b.np + tz] += (float)wc[cz] * d;
      if (ln[tn] == q) b.cnt[(size_t)f * b.np + tn] += (float)wc[cn];
    }
  }
}

// Stencil plane of the pair (p, p + th - 1): NE, or S where the template has two rows and the offsets
// fall together.
__device__ __forceinline__ int rc_ne(int th) { return th == 2 ? 1 : 2; }

// Mask (column sums of ww > 0 and a finite first guess) and the first iterate of every pixel. Grid:
// (blocks, frames).
__global__ void __launch_bounds__(256) k_rc_mask(RcBufs b) {
  const int f = blockIdx.y, th = b.th, np = b.np, ne = rc_ne(th);
  const double* ww = b.ww + (size_t)f * np * kRcStencil;
  const double *S = ww + np, *NE = ww + (size_t)ne * np, *E = ww + (size_t)3 * np, *SE = ww + (size_t)4 * np;
  float* x = rc_iterate(b, 0, f);
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < np; p += gridDim.x * blockDim.x) {
    double s = ww[p];  // (no entry is negative)
    if (p >= 1) s += S[p - 1];
    if (p + 1 < np) s += S[p];
    if (p >= th - 1) s += NE[p - th + 1];
    if (p + th - 1 < np) s += NE[p];
    if (p >= th) s += E[p - th];
    if (p + th < np) s += E[p];
    if (p >= th + 1) s += SE[p - th - 1];
    if (p + th + 1 < np) s += SE[p];
    const size_t e = (size_t)f * np + p;
    const float iv = b.z[e] / b.cnt[e];
    b.mask[e] = (s > 0.0 && !isnan(iv)) ? 1 : 0;
    const int c = p / th;
    x[rc_place(b, p - c * th, c)] = isnan(iv) ? 0.0f : iv;
  }
}

// FP32 coefficients of every pixel: the eight neighbour terms and L; and Le. Q(p, q) of the masked system
// is ww + regfac GtG (vertical pairs vfac^2) with the rows and columns of unmasked pixels zero. Grid:
// (blocks, frames).
__global__ void __launch_bounds__(256) k_rc_coef(RcBufs b, double regfac, double vf2) {
  const int f = blockIdx.y, th = b.th, tw = b.tw, np = b.np, ne = rc_ne(th);
  const double* ww = b.ww + (size_t)f * np * kRcStencil;
  const double *S = ww + np, *NE = ww + (size_t)ne * np, *E = ww + (size_t)3 * np, *SE = ww + (size_t)4 * np;
  const uint8_t* mk = b.mask + (size_t)f * np;
  const double rh = -regfac, rv = -__dmul_rn(regfac, vf2);
  const size_t plane = 4 * (size_t)b.nq;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < np; p += gridDim.x * blockDim.x) {
    const int c = p / th, r = p - c * th;
    // (the entries of a quarter plane past the template's last row or column are never read)
    float* cf = b.coef + (size_t)f * kRcTerms * plane + rc_place(b, r, c);
    const bool m = mk[p] != 0;
    float R = 0.0f;
    if (m) {
      const int nh = (c > 0) + (c < tw - 1), nv = (r > 0) + (r < th - 1);
      R = (float)__dadd_rn(ww[p], __dmul_rn(regfac, (double)nh + (double)nv * vf2));
    }
    // the term of neighbour q within the reference's finders' bounds (steady_scan.m:677-723), its stencil
    // entry w and regulariser
    auto term = [&](int j, bool ok, int q, const double* w, int at, double reg) {
      float t = 0.0f;
      if (R != 0.0f && ok) t = (mk[q] ? (float)__dadd_rn(w[at], reg) : 0.0f) / R;
      cf[j * plane] = t;
    };
    // N NE E SE S SW W NW; the finders' 1-based bounds (p + 1 = their index)
    term(0, r > 0, p - 1, S, p - 1, rv);
    term(1, r > 0 && p + th < np, p + th - 1, NE, p, 0.0);
    term(2, p + th < np, p + th, E, p, rh);
    term(3, r < th - 1 && p + th + 2 < np, p + th + 1, SE, p, 0.0);
    term(4, r < th - 1, p + 1, S, p, rv);
    term(5, r < th - 1 && p >= th - 1, p - th + 1, NE, p - th + 1, 0.0);
    term(6, p >= th, p - th, E, p - th, rh);
    term(7, p >= th + 1, p - th - 1, SE, p - th - 1, 0.0);
    const float lf = m ? (float)b.wy[(size_t)f * np + p] : 0.0f;
    float L = lf / R;
    if (!isfinite(L)) L = 0.0f;
    cf[8 * plane] = L;
    b.le[(size_t)f * np + p] = lf;
  }
}

// One colour of one sweep, iterate `it` (slot `snew`) from its predecessor (slot `sold`), of the frames
// that sweep that far (limit[f] >= it). A colour's eight neighbours are of the other colours: the ones
// before it come from the new iterate, the ones after it from the old. Neighbours outside the template
// have zero terms. Bound: HBM, 36 B of terms per pixel (pixel by pixel in memory, 10 floats each, a
// colour of 64 frames of 512 x 512 took 48 us; colour by colour 41.5 us, 5.2 TB/s).
template <int COLOUR>
__global__ void __launch_bounds__(256) k_rc_sweep(RcBufs b, int it, int sold, int snew, const int* __restrict__ limit) {
  const int f = blockIdx.y;
  if (limit[f] < it) return;
  constexpr int pr = COLOUR >> 1, pc = COLOUR & 1;
  // N NE E SE S SW W NW
  constexpr int dr[8] = {-1, -1, 0, 1, 1, 1, 0, -1}, dc[8] = {0, 1, 1, 1, 0, -1, -1, -1};
  const int th = b.th, tw = b.tw, rh = b.rh;
  const size_t nq = b.nq;
  const float* xo = rc_iterate(b, sold, f);
  float* xn = rc_iterate(b, snew, f);
  const float* cf = b.coef + (size_t)f * kRcTerms * 4 * nq + (size_t)COLOUR * nq;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < b.nq; k += gridDim.x * blockDim.x) {
    const int j = k / rh, i = k - j * rh, r = 2 * i + pr, c = 2 * j + pc;
    if (r >= th || c >= tw) continue;
    float v[8], t[8];
#pragma unroll
    for (int q = 0; q < 8; q++) {
      constexpr auto colour_of = [](int a, int e) { return (a & 1) * 2 + (e & 1); };
      const int qc = colour_of(pr + dr[q] + 2, pc + dc[q] + 2);
      const int qi = i + ((pr + dr[q] + 2) >> 1) - 1, qj = j + ((pc + dc[q] + 2) >> 1) - 1;
      const bool in = (unsigned)(r + dr[q]) < (unsigned)th && (unsigned)(c + dc[q]) < (unsigned)tw;
      const float* x = (qc < COLOUR ? xn : xo) + qc * nq;
      v[q] = x[in ? qi + rh * qj : k];  // (outside: any value of the plane, selected away)
      if (!in) v[q] = 0.0f;
      t[q] = __ldg(cf + (size_t)q * 4 * nq + k);
    }
    const float L = __ldg(cf + (size_t)8 * 4 * nq + k);
    float s = 0.0f;
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const float a = v[q] * t[q];
      s = q == 0 ? a : s + a;
    }
    xn[(size_t)COLOUR * nq + k] = L - s;
  }
}

// Linear energy terms of iterates it0 .. it0 + nit - 1 (slots sl.x ..) of the frames that have swept that
// far: FP32 sums of Le_p x_p, kRcParts CTAs per frame over fixed pixel ranges. Bound: HBM, 20 B per
// pixel (four iterates of 64 frames of 512 x 512: 65 us, 5.2 TB/s; 99 with each iterate's load under a
// branch on nit).
__global__ void __launch_bounds__(256) k_rc_linear(RcBufs b, int it0, int nit, int4 sl, const int* __restrict__ limit) {
  const int f = blockIdx.y;
  if (limit[f] < it0 + nit - 1) return;
  const int th = b.th, np = b.np;
  const float* le = b.le + (size_t)f * np;
  // (past the last of nit, the first's again: every load is unconditional)
  const float* xs[kRcBatch] = {rc_iterate(b, sl.x, f), rc_iterate(b, nit > 1 ? sl.y : sl.x, f),
                               rc_iterate(b, nit > 2 ? sl.z : sl.x, f), rc_iterate(b, nit > 3 ? sl.w : sl.x, f)};
  const int per = (np + kRcParts - 1) / kRcParts, a = blockIdx.x * per, e = min(np, a + per);
  float ls[kRcBatch] = {};
  int c = (a + (int)threadIdx.x) / th, r = a + (int)threadIdx.x - c * th;
#pragma unroll 4
  for (int p = a + threadIdx.x; p < e; p += blockDim.x) {
    const int at = ((r & 1) * 2 + (c & 1)) * b.nq + (r >> 1) + b.rh * (c >> 1);  // (4 nq < 2^31)
    const float l = le[p];  // zero at unmasked pixels
    for (r += blockDim.x; r >= th; r -= th) c++;
#pragma unroll
    for (int k = 0; k < kRcBatch; k++) ls[k] = fmaf(l, xs[k][at], ls[k]);
  }
  __shared__ float sv[kRcBatch][256];
#pragma unroll
  for (int k = 0; k < kRcBatch; k++) sv[k][threadIdx.x] = ls[k];
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o)
#pragma unroll
      for (int k = 0; k < kRcBatch; k++) sv[k][threadIdx.x] += sv[k][threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x < nit) b.part_l[((size_t)f * kRcBatch + threadIdx.x) * kRcParts + blockIdx.x] = sv[threadIdx.x][0];
}

// Quadratic energy terms of those iterates: FP64 sums of x_p (Q x)_p over masked p, each pair of pixels
// once. A thread takes a 2 x 2 quad, the same place of the four quarter planes, so that consecutive
// lanes read consecutive floats of an iterate, a quad's 11 samples are converted once each, and its 20
// stencil entries (five times an iterate's bytes) serve nit iterates. Bound: load latency at 16 warps
// per SM (128 registers); so no load waits for another or for a branch, and the next iterate's samples
// are under way while one is summed. Four iterates of 64 frames of 512 x 512 (147 us of HBM time):
// 243 us; 376 with each load under its own bounds check. One iterate at a time, with a thread and 20
// conversions per pixel, took 4 x 125. kRcParts CTAs per frame.
__global__ void __launch_bounds__(256, 2) k_rc_quadratic(RcBufs b, int it0, int nit, int4 sl, const int* __restrict__ limit,
                                                      double regfac, double vf2) {
  const int f = blockIdx.y;
  if (limit[f] < it0 + nit - 1) return;
  const int th = b.th, tw = b.tw, np = b.np, rh = b.rh;
  const size_t nq = b.nq;
  const double* ww = b.ww + (size_t)f * np * kRcStencil;
  const uint8_t* mk = b.mask + (size_t)f * np;
  const int s_ne = rc_ne(th);
  const bool paired = (th & 1) == 0;  // then every column, plane and frame of ww starts on 16 bytes
  double qs[kRcBatch] = {};
  for (int k = blockIdx.x * 256 + threadIdx.x; k < b.nq; k += kRcParts * 256) {
    const int j = k / rh, i = k - j * rh, r0 = 2 * i, c0 = 2 * j;
    const bool up = r0 > 0, down = r0 + 2 < th, low = r0 + 1 < th, right = c0 + 2 < tw, mid = c0 + 1 < tw;
    // Every load is unconditional, from a clamped place, and its value selected afterwards, so that the
    // loads of a quad are in flight together.
    // The stencil entries of the quad's pixels, two rows at a time.
    double2 w[2][kRcStencil];
    const size_t p0 = (size_t)c0 * th + r0, p1 = mid ? p0 + th : p0;
    if (paired) {
#pragma unroll
      for (int s = 0; s < kRcStencil; s++) {
        const double* wp = ww + (size_t)(s == 2 ? s_ne : s) * np;
        w[0][s] = *reinterpret_cast<const double2*>(wp + p0);
        w[1][s] = *reinterpret_cast<const double2*>(wp + p1);
      }
    } else {
#pragma unroll
      for (int s = 0; s < kRcStencil; s++) {
        const double* wp = ww + (size_t)(s == 2 ? s_ne : s) * np;
        w[0][s] = make_double2(wp[p0], wp[p0 + low]);
        w[1][s] = make_double2(wp[p1], wp[p1 + low]);
      }
    }
    // masks of the quad and its neighbours: rows r0 - 1 .. r0 + 2, columns c0 .. c0 + 2
    const bool row_in[4] = {up, true, low, down}, col_in[3] = {true, mid, right};
    bool m[4][3];
#pragma unroll
    for (int e = 0; e < 3; e++)
#pragma unroll
      for (int a = 0; a < 4; a++) {
        const bool in = row_in[a] && col_in[e];
        m[a][e] = (mk[in ? p0 + (size_t)e * th + a - 1 : p0] != 0) & in;
      }
    // iterate t's samples of the quad and its neighbours (past the last of nit, the first's again)
    const int rt = right ? rh : 0, dn = down ? 1 : 0;
    auto samples = [&](int t, float (&o)[11]) {
      const int slot = t >= nit ? sl.x : t == 0 ? sl.x : t == 1 ? sl.y : t == 2 ? sl.z : sl.w;
      const float* A = rc_iterate(b, slot, f) + k;
      const float *B = A + nq, *C = A + 2 * nq, *D = A + 3 * nq;
      o[0] = A[0], o[1] = B[0], o[2] = C[0], o[3] = D[0], o[4] = A[rt], o[5] = C[rt], o[6] = A[dn], o[7] = B[dn];
      o[8] = A[rt + dn], o[9] = D[up ? -1 : 0], o[10] = C[up ? rt - 1 : rt];
    };
    const bool in_x[11] = {true, mid,          low,           low && mid, right,      right && low,
                           down, down && mid, down && right, up && mid,  up && right};
    float x[2][11];
    samples(0, x[0]);
    // Q(p, q) of the quad's pixels (r0 + dr, c0 + dc) with themselves and their S, NE, E, SE neighbours
    double q[2][2][kRcStencil];
#pragma unroll
    for (int dr = 0; dr < 2; dr++)
#pragma unroll
      for (int dc = 0; dc < 2; dc++) {
        double* v = q[dr][dc];
        const int r = r0 + dr, c = c0 + dc;
        const bool own = m[1 + dr][dc];
        auto at = [&](int s) { return dr ? w[dc][s].y : w[dc][s].x; };
        const int nh = (c > 0) + (c < tw - 1), nv = (r > 0) + (r < th - 1);
        v[0] = own ? at(0) + regfac * ((double)nh + (double)nv * vf2) : 0.0;
        v[1] = own && m[2 + dr][dc] ? at(1) - regfac * vf2 : 0.0;
        if (th == 2) v[1] += v[1];  // (p + 1 and p + th - 1 are both summed there)
        v[2] = own && m[dr][dc + 1] ? at(2) : 0.0;
        v[3] = own && m[1 + dr][dc + 1] ? at(3) - regfac : 0.0;
        v[4] = own && m[2 + dr][dc + 1] ? at(4) : 0.0;
      }
#pragma unroll
    for (int t = 0; t < kRcBatch; t++) {
      // rows r0 - 1 .. r0 + 2, columns c0 .. c0 + 2; the next iterate's samples arrive meanwhile
      double v[11];
#pragma unroll
      for (int e = 0; e < 11; e++) v[e] = in_x[e] ? x[t & 1][e] : 0.f;
      const double a0 = v[0], b0 = v[1], c_0 = v[2], d0 = v[3], a_r = v[4], c_r = v[5], a_d = v[6], b_d = v[7], a_dr = v[8],
                   d_u = v[9], c_ur = v[10];
      if (t + 1 < kRcBatch) samples(t + 1, x[(t + 1) & 1]);
      auto px = [](const double (&v)[kRcStencil], double p, double s, double ne, double e, double se) {
        return p * (v[0] * p + 2.0 * (v[1] * s + v[2] * ne + v[3] * e + v[4] * se));
      };
      qs[t] += (px(q[0][0], a0, c_0, d_u, b0, d0) + px(q[0][1], b0, d0, c_ur, a_r, c_r)) +
               (px(q[1][0], c_0, a_d, b0, d0, b_d) + px(q[1][1], d0, b_d, a_r, c_r, a_dr));
    }
  }
  __shared__ double sq[kRcBatch][8];
#pragma unroll
  for (int t = 0; t < kRcBatch; t++) {
    const double v = warp_sum(qs[t]);
    if ((threadIdx.x & 31) == 0) sq[t][threadIdx.x >> 5] = v;
  }
  __syncthreads();
  if (threadIdx.x < nit) {
    double v = 0.0;
    for (int w = 0; w < 8; w++) v += sq[threadIdx.x][w];
    b.part[((size_t)f * kRcBatch + threadIdx.x) * kRcParts + blockIdx.x] = v;
  }
}

// The energies of those iterates (a thread each) from their partial sums in a fixed order.
__global__ void k_rc_total(RcBufs b, int nf, int it0, int nit, const int* __restrict__ limit, float* __restrict__ energy) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x, f = e / kRcBatch, k = e - f * kRcBatch;
  if (f >= nf || k >= nit || limit[f] < it0 + nit - 1) return;
  double q = 0.0;
  float l = 0.0f;
  for (int i = 0; i < kRcParts; i++) {
    q += b.part[(size_t)e * kRcParts + i];
    l += b.part_l[(size_t)e * kRcParts + i];
  }
  energy[e] = (float)(q - 2.0 * (double)l);
}

// Masked pixels of every frame (a frame with none is skipped, as the reference's `continue`); grid
// (blocks, frames), one atomic per CTA.
__global__ void __launch_bounds__(256) k_rc_count(RcBufs b, int* __restrict__ count) {
  const int f = blockIdx.y;
  const uint8_t* mk = b.mask + (size_t)f * b.np;
  int c = 0;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < b.np; p += gridDim.x * blockDim.x) c += mk[p] ? 1 : 0;
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  __shared__ int sc[8];
  if ((threadIdx.x & 31) == 0) sc[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += sc[w];
    if (t) atomicAdd(count + f, t);
  }
}

// Outputs of the chunk's frames: the iterate in slot[f] (below 0: zeros), NaN outside the mask.
template <class OutT>
__global__ void __launch_bounds__(256) k_rc_out(RcBufs b, int nf, OutT* __restrict__ out, uint8_t* __restrict__ mk_out,
                                                const int* __restrict__ slot, const int* __restrict__ skip) {
  const size_t total = (size_t)b.np * nf;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
    const int f = (int)(e / b.np), p = (int)(e - (size_t)f * b.np);
    const bool m = b.mask[e] && !skip[f];
    float v = 0.0f;
    if (m && slot[f] >= 0) v = rc_iterate(b, slot[f], f)[rc_place(b, p % b.th, p / b.th)];
    out[e] = m ? (OutT)v : (OutT)NAN;
    if (mk_out) mk_out[e] = m ? 1 : 0;
  }
}

}  // namespace ss
