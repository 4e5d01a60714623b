// Mixed-precision pair kernel: the pair sums, strain rates and heat fluxes in FP32, on
// particle coordinates stored relative to the origin of their own cell; the predictor,
// corrector (leap-frog accumulation), JC return map and the tool-force reduction stay FP64.
//
// Same neighbour set and order as the plain form (interactions_gpu.cu:147-345); the
// differences are the arithmetic type and these exact rewrites:
//   * x_ij = (ci - cj) * dx + (xi_rel - xj_rel) and y_ij likewise: a small integer times the
//     cell size plus a difference of in-cell offsets, instead of a difference of absolute
//     coordinates;
//   * (e_ij . grad W) / r = der * fac (Brookshaw), one rsqrt per pair for 1/r;
//   * temperatures are stored relative to the initial temperature, so Ti - Tj keeps its
//     digits near it.
// Its error against the FP64 form is measured and reported, not assumed.
#pragma once

#include "mf_kernels.cuh"

namespace mf {

// the marks in a record's first word (F_ROW, F_H)
__device__ __forceinline__ bool f_blanked(const float4 &b0) { return b0.z != b0.z; }
__device__ __forceinline__ bool f_tool(const float4 &b0) { return __float_as_int(b0.z) < 0; }
__device__ __forceinline__ bool f_nonfinite(const float4 &b0) { return __float_as_int(b0.w) < 0; }

// the i particle's values and the pair sums of one thread
struct mixed_i {
  float x, y, row, sxy, Rxy, h, rho, c, T;  // row: cell row + 1
  float2 nv, sd, Rd;                        // (-vx, -vy), (sxx, syy), (Rxx, Ryy)
  float h1, fourh2;
  // the spline's coefficients: W / W(dp) for q > 1 (w_out (2 - q)^6) and q <= 1 (w_in (1 - 1.5 q^2 +
  // 0.75 q^3)), (dW/dr) / r for q > 1 (d_out (2 - q)^2 / r) and q <= 1 (d_in (1 - 0.75 q))
  float w_out, w_in, d_out, d_in;
  bool mech, thermal, nonfinite;
};
// The constant factors of a sum are applied once at the end: the stress sums without the mass, the
// viscosity sums without -2 mass, XSPH without 2 mass eps W(dp), the Brookshaw sum without its factor 2.
struct mixed_acc {
  float2 v14;  // (vdx, vdw)
  float vdy, vdz;
  float2 s14;  // (sdx, sdw)
  float sdy, sdz;
  float vtx, vty, xtx, xty;
  float T_lapl;
};
struct mixed_const {
  float alpha4, beta4, eta4;  // alpha / 4, beta / 4, eta^2 / 4
};

// r^2 with its one fused multiply-add written out, so that every kernel that tests or uses a
// pair's distance (window, list build, list) rounds it the same way
__device__ __forceinline__ float dist2(float x, float y) { return fmaf(x, x, __fmul_rn(y, y)); }
// offset of a record's particle from particle i, dcol columns of cells (i's - j's) and the rows'
// difference away: the in-cell offsets' difference first, then one rounding
__device__ __forceinline__ float offset_x(const mixed_i &I, const float4 &b0, float dcol, float dxc) {
  return fmaf(dcol, dxc, I.x - b0.x);
}
__device__ __forceinline__ float offset_y(const mixed_i &I, const float4 &b0, float dxc) {
  return fmaf(I.row - fabsf(b0.z), dxc, I.y - b0.y);
}

// One neighbour j (records b0..b3) of particle i at offset (xij, yij): the reference's cubic spline
// (kernels.cuh:30-70; its value (2 - q)^6 / 4 for q > 1 is sic), both branches evaluated and selected,
// with the constants folded into the coefficients (1 / r cancels for q <= 1). SELECT: both branches
// evaluated and selected (the list form, 48.2 against 50.1 us at 176,695 particles; the window form's
// lanes take the branches together more often and lose by it, 201 against 191 us at 577,555). Every
// multiply-add is written out. Packed pairs (two multiply-adds an issue) stand only where both
// operands already lie in register pairs, as words of a record or sums side by side: the moves that
// built pairs of duplicated factors cost the ALU pipe more than they gave back (1,100 against 1,770
// integer instructions a particle at 577,555; 24-system batch 181.5 all scalar, 179.3 us so).
template <bool SELECT>
__device__ __forceinline__ void mixed_interact(const mixed_i &I, const mixed_const &K, mixed_acc &a, float xij,
                                               float yij, const float4 &b0, const float4 &b1, const float4 &b2,
                                               const float4 &b3) {
  const float rr2 = dist2(xij, yij);
  // outside the support (candidates taken because a record holds a NaN or Inf) W = 0
  const bool in_support = !(rr2 >= I.fourh2 || rr2 < 1e-8f);
  float w = 0.f, dwr = 0.f;  // W / W(dp), (dW/dr) / r
  auto kernel = [&](float rinv) {
    const float qq = __fmul_rn(__fmul_rn(rr2, rinv), I.h1);
    const float t = 2.f - qq, t2 = __fmul_rn(t, t);
    if (SELECT) {
      const float val_out = __fmul_rn(__fmul_rn(t2, t2), __fmul_rn(I.w_out, t2));
      const float val_in = __fmul_rn(I.w_in, fmaf(__fmul_rn(qq, qq), fmaf(0.75f, qq, -1.5f), 1.f));
      const float der_out = __fmul_rn(__fmul_rn(I.d_out, t2), rinv);
      const float der_in = __fmul_rn(I.d_in, fmaf(-0.75f, qq, 1.f));
      w = qq > 1.f ? val_out : val_in;
      dwr = qq > 1.f ? der_out : der_in;
    } else if (qq > 1.f) {
      w = __fmul_rn(__fmul_rn(t2, t2), __fmul_rn(I.w_out, t2));
      dwr = __fmul_rn(__fmul_rn(I.d_out, t2), rinv);
    } else {
      w = __fmul_rn(I.w_in, fmaf(__fmul_rn(qq, qq), fmaf(0.75f, qq, -1.5f), 1.f));
      dwr = __fmul_rn(I.d_in, fmaf(-0.75f, qq, 1.f));
    }
  };
  if (in_support) kernel(rsqrtf(rr2));
  const float wx = __fmul_rn(dwr, xij), wy = __fmul_rn(dwr, yij);
  const float volj = b3.z;
  if (I.mech && !f_tool(b0)) {
    const float2 dv = __fadd2_rn(make_float2(b1.x, b1.y), I.nv);
    const float dvx = dv.x, dvy = dv.y;
    const float2 w2v = make_float2(wx, wy);
    const float ax = __fmul_rn(dvx, volj), ay = __fmul_rn(dvy, volj);
    a.v14 = __ffma2_rn(make_float2(ax, ay), w2v, a.v14);
    a.vdy = fmaf(ax, wy, a.vdy);
    a.vdz = fmaf(ay, wx, a.vdz);
    const float w2 = __fmul_rn(w, w), fab = __fmul_rn(w2, w2);
    const float2 Rs = __fadd2_rn(I.Rd, make_float2(b2.z, b2.w)), ss = __fadd2_rn(I.sd, make_float2(b2.x, b2.y));
    const float2 sd2 = make_float2(fmaf(fab, Rs.x, ss.x), fmaf(fab, Rs.y, ss.y));
    const float sxy = fmaf(fab, I.Rxy + b1.w, I.sxy + b1.z);
    a.s14 = __ffma2_rn(sd2, w2v, a.s14);
    a.sdz = fmaf(sxy, wx, a.sdz);
    a.sdy = fmaf(sxy, wy, a.sdy);
    const float nvr = fmaf(dvx, xij, __fmul_rn(dvy, yij));  // -v_ij . x_ij
    const float irho = __fdividef(1.f, I.rho + b3.x);        // half of 1 / rho_ij
    if (nvr > 0.f) {  // Monaghan viscosity for approaching pairs: pi_ij / 2
      const float hh = I.h + fabsf(b0.w);                    // 2 h_ij
      const float mu2 = __fmul_rn(__fmul_rn(hh, nvr), __fdividef(1.f, fmaf(__fmul_rn(K.eta4, hh), hh, rr2)));
      const float pi = __fmul_rn(__fmul_rn(fmaf(K.beta4, mu2, __fmul_rn(K.alpha4, I.c + b3.y)), mu2), irho);
      a.vtx = fmaf(pi, wx, a.vtx);
      a.vty = fmaf(pi, wy, a.vty);
    }
    const float xs = __fmul_rn(w, irho);
    a.xtx = fmaf(xs, dvx, a.xtx);
    a.xty = fmaf(xs, dvy, a.xty);
  }
  // Brookshaw: 2 (m/rho_j)(Ti - Tj)(e_ij . grad W)/r with (e_ij . grad W)/r = dwr
  if (I.thermal && rr2 > 1e-16f) a.T_lapl = fmaf(__fmul_rn(volj, I.T - b3.w), dwr, a.T_lapl);
}

// Records of the candidates in global memory, read through the read-only path (word k of
// record j among N at recf_word(k, j, N)). (A block's candidates staged in shared memory by bulk copies
// on one mbarrier measured 25-30 % slower on the ~150k-particle cut: fewer resident warps and
// the copy's wait before any arithmetic, against loads that L1 already served 84 % of.)
struct rec_global {
  const float4 *__restrict__ r0;    // word 0
  const float4 *__restrict__ rest;  // the tiles of words 1..3
  __device__ __forceinline__ explicit rec_global(const float *recf, int N)
      : r0(reinterpret_cast<const float4 *>(recf)), rest(r0 + recf_word(1, 0, N)) {}
  __device__ __forceinline__ float4 p0(int j) const { return __ldg(r0 + j); }
  __device__ __forceinline__ void words(int j, float4 &b1, float4 &b2, float4 &b3) const {
    const float4 *t = rest + ((size_t)(j >> 5) * 96 + (size_t)(j & 31));
    b1 = __ldg(t); b2 = __ldg(t + 32); b3 = __ldg(t + 64);
  }
  __device__ __forceinline__ void all(int j, float4 &b0, float4 &b1, float4 &b2, float4 &b3) const {
    b0 = p0(j);
    words(j, b1, b2, b3);
  }
};

// Neighbour list of particle q (its G lanes, sub = lane), built on a step that sorted: the
// candidates within 2 h_i + skin over the 7x7 cells around its own (the 5x5 window widened by one
// cell, which covers that radius for h_i up to the cell size), blanked ones left out, non-finite
// ones kept (their pair terms carry the NaN). Columns in x order and each column's range in array
// order. Called by whole warps; `on`: the particle gets a list.
template <int G>
__device__ __forceinline__ void build_list(const dev_buffers &D, const rec_global &REC, int q, int sub, bool on,
                                           const mixed_i &I, const geom &g, int gi, int gj, float dxc, float skin) {
  const float R = 2.f * I.h + skin;
  const float R2 = R * R;
  const int low_j = gj - 3 < 0 ? 0 : gj - 3;
  const int high_j = gj + 4 > g.ny ? g.ny : gj + 4;
  unsigned *row = D.nlist + (size_t)q * LIST_CAP;
  int cnt = 0;
  for (int c = -3; c <= 3; ++c) {
    const int ii = gi + c;
    const bool in = on && ii >= 0 && ii < g.nx;
    const int j0 = in ? __ldg(D.off + ii * g.ny + low_j) : 0;
    const int j1 = in ? __ldg(D.off + ii * g.ny + high_j) : 0;
    const float dcol = (float)-c;
    const unsigned tag = (unsigned)(3 - c) << LIST_INDEX_BITS;
    for (int jb = j0; G == 1 ? jb < j1 : __any_sync(0xffffffffu, jb < j1); jb += G) {
      const int j = jb + sub;
      bool take = false;
      if (j < j1) {
        const float4 b0 = REC.p0(j);
        take = !f_blanked(b0) && (!(dist2(offset_x(I, b0, dcol, dxc), offset_y(I, b0, dxc)) >= R2) || f_nonfinite(b0));
      }
      unsigned m = 1u, below = 0u;
      if (G > 1) {
        m = (__ballot_sync(0xffffffffu, take) >> (lane_id() & ~(unsigned)(G - 1))) & ((1u << G) - 1u);
        below = __popc(m & ((1u << sub) - 1u));
      }
      if (take && cnt + (int)below < LIST_CAP) row[cnt + below] = (unsigned)j | tag;
      cnt += G > 1 ? __popc(m) : (take ? 1 : 0);
    }
  }
  if (!on || sub != 0) return;
  if (cnt > LIST_CAP) {
    atomicOr(&D.st->error_flags, ERR_LIST_OVERFLOW);
    cnt = LIST_CAP;
  }
  D.ncount[q] = cnt;
}

// The neighbour-list invariant by brute force (a diagnostic: all N^2 pairs). k_list_abs puts
// every particle's position in FP64 from its pair record (origin of the cell of the last sort
// plus the FP32 offset); k_list_check then requires of every particle i that has a list (not
// blanked, finite, not a tool particle without heat conduction) that each unblanked, finite j
// closer than 2 h_i (h_i of the record, less a 1e-5 relative margin; the pair kernel's
// zero-distance cut-off 1e-8 left out) is among the ncount[i] entries of its row.
// out[0] += such pairs, out[1] += those missing from the lists.
static __global__ void k_list_abs(int N, dev_buffers D, double2 *abs) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= N) return;
  const float4 b0 = reinterpret_cast<const float4 *>(D.recf)[recf_word(0, j, N)];
  const geom g = *D.g;
  const int hj = D.hash_cur[j];
  const int cx = hj / g.ny, cy = hj - cx * g.ny;
  const double dxf = (double)(float)g.dx;
  abs[j] = make_double2(g.bbmin_x + cx * dxf + (double)b0.x, g.bbmin_y + cy * dxf + (double)b0.y);
}

static __global__ void k_list_check(params P, dev_buffers D, const double2 *__restrict__ abs,
                                    unsigned long long *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= P.N) return;
  const float4 *__restrict__ r0 = reinterpret_cast<const float4 *>(D.recf);
  const float4 bi = r0[recf_word(0, i, P.N)];
  if (f_blanked(bi) || f_nonfinite(bi)) return;
  if (f_tool(bi) && P.thermal_solver != MF_THERMAL_BROOKSHAW) return;  // no pair sums
  const double h = (double)bi.w;
  const double lim = 4. * h * h * (1. - 1e-5);
  const double2 xi = abs[i];
  const unsigned *row = D.nlist + (size_t)i * LIST_CAP;
  const int cnt = min(D.ncount[i], LIST_CAP);
  unsigned long long pairs = 0, missing = 0;
  for (int j = 0; j < P.N; ++j) {
    if (j == i) continue;
    const float4 bj = r0[recf_word(0, j, P.N)];
    if (f_blanked(bj) || f_nonfinite(bj)) continue;
    const double2 xj = abs[j];
    const double dx = xi.x - xj.x, dy = xi.y - xj.y;
    const double rr2 = dx * dx + dy * dy;
    if (!(rr2 < lim) || rr2 < 1e-8) continue;
    ++pairs;
    bool found = false;
    for (int k = 0; k < cnt && !found; ++k) found = (row[k] & LIST_INDEX_MASK) == (unsigned)j;
    if (!found) ++missing;
  }
  if (pairs) atomicAdd(out, pairs);
  if (missing) atomicAdd(out + 1, missing);
}

// The i particle of slot q: its records and the constants of its sums. False when q has no
// pair sums (past the end, blanked, a tool particle without Brookshaw heat).
__device__ __forceinline__ bool mixed_begin(const params &P, const dev_buffers &D, int q, mixed_i &I,
                                            mixed_const &K, double &thermal_alpha) {
  if (q >= P.N) return false;
  const float4 *__restrict__ r0 = reinterpret_cast<const float4 *>(D.recf);
  const float4 a0 = __ldg(r0 + recf_word(0, q, P.N));  // x, y, row, h
  if (f_blanked(a0)) return false;
  const bool tool_i = f_tool(a0);
  const bool brookshaw = P.thermal_solver == MF_THERMAL_BROOKSHAW;
  if (!brookshaw && tool_i) return false;
  const float4 a1 = __ldg(r0 + recf_word(1, q, P.N));  // vx, vy, sxy, Rxy
  const float4 a2 = __ldg(r0 + recf_word(2, q, P.N));  // sxx, syy, Rxx, Ryy
  const float4 a3 = __ldg(r0 + recf_word(3, q, P.N));  // rho, c, vol, T - T_init

  K.alpha4 = 0.25f * (float)P.corr.alpha;
  K.beta4 = 0.25f * (float)P.corr.beta;
  const float eta = (float)P.corr.eta;
  K.eta4 = 0.25f * eta * eta;
  thermal_alpha = 0.;
  if (brookshaw) thermal_alpha = !tool_i ? P.trml_wp.alpha : (P.thermal_tool_on ? P.trml_tool.alpha : 0.);

  I.thermal = thermal_alpha != 0.;
  I.nonfinite = f_nonfinite(a0);
  I.mech = !tool_i;
  I.x = a0.x; I.y = a0.y; I.row = fabsf(a0.z); I.h = fabsf(a0.w);
  I.nv = make_float2(-a1.x, -a1.y);
  I.sd = make_float2(a2.x, a2.y); I.sxy = a1.z;
  I.Rd = make_float2(a2.z, a2.w); I.Rxy = a1.w;
  I.rho = a3.x; I.c = a3.y; I.T = I.thermal ? a3.w : 0.f;
  // the spline's constants from the FP64 smoothing length, rounded once: an error of the rounded h
  // would enter every gradient four times over, all with the same sign
  const double h = D.B.h[q], h1 = 1. / h, fac = 0.454728408833987 * h1 * h1, w_in = fac * P.inv_wdeltap;
  I.h1 = (float)h1;
  I.fourh2 = (float)(4. * h * h);
  I.w_in = (float)w_in;
  I.w_out = (float)(0.25 * w_in);
  I.d_in = (float)(-3. * h1 * h1 * fac);
  I.d_out = (float)(-0.75 * h1 * fac);
  return true;
}

// the rates of slot q from its pair sums: Jaumann stress rate, continuity, momentum, advection
// and heat (actions_gpu.cu:100-132, interactions_gpu.cu:331-345)
__device__ __forceinline__ void mixed_end(const params &P, const dev_buffers &D, int q, int p, const mixed_i &I,
                                          const mixed_acc &acc, double thermal_alpha) {
  const float mass = (float)P.phys.mass;
  const float m2 = 2.f * mass, m_eps = (float)P.corr.xspheps * m2 * (float)P.corr.wdeltap;
  const float vdx = acc.v14.x, vdy = acc.vdy, vdz = acc.vdz, vdw = acc.v14.y;
  const float sdx = mass * acc.s14.x, sdy = mass * acc.sdy, sdz = mass * acc.sdz, sdw = mass * acc.s14.y;
  const float vtx = -m2 * acc.vtx, vty = -m2 * acc.vty;
  const float xtx = m_eps * acc.xtx, xty = m_eps * acc.xty, T_lapl = 2.f * acc.T_lapl;
  const bool mech_i = I.mech, thermal = I.thermal;
  const float rhoi = I.rho;

  const state_set &B = D.B;
  if (P.keep_derivs) {
    D.S_der[q] = make_double4(sdx, sdy, sdz, sdw);
    D.v_der[q] = make_double4(vdx, vdy, vdz, vdw);
  }
  if (mech_i) {
    const double4 S = B.S[q];
    const float G = (float)P.phys.G;
    const float e01 = 0.5f * (vdy + vdz);
    const float w01 = 0.5f * (vdz - vdy);
    const float t3 = (1.f / 3.f) * (vdx + vdw);
    const float Sxx = (float)S.x, Sxy = (float)S.y, Syy = (float)S.z;
    const float g2 = 2.f * G;
    // Jaumann rate with omega_10 = -omega_01 (actions_gpu.cu:120-132)
    const float tx = g2 * (vdx - t3) - 2.f * w01 * Sxy;
    const float ty = g2 * e01 + w01 * (Sxx - Syy);
    const float tz = g2 * (vdw - t3) + 2.f * w01 * Sxy;
    const float tw = -g2 * t3;
    B.S_t[q] = make_double4(tx, ty, tz, tw);
    B.rho_t[q] = -(double)rhoi * (double)(vdx + vdw);
    double2 fc, ft;
    prev_contact_forces(P, D, q, p, B.flags[q], fc, ft);
    const double2 vp = B.vel[q];
    double2 vel_t = make_double2((double)(vtx + (sdx + sdy)), (double)(vty + (sdz + sdw)));
    if (fc.x != 0. || fc.y != 0. || ft.x != 0. || ft.y != 0.) {  // (few particles touch the tool)
      const double m = P.phys.mass;
      vel_t.x = vel_t.x + fc.x / m + ft.x / m;
      vel_t.y = vel_t.y + fc.y / m + ft.y / m;
    }
    B.vel_t[q] = vel_t;
    B.pos_t[q] = make_double2((double)xtx + vp.x, (double)xty + vp.y);
  } else {
    B.vel_t[q] = make_double2(vtx, vty);
    B.pos_t[q] = make_double2(xtx, xty);
  }
  if (thermal) B.T_t[q] = thermal_alpha * (double)T_lapl;
}

// A particle's contributing neighbours in shared memory, in the order of the window, filled by its
// G lanes. Its sums have T parts: neighbour number n (counted in that order) belongs to part n mod T,
// each part is summed in order, and the parts are added up in order. Where T lanes share the
// particle (G = T) each takes a part; one lane (G = 1, the batched kernels) takes them one after the
// other and gets the same bits. The neighbours and their order do not depend on whether the window
// or the particle's neighbour list was searched.
// An entry is the neighbour's index and the column offset of the pair's cells (i's - j's) + 3.
template <int G>
struct mixed_rows {
  static constexpr int CAP = G == 1 ? 41 : 64 + G;  // entries (rows on distinct banks)
};
constexpr int ROW_INDEX_BITS = 29;
constexpr unsigned ROW_INDEX_MASK = (1u << ROW_INDEX_BITS) - 1u;
// words of a block's rows, whatever its lanes per particle
template <int BS>
struct mixed_shared {
  static constexpr int WORDS = BS * mixed_rows<1>::CAP;
};

__device__ __forceinline__ void acc_add(mixed_acc &a, const mixed_acc &b) {
  a.v14.x += b.v14.x; a.vdy += b.vdy; a.vdz += b.vdz; a.v14.y += b.v14.y;
  a.s14.x += b.s14.x; a.sdy += b.sdy; a.sdz += b.sdz; a.s14.y += b.s14.y;
  a.vtx += b.vtx; a.vty += b.vty; a.xtx += b.xtx; a.xty += b.xty;
  a.T_lapl += b.T_lapl;
}
__device__ __forceinline__ void acc_zero(mixed_acc &a) {
  a.v14 = a.s14 = make_float2(0.f, 0.f); a.vdy = a.vdz = a.sdy = a.sdz = 0.f;
  a.vtx = a.vty = a.xtx = a.xty = a.T_lapl = 0.f;
}

// called by whole warps
template <int G>
__device__ __forceinline__ void row_append(unsigned *row, int &cnt, int sub, bool take, unsigned entry) {
  if (G == 1) {
    if (take) row[cnt++] = entry;
    return;
  }
  const unsigned m = (__ballot_sync(0xffffffffu, take) >> (lane_id() & ~(unsigned)(G - 1))) & ((1u << G) - 1u);
  if (take) row[cnt + __popc(m & ((1u << sub) - 1u))] = entry;
  cnt += __popc(m);
}

// entries first, first + step, ... of a row of cnt
__device__ __forceinline__ void row_sum(const rec_global &R, const unsigned *row, int first, int step, int cnt,
                                        const mixed_i &I, const mixed_const &K, float dxc, mixed_acc &acc) {
  for (int k = first; k < cnt; k += step) {
    const unsigned e = row[k];
    float4 b0, b1, b2, b3;
    R.all((int)(e & ROW_INDEX_MASK), b0, b1, b2, b3);
    const float dcol = (float)((int)(e >> ROW_INDEX_BITS) - 3);
    mixed_interact<false>(I, K, acc, offset_x(I, b0, dcol, dxc), offset_y(I, b0, dxc), b0, b1, b2, b3);
  }
}

// The row's entries (numbers base, base + 1, ...) into the lane's part of the sums.
template <int G>
__device__ __forceinline__ void row_drain(const rec_global &R, const unsigned *row, int &cnt, int &base, int sub,
                                          const mixed_i &I, const mixed_const &K, float dxc, mixed_acc &acc) {
  if (G > 1) __syncwarp();
  row_sum(R, row, (sub - base) & (G - 1), G, cnt, I, K, dxc, acc);
  base += cnt;
  cnt = 0;
  if (G > 1) __syncwarp();
}

// One lane's T parts, one after the other, added up in acc at the last drain of the particle. Rows
// that overflow (more than CAP neighbours) keep their unfinished parts in local memory meanwhile.
template <int T>
__device__ __forceinline__ void row_drain_parts(const rec_global &R, const unsigned *row, int &cnt, int &base,
                                                bool last, mixed_acc *part, const mixed_i &I, const mixed_const &K,
                                                float dxc, mixed_acc &acc) {
  const bool kept = base != 0;
#pragma unroll 1
  for (int r = 0; r < T; ++r) {
    mixed_acc s;
    acc_zero(s);
    if (kept) s = part[r];
    row_sum(R, row, (r - base) & (T - 1), T, cnt, I, K, dxc, s);
    if (!last) part[r] = s;
    else if (r == 0) acc = s;
    else acc_add(acc, s);
  }
  base += cnt;
  cnt = 0;
}

// The 5x5 window's pair sums (interactions_gpu.cu:147-345) of a particle's G lanes, in two passes
// like the FP64 kernel's (pair_fp64_body): the candidates that contribute, by the same FP32 test
// that the pair term makes, into the row, then the row's entries, so that a warp's lanes run their
// ~28 pair terms together instead of each column's separately. Called by whole warps; `on`: the
// particle takes part.
template <int G, int T>
__device__ __forceinline__ void mixed_window(const dev_buffers &D, const rec_global &R, int N, int sub, unsigned *row,
                                             bool on, const mixed_i &I, const mixed_const &K, const geom &g, int gi,
                                             int gj, float dxc, mixed_acc &acc) {
  constexpr int U = CAND_STEP / G;
  static_assert(G == T || G == 1, "a lane per part, or one lane");
  const int low_j = gj - 2 < 0 ? 0 : gj - 2;
  const int high_j = gj + 3 > g.ny ? g.ny : gj + 3;
  int cnt = 0, base = 0;
  mixed_acc part[G == T ? 1 : T];
  auto drain = [&](bool last) {
    if (G == T) row_drain<G>(R, row, cnt, base, sub, I, K, dxc, acc);
    else row_drain_parts<T>(R, row, cnt, base, last, part, I, K, dxc, acc);
  };
  auto bounds = [&](int c, int &j0, int &j1) {  // window column c's particles
    const int ii = gi - 2 + c;
    const bool in = on && ii >= 0 && ii < g.nx;
    j0 = in ? __ldg(D.off + ii * g.ny + low_j) : 0;
    j1 = in ? __ldg(D.off + ii * g.ny + high_j) : 0;
  };
  int n0, n1;
  bounds(0, n0, n1);
#pragma unroll 1
  for (int c = 0; c < 5; ++c) {
    const int j0 = n0, j1 = n1;
    if (c < 4) bounds(c + 1, n0, n1);  // the next column's bounds, in flight during this one
    const float dcol = (float)(2 - c);
    const unsigned tag = (unsigned)(5 - c) << ROW_INDEX_BITS;
    for (int jb = j0; __any_sync(0xffffffffu, jb < j1); jb = next_round(jb, N)) {
      if (__any_sync(0xffffffffu, cnt > mixed_rows<G>::CAP - CAND_STEP)) drain(false);
      float4 b[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        b[u] = R.p0(jb + u * G + sub);  // (past the column's end: not used)
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int j = jb + u * G + sub;
        const float rr2 = dist2(offset_x(I, b[u], dcol, dxc), offset_y(I, b[u], dxc));
        // (false for a blanked particle's NaN row)
        bool take = rr2 < I.fourh2 && rr2 >= 1e-8f;
        if (I.nonfinite || f_nonfinite(b[u])) take = !f_blanked(b[u]);
        row_append<G>(row, cnt, sub, j < j1 && take, (unsigned)j | tag);
      }
    }
  }
  drain(true);
}

// A list step's pair sums: the row of the particle's neighbour list in place of the window; each
// entry passes the same support test as a window candidate. One lane per particle sums as it reads,
// with a software pipeline: the next entry's four record words are in flight while one entry is
// summed (past the count, the particle's own record, always a valid address; measured on the
// ~150k-particle cut: pair kernel 48.1 against 50.1 us at 5 blocks per SM). Several lanes search
// the list as they search the window. Called by whole warps; `on`: the particle takes part.
template <int G>
__device__ __forceinline__ void mixed_list(const dev_buffers &D, const rec_global &R, int q, int sub, unsigned *srow,
                                           bool on, const mixed_i &I, const mixed_const &K, float dxc, mixed_acc &acc) {
  const unsigned self = (unsigned)q | (3u << LIST_INDEX_BITS);
  auto take = [&](const float4 &b0, float xij, float yij) {
    const float rr2 = dist2(xij, yij);
    return f_nonfinite(b0) ? !f_blanked(b0) : rr2 < I.fourh2 && rr2 >= 1e-8f;  // (false for a blanked NaN row)
  };
  auto xij_of = [&](unsigned e, const float4 &b0) {
    return offset_x(I, b0, (float)((int)(e >> LIST_INDEX_BITS) - 3), dxc);
  };
  const int cnt = on ? D.ncount[q] : 0;
  if (G == 1) {
    // a particle's row is contiguous: four entries per 16-byte load
    const uint4 *row = reinterpret_cast<const uint4 *>(D.nlist + (size_t)q * LIST_CAP);
    uint4 e4 = row[0];  // (a row is LIST_CAP entries: the first four are always there)
    float4 c0, c1, c2, c3;
    R.all((int)((cnt > 0 ? e4.x : self) & LIST_INDEX_MASK), c0, c1, c2, c3);
    for (int k0 = 0; k0 < cnt; k0 += 4) {
      const unsigned ev[4] = {e4.x, e4.y, e4.z, e4.w};
      if (k0 + 4 < cnt) e4 = row[(k0 >> 2) + 1];  // the next four, in flight during these
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const bool live = k0 + u < cnt;
        const unsigned e = live ? ev[u] : self;
        const unsigned en = (k0 + u + 1 < cnt) ? (u < 3 ? ev[u + 1] : e4.x) : self;
        const float4 b0 = c0, b1 = c1, b2 = c2, b3 = c3;
        R.all((int)(en & LIST_INDEX_MASK), c0, c1, c2, c3);
        const float xij = xij_of(e, b0), yij = offset_y(I, b0, dxc);
        if (live && take(b0, xij, yij)) mixed_interact<true>(I, K, acc, xij, yij, b0, b1, b2, b3);
      }
    }
    return;
  }
  constexpr int U = 8 / G;
  static_assert(G == 1 || LIST_CAP <= mixed_rows<G>::CAP, "a whole list fits a row");
  const unsigned *row = D.nlist + (size_t)q * LIST_CAP;
  int n = 0, base = 0;
  for (int k0 = 0; __any_sync(0xffffffffu, k0 < cnt); k0 += 8) {
    unsigned e[U];
    float4 b[U];
#pragma unroll
    for (int u = 0; u < U; ++u) e[u] = k0 + u * G + sub < cnt ? row[k0 + u * G + sub] : self;
#pragma unroll
    for (int u = 0; u < U; ++u) b[u] = R.p0((int)(e[u] & LIST_INDEX_MASK));
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool in = take(b[u], xij_of(e[u], b[u]), offset_y(I, b[u], dxc));
      row_append<G>(srow, n, sub, k0 + u * G + sub < cnt && in,
                    (e[u] & LIST_INDEX_MASK) | (e[u] >> LIST_INDEX_BITS << ROW_INDEX_BITS));
    }
  }
  row_drain<G>(R, srow, n, base, sub, I, K, dxc, acc);
}

// The mixed pair sums, in T parts, of the particles of block bk.x (BS threads, G lanes per particle;
// s_list: mixed_shared<BS>::WORDS words). LIST: the neighbour-list form (steps with P.verlet): a step that
// sorts sums over the window, exactly as the form without lists, and builds the lists; the steps
// that keep the order sum over the lists (a particle with a non-finite record over the window).
template <int BS, int G, int T, bool LIST>
__device__ __forceinline__ void pair_mixed_body(const params &P, const dev_buffers &D, blk bk, unsigned *s_list) {
  const int sub = (int)threadIdx.x & (G - 1);
  const int q = bk.x * (BS / G) + (int)threadIdx.x / G;
  const int qc = q < P.N ? q : P.N - 1;
  unsigned *const row = s_list + (int)threadIdx.x / G * mixed_rows<G>::CAP;
  mixed_i I;
  mixed_const K;
  double thermal_alpha;
  const bool act = mixed_begin(P, D, qc, I, K, thermal_alpha) && q < P.N;
  if (!__any_sync(0xffffffffu, act)) return;
  const rec_global R(D.recf, P.N);
  // the particle's slot at the start of the step (its last contact forces are read there at the
  // end): loaded now, so that the load's latency passes during the sums; a list step without a
  // sort keeps the order
  const bool sorting = !LIST || D.st->sort_now;
  const int p = sorting ? __ldg(D.perm + qc) : qc;

  const geom g = *D.g;
  const float dxc = (float)g.dx;
  const int gi = D.col[qc];
  const int gj = (int)I.row - 1;

  mixed_acc acc;
  acc_zero(acc);

  const bool window = act && (sorting || I.nonfinite);
  if (LIST && !sorting) {
    mixed_list<G>(D, R, qc, sub, row, act && !window, I, K, dxc, acc);
    __syncwarp();
  }
  if (!LIST || __any_sync(0xffffffffu, window))
    mixed_window<G, T>(D, R, P.N, sub, row, window, I, K, g, gi, gj, dxc, acc);
  if (LIST && sorting) build_list<G>(D, R, qc, sub, act && !I.nonfinite, I, g, gi, gj, dxc, P.skin);
  if (G > 1) {  // the lanes' parts, added up in order by the particle's first lane
    const mixed_acc own = acc;
#pragma unroll
    for (int r = 1; r < G; ++r) {
      mixed_acc o;
      o.v14.x = __shfl_down_sync(0xffffffffu, own.v14.x, r); o.vdy = __shfl_down_sync(0xffffffffu, own.vdy, r);
      o.vdz = __shfl_down_sync(0xffffffffu, own.vdz, r); o.v14.y = __shfl_down_sync(0xffffffffu, own.v14.y, r);
      o.s14.x = __shfl_down_sync(0xffffffffu, own.s14.x, r); o.sdy = __shfl_down_sync(0xffffffffu, own.sdy, r);
      o.sdz = __shfl_down_sync(0xffffffffu, own.sdz, r); o.s14.y = __shfl_down_sync(0xffffffffu, own.s14.y, r);
      o.vtx = __shfl_down_sync(0xffffffffu, own.vtx, r); o.vty = __shfl_down_sync(0xffffffffu, own.vty, r);
      o.xtx = __shfl_down_sync(0xffffffffu, own.xtx, r); o.xty = __shfl_down_sync(0xffffffffu, own.xty, r);
      o.T_lapl = __shfl_down_sync(0xffffffffu, own.T_lapl, r);
      acc_add(acc, o);
    }
  }
  if (act && sub == 0) mixed_end(P, D, q, p, I, acc, thermal_alpha);
}

// Parts of a particle's sums, and lanes per particle of the single-system kernels: as many as let
// every particle's lanes be resident at once, then one; see pair64_lanes. The sorted and the list form
// give the same bits, so one rule serves both: the four-lane limit is the window form's (24 warps per
// SM on 148 SMs: 28,416 particles; the list form's own, at 20 warps, is 23,680), the two-lane limit the
// list form's (47,360; the window form's own is 56,832). Between them the other form gives away up to
// 6 %. Step in us, sorted every step, at 4 / 2 / 1 lanes: 7,090 particles 32.9 / 34.9 / 39.0; 23,437
// 35.4 / 37.6 / 41.3; 27,963 37.0 / 37.2 / 41.1; 28,957 39.3 / 39.0 / 41.3; 35,947 43.1 / 40.5 / 43.0;
// 47,207 46.2 / 43.2 / 45.3; 47,978 46.5 / 43.3 / 45.2; 56,867 49.3 / 46.4 / 49.4; 64,105 52.3 / 49.3 /
// 47.7; on lists: 28.8 / 31.4 / 36.6; 30.9 / 33.9 / 38.8; 35.9 / 34.0 / 39.1; 37.0 / 35.4 / 39.5; 37.4 /
// 35.4 / 40.5; 39.5 / 37.8 / 43.0; 43.2 / 43.9 / 43.6; 46.1 / 48.0 / 43.6; 47.0 / 49.3 / 44.5.
// (Before, one thread per particle: pair stage 22.0 on lists at 6,149, 32.8 sorted at 45,052.)
// A batch of many small systems fills the GPU anyway and runs the pair sums at one lane, in as many
// parts (24 systems of 2.8k to 38k particles: 196 us a step at one lane, 209 at two, 253 at four).
__host__ __device__ constexpr int mixed_parts(int N) { return N <= 28416 ? 4 : N <= 47360 ? 2 : 1; }

// blocks per SM: the window form at 6 (80 registers, no spills), the list form at 5 (96 registers,
// its software pipeline; at 4 with 113 registers 54 against 48 us)
template <int G, bool LIST>
static __global__ void __launch_bounds__(PAIR_BLOCK, LIST ? 5 : 6) k_pair_mixed(params P, dev_buffers D) {
  MF_PDL_WAIT();
  MF_PDL_TRIGGER();
  __shared__ unsigned s_list[PAIR_BLOCK / G * mixed_rows<G>::CAP];
  pair_mixed_body<PAIR_BLOCK, G, G, LIST>(P, D, grid_blk(), s_list);
}

// PSE heat Laplacian (interactions_gpu.cu:88-144, kernels.cuh:72-89) in FP32 for the mixed
// form, on the FP32 records: the same window (every particle of the 5x5 cells, blanked ones
// included, no support cut-off) and the same alpha through the half-length texture binding;
// the Gaussian from the hardware's 2^x, its exponent's factor rounded once from the FP64 smoothing
// length, temperatures relative to the initial temperature. G lanes per particle as in pse_body.
// It is bound by instructions (56 candidates of a particle), so a round of 8 candidates is read at
// constant offsets from one address (past the column's end what is read is not used), and a blanked
// candidate, whose record holds no row, is noticed by the NaN it leaves and the round done again.
// Measured at 577,555 particles: 54.9 us before (41 instructions a candidate), 46.4 so.
template <int BS, int G>
__device__ __forceinline__ void pse_mixed_body(const params &P, const dev_buffers &D, blk bk) {
  constexpr int U = 8 / G;
  const int sub = (int)threadIdx.x & (G - 1);
  const rec_global R(D.recf, P.N);
  const float2 *__restrict__ heat = D.heat;
  const int N = P.N;
  const geom g = *D.g;
  const float dxc = (float)g.dx;
  const long long tex_elems = ((long long)sizeof(int) * P.N) / 8;
  const int q = bk.x * (BS / G) + (int)threadIdx.x / G, qc = min(q, N - 1);
  const float4 a0 = R.p0(qc);  // x, y, row, h
  const float Ti = __ldg(heat + qc).y;
  const double h = D.B.h[qc], h2 = h * h;
  const float k2 = (float)(-1.4426950408889634 / h2);  // exp(-r^2 / h^2) = 2^(k2 r^2)
  const bool act = q < N && !f_blanked(a0);
  const float row = fabsf(a0.z);
  const int gi = D.col[qc], gj = (int)row - 1;
  const int low_j = max(gj - 2, 0), high_j = min(gj + 3, g.ny);
  float sum = 0.f;
  auto term = [&](const float4 &b0, float jrow, const float2 &b, float dcol) {
    const float xij = fmaf(dcol, dxc, a0.x - b0.x), yij = fmaf(row - jrow, dxc, a0.y - b0.y);
    float w;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(w) : "f"(__fmul_rn(dist2(xij, yij), k2)));
    return make_float2(__fmul_rn(b.y - Ti, b.x), w);
  };
  if (act) {
    for (int ii = max(gi - 2, 0); ii < min(gi + 3, g.nx); ++ii) {
      const int j0 = __ldg(D.off + ii * g.ny + low_j);
      const int j1 = __ldg(D.off + ii * g.ny + high_j);
      const float dcol = (float)(gi - ii);
      for (int jb = j0 + sub; jb < j1; jb += 8) {
        float4 b0[U];
        float2 b[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          b0[u] = R.p0(jb + u * G);
          b[u] = __ldg(heat + (jb + u * G));
        }
        const float before = sum;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const float2 t = term(b0[u], fabsf(b0[u].z), b[u], dcol);
          if (jb + u * G < j1) sum = fmaf(t.x, t.y, sum);
        }
        if (sum != sum) {  // a blanked candidate (or a NaN): its row from its cell
          sum = before;
          for (int j = jb; j < min(jb + 8, j1); j += G) {
            const float4 c0 = R.p0(j);
            const float jrow = f_blanked(c0) ? (float)(D.hash_cur[j] - ii * g.ny + 1) : fabsf(c0.z);
            const float2 t = term(c0, jrow, __ldg(heat + j), dcol);
            sum = fmaf(t.x, t.y, sum);
          }
        }
      }
    }
  }
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (act && sub == 0) {
    const bool tool_i = q < tex_elems ? f_tool(a0) : false;
    const double alpha = tool_i ? P.trml_tool.alpha : P.trml_wp.alpha;
    D.B.T_t[q] = alpha * (4. / 3.14159265358979323846 / (h2 * h2) * (double)sum);
  }
}

template <int G>
static __global__ void __launch_bounds__(PAIR_BLOCK) k_pse_mixed(params P, dev_buffers D) {
  MF_PDL_WAIT();
  MF_PDL_TRIGGER();
  pse_mixed_body<PAIR_BLOCK, G>(P, D, grid_blk());
}

}  // namespace mf
