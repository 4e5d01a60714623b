// Differentiable form: the FP64 leap-frog step (leap_frog.cu:94-155) carried out on dual
// numbers, so that every state variable also carries its derivative with respect to one of the
// Johnson-Cook parameters A, B, n, C, m or the friction coefficient mu. Forward-mode
// (tangent) propagation: the derivative of the window-averaged tool force follows the state
// through every step, the cell-list sort included (a permutation), with no checkpoints.
//
// Several directions run side by side: every kernel's grid has one row of blocks per direction
// (blockIdx.y), each on its own copy of the dual state, sharing the cell lists (the values are the
// same in all). A thread then carries one direction's duals: on a thread with all six the pair
// sums alone need more registers than there are, and 23k particles fill a quarter of the GPU. The
// repeated value arithmetic is a third of a direction's. Layout: one 16-byte (value, derivative)
// plane per scalar, so that a warp's loads are coalesced (one record of all scalars per particle
// cost a cache line per lane and scalar).
//
// The kernels restate the step of mf_kernels.cuh in dual arithmetic: gather + predictor + EOS +
// artificial stress, the pair sums with the rates (same neighbour lists, lanes per particle and
// division-free pair term), and the corrector .. boundary conditions with the secant return map
// iterated on duals, the tool force and the next step's cell counts. The cell lists come from the
// product's own kernels (k_scan, k_scatter and the stable rank) run on the value positions.
// Supported: locked grid (Green order), Brookshaw or no heat conduction, the Johnson-Cook law.
//
// Per step at 23,416 particles and six directions, before (one thread per particle with all six)
// and so: pair sums 974 / 213 us, force sum 281 us (one thread walking the block sums) / in the
// finish kernel, finish 98 / 42 us, gather 82 / 17 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <utility>

#include "mf_dual.cuh"
#include "mf_tangent.h"
#include "mfree_b200.h"

namespace mf {
namespace tg {

namespace {

// planes of a state, N duals each
enum : int {
  POSX = 0, POSY, VELX, VELY, SXX, SXY, SYY, SZZ, RHO, TEMP, EPS, EPSD, FCX, FCY, FTX, FTY,
  PTX, PTY, VTX, VTY, STX, STXY, STY, STZ, RHOT, TT, PLANES
};
// planes of the neighbour records (predicted state), in tiles of 32 particles; the last one holds
// (h, flags)
enum : int { N_X = 0, N_Y, N_VX, N_VY, N_SXX, N_SXY, N_SYY, N_RXX, N_RXY, N_RYY, N_RHO, N_C, N_VOL, N_T, N_HF, N_PLANES };

// what all directions share
struct shared_state {
  double *h;        // smoothing length
  unsigned *flags;  // fixed / blanked / tool bits
};

struct tbuf {
  dual *a, *b;  // state at the start of the step / in the new order: PLANES x N per direction
  shared_state sa, sb;
  unsigned *fl;    // the sorted flags of this step
  dual *n;         // contact normal, position-indexed: 2 x N per direction
  dual *pp;        // predictor pressure: N per direction
  dual *rec;       // neighbour records: rec_planes per direction
  float4 *cand;    // FP32 candidate records (mf_kernels.cuh, rec_cand)
  dual *blk;       // per-block force partials (4 per block) per direction
  dual *wsum;      // window sums of (Fc, Ff) per direction
  unsigned *tick;  // per direction: blocks that have left their partials
};

// the differentiated parameters, seeded in one direction
struct tparams {
  dual A, B, n, C, m, mu;
};
constexpr int MAX_DIRECTIONS = 6;
struct tparam_set {
  tparams t[MAX_DIRECTIONS];
};

__host__ __device__ __forceinline__ size_t rec_planes(int N) { return (size_t)((N + 31) / 32) * 32 * N_PLANES; }
__device__ __forceinline__ size_t rec_at(int k, int j) {
  return (size_t)(j >> 5) * (N_PLANES * 32) + (size_t)(k * 32 + (j & 31));
}
__device__ __forceinline__ dual load(const dual *p) {
  const double2 x = __ldg(reinterpret_cast<const double2 *>(p));
  return dual{x.x, x.y};
}

// cell hash of a position (grid.cu:34-51), clamped to the grid
__device__ __forceinline__ int cell_of(const geom &g, double x, double y) {
  const int ix = __double2int_rz((x - g.bbmin_x) / g.dx), iy = __double2int_rz((y - g.bbmin_y) / g.dx);
  const long long hh = (long long)ix * (long long)g.ny + (long long)iy;
  return (int)(hh < 0 ? 0 : hh >= g.num_cell ? g.num_cell - 1 : hh);
}

// the context's state into every direction's dual planes, and the first step's cell counts
__global__ void __launch_bounds__(BLOCK) k_t_start(int N, state_set S, const double2 *n, const int *hash, dev_buffers D,
                                                   tbuf T) {
  const int q = blockIdx.x * BLOCK + threadIdx.x, dir = blockIdx.y;
  if (q >= N) return;
  dual *a = T.a + (size_t)dir * PLANES * N + q;
  auto put = [&](int k, double v) { a[(size_t)k * N] = dconst(v); };
  auto put2 = [&](int k, double2 v) {
    put(k, v.x);
    put(k + 1, v.y);
  };
  auto put4 = [&](int k, double4 v) {
    put(k, v.x);
    put(k + 1, v.y);
    put(k + 2, v.z);
    put(k + 3, v.w);
  };
  const double2 pos = S.pos[q];
  const unsigned f = S.flags[q];
  put2(POSX, pos);
  put2(VELX, S.vel[q]);
  put4(SXX, S.S[q]);
  put(RHO, S.rho[q]);
  put(TEMP, S.T[q]);
  put(EPS, S.eps_pl[q]);
  put(EPSD, S.eps_pl_dot[q]);
  put2(FCX, S.fc[q]);
  put2(FTX, S.ft[q]);
  put2(PTX, S.pos_t[q]);
  put2(VTX, S.vel_t[q]);
  put4(STX, S.S_t[q]);
  put(RHOT, S.rho_t[q]);
  put(TT, S.T_t[q]);
  dual *nn = T.n + (size_t)dir * 2 * N;
  nn[q] = dconst(n[q].x);
  nn[N + q] = dconst(n[q].y);
  if (dir != 0) return;
  T.sa.h[q] = S.h[q];
  T.sa.flags[q] = f;
  const int hq = hash[q];
  D.hash_cur[q] = hq;
  // blanked particles keep their previous hash (grid.cu:39-41)
  const int hsh = (f & FLAG_BLANKED) ? min(max(hq, 0), D.g->num_cell - 1) : cell_of(*D.g, pos.x, pos.y);
  D.hash_new[q] = hsh;
  count_particle(D.count, D.tsum_r, hsh);
}

// artificial stress (actions_gpu.cu:35-39, 53-97) on duals; the derivatives of the angle and its
// sine and cosine only where a principal stress is tensile (elsewhere R is zero)
__device__ __forceinline__ void t_artificial_stress(const dual &rhoi21, const dual &sxx, const dual &sxy,
                                                    const dual &syy, double eps, dual &Rxx, dual &Rxy, dual &Ryy) {
  Rxx = Rxy = Ryy = dconst(0.);
  const double theta = 0.5 * (double)atan2f((float)(2. * sxy.v), (float)(sxx.v - syy.v));
  const double c = (double)cosf((float)theta), s = (double)sinf((float)theta);
  const double vxx = c * c * sxx.v + 2.0 * c * s * sxy.v + s * s * syy.v;
  const double vyy = s * s * sxx.v - 2.0 * c * s * sxy.v + c * c * syy.v;
  if (!(vxx > 0) && !(vyy > 0)) return;
  const dual th = 0.5 * datan2f_narrow(2. * sxy, sxx - syy);
  const dual ct = dcosf_narrow(th), st = dsinf_narrow(th);
  const dual ct2 = ct * ct, st2 = st * st;
  const dual rot_sxx = ct2 * sxx + 2.0 * ct * st * sxy + st2 * syy;
  const dual rot_syy = st2 * sxx - 2.0 * ct * st * sxy + ct2 * syy;
  dual rot_rxx = dconst(0.), rot_ryy = dconst(0.);
  if (rot_sxx.v > 0) rot_rxx = -eps * rot_sxx * rhoi21;
  if (rot_syy.v > 0) rot_ryy = -eps * rot_syy * rhoi21;
  Rxx = ct2 * rot_rxx + st2 * rot_ryy;
  Rxy = ct * st * (rot_rxx - rot_ryy);
  Ryy = st2 * rot_rxx + ct2 * rot_ryy;
}

// gather into the new order + predictor + EOS + artificial stress + records. Writes only what the
// later kernels read in the new order: the records, the predicted stress, the pressure, and the
// rates of the particles whose rates the pair pass does not (all) write.
__global__ void __launch_bounds__(128) k_t_reorder(params P, dev_buffers D, tbuf T) {
  MF_PDL_WAIT();
  MF_PDL_TRIGGER();
  const int t = blockIdx.x * blockDim.x + threadIdx.x, dir = blockIdx.y, N = P.N;
  if (t >= N) return;
  const int4 u = D.perm_u[t];
  const int p = u.x;
  const int q = u.z + stable_rank(D.perm_u, u);  // the particle's stable slot in its cell
  const unsigned f = T.sa.flags[p];
  const double h = T.sa.h[p];
  const bool blanked = f & FLAG_BLANKED, tool = f & FLAG_TOOL;
  const dual *a = T.a + (size_t)dir * PLANES * N + p;
  dual *b = T.b + (size_t)dir * PLANES * N + q;
  auto at = [&](int k) { return load(a + (size_t)k * N); };
  const double hdt = blanked ? 0. : 0.5 * P.dt;  // predict (leap_frog.cu:42-66)
  auto ahead = [&](int k, int kt) {
    const dual x = at(k);
    if (blanked) return x;
    return x + hdt * at(kt);
  };
  dual s[4], pos[2], vel[2];
  for (int k = 0; k < 2; ++k) {
    pos[k] = ahead(POSX + k, PTX + k);
    vel[k] = ahead(VELX + k, VTX + k);
  }
  for (int k = 0; k < 3; ++k) {
    s[k] = ahead(SXX + k, STX + k);
    b[(size_t)(SXX + k) * N] = s[k];
  }
  const dual rho = ahead(RHO, RHOT), temp = ahead(TEMP, TT);
  if (blanked || tool) {
    for (int k = PTX; k < PLANES; ++k) b[(size_t)k * N] = at(k);
  } else if (P.trml_wp.alpha == 0.) {
    b[(size_t)TT * N] = at(TT);
  }
  const dual rho21 = 1. / (rho * rho);
  dual prs = dconst(0.), Rxx = dconst(0.), Rxy = dconst(0.), Ryy = dconst(0.);
  if (!tool) {
    prs = P.eos_c0 * P.eos_c0 * (rho - P.phys.rho0);
    t_artificial_stress(rho21, s[0] - prs, s[1], s[2] - prs, P.corr.stresseps, Rxx, Rxy, Ryy);
  }
  T.pp[(size_t)dir * N + q] = prs;
  dual *rec = T.rec + dir * rec_planes(N);
  auto put = [&](int k, const dual &x) { rec[rec_at(k, q)] = x; };
  put(N_X, pos[0]); put(N_Y, pos[1]); put(N_VX, vel[0]); put(N_VY, vel[1]);
  put(N_SXX, (s[0] - prs) * rho21); put(N_SXY, s[1] * rho21); put(N_SYY, (s[2] - prs) * rho21);
  put(N_RXX, Rxx); put(N_RXY, Rxy); put(N_RYY, Ryy);
  put(N_RHO, rho);
  put(N_C, dsqrtf_narrow(P.phys.K / rho));
  put(N_VOL, P.phys.mass / rho);
  put(N_T, temp);
  rec[rec_at(N_HF, q)] = dual{h, __longlong_as_double((long long)f)};
  if (dir != 0) return;
  if (t == u.z) D.count[u.y] = 0;
  D.perm[q] = p;
  D.hash_cur[q] = u.y;
  T.sb.h[q] = h;
  T.fl[q] = f;
  // the pair kernel's candidate record (as in predict_particle)
  const geom g = *D.g;
  const int ci = u.y / g.ny, cj = u.y - ci * g.ny;
  const double rx = pos[0].v - (g.bbmin_x + ci * g.dx), ry = pos[1].v - (g.bbmin_y + cj * g.dx);
  const bool any = !cand_counts_cells(g) || !(fabs(rx) <= 4. * g.dx && fabs(ry) <= 4. * g.dx) ||
                   !(fabs(rho.v) >= 1e-30 && fabs(rho.v) <= 1e30) || !(h >= 1e-15 && h <= 1e15);
  T.cand[q] = make_float4(blanked ? __int_as_float(0x7f800000) : any ? __int_as_float(0x7fffffff) : (float)rx, (float)ry,
                          __uint_as_float(((unsigned)ci & CAND_COLUMN) | (tool ? CAND_TOOL : 0u) | (any ? CAND_ANY : 0u)), (float)cj);
}

// 1 / x on duals (rcp64 unless the value may lie outside float's range)
__device__ __forceinline__ dual drcp(const dual &x, bool careful) {
  const double r = careful ? 1. / x.v : rcp64(x.v);
  return dual{r, -(r * r) * x.d};
}

struct tpair_i {
  dual x, y, vx, vy, sxx, sxy, syy, Rxx, Rxy, Ryy, rho, c, T;
  double h, h1, fourh2, fac;
  bool tool, thermal;
};
struct tpair_acc {
  dual v[4], s[4], vt[2], xt[2], T;
};

// neighbour j added to particle i's sums (pair64_add on duals; outside the support nothing)
__device__ __forceinline__ void tpair_add(const params &P, const tpair_i &I, const dual *rec, int j, bool tool_j,
                                          bool careful, tpair_acc &a) {
  const dual *r = rec + rec_at(0, j);
  auto at = [&](int k) { return load(r + k * 32); };
  const dual xij = I.x - at(N_X), yij = I.y - at(N_Y);
  const dual rr2 = xij * xij + yij * yij;
  if (rr2.v >= I.fourh2 || rr2.v < 1e-8) return;
  // rad = (double)sqrtf((float)rr2); its derivative is the exact root's, 1 / sqrt(rr2) by one
  // third-order step from 1 / rad
  const float radf = sqrtf((float)rr2.v);
  const double irad_v = rcp64_from((double)radf, radf);
  const double e = fma(-rr2.v, irad_v * irad_v, 1.);
  const double isq = fma(irad_v, e * fma(e, 0.375, 0.5), irad_v);
  const dual rad{(double)radf, 0.5 * isq * rr2.d};
  const dual irad{irad_v, -(irad_v * irad_v) * rad.d};
  const dual qq = rad * I.h1;
  dual w, dwr;
  if (qq.v > 1.) {
    const dual t = 2. - qq, t2 = t * t;
    w = (0.25 * I.fac) * (t2 * t2 * t2);
    dwr = (-0.75 * I.h1 * I.fac) * (t2 * irad);
  } else {
    w = I.fac * (1. - 1.5 * (qq * qq) * (1. - 0.5 * qq));
    dwr = (-3. * I.h1 * I.h1 * I.fac) * (1. - 0.75 * qq);
  }
  const dual wx = dwr * xij, wy = dwr * yij;
  const dual volj = at(N_VOL);
  if (!I.tool && !tool_j) {
    const dual dvx = at(N_VX) - I.vx, dvy = at(N_VY) - I.vy;
    const dual ax = dvx * volj, ay = dvy * volj;
    a.v[0] += ax * wx;
    a.v[1] += ax * wy;
    a.v[2] += ay * wx;
    a.v[3] += ay * wy;
    dual fab = w * P.inv_wdeltap;
    fab = fab * fab;
    fab = fab * fab;
    const dual sxx = (I.sxx + at(N_SXX)) + fab * (I.Rxx + at(N_RXX));
    const dual sxy = (I.sxy + at(N_SXY)) + fab * (I.Rxy + at(N_RXY));
    const dual syy = (I.syy + at(N_SYY)) + fab * (I.Ryy + at(N_RYY));
    a.s[0] += sxx * wx;
    a.s[1] += sxy * wy;
    a.s[2] += sxy * wx;
    a.s[3] += syy * wy;
    const dual nvr = dvx * xij + dvy * yij;
    const dual irho = drcp(I.rho + at(N_RHO), careful);
    if (nvr.v > 0.) {
      const double hij = 0.5 * (I.h + load(r + N_HF * 32).v);
      const dual nmu = hij * nvr * drcp(rr2 + P.eta2 * hij * hij, careful);
      const dual pi = ((P.alpha_half * (I.c + at(N_C))) + P.corr.beta * nmu) * nmu * irho;
      a.vt[0] += pi * wx;
      a.vt[1] += pi * wy;
    }
    const dual xs = w * irho;
    a.xt[0] += xs * dvx;
    a.xt[1] += xs * dvy;
  }
  if (I.thermal) a.T += (volj * (I.T - at(N_T))) * dwr;
}

__device__ __forceinline__ dual sum_lanes(dual x, int o) {
  return dual{x.v + __shfl_xor_sync(0xffffffffu, x.v, o), x.d + __shfl_xor_sync(0xffffffffu, x.d, o)};
}

// pair sums over the 5x5 window (interactions_gpu.cu:147-345) and the rates
// (actions_gpu.cu:99-224), on duals: the two passes of pair_fp64_body with G lanes per particle
// (in 64-thread blocks at 4 per SM, 214 registers and no spills: 2,991 us for the ten-step six-direction
// pass at 23,416 particles; at 5, 168 registers and 64 B of spills, 3,148; at 8 3,046)
constexpr int T_PAIR_BLOCK = 64;
template <int G>
__global__ void __launch_bounds__(T_PAIR_BLOCK, 4) k_t_pair(params P, dev_buffers D, tbuf T) {
  MF_PDL_WAIT();
  MF_PDL_TRIGGER();
  using R_ = pair64_rows<G>;
  constexpr int GROUPS = T_PAIR_BLOCK / G, U = R_::U, LANES = R_::LANES, HALF = R_::HALF,
                CAP = R_::CAP;
  __shared__ unsigned s_list[T_PAIR_BLOCK / LANES * CAP];
  const int N = P.N, dir = blockIdx.y;
  const int sub = (int)threadIdx.x & (G - 1), side = (int)threadIdx.x & (LANES - 1);
  unsigned *const row = s_list + (int)threadIdx.x / LANES * CAP;
  const int q = (int)blockIdx.x * GROUPS + (int)threadIdx.x / G;
  const int qc = q < N ? q : N - 1;
  const float4 *__restrict__ cand = T.cand;
  const dual *__restrict__ rec = T.rec + dir * rec_planes(N);
  const float4 ci = __ldg(cand + qc);
  auto at = [&](int k) { return load(rec + rec_at(k, qc)); };
  const dual hf = at(N_HF);
  const unsigned fi = (unsigned)__double_as_longlong(hf.d), marks = __float_as_uint(ci.z);
  const bool act = q < N && !(fi & FLAG_BLANKED), any_i = marks & CAND_ANY;
  const geom g = *D.g;
  const float dxc = (float)g.dx;
  const float Rf = 2.00001f * (float)hf.v + 1e-5f * dxc;  // as in pair_fp64_body
  const float R2 = Rf * Rf;
  const float xi = any_i ? __int_as_float(0x7fffffff) : ci.x;
  int gi = (int)(marks & CAND_COLUMN), gj = (int)ci.w;
  if (!cand_counts_cells(g)) {
    const int c = D.hash_cur[qc];
    gi = c / g.ny;
    gj = c - gi * g.ny;
  }
  const int low_j = max(gj - 2, 0), high_j = min(gj + 3, g.ny);
  tpair_i I;
  I.tool = fi & FLAG_TOOL;
  const double alpha = !I.tool ? P.trml_wp.alpha : (P.thermal_tool_on ? P.trml_tool.alpha : 0.);
  I.thermal = alpha != 0.;
  I.x = at(N_X); I.y = at(N_Y); I.vx = at(N_VX); I.vy = at(N_VY);
  I.sxx = at(N_SXX); I.sxy = at(N_SXY); I.syy = at(N_SYY);
  I.Rxx = at(N_RXX); I.Rxy = at(N_RXY); I.Ryy = at(N_RYY);
  I.rho = at(N_RHO); I.c = at(N_C); I.T = at(N_T);
  I.h = hf.v;
  I.h1 = 1. / I.h;
  I.fourh2 = 4. * I.h * I.h;
  I.fac = 0.454728408833987 * I.h1 * I.h1;
  tpair_acc a;
#pragma unroll
  for (int k = 0; k < 4; ++k) a.v[k] = a.s[k] = dconst(0.);
  a.vt[0] = a.vt[1] = a.xt[0] = a.xt[1] = a.T = dconst(0.);
  int cnt = 0, c = -1, jb = 0, j1 = 0;  // entries; the column, its next candidate and its end
  do {
    // fill the rows: until the window is exhausted or a row could overflow
    bool more = true;
    while (more) {
      while (jb >= j1 && c < 5) {  // to the next column with candidates
        ++c;
        const int ii = gi - 2 + c;
        const bool in = act && c < 5 && ii >= 0 && ii < g.nx;
        jb = in ? __ldg(D.off + ii * g.ny + low_j) : 0;
        j1 = in ? __ldg(D.off + ii * g.ny + high_j) : 0;
      }
      const float ox = fmaf((float)(2 - c), dxc, xi);
      float4 b[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        b[u] = __ldg(cand + (jb + u * G + sub));  // (past the column's end: not used)
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int j = jb + u * G + sub;
        const float xij = ox - b[u].x;
        const float yij = fmaf(ci.w - b[u].w, dxc, ci.y - b[u].y);
        const float rr2 = fmaf(xij, xij, yij * yij);
        if (j < j1 && !(rr2 > R2) && j != q) {
          row[side ? CAP - 1 - cnt : cnt] = (unsigned)j | (__float_as_uint(b[u].z) & (CAND_TOOL | CAND_ANY));
          ++cnt;
        }
      }
      jb = next_round(jb, N);
      more = __any_sync(0xffffffffu, c < 5) && !__any_sync(0xffffffffu, cnt > HALF - U);
    }
    if (LANES > 1) __syncwarp();
    const int other = LANES > 1 ? __shfl_xor_sync(0xffffffffu, cnt, 1) : 0;
    const int front = side ? other : cnt, n = cnt + other;
    for (int k = side; k < n; k += LANES) {
      const unsigned e = row[k < front ? k : CAP - 1 - (k - front)];
      const int j = (int)(e & CAND_COLUMN);
      const bool careful = (e & CAND_ANY) || any_i;
      if (careful && ((unsigned)__double_as_longlong(load(rec + rec_at(N_HF, j)).d) & FLAG_BLANKED)) continue;
      tpair_add(P, I, rec, j, e & CAND_TOOL, careful, a);
    }
    cnt = 0;
    if (LANES > 1) __syncwarp();
  } while (__any_sync(0xffffffffu, c < 5));
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      a.v[k] = sum_lanes(a.v[k], o);
      a.s[k] = sum_lanes(a.s[k], o);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      a.vt[k] = sum_lanes(a.vt[k], o);
      a.xt[k] = sum_lanes(a.xt[k], o);
    }
    a.T = sum_lanes(a.T, o);
  }
  if (!act || sub != 0) return;
  dual *b = T.b + (size_t)dir * PLANES * N + q;
  auto put = [&](int k, const dual &x) { b[(size_t)k * N] = x; };
  if (!I.tool) {
    // Jaumann rate (actions_gpu.cu:99-133); the structurally zero GLM entries dropped
    const dual vdx = a.v[0], vdy = a.v[1], vdz = a.v[2], vdw = a.v[3];
    const dual e01 = 0.5 * (vdy + vdz), w01 = 0.5 * (vdz - vdy), w10 = 0.5 * (vdy - vdz);
    const dual t3 = (1. / 3.) * (vdx + vdw);
    const double g2 = 2. * P.phys.G, mass = P.phys.mass, m2 = 2. * mass, m_eps = P.corr.xspheps * m2;
    const dual Sxx = b[(size_t)SXX * N], Sxy = b[(size_t)SXY * N], Syy = b[(size_t)SYY * N];
    put(STX, g2 * (vdx - t3) + w10 * Sxy + Sxy * w10);
    put(STXY, g2 * e01 + w01 * Sxx + Syy * w10);
    put(STY, g2 * (vdw - t3) + w01 * Sxy + Sxy * w01);
    put(STZ, g2 * (0. - t3));
    put(RHOT, -(I.rho * (vdx + vdw)));
    // the last step's contact forces stay with the start state
    const dual *s = T.a + (size_t)dir * PLANES * N + D.perm[q];
    auto force = [&](int k) { return load(s + (size_t)k * N) / mass; };
    put(VTX, (-m2) * a.vt[0] + (mass * a.s[0] + mass * a.s[1] + force(FCX) + force(FTX)));
    put(VTY, (-m2) * a.vt[1] + (mass * a.s[2] + mass * a.s[3] + force(FCY) + force(FTY)));
    put(PTX, m_eps * a.xt[0] + I.vx);
    put(PTY, m_eps * a.xt[1] + I.vy);
  } else {
    put(PTX, dconst(0.));
    put(PTY, dconst(0.));
    put(VTX, dconst(0.));
    put(VTY, dconst(0.));
  }
  if (I.thermal) put(TT, (2. * alpha) * a.T);
}

// the factor of the Johnson-Cook yield stress (plasticity.cuh:30-46) that depends on the
// temperature alone
__device__ __forceinline__ dual t_term_c(const params &P, const tparams &TP, const dual &t) {
  const mf_joco_constants &jc = P.joco;
  return 1.0 - dpow((t - jc.Tref) / (jc.Tmelt - jc.Tref), TP.m);
}
__device__ __forceinline__ dual t_sigma_yield(const params &P, const tparams &TP, const dual &eps_pl,
                                              const dual &eps_pl_dot, const dual &term_c) {
  const dual Term_A = TP.A + TP.B * dpow(eps_pl, TP.n);
  const dual eps_dot = eps_pl_dot / P.joco.eps_dot_ref;
  const dual Term_B = eps_dot.v > 1.0 ? 1.0 + TP.C * dlog(eps_dot) : dpow(1.0 + eps_dot, TP.C);
  return Term_A * Term_B * term_c;
}

// secant radial return (plasticity.cuh:74-119) iterated on duals: the derivative of the
// iterate the reference returns
__device__ __noinline__ dual t_solve_secant(const params &P, const tparams &TP, dual init, dual norm_Strial,
                                            dual eps_pl_init, dual term_c, double delta_t, double mu) {
  const double s23 = sqrt(2.0 / 3.0), tol = 1e-6;
  dual dl = init, dl_old = init;
  int iter = 0;
  while (true) {
    const dual dl_1 = dl * 1.01;
    const dual e0 = eps_pl_init + s23 * dfmax0(dl), ed0 = s23 * dfmax0(dl) / delta_t;
    const dual e1 = eps_pl_init + s23 * dfmax0(dl_1), ed1 = s23 * dfmax0(dl_1) / delta_t;
    const dual g = norm_Strial - 2 * mu * dl - s23 * t_sigma_yield(P, TP, e0, ed0, term_c);
    const dual g_1 = norm_Strial - 2 * mu * dl_1 - s23 * t_sigma_yield(P, TP, e1, ed1, term_c);
    const dual slope = (g - g_1) / (dl - dl_1);
    dl_old = dl;
    dl = dl - g / slope;
    if (dl.v < 0.) dl = -0.1 * dl;
    if (fabs(dl.v - dl_old.v) < tol) return dl;
    if (iter > 100) return dl;
    iter++;
  }
}

// contact (tool_gpu.cu:87-207) on duals; the closest feature is chosen on values
__device__ __noinline__ bool t_contact(const mf_tool_state &TL, const dual &qx, const dual &qy, dual &cpx, dual &cpy,
                                       dual &nx, dual &ny) {
  double cpxv, cpyv, nxv, nyv;
  if (!establish_contact(TL, qx.v, qy.v, cpxv, cpyv, nxv, nyv)) return false;
  // repeat the selection of establish_contact to know which feature won
  const bool has_fillet = TL.num_seg == 5;
  double depth = 3.402823466e+38;
  int best = -1;
  for (int i = 0; i < TL.num_seg; i++) {
    double d;
    if (TL.seg[i].vertical) d = fabs(TL.seg[i].left[0] - qx.v);
    else if (has_fillet && i == 2) d = circle_segment_distance(TL.fillet, qx.v, qy.v);
    else {
      const double bb = -1, cc = TL.seg[i].b, aa = TL.seg[i].a;
      const double px = (bb * (bb * qx.v - aa * qy.v) - aa * cc) / (aa * aa + bb * bb);
      const double py = (aa * (-bb * qx.v + aa * qy.v) - bb * cc) / (aa * aa + bb * bb);
      d = sqrt((px - qx.v) * (px - qx.v) + (py - qy.v) * (py - qy.v));
    }
    if (d < depth) { depth = d; best = i; }
  }
  if (best < 0) return false;
  const mf_segment &s = TL.seg[best];
  if (s.vertical) {
    nx = dconst(nxv);
    ny = dconst(nyv);
    cpx = dconst(s.left[0]);
    cpy = qy;
  } else if (has_fillet && best == 2) {
    const dual vx = qx - TL.fillet.p[0], vy = qy - TL.fillet.p[1];
    const dual inv = 1. / dsqrt(vx * vx + vy * vy);
    nx = vx * inv;
    ny = vy * inv;
    cpx = TL.fillet.p[0] + nx * TL.fillet.r;
    cpy = TL.fillet.p[1] + ny * TL.fillet.r;
  } else {
    const double bb = -1, cc = s.b, aa = s.a;
    cpx = (bb * (bb * qx - aa * qy) - aa * cc) / (aa * aa + bb * bb);
    cpy = (aa * (-bb * qx + aa * qy) - bb * cc) / (aa * aa + bb * bb);
    nx = dconst(-s.n[0]);
    ny = dconst(-s.n[1]);
  }
  return true;
}

// corrector .. invalidate (leap_frog.cu:68-92, actions_gpu.cu:135-349, tool_gpu.cu:151-221)
// on duals, the step's tool force (report_force, output.cu:31-39; per block, then by the
// direction's last block in block order) and the next step's cell counts
// (The parameters are __grid_constant__: the out-of-line contact and secant functions take them by
// reference, and copies of them in every thread's local memory wrote 100 MB a launch: 2,991 us for
// the pass above, 2,782 without.)
constexpr int T_FINISH_BLOCK = 128;
__global__ void __launch_bounds__(T_FINISH_BLOCK)
    k_t_finish(const __grid_constant__ params P, const __grid_constant__ dev_buffers D, const __grid_constant__ tbuf T,
               const __grid_constant__ tparam_set TPS, const __grid_constant__ mf_tool_state TL, int accumulate) {
  MF_PDL_WAIT();
  MF_PDL_TRIGGER();
  __shared__ dual sh[4][T_FINISH_BLOCK];
  __shared__ bool s_last;
  const int N = P.N, dir = blockIdx.y, tid = threadIdx.x;
  const int q = blockIdx.x * T_FINISH_BLOCK + tid;
  const tparams &TP = TPS.t[dir];
  dual fc[2] = {dconst(0.), dconst(0.)}, ft[2] = {dconst(0.), dconst(0.)};
  if (q < N) {
    const double dt = P.dt;
    dual *b = T.b + (size_t)dir * PLANES * N + q;
    const dual *a = T.a + (size_t)dir * PLANES * N + D.perm[q];
    dual *nn = T.n + (size_t)dir * 2 * N + q;
    auto A = [&](int k) { return load(a + (size_t)k * N); };
    auto rate = [&](int k) { return b[(size_t)k * N]; };
    auto put = [&](int k, const dual &x) { b[(size_t)k * N] = x; };
    unsigned f = T.fl[q];
    const bool blanked = f & FLAG_BLANKED, tool = f & FLAG_TOOL, fixed = f & FLAG_FIXED;
    dual pos[2] = {A(POSX), A(POSY)}, vel[2] = {A(VELX), A(VELY)};
    dual S[4] = {A(SXX), A(SXY), A(SYY), A(SZZ)};
    dual rho = A(RHO), Tm = A(TEMP);
    bool bad = false;  // invalidate (actions_gpu.cu:317-349)
    auto step = [&](dual &x, int k) {
      const dual r = rate(k);
      x = x + dt * r;
      bad = bad || isnaninf(r.v);
    };
    if (!blanked) {
      for (int k = 0; k < 2; ++k) {
        step(pos[k], PTX + k);
        step(vel[k], VTX + k);
      }
      if (!tool && fixed) bad = false;  // their kinematic rates are zeroed below, before the test
      for (int k = 0; k < 4; ++k) step(S[k], STX + k);
      step(rho, RHOT);
      step(Tm, TT);
    }
    dual eps_pl = A(EPS), eps_pl_dot = A(EPSD);
    fc[0] = A(FCX); fc[1] = A(FCY);
    ft[0] = A(FTX); ft[1] = A(FTY);
    if (P.has_tool && P.fric_heat && !tool) {  // friction heat (actions_gpu.cu:135-162)
      const dual f2 = ft[0] * ft[0] + ft[1] * ft[1];
      if (sqrtf((float)f2.v) != 0.f) {
        const dual f_fric_mag = dsqrtf_narrow(f2);
        const dual vdx = vel[0] - TL.vel[0], vdy = vel[1] - TL.vel[1];
        const dual vdn = vdx * nn[0] + vdy * nn[N];
        const dual vrx = vdx - vdn, vry = vdy - vdn;
        const dual v_rel_mag = dsqrtf_narrow(vrx * vrx + vry * vry);
        Tm += P.trml_wp.eta * dt * f_fric_mag * v_rel_mag / (P.trml_wp.cp * P.phys.mass);
      }
    }
    if (P.plastic && !tool) {  // JC radial return (actions_gpu.cu:226-285)
      const double mu = P.phys.G;
      const double pr = T.pp[(size_t)dir * N + q].v;
      const double cxx = S[0].v - pr, cyy = S[2].v - pr, czz = S[3].v - pr, cxy = S[1].v;
      const double svm = (double)sqrtf(
          (float)((cxx * cxx + cyy * cyy + czz * czz) - cxx * cyy - cxx * czz - cyy * czz + 3.0 * cxy * cxy));
      // the yield test's value alone decides; first the FP32 lower bound of the flow stress (as in
      // the product's finish kernel)
      bool elastic = false;
      if (P.jc_lower_bound) {
        const mf_joco_constants &JC = P.joco;
        const float theta_f = (float)(Tm.v - JC.Tref) * (1.f / (float)(JC.Tmelt - JC.Tref));
        elastic = svm < 0.999 * JC.A * (1.0 - 1.00001 * (double)powf(theta_f, (float)JC.m));
      }
      if (!elastic) {
        const dual term_c = t_term_c(P, TP, Tm);
        elastic = svm < t_sigma_yield(P, TP, dconst(eps_pl.v), dconst(eps_pl_dot.v), term_c).v;
        if (!elastic) {
          const dual Sxx = S[0], Syy = S[2], Szz = S[3], Sxy = S[1];
          const dual norm_Strial = dsqrtf_narrow(Sxx * Sxx + Syy * Syy + Szz * Szz + Sxy * Sxy);
          dual init = eps_pl_dot * dt * sqrt(2. / 3.);
          if (!(init.v > 1e-8)) init = dconst(fmax(init.v, 1e-8));
          const dual dl = t_solve_secant(P, TP, init, norm_Strial, eps_pl, term_c, dt, mu);
          // (double)(sqrtf(2/3) * fmaxf((float)dl, 0)): float-rounded value, exact derivative
          const float s23f = sqrtf((float)(2.0 / 3.0));
          const double inc_v = (double)(s23f * fmaxf((float)dl.v, 0.f));
          const dual inc = dl.v > 0. ? dchain(inc_v, sqrt(2.0 / 3.0), dl) : dconst(inc_v);
          const dual eps_pl_new = eps_pl + inc;
          const dual eps_pl_dot_new = inc / dt;
          S[0] = Sxx - Sxx / norm_Strial * dl * 2. * mu;
          S[2] = Syy - Syy / norm_Strial * dl * 2. * mu;
          S[3] = Szz - Szz / norm_Strial * dl * 2. * mu;
          S[1] = Sxy - Sxy / norm_Strial * dl * 2. * mu;
          if (P.trml_wp.tq != 0.) {
            const dual sY = t_sigma_yield(P, TP, eps_pl_new, eps_pl_dot_new, term_c);
            Tm += P.trml_wp.tq / (P.trml_wp.cp * rho) * (eps_pl_new - eps_pl) * sY;
          }
          eps_pl = eps_pl_new;
          eps_pl_dot = eps_pl_dot_new;
        }
      }
      if (elastic) eps_pl_dot = dconst(0.);
    }
    if (P.has_tool) {
      if (tool) {
        pos[0] += dt * TL.vel[0];
        pos[1] += dt * TL.vel[1];
      } else {
        dual cpx, cpy, nx = dconst(0.), ny = dconst(0.);
        if (!t_contact(TL, pos[0], pos[1], cpx, cpy, nx, ny)) {
          fc[0] = fc[1] = ft[0] = ft[1] = dconst(0.);
        } else {
          const double dt2 = dt * dt;
          const dual gN = (pos[0] - cpx) * nx + (pos[1] - cpy) * ny;
          const dual sc = -TL.slave_mass * gN;
          const dual fNx = sc * nx / dt2 * TL.contact_alpha, fNy = sc * ny / dt2 * TL.contact_alpha;
          dual fTx = dconst(0.), fTy = dconst(0.);
          if (TP.mu.v != 0.) {
            const dual vx = vel[0] - TL.vel[0], vy = vel[1] - TL.vel[1];
            const dual vrx = vx - vx * nx, vry = vy - vy * ny;
            const double ks = TL.contact_alpha * TL.slave_mass;
            const dual kx = ks * vrx / dt, ky = ks * vry / dt;
            const dual fy = TP.mu * dsqrt(fNx * fNx + fNy * fNy);
            const dual fsx = ft[0] - kx, fsy = ft[1] - ky;
            const dual lfs = dsqrt(fsx * fsx + fsy * fsy);
            if (lfs.v > fy.v) {
              fTx = fy * fsx / lfs;
              fTy = fy * fsy / lfs;
            } else {
              fTx = fsx;
              fTy = fsy;
            }
          }
          fc[0] = fNx; fc[1] = fNy; ft[0] = fTx; ft[1] = fTy;
        }
        nn[0] = nx;
        nn[N] = ny;
      }
    }
    if (!tool && fixed) {  // boundary conditions (actions_gpu.cu:287-311)
      vel[0] = vel[1] = fc[0] = fc[1] = dconst(0.);
      for (int k = 0; k < 4; ++k) put(PTX + k, dconst(0.));
    }
    if (P.thermal_bc && fixed) Tm = dconst(P.trml_wp.T_init);
    if (!blanked && bad) f |= FLAG_BLANKED;
    for (int k = 0; k < 2; ++k) {
      put(POSX + k, pos[k]);
      put(VELX + k, vel[k]);
      put(FCX + k, fc[k]);
      put(FTX + k, ft[k]);
    }
    for (int k = 0; k < 4; ++k) put(SXX + k, S[k]);
    put(RHO, rho);
    put(TEMP, Tm);
    put(EPS, eps_pl);
    put(EPSD, eps_pl_dot);
    if (dir == 0) {  // flags, and the next step's hash and count
      T.sb.flags[q] = f;
      const int hsh = (f & FLAG_BLANKED) ? D.hash_cur[q] : cell_of(*D.g, pos[0].v, pos[1].v);
      D.hash_new[q] = hsh;
      count_particle(D.count, D.tsum_w, hsh);
    }
  }
  // the block's forces; blocks without contact (nearly all) leave zeros
  const bool nz = fc[0].v != 0. || fc[1].v != 0. || ft[0].v != 0. || ft[1].v != 0. || fc[0].d != 0. ||
                  fc[1].d != 0. || ft[0].d != 0. || ft[1].d != 0.;
  const int nb = gridDim.x;
  dual *blk = T.blk + (size_t)dir * 4 * nb;
  auto tree = [&]() {  // sh[k][0] = the sum over the block
    __syncthreads();
    for (int s = T_FINISH_BLOCK / 2; s > 0; s >>= 1) {
      if (tid < s)
        for (int k = 0; k < 4; ++k) sh[k][tid] = sh[k][tid] + sh[k][tid + s];
      __syncthreads();
    }
  };
  if (__syncthreads_or(nz)) {
    sh[0][tid] = fc[0]; sh[1][tid] = fc[1]; sh[2][tid] = ft[0]; sh[3][tid] = ft[1];
    tree();
  } else if (tid == 0) {
    for (int k = 0; k < 4; ++k) sh[k][0] = dconst(0.);
  }
  if (tid == 0) {
    for (int k = 0; k < 4; ++k) blk[4 * blockIdx.x + k] = sh[k][0];
    __threadfence();
    s_last = atomicAdd(&T.tick[dir], 1u) == (unsigned)nb - 1u;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  dual r[4] = {dconst(0.), dconst(0.), dconst(0.), dconst(0.)};
  for (int v = tid; v < nb; v += T_FINISH_BLOCK)
    for (int k = 0; k < 4; ++k) {
      const double2 x = __ldcg(reinterpret_cast<const double2 *>(blk + 4 * v + k));
      r[k] += dual{x.x, x.y};
    }
  for (int k = 0; k < 4; ++k) sh[k][tid] = r[k];
  tree();
  if (tid == 0) {
    T.tick[dir] = 0u;
    if (accumulate) {
      T.wsum[2 * dir] += sh[0][0] + sh[2][0];
      T.wsum[2 * dir + 1] += sh[1][0] + sh[3][0];
    }
  }
}

// lays arrays out one after the other in one allocation (256-byte aligned); with base = nullptr
// it only measures
struct arena {
  char *base;
  size_t at = 0;
  template <class X>
  void get(X *&p, size_t n) {
    at = (at + 255) & ~(size_t)255;
    p = base ? reinterpret_cast<X *>(base + at) : nullptr;
    at += n * sizeof(X);
  }
};

// each kernel may be scheduled while the previous one drains: launched one by one, not from a graph, the
// steps lose more to the gaps than the early start's uneven spread costs (1,045 against 1,143 us for
// 16 steps of 6,149 particles with the pair and finish kernels in turn)
template <typename... KArgs, typename... Args>
cudaError_t launch(cudaStream_t stream, void (*kernel)(KArgs...), dim3 grid, int block, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)block);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Lanes per particle of the pair kernel, by the particle count alone, so that a pass with one
// direction and one with six add each direction up alike. As many as let one direction's lanes be
// resident at once (4 blocks of 64 per SM: 9,472 particles at 4, 18,944 at 2), the four-lane limit
// lower, because six directions fill the GPU anyway and lose by four lanes at every size. Step in us
// at 4 / 2 / 1 lanes, one direction: 3,467 particles 68 / 75 / 95; 8,329 68 / 79 / 99; 11,233 86 / 81 /
// 101; 18,822 92 / 85 / 108; 23,437 108 / 104 / 107; 31,203 124 / 115 / 112; six: 97 / 91 / 103; 152 /
// 137 / 145; 196 / 170 / 162; 303 / 252 / 229; 368 / 304 / 278; 483 / 396 / 355.
constexpr int lanes(int N) { return N <= 8192 ? 4 : N <= 18944 ? 2 : 1; }

// Work memory kept for a context's next call; a larger one is given back, so that contexts with many
// particles do not hold several GB each while they step.
constexpr size_t KEEP_BYTES = (size_t)1 << 30;

}  // namespace

void release(workspace &ws) {
  if (ws.mem) cudaFree(ws.mem);
  ws.mem = nullptr;
  ws.bytes = 0;
}

int run_mean_force(const params &P_in, const dev_buffers &C, const state_set &now, mf_tool_state TL, int max_cell,
                   cudaStream_t stream, workspace &ws, int skip_steps, int window_steps, const int *directions,
                   int n_directions, double out_mean[2], double *out_dmean, int *cuda_err) {
  params P = P_in;
  P.staged = 0;
  P.verlet = 0;
  const int N = P.N, nd = std::max(1, n_directions);
  const int scan_tiles = (max_cell + SCAN_TILE - 1) / SCAN_TILE + 1;
  const int nf = (N + T_FINISH_BLOCK - 1) / T_FINISH_BLOCK;
  tbuf T{};
  dev_buffers D{};
  D.g = C.g;
  // the arrays that start at zero come first
  auto lay_out = [&](arena &m) {
    m.get(T.wsum, 2 * (size_t)nd);
    m.get(T.tick, (size_t)nd);
    m.get(D.st, 1);
    m.get(D.count, (size_t)max_cell);
    m.get(D.tsum_r, (size_t)scan_tiles);
    m.get(D.tsum_w, (size_t)scan_tiles);
    const size_t zeroed = m.at;
    m.get(D.off, (size_t)max_cell + 1);
    m.get(D.hash_cur, (size_t)N);
    m.get(D.hash_new, (size_t)N);
    m.get(D.perm, (size_t)N);
    m.get(D.perm_u, (size_t)N);
    m.get(T.sa.h, (size_t)N);
    m.get(T.sb.h, (size_t)N);
    m.get(T.sa.flags, (size_t)N);
    m.get(T.sb.flags, (size_t)N);
    m.get(T.fl, (size_t)N);
    m.get(T.cand, (size_t)N + CAND_PAD);
    m.get(T.blk, 4 * (size_t)nf * nd);
    m.get(T.n, 2 * (size_t)N * nd);
    m.get(T.pp, (size_t)N * nd);
    m.get(T.rec, rec_planes(N) * nd);
    m.get(T.a, (size_t)PLANES * N * nd);
    m.get(T.b, (size_t)PLANES * N * nd);
    return zeroed;
  };
  arena measure{nullptr};
  lay_out(measure);
  cudaError_t e = cudaSuccess;
  if (ws.bytes < measure.at) {
    release(ws);
    e = cudaMalloc(&ws.mem, measure.at);
    if (e != cudaSuccess) {
      ws.mem = nullptr;
      cudaGetLastError();
      *cuda_err = (int)e;
      return e == cudaErrorMemoryAllocation ? MF_ERR_NOMEM : MF_ERR_CUDA;
    }
    ws.bytes = measure.at;
  }
  arena place{(char *)ws.mem};
  const size_t zeroed = lay_out(place);
  tparam_set TPS{};
  const mf_joco_constants &jc = P.joco;
  for (int k = 0; k < nd; ++k) {
    const int dir = k < n_directions ? directions[k] : -1;
    auto seed = [dir](double v, int which) { return dual{v, dir == which ? 1. : 0.}; };
    TPS.t[k] = tparams{seed(jc.A, 0), seed(jc.B, 1), seed(jc.n, 2), seed(jc.C, 3), seed(jc.m, 4), seed(TL.mu, 5)};
  }
  const dim3 g128((unsigned)((N + 127) / 128), (unsigned)nd), g256((unsigned)((N + BLOCK - 1) / BLOCK), (unsigned)nd);
  const int G = lanes(N), per = T_PAIR_BLOCK / G;
  const dim3 gpair((unsigned)((N + per - 1) / per), (unsigned)nd), gfin((unsigned)nf, (unsigned)nd);
  e = cudaMemsetAsync(ws.mem, 0, zeroed, stream);
  if (e == cudaSuccess)
    k_t_start<<<g256, BLOCK, 0, stream>>>(N, now, C.n, C.hash_cur, D, T);
  if (e == cudaSuccess) e = cudaGetLastError();
  for (int step = 0; step < skip_steps + window_steps && e == cudaSuccess; ++step) {
    e = launch(stream, k_scan, dim3((unsigned)scan_tiles), SCAN_THREADS, D, N, 0);
    if (e == cudaSuccess) e = launch(stream, k_scatter, dim3(g256.x), BLOCK, N, D, 0);
    if (e == cudaSuccess) e = launch(stream, k_t_reorder, g128, 128, P, D, T);
    if (e == cudaSuccess)
      e = G == 4   ? launch(stream, k_t_pair<4>, gpair, T_PAIR_BLOCK, P, D, T)
          : G == 2 ? launch(stream, k_t_pair<2>, gpair, T_PAIR_BLOCK, P, D, T)
                   : launch(stream, k_t_pair<1>, gpair, T_PAIR_BLOCK, P, D, T);
    if (P.has_tool) mf_tool_translate(&TL, P.dt);  // tool::update_tool, before contact
    if (e == cudaSuccess)
      e = launch(stream, k_t_finish, gfin, T_FINISH_BLOCK, P, D, T, TPS, TL, step >= skip_steps ? 1 : 0);
    std::swap(D.tsum_r, D.tsum_w);  // the scan zeroed the one the finish kernel then added to
    std::swap(T.a, T.b);
    std::swap(T.sa, T.sb);
  }
  dual w[2 * MAX_DIRECTIONS];
  dev_status st;
  if (e == cudaSuccess) e = cudaMemcpyAsync(w, T.wsum, sizeof(dual) * 2 * nd, cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&st, D.st, sizeof(st), cudaMemcpyDeviceToHost, stream);
  const cudaError_t es = cudaStreamSynchronize(stream);
  if (e == cudaSuccess) e = es;
  if (ws.bytes > KEEP_BYTES) release(ws);
  if (e != cudaSuccess) {
    *cuda_err = (int)e;
    return MF_ERR_CUDA;
  }
  if (st.error_flags) return MF_ERR_CUDA;
  out_mean[0] = w[0].v / window_steps;
  out_mean[1] = w[1].v / window_steps;
  for (int k = 0; k < n_directions; ++k) {  // d(mean Fc), d(mean Ff) at [2k], [2k + 1]
    out_dmean[2 * k] = w[2 * k].d / window_steps;
    out_dmean[2 * k + 1] = w[2 * k + 1].d / window_steps;
  }
  return MF_OK;
}

}  // namespace tg
}  // namespace mf
