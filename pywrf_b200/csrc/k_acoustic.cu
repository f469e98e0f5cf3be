// Acoustic (small) time step (wrf_dynamics.py:3152-3930, wrf_boundary.py:244-400).
//   k_ssp2d / k_ssp3d   small_step_prep (2-D masses, then 3-D perturbation form)
//   k_p_rho0            calc_p_rho before the first substep
//   k_coef_w            calc_coef_w: tridiagonal coefficients + forward sweep
//   k_advance_uv        advance_uv + spec_bdyupdate(u), (v)
//   k_acoustic_col      advance_mu_t, advance_w, sumflux, spec_bdyupdate of
//                       t / mu / muts / ph and calc_p_rho of one substep
//   k_mu_uv_1 / k_ssfinish  calc_mu_uv_1, small_step_finish
// The vertical recurrences (mass divergence sum, ww scan, Thomas sweeps) run
// sequentially per column in the reference's order.
#include <type_traits>
#include "kernels.cuh"
#include "tma.cuh"

namespace wrf {

__global__ void k_ssp2d(Grid g, S s, int rk_step) {
  WRF_COLUMN_INDEX(g, j, i);
  const int c = g.i2(j, i);
  const int jts = g.jds, jme = g.jde - 1, its = g.ids, ime = g.ide - 1, ieu = g.ide, jev = g.jde;
  float* mu = s[WF_MU];
  float* mu1 = s[WF_MU_1];
  const float* mub = s[WF_MUB];
  const bool t2 = j >= jts && j < jme && i >= its && i < ime;
  if (rk_step == 1) {
    if (t2) {
      const float m2 = mu[c];
      mu1[c] = m2;
      s[WF_MUDF][c] = 0.f;
      s[WF_MUTS][c] = mub[c] + m2;
      s[WF_MU_SAVE][c] = m2;
      mu[c] = 0.f;
    }
    if (j >= jts && j < jme && i >= its && i < ieu) s[WF_MUUS][c] = s[WF_MUU][c];
    if (j >= jts && j < jev && i >= its && i < ime) s[WF_MUVS][c] = s[WF_MUV][c];
  } else {
    if (t2) {
      s[WF_MUTS][c] = mub[c] + mu1[c];
      const float m2 = mu[c];
      s[WF_MU_SAVE][c] = m2;
      mu[c] = mu1[c] - m2;
    }
    if (j >= jts && j < jme && i >= its && i < ieu)
      s[WF_MUUS][c] = 0.5f * (mub[c] + mu1[c] + mub[c - 1] + mu1[c - 1]);
    if (j >= jts && j < jev && i >= its && i < ieu)
      s[WF_MUVS][c] = 0.5f * (mub[c] + mu1[c] + mub[c - g.nx] + mu1[c - g.nx]);
  }
}

// all operands are loaded before any store (the stores would otherwise hold
// back the later fields' loads); in stage 1 the *_1 copies are the values
// just read
__global__ void k_ssp3d(Grid g, S s, int rk_step) {
  WRF_POINT_INDEX(g, k, j, i);
  const int nz = g.nz, ktf = nz - 1;
  const int jts = g.jds, jme = g.jde - 1, its = g.ids, ime = g.ide - 1, ieu = g.ide, jev = g.jde;
  const int c = g.i2(j, i);
  const size_t p = (size_t)k * g.ny * g.nx + c;
  const bool t2 = j >= jts && j < jme && i >= its && i < ime;
  const bool du = k < ktf && j >= jts && j < jme && i >= its && i < ieu;
  const bool dv = k < ktf && j >= jts && j < jev && i >= its && i < ime;
  const bool r1 = rk_step == 1;
  float u2 = 0.f, u1 = 0.f, muus = 0.f, muu = 0.f, mfuy = 1.f;
  if (du) {
    u2 = s[WF_U][p];
    u1 = r1 ? u2 : s[WF_U_1][p];
    muus = s[WF_MUUS][c];
    muu = s[WF_MUU][c];
    mfuy = s[WF_MSFUY][c];
  }
  float v2 = 0.f, v1 = 0.f, muvs = 0.f, muv = 0.f, mvxi = 0.f;
  if (dv) {
    v2 = s[WF_V][p];
    v1 = r1 ? v2 : s[WF_V_1][p];
    muvs = s[WF_MUVS][c];
    muv = s[WF_MUV][c];
    mvxi = s[WF_MSFVX_INV][c];
  }
  float muts = 0.f, mut = 0.f, pbv = 0.f, ppv = 0.f, altv = 1.f, t2v = 0.f, t1 = 0.f;
  float w2 = 0.f, w1 = 0.f, mfty = 1.f, ph2 = 0.f, ph1 = 0.f, wwv = 0.f;
  if (t2) {
    muts = s[WF_MUTS][c];
    mut = s[WF_MUT][c];
    if (k < ktf) {
      pbv = s[WF_PB][p];
      ppv = s[WF_P][p];
      altv = s[WF_ALT][p];
      t2v = s[WF_T][p];
      t1 = r1 ? t2v : s[WF_T_1][p];
    }
    w2 = s[WF_W][p];
    w1 = r1 ? w2 : s[WF_W_1][p];
    mfty = s[WF_MSFTY][c];
    ph2 = s[WF_PH][p];
    ph1 = r1 ? ph2 : s[WF_PH_1][p];
    wwv = s[WF_WW][p];
  }
  if (du) {
    if (r1) s[WF_U_1][p] = u2;
    s[WF_U_SAVE][p] = u2;
    s[WF_U][p] = (muus * u1 - muu * u2) / mfuy;
  }
  if (dv) {
    if (r1) s[WF_V_1][p] = v2;
    s[WF_V_SAVE][p] = v2;
    s[WF_V][p] = (muvs * v1 - muv * v2) * mvxi;
  }
  if (t2) {
    if (k < ktf) {
      s[WF_C2A][p] = (float)CPOVCV * (pbv + ppv) / altv;
      if (r1) s[WF_T_1][p] = t2v;
      s[WF_T_SAVE][p] = t2v;
      s[WF_T][p] = muts * t1 - mut * t2v;
    }
    if (r1) s[WF_W_1][p] = w2;
    s[WF_W_SAVE][p] = w2;
    s[WF_W][p] = (muts * w1 - mut * w2) / mfty;
    if (r1) s[WF_PH_1][p] = ph2;
    s[WF_PH_SAVE][p] = ph2;
    s[WF_PH][p] = ph1 - ph2;
    s[WF_WW1][p] = wwv;
  }
}

// calc_p_rho at the start of the acoustic steps (wrf_dynamics.py:3269-3313,
// step 0): al and p from the prepared state; pm1 becomes a copy of the whole
// new p (the later substeps run inside k_acoustic_col)
__global__ void k_p_rho0(Grid g, S s) {
  WRF_POINT_INDEX(g, k, j, i);
  const int ktf = g.nz - 1;
  const int c = g.i2(j, i);
  const size_t lev = (size_t)g.ny * g.nx;
  const size_t p = k * lev + c;
  float* pp = s[WF_P];
  float pnew = pp[p];
  if (k < ktf && j >= g.jds && j < g.jde - 1 && i >= g.ids && i < g.ide - 1) {
    // operands first, then the stores
    const float muts = s[WF_MUTS][c], mu = s[WF_MU][c];
    const float alt = s[WF_ALT][p], t1 = s[WF_T_SAVE][p];
    const float* ph = s[WF_PH];
    const float phu = ph[p + lev], phk = ph[p], rdnw = s[WF_RDNW][k];
    const float c2 = s[WF_C2A][p], tk = s[WF_T][p];
    const float al = -1.0f / muts * (alt * mu + rdnw * (phu - phk));
    pnew = c2 * (alt * (tk - mu * t1) / (muts * ((float)T0 + t1)) - al);
    s[WF_AL][p] = al;
    pp[p] = pnew;
  }
  s[WF_PM1][p] = pnew;
}

// calc_coef_w: a block owns 32 adjacent mass columns of one row (a warp's
// lanes) and 8 level groups (its warps).  The per-level coefficients a, b, c
// are formed over levels in parallel, every operand of a thread's levels in
// flight at once; one warp then runs the recurrence alpha = 1 / (b - a
// gamma), gamma = c alpha from shared memory in the reference's order, and
// the levels are stored in parallel again.  Five field passes: the earlier
// one-thread-per-column form waited on a memory round trip every few levels
// and, below about 20 000 columns, left most of the chip idle.  Divisions by
// mut^2 and the reciprocals are in their correctly rounded forms.
constexpr int kCwTX = 32, kCwKT = 8;

__global__ void __launch_bounds__(kCwTX* kCwKT) k_coef_w(Grid g, S s, float dts, int i0) {
  extern __shared__ float cw_smem[];
  const int nz = g.nz;
  const int tx = threadIdx.x % kCwTX, tk = threadIdx.x / kCwTX;
  float* const sa = cw_smem + tx;                  // [nz][32]: a
  float* const sb = sa + nz * kCwTX;               // b, then alpha
  float* const sc = sb + nz * kCwTX;               // c, then gamma
  const int i = i0 + blockIdx.x * kCwTX + tx, j = g.jds + blockIdx.y;
  const bool col = i >= g.ids && i < g.ide - 1;
  const int c = col ? g.i2(j, i) : g.i2(j, g.ids);
  const size_t lev = g.n2();
  const double cofd = (0.5 * (double)dts * G * (1.0 + (double)g.epssm)) * (0.5 * (double)dts * G * (1.0 + (double)g.epssm));
  const float cof = (float)cofd, cofm2 = (float)(-2.0 * cofd), cof2 = (float)(2.0 * cofd);
  const float* cqw = s[WF_CQW];
  const float* c2a = s[WF_C2A];
  const float* rdn = s[WF_RDN];
  const float* rdnw = s[WF_RDNW];
  float* a = s[WF_A];
  float* alpha = s[WF_ALPHA];
  float* gamma = s[WF_GAMMA];
  const float mut = __ldg(&s[WF_MUT][c]);
  const float c2t = __ldg(&c2a[(nz - 2) * lev + c]);
  const float mm = mut * mut, r_mm = __frcp_rn(mm);
#pragma unroll 4
  for (int k = 1 + tk; k < nz - 1; k += kCwKT) {
    const size_t p = k * lev + c;
    const float cw = __ldg(&cqw[p]), c2k = __ldg(&c2a[p]), c2m = __ldg(&c2a[p - lev]);
    const float rk = __ldg(&rdn[k]), rwk = __ldg(&rdnw[k]), rwm = __ldg(&rdnw[k - 1]);
    sa[k * kCwTX] = k >= 2 ? divc(-cw * cof * rk * rwm * c2m, mm, r_mm) : 0.f;
    sb[k * kCwTX] = 1.0f + cw * cof * rk * (divc(rwk * c2k, mm, r_mm) + divc(rwm * c2m, mm, r_mm));
    sc[k * kCwTX] = divc(-cw * cof * rk * rwk * c2k, mm, r_mm);
  }
  __syncthreads();
  if (tk == 0) {
    const float lid = g.top_lid ? 0.f : 1.f;
    const float rwt = __ldg(&rdnw[nz - 2]);
    const float atop = divc(cofm2 * (rwt * rwt) * c2t * lid, mm, r_mm);
    float gm = 0.f;
#pragma unroll 8
    for (int k = 1; k < nz - 1; ++k) {
      const float al = __frcp_rn(sb[k * kCwTX] - sa[k * kCwTX] * gm);
      sb[k * kCwTX] = al;
      gm = sc[k * kCwTX] * al;
      sc[k * kCwTX] = gm;
    }
    const float btop = 1.0f + divc(cof2 * (rwt * rwt) * c2t, mm, r_mm);
    sa[(nz - 1) * kCwTX] = atop;
    sb[(nz - 1) * kCwTX] = __frcp_rn(btop - atop * gm);
    sc[(nz - 1) * kCwTX] = 0.f;
    sc[0] = 0.f;
  }
  __syncthreads();
  if (!col) return;
#pragma unroll 4
  for (int k = tk; k < nz; k += kCwKT) {
    const size_t p = k * lev + c;
    if (k > 0) {
      a[p] = sa[k * kCwTX];
      alpha[p] = sb[k * kCwTX];
    }
    gamma[p] = sc[k * kCwTX];
  }
}

// columns of a 32-wide block start on a 32-byte sector when the rows do
static void run_coef_w(const Grid& g, const S& s, float dts, cudaStream_t st) {
  const int i0 = g.nx % 8 == 0 ? g.ids / 8 * 8 : g.ids;
  k_coef_w<<<dim3((g.ide - 1 - i0 + kCwTX - 1) / kCwTX, g.jde - 1 - g.jds), kCwTX * kCwKT,
             3 * g.nz * kCwTX * sizeof(float), st>>>(g, s, dts, i0);
}

// advance_uv for rows that are no multiple of 16 bytes (and the cross-check of
// the tensor-map form below): a thread marches LZ levels of its column,
// its ph, p and vertical averages carried in registers and its map factors,
// with their divisions, formed once.  A thread per point loaded two and a half
// times as much and waited for it in two rounds, the second behind u's store:
// 19.7 -> 12.4 us per launch at 131x131x35, 14.3 -> 10.1 at 101x101x35.
template <int LZ>
__global__ void __launch_bounds__(128) k_advance_uv(Grid g, S s, float dts) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
  const int nz = g.nz, ktf = nz - 1, nx = g.nx;
  const size_t lev = g.n2();
  const int ids = g.ids, ide = g.ide, jds = g.jds, jde = g.jde;
  const int k0 = blockIdx.z * LZ, k1 = min(k0 + LZ, ktf);
  if (i >= nx || j >= g.ny) return;
  // updated points, and the specified rows (spec_bdyupdate)
  const bool uin = j >= jds + 1 && j < jde - 2 && i >= ids + 1 && i < ide - 1;
  const bool vin = j >= jds + 1 && j < jde - 1 && i >= ids + 1 && i < ide - 2;
  const bool us = uin || ((j == jds || j == jde - 2) && i >= ids && i < ide) ||
                  (j >= jds + 1 && j < jde - 2 && (i == ids || i == ide - 1));
  const bool vs = vin || ((j == jds || j == jde - 1) && i >= ids && i < ide - 1) ||
                  (j >= jds + 1 && j < jde - 1 && (i == ids || i == ide - 2));
  if (!us && !vs) return;
  const int c = j * nx + i, w = c - 1, so = c - nx;
  const float *pp = s[WF_P], *pb = s[WF_PB], *ph = s[WF_PH], *php = s[WF_PHP], *alt = s[WF_ALT], *al = s[WF_AL];
  const float *mu = s[WF_MU], *mudf = s[WF_MUDF], *fnm = s[WF_FNM], *fnp = s[WF_FNP];
  float *const U = s[WF_U], *const V = s[WF_V];
  const float rdx = g.rdx, rdy = g.rdy;
  auto dpn0 = [&](int kk, int cb) {
    auto sum = [&](int l) { return __ldg(pp + l * lev + c) + __ldg(pp + l * lev + cb); };
    if (kk == 0) return 0.5f * (g.cf1 * sum(0) + g.cf2 * sum(1) + g.cf3 * sum(2));
    return 0.5f * (__ldg(fnm + kk) * sum(kk) + __ldg(fnp + kk) * sum(kk - 1));
  };
  float cu = 0.f, ru = 0.f, mu_u = 0.f, md_u = 0.f, cv = 0.f, rv = 0.f, mu_v = 0.f, md_v = 0.f;
  float ph_c = 0.f, ph_w = 0.f, ph_s = 0.f, p_c = 0.f, p_w = 0.f, p_s = 0.f, dpn_u = 0.f, dpn_v = 0.f;
  if (uin || vin) {
    ph_c = __ldg(ph + k0 * lev + c);
    p_c = __ldg(pp + k0 * lev + c);
  }
  if (uin) {
    const float mfy = __ldg(&s[WF_MSFUY][c]), r = __ldg(&s[WF_MSFUX][c]) / mfy;
    md_u = (float)(-(double)g.emdiv * g.dxd) * (__ldg(mudf + c) - __ldg(mudf + w)) / mfy;
    cu = r * 0.5f * rdx * __ldg(&s[WF_MUU][c]);
    ru = r * rdx;
    mu_u = 0.5f * (__ldg(mu + w) + __ldg(mu + c));
    ph_w = __ldg(ph + k0 * lev + w);
    p_w = __ldg(pp + k0 * lev + w);
    dpn_u = dpn0(k0, w);
  }
  if (vin) {
    const float r = __ldg(&s[WF_MSFVY][c]) / __ldg(&s[WF_MSFVX][c]);
    md_v = (float)(-(double)g.emdiv * g.dyd) * (__ldg(mudf + c) - __ldg(mudf + so)) * __ldg(&s[WF_MSFVX_INV][c]);
    cv = r * 0.5f * rdy * __ldg(&s[WF_MUV][c]);
    rv = r * rdy;
    mu_v = 0.5f * (__ldg(mu + so) + __ldg(mu + c));
    ph_s = __ldg(ph + k0 * lev + so);
    p_s = __ldg(pp + k0 * lev + so);
    dpn_v = dpn0(k0, so);
  }
  for (int k = k0; k < k1; ++k) {
    const size_t o = k * lev, q = o + c;
    const float rdk = __ldg(&s[WF_RDNW][k]);
    const bool top = k + 1 == ktf;
    const float fm1 = top ? 0.f : __ldg(fnm + k + 1), fp1 = top ? 0.f : __ldg(fnp + k + 1);
    float hu = 0.f, pu = 0.f, altc = 0.f, alc = 0.f, pbc = 0.f, phpc = 0.f;
    if (uin || vin) {
      hu = __ldg(ph + q + lev);
      pu = __ldg(pp + q + lev);
      altc = __ldg(alt + q);
      alc = __ldg(al + q);
      pbc = __ldg(pb + q);
      phpc = __ldg(php + q);
    }
    float un = 0.f, vn = 0.f;
    if (us) un = U[q] + dts * __ldg(&s[WF_RU_TEND][q]);
    if (vs) vn = V[q] + dts * __ldg(&s[WF_RV_TEND][q]);
    if (uin) {
      const size_t n = o + w;
      const float hn = __ldg(ph + n + lev), pn = __ldg(pp + n + lev);
      const float up = top ? 0.f : 0.5f * (fm1 * (pu + pn) + fp1 * (p_c + p_w));
      float dp = cu * (((hu - hn) + (ph_c - ph_w)) + (altc + __ldg(alt + n)) * (p_c - p_w) +
                       (alc + __ldg(al + n)) * (pbc - __ldg(pb + n)));
      dp = dp + ru * (phpc - __ldg(php + n)) * (rdk * (up - dpn_u) - mu_u);
      un = un - dts * __ldg(&s[WF_CQU][q]) * dp + md_u;
      ph_w = hn;
      p_w = pn;
      dpn_u = up;
    }
    if (vin) {
      const size_t n = o + so;
      const float hn = __ldg(ph + n + lev), pn = __ldg(pp + n + lev);
      const float up = top ? 0.f : 0.5f * (fm1 * (pu + pn) + fp1 * (p_c + p_s));
      float dp = cv * (((hu - hn) + (ph_c - ph_s)) + (altc + __ldg(alt + n)) * (p_c - p_s) +
                       (alc + __ldg(al + n)) * (pbc - __ldg(pb + n)));
      dp = dp + rv * (phpc - __ldg(php + n)) * (rdk * (up - dpn_v) - mu_v);
      vn = vn - dts * __ldg(&s[WF_CQV][q]) * dp + md_v;
      ph_s = hn;
      p_s = pn;
      dpn_v = up;
    }
    if (us) U[q] = un;
    if (vs) V[q] = vn;
    ph_c = hu;
    p_c = pu;
  }
}

// advance_uv, tensor-map form (nx a multiple of 4): a block of 32 x 8
// threads owns 32 x 8 columns (u and v points (j, i)) and a chunk of levels.
// Per level one thread loads boxes of alt, al, pb, php at k and ph, p at k+1
// (40 x 9 from x = floor4(i0 - 1), y = j0 - 1: every point's i-1 and j-1
// neighbours) into an mbarrier ring two levels ahead; ph(k), p(k) and the
// vertical pressure averages dpn(k) come from the level below in registers
// (each is the same operation on the same operands as in k_advance_uv), and
// the thread's own u, v, tendencies and cq are loaded a level ahead.  Every
// wait on a box is bounded; a block whose wait runs out fills the levels it
// leaves with NaN, drains its copies and adds 1 to STATUS[WRF_ST_WAIT].
constexpr int kUvTX = 32, kUvTY = 8, kUvBW = 40, kUvBH = kUvTY + 1;
constexpr int kUvNB = 6;                 // boxes per level: alt al pb php (k), ph p (k+1)
constexpr int kUvSlot = 384;             // floats per box slot (1536 B >= 40 x 9 x 4)
constexpr int kUvOW = 36, kUvOH = kUvTY;  // the thread's own u, ru_tend, v, rv_tend, cqu, cqv at k
constexpr int kUvNO = 6, kUvOSlot = kUvOW * kUvOH;  // 1152 B, a 128-byte multiple
constexpr int kUvRing = 3, kUvKCH = 7;
constexpr uint32_t kUvBytes = kUvNB * kUvBW * kUvBH * 4 + kUvNO * kUvOW * kUvOH * 4;
constexpr long long kUvWaitCycles = 4000000000LL;
static_assert(kUvBW * kUvBH <= kUvSlot && (kUvOSlot * 4) % 128 == 0, "ring slots hold one box, 128-byte aligned");

struct UvTmaArgs {
  CUtensorMap alt, al, pb, php, ph, pp;
  CUtensorMap own[kUvNO];  // u, ru_tend, v, rv_tend, cqu, cqv
  int nchunk, expired;     // expired: every wait counts as run out
};

__global__ void __launch_bounds__(kUvTX * kUvTY, 4) k_advance_uv_tma(Grid g, S s, float dts,
                                                                     const __grid_constant__ UvTmaArgs a) {
  __shared__ __align__(128) float box[kUvRing][kUvNB][kUvSlot];
  __shared__ __align__(128) float obox[kUvRing][kUvNO][kUvOSlot];
  __shared__ uint64_t bar[kUvRing];
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * kUvTX + tx;
  const int nx = g.nx, ny = g.ny, nz = g.nz, ktf = nz - 1;
  const int ids = g.ids, ide = g.ide, jds = g.jds, jde = g.jde;
  const int i0 = ids + blockIdx.x * kUvTX, j0 = jds + blockIdx.y * kUvTY;
  const int i = i0 + tx, j = j0 + ty;
  const int mx = (i0 - 1) & ~3, om = i0 - mx;
  const int ox = i0 & ~3, oo = i0 - ox;
  const int k0 = blockIdx.z * ktf / a.nchunk, k1 = (blockIdx.z + 1) * ktf / a.nchunk;
  const size_t lev = (size_t)ny * nx;
  const bool uin = j >= jds + 1 && j < jde - 2 && i >= ids + 1 && i < ide - 1;
  const bool uspec = ((j == jds || j == jde - 2) && i >= ids && i < ide) ||
                     (j >= jds + 1 && j < jde - 2 && (i == ids || i == ide - 1));
  const bool vin = j >= jds + 1 && j < jde - 1 && i >= ids + 1 && i < ide - 2;
  const bool vspec = ((j == jds || j == jde - 1) && i >= ids && i < ide - 1) ||
                     (j >= jds + 1 && j < jde - 1 && (i == ids || i == ide - 2));
  const bool wu = uin || uspec, wv = vin || vspec;
  const int c = min(j, ny - 1) * nx + min(i, nx - 1);
  const float* pp = s[WF_P];
  const float* ph = s[WF_PH];
  const float* fnm = s[WF_FNM];
  const float* fnp = s[WF_FNP];
  const float* rdnw = s[WF_RDNW];
  float* U = s[WF_U];
  float* V = s[WF_V];
  const float rdx = g.rdx, rdy = g.rdy;

  if (tid == 0) {
    for (int r = 0; r < kUvRing; ++r) tma::mbar_init(&bar[r], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  auto issue = [&](int k, int r) {
    tma::mbar_expect_tx(&bar[r], kUvBytes);
    tma::load_4d(box[r][0], &a.alt, mx, j0 - 1, k, 0, &bar[r]);
    tma::load_4d(box[r][1], &a.al, mx, j0 - 1, k, 0, &bar[r]);
    tma::load_4d(box[r][2], &a.pb, mx, j0 - 1, k, 0, &bar[r]);
    tma::load_4d(box[r][3], &a.php, mx, j0 - 1, k, 0, &bar[r]);
    tma::load_4d(box[r][4], &a.ph, mx, j0 - 1, k + 1, 0, &bar[r]);
    tma::load_4d(box[r][5], &a.pp, mx, j0 - 1, k + 1, 0, &bar[r]);
    for (int f = 0; f < kUvNO; ++f) tma::load_4d(obox[r][f], &a.own[f], ox, j0, k, 0, &bar[r]);
  };
  int hi = k0 - 1;
  if (tid == 0) {
    for (int k = k0; k < min(k0 + kUvRing - 1, k1); ++k) issue(k, k - k0);
    hi = min(k0 + kUvRing - 1, k1) - 1;
  }
  // per-column constants, in the association order of k_advance_uv
  float mudf_u = 0.f, cu = 0.f, ru = 0.f, muav_u = 0.f, mudf_v = 0.f, cv = 0.f, rv = 0.f, muav_v = 0.f;
  if (uin) {
    const float* mudf = s[WF_MUDF];
    const float* mu = s[WF_MU];
    mudf_u = (float)(-(double)g.emdiv * g.dxd) * (__ldg(&mudf[c]) - __ldg(&mudf[c - 1])) / __ldg(&s[WF_MSFUY][c]);
    const float r = __ldg(&s[WF_MSFUX][c]) / __ldg(&s[WF_MSFUY][c]);
    cu = r * 0.5f * rdx * __ldg(&s[WF_MUU][c]);
    ru = r * rdx;
    muav_u = 0.5f * (__ldg(&mu[c - 1]) + __ldg(&mu[c]));
  }
  if (vin) {
    const float* mudf = s[WF_MUDF];
    const float* mu = s[WF_MU];
    mudf_v = (float)(-(double)g.emdiv * g.dyd) * (__ldg(&mudf[c]) - __ldg(&mudf[c - nx])) * __ldg(&s[WF_MSFVX_INV][c]);
    const float r = __ldg(&s[WF_MSFVY][c]) / __ldg(&s[WF_MSFVX][c]);
    cv = r * 0.5f * rdy * __ldg(&s[WF_MUV][c]);
    rv = r * rdy;
    muav_v = 0.5f * (__ldg(&mu[c - nx]) + __ldg(&mu[c]));
  }
  // ph(k), p(k) at (j, i), (j, i-1), (j-1, i) and dpn(k) of the u and v points
  const int cw = (uin || vin) ? c - 1 : c, cs = (uin || vin) ? c - nx : c;
  float ph_c = 0.f, ph_w = 0.f, ph_s = 0.f, p_c = 0.f, p_w = 0.f, p_s = 0.f, dpn_u = 0.f, dpn_v = 0.f;
  if (uin || vin) {
    const size_t q = (size_t)k0 * lev;
    ph_c = __ldg(&ph[q + c]);
    ph_w = __ldg(&ph[q + cw]);
    ph_s = __ldg(&ph[q + cs]);
    p_c = __ldg(&pp[q + c]);
    p_w = __ldg(&pp[q + cw]);
    p_s = __ldg(&pp[q + cs]);
    if (k0 == 0) {  // dpn(0): cf1..cf3 over the three lowest levels
      const float a1 = __ldg(&pp[lev + c]), a2 = __ldg(&pp[2 * lev + c]);
      const float w1 = __ldg(&pp[lev + cw]), w2 = __ldg(&pp[2 * lev + cw]);
      const float s1 = __ldg(&pp[lev + cs]), s2 = __ldg(&pp[2 * lev + cs]);
      dpn_u = 0.5f * (g.cf1 * (p_c + p_w) + g.cf2 * (a1 + w1) + g.cf3 * (a2 + w2));
      dpn_v = 0.5f * (g.cf1 * (p_c + p_s) + g.cf2 * (a1 + s1) + g.cf3 * (a2 + s2));
    } else if (k0 < nz - 1) {
      const float fm = __ldg(&fnm[k0]), fp = __ldg(&fnp[k0]);
      const size_t qm = q - lev;
      dpn_u = 0.5f * (fm * (p_c + p_w) + fp * (__ldg(&pp[qm + c]) + __ldg(&pp[qm + cw])));
      dpn_v = 0.5f * (fm * (p_c + p_s) + fp * (__ldg(&pp[qm + c]) + __ldg(&pp[qm + cs])));
    }
  }
  const int oA = (ty + 1) * kUvBW + om + tx;
  const int oO = ty * kUvOW + oo + tx;  // (j, i) in an own-value box
  int kstop = a.expired ? k0 : k1, slot = 0;
  uint32_t par = 0;
  for (int k = a.expired ? k1 : k0; k < k1; ++k) {
    const float rdk = __ldg(&rdnw[k]);
    const float fm1 = k + 1 < nz - 1 ? __ldg(&fnm[k + 1]) : 0.f, fp1 = k + 1 < nz - 1 ? __ldg(&fnp[k + 1]) : 0.f;
    const bool ok = tma::mbar_wait_bounded(&bar[slot], par, kUvWaitCycles);
    if (__syncthreads_or(!ok)) {
      kstop = k;
      break;
    }
    // every thread is past level k-1: its slot takes level k + kUvRing - 1
    if (tid == 0 && k + kUvRing - 1 < k1) {
      issue(k + kUvRing - 1, slot == 0 ? kUvRing - 1 : slot - 1);
      hi = k + kUvRing - 1;
    }
    const float* B = box[slot][0];
    const size_t p = (size_t)k * lev + c;
    const float u0 = obox[slot][0][oO], rt0 = obox[slot][1][oO], v0 = obox[slot][2][oO];
    const float vt0 = obox[slot][3][oO], qu0 = obox[slot][4][oO], qv0 = obox[slot][5][oO];
    float pu_c = 0.f, pu_w = 0.f, pu_s = 0.f, hu_c = 0.f, hu_w = 0.f, hu_s = 0.f;
    if (uin || vin) {
      hu_c = B[4 * kUvSlot + oA];
      pu_c = B[5 * kUvSlot + oA];
      hu_w = B[4 * kUvSlot + oA - 1];
      pu_w = B[5 * kUvSlot + oA - 1];
      hu_s = B[4 * kUvSlot + oA - kUvBW];
      pu_s = B[5 * kUvSlot + oA - kUvBW];
    }
    float unew = 0.f, vnew = 0.f;
    if (uin) {
      const float u = u0 + dts * rt0;
      const float alt_c = B[oA], alt_w = B[oA - 1];
      const float al_c = B[kUvSlot + oA], al_w = B[kUvSlot + oA - 1];
      const float pb_c = B[2 * kUvSlot + oA], pb_w = B[2 * kUvSlot + oA - 1];
      const float php_c = B[3 * kUvSlot + oA], php_w = B[3 * kUvSlot + oA - 1];
      const float dpn_up = k + 1 == nz - 1 ? 0.f : 0.5f * (fm1 * (pu_c + pu_w) + fp1 * (p_c + p_w));
      float dp = cu * (((hu_c - hu_w) + (ph_c - ph_w)) + (alt_c + alt_w) * (p_c - p_w) + (al_c + al_w) * (pb_c - pb_w));
      dp = dp + ru * (php_c - php_w) * (rdk * (dpn_up - dpn_u) - muav_u);
      unew = u - dts * qu0 * dp + mudf_u;
      dpn_u = dpn_up;
    } else if (uspec) {
      unew = u0 + dts * rt0;  // spec_bdyupdate(u)
    }
    if (vin) {
      const float v = v0 + dts * vt0;
      const float alt_c = B[oA], alt_s = B[oA - kUvBW];
      const float al_c = B[kUvSlot + oA], al_s = B[kUvSlot + oA - kUvBW];
      const float pb_c = B[2 * kUvSlot + oA], pb_s = B[2 * kUvSlot + oA - kUvBW];
      const float php_c = B[3 * kUvSlot + oA], php_s = B[3 * kUvSlot + oA - kUvBW];
      const float dpn_up = k + 1 == nz - 1 ? 0.f : 0.5f * (fm1 * (pu_c + pu_s) + fp1 * (p_c + p_s));
      float dp = cv * (((hu_c - hu_s) + (ph_c - ph_s)) + (alt_c + alt_s) * (p_c - p_s) + (al_c + al_s) * (pb_c - pb_s));
      dp = dp + rv * (php_c - php_s) * (rdk * (dpn_up - dpn_v) - muav_v);
      vnew = v - dts * qv0 * dp + mudf_v;
      dpn_v = dpn_up;
    } else if (vspec) {
      vnew = v0 + dts * vt0;  // spec_bdyupdate(v)
    }
    if (wu) U[p] = unew;
    if (wv) V[p] = vnew;
    ph_c = hu_c;
    ph_w = hu_w;
    ph_s = hu_s;
    p_c = pu_c;
    p_w = pu_w;
    p_s = pu_s;
    if (++slot == kUvRing) {
      slot = 0;
      par ^= 1u;
    }
  }
  if (kstop == k1) return;
#pragma unroll 1
  for (int k = kstop; k < k1; ++k) {
    const size_t p = (size_t)k * lev + c;
    if (wu) U[p] = tma::unfinished();
    if (wv) V[p] = tma::unfinished();
  }
  if (tid == 0) {
    for (int k = kstop; k <= hi; ++k)
      tma::mbar_wait_bounded(&bar[(k - k0) % kUvRing], ((k - k0) / kUvRing) & 1, kUvWaitCycles);
    if (s[WF_STATUS]) atomicAdd(reinterpret_cast<int*>(s[WF_STATUS]) + WRF_ST_WAIT, 1);
  }
}

// Fused acoustic column update of one substep: advance_mu_t, advance_w,
// sumflux, spec_bdyupdate of t / mu / muts / ph, calc_p_rho
// (wrf_dynamics.py:3528-3839, 3269-3313; wrf_boundary.py:244-355).  A block
// owns kColTX adjacent columns of one row; thread (tx, tk) handles the levels
// k = tk, tk + kColKT, ... of column tx.  The explicit parts run over levels
// in parallel; the vertical recurrences (column mass divergence sum, ww scan,
// Thomas sweeps) run sequentially per column in the reference's order, from
// separate shared arrays so that their loads pipeline.  Small blocks and few
// registers let several blocks share an SM, which overlaps one block's
// sweeps with the memory phases of the others.  No column reads another
// column's result of this kernel; zero_grad_bdy(w) follows in the substep's
// halo launch (k_bc).
// Divisions by per-column constants use the correctly rounded form divc with
// the column's reciprocals (__frcp_rn).
constexpr int kColTX = 16, kColKT = 16;

// NQ = ceil(nz / kColKT) level slots per thread.  Phases that store to global
// memory first load every slot's operands into registers and only then
// compute and store: the loads of a thread's levels are then all in flight at
// once (the compiler cannot hoist a later level's loads above an earlier
// level's stores through possibly aliasing field pointers).
#ifndef WRF_COL_MINB
#define WRF_COL_MINB 4
#endif
template <int NQ>
__global__ void __launch_bounds__(kColTX * kColKT, WRF_COL_MINB) k_acoustic_col(Grid g, S s, float dts, int iteration, int nsub,
                                                                             int i0) {
  constexpr int NZ = NQ * kColKT;  // nz <= NZ
  __shared__ float sdw[NZ][kColTX], sww[NZ][kColTX], st2av[NZ][kColTX], srhs[NZ][kColTX];
  __shared__ float sa[NZ][kColTX], salpha[NZ][kColTX], sgamma[NZ][kColTX], sph[NZ][kColTX];
  __shared__ float swd[NZ][kColTX];
  __shared__ float pdnw[kMaxNz], prdnw[kMaxNz], prdn[kMaxNz], pfnm[kMaxNz], pfnp[kMaxNz];
  __shared__ float smuave[kColTX], smuts[kColTX], smu[kColTX];
  const int nz = g.nz, kend = nz - 1, nx = g.nx;
  const int ids = g.ids, ide = g.ide, jds = g.jds, jde = g.jde;
  const int tx = threadIdx.x % kColTX, tk = threadIdx.x / kColTX;
  const int i = i0 + blockIdx.x * kColTX + tx;      // i0 <= ids: whole sectors where the rows allow it
  const int j = jds + blockIdx.y;
  const bool col = i >= ids && i < ide;             // j < jde by the grid
  const bool inner = col && j >= jds + 1 && j < jde - 2 && i >= ids + 1 && i < ide - 2;
  const bool spec = col && (((j == jds || j == jde - 2) && i < ide - 1) || (j >= jds + 1 && j < jde - 2 && (i == ids || i == ide - 2)));
  const bool mass = inner || spec;
  const int c = col ? g.i2(j, i) : 0;
  const int lev = g.ny * nx;
  for (int e = threadIdx.x; e < nz; e += kColTX * kColKT) {
    pdnw[e] = __ldg(&s[WF_DNW][e]);
    prdnw[e] = __ldg(&s[WF_RDNW][e]);
    prdn[e] = __ldg(&s[WF_RDN][e]);
    pfnm[e] = __ldg(&s[WF_FNM][e]);
    pfnp[e] = __ldg(&s[WF_FNP][e]);
  }
  float* t = s[WF_T];
  const float* ft = s[WF_T_TEND];
  const float* t1 = s[WF_T_SAVE];
  float* ww = s[WF_WW];
  const float* ww1 = s[WF_WW1];
  const float* u = s[WF_U];
  const float* v = s[WF_V];
  const float msftx = col ? __ldg(&s[WF_MSFTX][c]) : 1.f, msfty = col ? __ldg(&s[WF_MSFTY][c]) : 1.f;
  const float mut = col ? __ldg(&s[WF_MUT][c]) : 1.f;
  const float mu_tend = col ? __ldg(&s[WF_MU_TEND][c]) : 0.f;
  const float r_msfty = __frcp_rn(msfty), r_mut = __frcp_rn(mut);
  const float ep = g.epssm;
  const float ep1 = (float)(1.0 + (double)ep), em1 = (float)(1.0 - (double)ep);
#ifndef WRF_COL_NOPREFETCH
  // Ask L2 for what the later phases of this thread's levels will load: the
  // requests need no registers, and the phases after the column sweeps then
  // find their operands in L2 instead of waiting on DRAM one phase at a time.
  if (col) {
    auto pf = [](const float* a) { asm volatile("prefetch.global.L2 [%0];" ::"l"(a)); };
    const float* fields[] = {ww1, ww, t1, t, ft, s[WF_PH], s[WF_A], s[WF_ALPHA], s[WF_GAMMA], s[WF_PH_SAVE],
                             s[WF_PHB], s[WF_PH_TEND], s[WF_W], s[WF_RW_TEND], s[WF_C2A], s[WF_ALT], s[WF_CQW],
                             s[WF_W_SAVE], s[WF_PM1], s[WF_RU_M], s[WF_RV_M], s[WF_WW_M]};
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int k = tk + q * kColKT;
      if (k >= nz) continue;
      const int p = k * lev + c;
#pragma unroll
      for (const float* f : fields) pf(f + p);
      if (inner) {
        pf(t1 + p + nx);
        pf(t1 + p - nx);
        pf(v + p + nx);
      }
    }
  }
#endif

  // --- A: horizontal mass-flux divergence per level (inner) / spec t, mu, muts
  if (inner) {
    const float* u1 = s[WF_U_SAVE];
    const float* v1 = s[WF_V_SAVE];
    const float muvn = __ldg(&s[WF_MUV][c + nx]), mvin = __ldg(&s[WF_MSFVX_INV][c + nx]);
    const float muv0 = __ldg(&s[WF_MUV][c]), mvi0 = __ldg(&s[WF_MSFVX_INV][c]);
    const float muup = __ldg(&s[WF_MUU][c + 1]), mfup = __ldg(&s[WF_MSFUY][c + 1]);
    const float muu0 = __ldg(&s[WF_MUU][c]), mfu0 = __ldg(&s[WF_MSFUY][c]);
    const float r_mfup = __frcp_rn(mfup), r_mfu0 = __frcp_rn(mfu0);
    const float rdx = g.rdx, rdy = g.rdy;
    float vn[NQ], v1n[NQ], v0[NQ], v10[NQ], ue[NQ], u1e[NQ], u0[NQ], u10[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int k = tk + q * kColKT;
      if (k >= kend) continue;
      const int p = k * lev + c;
      vn[q] = __ldg(&v[p + nx]);
      v1n[q] = __ldg(&v1[p + nx]);
      v0[q] = __ldg(&v[p]);
      v10[q] = __ldg(&v1[p]);
      ue[q] = __ldg(&u[p + 1]);
      u1e[q] = __ldg(&u1[p + 1]);
      u0[q] = __ldg(&u[p]);
      u10[q] = __ldg(&u1[p]);
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int k = tk + q * kColKT;
      if (k >= kend) continue;
      sdw[k][tx] = msftx * msfty *
                   (rdy * ((vn[q] + muvn * v1n[q] * mvin) - (v0[q] + muv0 * v10[q] * mvi0)) +
                    rdx * ((ue[q] + divc(muup * u1e[q], mfup, r_mfup)) - (u0[q] + divc(muu0 * u10[q], mfu0, r_mfu0))));
    }
  } else if (spec) {
    for (int k = tk; k < kend; k += kColKT) {
      const int p = k * lev + c;
      t[p] = t[p] + dts * __ldg(&ft[p]);
    }
    if (tk == 0) {
      const float mu = s[WF_MU][c] + dts * mu_tend;
      const float muts = s[WF_MUTS][c] + dts * mu_tend;
      s[WF_MU][c] = mu;
      s[WF_MUTS][c] = muts;
      smu[tx] = mu;
      smuts[tx] = muts;
    }
  }
  __syncthreads();
  // --- B: column mass tendency (sequential sum, reference order)
  if (inner && tk == 0) {
    float dmdt = 0.f;
#pragma unroll 8
    for (int k = 0; k < kend; ++k) dmdt = dmdt + pdnw[k] * sdw[k][tx];
    float mu = s[WF_MU][c];
    const float muave_old = mu;
    mu = mu + dts * (dmdt + mu_tend);
    const float muts = mut + mu;
    const float muave = 0.5f * (ep1 * mu + em1 * muave_old);
    s[WF_MU][c] = mu;
    s[WF_MUDF][c] = dmdt + mu_tend;
    s[WF_MUTS][c] = muts;
    s[WF_MUAVE][c] = muave;
    smu[tx] = mu;
    smuts[tx] = muts;
    smuave[tx] = muave;
    swd[0][tx] = dmdt;  // broadcast dmdt to the level threads
  }
  __syncthreads();
  // --- B2: increments of the ww scan in parallel, then the scan itself
  if (inner) {
    const float dmdt = swd[0][tx];
    for (int k = tk + 1; k < kend; k += kColKT)
      sww[k][tx] = divc(pdnw[k - 1] * (dmdt + sdw[k - 1][tx] + mu_tend), msfty, r_msfty);
  }
  __syncthreads();
  if (inner && tk == 0) {
    float wprev = ww[c];
    sww[0][tx] = wprev;
#pragma unroll 8
    for (int k = 1; k < kend; ++k) {
      wprev = wprev - sww[k][tx];
      sww[k][tx] = wprev;
    }
  }
  __syncthreads();
  // --- C: final ww (inner: scan - ww1)
  if (col) {
    float wv[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int k = tk + q * kColKT;
      if (k < nz) wv[q] = (inner && k < kend) ? __ldg(&ww1[k * lev + c]) : ww[k * lev + c];
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int k = tk + q * kColKT;
      if (k >= nz) continue;
      float w = wv[q];
      if (inner && k < kend) {
        w = sww[k][tx] - w;
        ww[k * lev + c] = w;
      }
      sww[k][tx] = w;
    }
  }
  __syncthreads();
  const float muave = inner ? smuave[tx] : 0.f;
  const float muts = mass ? smuts[tx] : 1.f;
  const float r_muts = __frcp_rn(muts);
  // --- C2: potential temperature and t_2ave; D1: wdwn, phi, coefficients
  if (inner) {
    const float cy = (float)(0.5 * g.rdyd), cx = (float)(0.5 * g.rdxd);
    float* t2a = s[WF_T_2SAVE];
    float t10[NQ], tup[NQ], tdn[NQ], told[NQ], ftk[NQ], vn[NQ], tn[NQ], v0[NQ], ts[NQ], ue[NQ], te[NQ], u0[NQ],
        tw[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int k = tk + q * kColKT;
      if (k >= kend) continue;
      const int p = k * lev + c;
      t10[q] = __ldg(&t1[p]);
      tup[q] = (k + 1 == nz - 1) ? 0.f : __ldg(&t1[p + lev]);
      tdn[q] = (k == 0) ? 0.f : __ldg(&t1[p - lev]);
      told[q] = t[p];
      ftk[q] = __ldg(&ft[p]);
      vn[q] = __ldg(&v[p + nx]);
      tn[q] = __ldg(&t1[p + nx]);
      v0[q] = __ldg(&v[p]);
      ts[q] = __ldg(&t1[p - nx]);
      ue[q] = __ldg(&u[p + 1]);
      te[q] = __ldg(&t1[p + 1]);
      u0[q] = __ldg(&u[p]);
      tw[q] = __ldg(&t1[p - 1]);
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int k = tk + q * kColKT;
      if (k >= kend) continue;
      const int p = k * lev + c;
      // wdtn(kk) = ww(kk) (fnm t1(kk) + fnp t1(kk-1)), zero at the bottom and top
      const float wup = (k + 1 == nz - 1) ? 0.f : sww[k + 1][tx] * (pfnm[k + 1] * tup[q] + pfnp[k + 1] * t10[q]);
      const float wdn = (k == 0) ? 0.f : sww[k][tx] * (pfnm[k] * t10[q] + pfnp[k] * tdn[q]);
      float tt = told[q] + msfty * dts * ftk[q];
      const float hy = cy * (vn[q] * (tn[q] + t10[q]) - v0[q] * (t10[q] + ts[q]));
      const float hx = cx * (ue[q] * (te[q] + t10[q]) - u0[q] * (t10[q] + tw[q]));
      tt = tt - dts * msfty * (msftx * (hy + hx) + prdnw[k] * (wup - wdn));
      t[p] = tt;
      float av = 0.5f * (ep1 * tt + em1 * told[q]);
      av = (av + muave * (float)T0) / (muts * ((float)T0 + t10[q]));
      t2a[p] = av;
      st2av[k][tx] = av;
    }
    const float* ph1 = s[WF_PH_SAVE];
    const float* phb = s[WF_PHB];
    float phv[NQ], av[NQ], alv[NQ], gav[NQ], p1[NQ], p1m[NQ], pb[NQ], pbm[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int k = tk + q * kColKT;
      if (k >= nz) continue;
      const int p = k * lev + c;
      phv[q] = s[WF_PH][p];
      av[q] = __ldg(&s[WF_A][p]);
      alv[q] = __ldg(&s[WF_ALPHA][p]);
      gav[q] = __ldg(&s[WF_GAMMA][p]);
      if (k >= 1 && k <= kend) {
        p1[q] = __ldg(&ph1[p]);
        p1m[q] = __ldg(&ph1[p - lev]);
        pb[q] = __ldg(&phb[p]);
        pbm[q] = __ldg(&phb[p - lev]);
      }
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int k = tk + q * kColKT;
      if (k >= nz) continue;
      sph[k][tx] = phv[q];
      sa[k][tx] = av[q];
      salpha[k][tx] = alv[q];
      sgamma[k][tx] = gav[q];
      // wdwn(k) = 0.5 (ww(k) + ww(k-1)) rdnw(k-1) (ph1(k) - ph1(k-1) + phb(k) - phb(k-1))
      if (k >= 1 && k <= kend)
        swd[k][tx] = 0.5f * (sww[k][tx] + sww[k - 1][tx]) * prdnw[k - 1] * (p1[q] - p1m[q] + pb[q] - pbm[q]);
    }
  }
  __syncthreads();
  // --- D2: right-hand side of the phi equation (inner)
  if (inner) {
    const float cw = (float)(0.5 * G * (1.0 - (double)ep));
    float ptv[NQ], wv[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int k = tk + q * kColKT;
      if (k < 1 || k >= nz) continue;
      ptv[q] = __ldg(&s[WF_PH_TEND][k * lev + c]);
      wv[q] = s[WF_W][k * lev + c];
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int k = tk + q * kColKT;
      if (k >= nz) continue;
      if (k == 0) {
        srhs[0][tx] = 0.f;
        continue;
      }
      float r = dts * (ptv[q] + cw * wv[q]);
      if (k < kend) r = r - dts * (pfnm[k] * swd[k + 1][tx] + pfnp[k] * swd[k][tx]);
      srhs[k][tx] = sph[k][tx] + divc(msfty * r, mut, r_mut);
    }
  }
  __syncthreads();
  // --- E: explicit part of w (inner)
  if (inner) {
    const float* c2a = s[WF_C2A];
    const float* alt = s[WF_ALT];
    const float msft_inv = 1.0f / msfty;
    const float cp = (float)(0.5 * (double)dts * G);
    const float cq = (float)((double)dts * G);
    if (tk == 0) {  // lower boundary: w from the terrain slope and near-surface winds
      const float* ht = s[WF_HT];
      auto cv = [&](int cc) { return g.cf1 * __ldg(&v[cc]) + g.cf2 * __ldg(&v[lev + cc]) + g.cf3 * __ldg(&v[2 * lev + cc]); };
      auto cu = [&](int cc) { return g.cf1 * __ldg(&u[cc]) + g.cf2 * __ldg(&u[lev + cc]) + g.cf3 * __ldg(&u[2 * lev + cc]); };
      const float h0 = __ldg(&ht[c]);
      sdw[0][tx] = msfty * 0.5f * g.rdy * ((__ldg(&ht[c + nx]) - h0) * cv(c + nx) + (h0 - __ldg(&ht[c - nx])) * cv(c)) +
                   msftx * 0.5f * g.rdx * ((__ldg(&ht[c + 1]) - h0) * cu(c + 1) + (h0 - __ldg(&ht[c - 1])) * cu(c));
    }
    float wkv[NQ], rwv[NQ], c2mv[NQ], almv[NQ], c2kv[NQ], alkv[NQ], cqv[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int k = tk + q * kColKT;
      if (k < 1 || k > kend) continue;
      const int p = k * lev + c;
      wkv[q] = s[WF_W][p];
      rwv[q] = __ldg(&s[WF_RW_TEND][p]);
      c2mv[q] = __ldg(&c2a[p - lev]);
      almv[q] = __ldg(&alt[p - lev]);
      if (k < kend) {
        c2kv[q] = __ldg(&c2a[p]);
        alkv[q] = __ldg(&alt[p]);
        cqv[q] = __ldg(&s[WF_CQW][p]);
      }
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int k = tk + q * kColKT;
      if (k < 1 || k > kend) continue;
      const float wk = wkv[q], rwk = rwv[q];
      const float c2m = c2mv[q], alm = almv[q];
      const float rdnw_m = prdnw[k - 1];
      float wl;
      if (k < kend) {
        const float c2k = c2kv[q], alk = alkv[q];
        const float X1 = divc(c2k * prdnw[k], mut, r_mut) * (ep1 * (srhs[k + 1][tx] - srhs[k][tx]) + em1 * (sph[k + 1][tx] - sph[k][tx]));
        const float X2 = divc(c2m * rdnw_m, mut, r_mut) * (ep1 * (srhs[k][tx] - srhs[k - 1][tx]) + em1 * (sph[k][tx] - sph[k - 1][tx]));
        wl = wk + dts * rwk + msft_inv * cqv[q] * (cp * prdn[k] * (X1 - X2)) +
             cq * msft_inv * (prdn[k] * (c2k * alk * st2av[k][tx] - c2m * alm * st2av[k - 1][tx]) - muave);
      } else {
        const float cm = (float)(-0.5 * (double)dts * G);
        wl = wk + dts * rwk +
             msft_inv * (divc(cm, mut, r_mut) * (rdnw_m * rdnw_m) * 2.0f * c2m *
                             (ep1 * (srhs[kend][tx] - srhs[kend - 1][tx]) + em1 * (sph[kend][tx] - sph[kend - 1][tx])) -
                         cq * (2.0f * rdnw_m * c2m * alm * st2av[kend - 1][tx] + muave));
      }
      sdw[k][tx] = wl;
    }
  }
  __syncthreads();
  // --- F: Thomas sweeps (sequential per column)
  if (inner && tk == 0) {
    float prev = sdw[0][tx];
#pragma unroll 8
    for (int k = 1; k <= kend; ++k) {
      prev = (sdw[k][tx] - sa[k][tx] * prev) * salpha[k][tx];
      sdw[k][tx] = prev;
    }
#pragma unroll 8
    for (int k = kend - 1; k >= 1; --k) {
      prev = sdw[k][tx] - sgamma[k][tx] * prev;
      sdw[k][tx] = prev;
    }
  }
  __syncthreads();
  // --- G: Rayleigh damping, w and phi (inner); spec phi; sumflux (all)
  float* ph = s[WF_PH];
  if (inner) {
    float* w = s[WF_W];
    const float* ph1 = s[WF_PH_SAVE];
    const float* phb = s[WF_PHB];
    const float gf = (float)G;
    constexpr float r_g = 1.0f / (float)G, r_hd = 1.0f / 5000.0f;
    const float hdepth = 5000.0f;
    const float dampmag = (float)((double)dts * 0.2);
    const float htop = divc(__ldg(&ph1[kend * lev + c]) + __ldg(&phb[kend * lev + c]), gf, r_g);
    const float hbot = htop - hdepth;
    const float hpi = (float)(0.5 * 3.14159265359);
    float p1v[NQ], pbv[NQ], wsv[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int k = tk + q * kColKT;
      if (k < 1 || k >= nz) continue;
      const int p = k * lev + c;
      p1v[q] = __ldg(&ph1[p]);
      pbv[q] = __ldg(&phb[p]);
      wsv[q] = __ldg(&s[WF_W_SAVE][p]);
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int k = tk + q * kColKT;
      if (k >= nz) continue;
      const int p = k * lev + c;
      if (k == 0) {
        w[c] = sdw[0][tx];
        continue;
      }
      const float hk = divc(p1v[q] + pbv[q], gf, r_g);
      float dwd = 0.f;
      if (hk >= hbot) {
        const float sn = sinf(divc(hpi * (hk - hbot), hdepth, r_hd));
        dwd = dampmag * (sn * sn);
      }
      const float num = sdw[k][tx] - dwd * mut * wsv[q];
      const float wk = dwd == 0.f ? num : num / (1.0f + dwd);  // x / 1 == x
      w[p] = wk;
      const float phk = srhs[k][tx] + divc(msfty * 0.5f * dts * gf * ep1 * wk, muts, r_muts);
      ph[p] = phk;
      sph[k][tx] = phk;
    }
  } else if (spec) {
    const float mu_old = muts - dts * mu_tend;
    const float* ph_save = s[WF_PH_SAVE];
    const float* ph_tend = s[WF_PH_TEND];
    float phv[NQ], ptv[NQ], psv[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int k = tk + q * kColKT;
      if (k >= nz) continue;
      const int p = k * lev + c;
      phv[q] = ph[p];
      ptv[q] = __ldg(&ph_tend[p]);
      psv[q] = __ldg(&ph_save[p]);
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int k = tk + q * kColKT;
      if (k >= nz) continue;
      const int p = k * lev + c;
      const float phk = divc(phv[q] * mu_old, muts, r_muts) + divc(dts * ptv[q], muts, r_muts) +
                        psv[q] * (divc(mu_old, muts, r_muts) - 1.0f);
      ph[p] = phk;
      sph[k][tx] = phk;
    }
  }
  if (col) {
    float* ru_m = s[WF_RU_M];
    float* rv_m = s[WF_RV_M];
    float* ww_m = s[WF_WW_M];
    const bool ur = j < jde - 1, vr = i < ide - 1, wr = ur && vr;
    const bool last = iteration == nsub;
    const float muuc = last && ur ? __ldg(&s[WF_MUU][c]) : 0.f, mfuc = last && ur ? __ldg(&s[WF_MSFUY][c]) : 1.f;
    const float muvc = last && vr ? __ldg(&s[WF_MUV][c]) : 0.f, mvic = last && vr ? __ldg(&s[WF_MSFVX_INV][c]) : 0.f;
    const float r_nsub = __frcp_rn((float)nsub), r_mfuc = __frcp_rn(mfuc);
    float am[NQ], bm[NQ], cm[NQ], uv[NQ], vv[NQ], us[NQ], vs[NQ], w1[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int k = tk + q * kColKT;
      if (k >= nz) continue;
      const int p = k * lev + c;
      am[q] = iteration == 1 ? 0.f : ru_m[p];
      bm[q] = iteration == 1 ? 0.f : rv_m[p];
      cm[q] = iteration == 1 ? 0.f : ww_m[p];
      const bool lv = k < nz - 1;
      uv[q] = lv && ur ? __ldg(&u[p]) : 0.f;
      vv[q] = lv && vr ? __ldg(&v[p]) : 0.f;
      us[q] = last && lv && ur ? __ldg(&s[WF_U_SAVE][p]) : 0.f;
      vs[q] = last && lv && vr ? __ldg(&s[WF_V_SAVE][p]) : 0.f;
      w1[q] = last && wr ? __ldg(&ww1[p]) : 0.f;
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int k = tk + q * kColKT;
      if (k >= nz) continue;
      const int p = k * lev + c;
      float a = am[q], b = bm[q], cc = cm[q];
      if (k < nz - 1 && ur) a = a + uv[q];
      if (k < nz - 1 && vr) b = b + vv[q];
      if (wr) cc = cc + sww[k][tx];
      if (last) {
        if (k < nz - 1 && ur) a = divc(a, (float)nsub, r_nsub) + divc(muuc * us[q], mfuc, r_mfuc);
        if (k < nz - 1 && vr) b = divc(b, (float)nsub, r_nsub) + muvc * vs[q] * mvic;
        if (wr) cc = divc(cc, (float)nsub, r_nsub) + w1[q];
      }
      ru_m[p] = a;
      rv_m[p] = b;
      ww_m[p] = cc;
    }
  }
  __syncthreads();
  // --- H: calc_p_rho with divergence damping (mass columns)
  if (mass) {
    const float mu = smu[tx];
    float* al = s[WF_AL];
    float* pp = s[WF_P];
    float* pm1 = s[WF_PM1];
    float altv[NQ], t1v[NQ], c2v[NQ], tv[NQ], pmv[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int k = tk + q * kColKT;
      if (k >= kend) continue;
      const int p = k * lev + c;
      altv[q] = __ldg(&s[WF_ALT][p]);
      t1v[q] = __ldg(&t1[p]);
      c2v[q] = __ldg(&s[WF_C2A][p]);
      tv[q] = t[p];
      pmv[q] = pm1[p];
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int k = tk + q * kColKT;
      if (k >= kend) continue;
      const int p = k * lev + c;
      const float alk = -r_muts * (altv[q] * mu + prdnw[k] * (sph[k + 1][tx] - sph[k][tx]));
      al[p] = alk;
      const float pnew = c2v[q] * (altv[q] * (tv[q] - mu * t1v[q]) / (muts * ((float)T0 + t1v[q])) - alk);
      pp[p] = pnew + g.smdiv * (pnew - pmv[q]);
      pm1[p] = pnew;
    }
  }
}


// The same update with one thread per column, for domains whose columns fill
// the GPU by themselves (acoustic_col_marches below).  Three sweeps per
// column, no block barriers: up (the divergence of every level and its sum,
// and the flux averages of u and v), up again (ww, theta, the right-hand
// sides and the Thomas forward sweep, each level as soon as its neighbours
// are known, the values of the levels around it carried in registers), down
// (the back substitution, phi, and calc_p_rho of each level).  Only two
// column arrays are kept, in shared memory ([nz][32] each): the divergence,
// overwritten by the eliminated right-hand side of w, and the right-hand side
// of phi.  The operands of a few levels are loaded together, so each resident
// warp keeps about twenty 128-byte lines in flight.  The tiled form above
// issues a third more instructions (predicates, addresses and reciprocals per
// level group, the sweeps by one warp of eight; 75 million warp instructions
// against 57 at 240x240x41) behind ten block barriers, but starts more loads
// at once where the columns are few.  Per launch, tiled and marching: 140 and
// 165 us at 240x240x41, 251 and 253 at 320x320x41, 411 and 374 at 320x320x61,
// 1091 and 828 at 512x512x61.
// The arithmetic is that of the tiled form, operation for operation.
constexpr int kMarchTX = 32;

__global__ void __launch_bounds__(kMarchTX, 13) k_acoustic_march(Grid g, S s, float dts, int iteration, int nsub,
                                                                 int i0) {
  extern __shared__ float march_smem[];
  const int nz = g.nz, kend = nz - 1, nx = g.nx;
  const int ids = g.ids, ide = g.ide, jds = g.jds, jde = g.jde;
  const int i = i0 + blockIdx.x * kMarchTX + threadIdx.x, j = jds + blockIdx.y;
  // the profiles: dnw, rdnw, rdn, fnm, fnp
  __shared__ float pd[5][kMaxNz];
  for (int e = threadIdx.x; e < nz; e += kMarchTX) {
    pd[0][e] = __ldg(&s[WF_DNW][e]);
    pd[1][e] = __ldg(&s[WF_RDNW][e]);
    pd[2][e] = __ldg(&s[WF_RDN][e]);
    pd[3][e] = __ldg(&s[WF_FNM][e]);
    pd[4][e] = __ldg(&s[WF_FNP][e]);
  }
  __syncwarp();
  if (i < ids || i >= ide) return;
  float* const sy = march_smem + threadIdx.x;           // divergence, then y of the Thomas sweep
  float* const sr = sy + nz * kMarchTX;                 // right-hand side of phi
  const bool inner = j >= jds + 1 && j < jde - 2 && i >= ids + 1 && i < ide - 2;
  const bool spec = ((j == jds || j == jde - 2) && i < ide - 1) || (j >= jds + 1 && j < jde - 2 && (i == ids || i == ide - 2));
  const int c = g.i2(j, i);
  const int lev = g.ny * nx;
  const float* __restrict__ u = s[WF_U];
  const float* __restrict__ v = s[WF_V];
  const float* __restrict__ t1 = s[WF_T_SAVE];
  const float* __restrict__ ft = s[WF_T_TEND];
  const float* __restrict__ ww1 = s[WF_WW1];
  const float* __restrict__ ph1 = s[WF_PH_SAVE];
  const float* __restrict__ phb = s[WF_PHB];
  const float* __restrict__ pht = s[WF_PH_TEND];
  const float* __restrict__ c2a = s[WF_C2A];
  const float* __restrict__ alt = s[WF_ALT];
  float* t = s[WF_T];
  float* ww = s[WF_WW];
  float* ph = s[WF_PH];
  const bool last = iteration == nsub;
  const float fsub = (float)nsub, r_nsub = __frcp_rn(fsub);
  const float msftx = __ldg(&s[WF_MSFTX][c]), msfty = __ldg(&s[WF_MSFTY][c]);
  const float mut = __ldg(&s[WF_MUT][c]);
  const float mu_tend = __ldg(&s[WF_MU_TEND][c]);
  const float ep = g.epssm;
  const float ep1 = (float)(1.0 + (double)ep), em1 = (float)(1.0 - (double)ep);

  // --- sweep 1: flux averages of u and v (all columns), divergence (inner)
  float dmdt = 0.f;
  {
    float* ru_m = s[WF_RU_M];
    float* rv_m = s[WF_RV_M];
    const float* __restrict__ u1 = s[WF_U_SAVE];
    const float* __restrict__ v1 = s[WF_V_SAVE];
    const bool ur = j < jde - 1, vr = i < ide - 1;
    const float muu0 = __ldg(&s[WF_MUU][c]), mfu0 = __ldg(&s[WF_MSFUY][c]);
    const float muv0 = __ldg(&s[WF_MUV][c]), mvi0 = __ldg(&s[WF_MSFVX_INV][c]);
    const float muup = inner ? __ldg(&s[WF_MUU][c + 1]) : 0.f, mfup = inner ? __ldg(&s[WF_MSFUY][c + 1]) : 1.f;
    const float muvn = inner ? __ldg(&s[WF_MUV][c + nx]) : 0.f, mvin = inner ? __ldg(&s[WF_MSFVX_INV][c + nx]) : 0.f;
    const float r_mfup = __frcp_rn(mfup), r_mfu0 = __frcp_rn(mfu0);
    const float msf = msftx * msfty, rdx = g.rdx, rdy = g.rdy;
    constexpr int B = 4;
    struct Ops { float u0, v0, u10, v10, ue, u1e, vn, v1n, a, b; };
    auto load = [&](int k, Ops& o) {
      const int p = k * lev + c;
      const bool lv = k < kend;
      o.u0 = lv ? __ldg(u + p) : 0.f;
      o.v0 = lv ? __ldg(v + p) : 0.f;
      const bool sv = lv && (inner || last);
      o.u10 = sv ? __ldg(u1 + p) : 0.f;
      o.v10 = sv ? __ldg(v1 + p) : 0.f;
      const bool in = lv && inner;
      o.ue = in ? __ldg(u + p + 1) : 0.f;
      o.u1e = in ? __ldg(u1 + p + 1) : 0.f;
      o.vn = in ? __ldg(v + p + nx) : 0.f;
      o.v1n = in ? __ldg(v1 + p + nx) : 0.f;
      o.a = iteration == 1 ? 0.f : ru_m[p];
      o.b = iteration == 1 ? 0.f : rv_m[p];
    };
    for (int kb = 0; kb < nz; kb += B) {
      Ops o[B];
#pragma unroll
      for (int q = 0; q < B; ++q)
        if (kb + q < nz) load(kb + q, o[q]);
#pragma unroll
      for (int q = 0; q < B; ++q) {
        const int k = kb + q;
        if (k >= nz) continue;
        const int p = k * lev + c;
        float a = o[q].a, b = o[q].b;
        if (k < kend) {
          if (ur) a = a + o[q].u0;
          if (vr) b = b + o[q].v0;
          if (last) {
            if (ur) a = divc(a, fsub, r_nsub) + divc(muu0 * o[q].u10, mfu0, r_mfu0);
            if (vr) b = divc(b, fsub, r_nsub) + muv0 * o[q].v10 * mvi0;
          }
        }
        ru_m[p] = a;
        rv_m[p] = b;
        if (inner && k < kend) {
          const float dw = msf * (rdy * ((o[q].vn + muvn * o[q].v1n * mvin) - (o[q].v0 + muv0 * o[q].v10 * mvi0)) +
                                  rdx * ((o[q].ue + divc(muup * o[q].u1e, mfup, r_mfup)) -
                                         (o[q].u0 + divc(muu0 * o[q].u10, mfu0, r_mfu0))));
          sy[k * kMarchTX] = dw;
          dmdt = dmdt + pd[0][k] * dw;
        }
      }
    }
  }
  float* ww_m = s[WF_WW_M];
  float* al = s[WF_AL];
  float* pp = s[WF_P];
  float* pm1 = s[WF_PM1];
  if (inner) {
    const float* __restrict__ ca = s[WF_A];
    const float* __restrict__ calpha = s[WF_ALPHA];
    const float* __restrict__ cgamma = s[WF_GAMMA];
    const float* __restrict__ rw = s[WF_RW_TEND];
    const float* __restrict__ cqw = s[WF_CQW];
    float* w = s[WF_W];
    float* t2a = s[WF_T_2SAVE];
    const float r_msfty = __frcp_rn(msfty), r_mut = __frcp_rn(mut);
    float mu = s[WF_MU][c];
    const float muave_old = mu;
    mu = mu + dts * (dmdt + mu_tend);
    const float muts = mut + mu;
    const float muave = 0.5f * (ep1 * mu + em1 * muave_old);
    s[WF_MU][c] = mu;
    s[WF_MUDF][c] = dmdt + mu_tend;
    s[WF_MUTS][c] = muts;
    s[WF_MUAVE][c] = muave;
    const float r_muts = __frcp_rn(muts);
    const float cy = (float)(0.5 * g.rdyd), cx = (float)(0.5 * g.rdxd);
    const float cw = (float)(0.5 * G * (1.0 - (double)ep));
    const float msft_inv = 1.0f / msfty;
    const float cp = (float)(0.5 * (double)dts * G);
    const float cq = (float)((double)dts * G);
    // lower boundary of w: the terrain slope and near-surface winds
    float w0;
    {
      const float* __restrict__ ht = s[WF_HT];
      auto cv = [&](int cc) { return g.cf1 * __ldg(&v[cc]) + g.cf2 * __ldg(&v[lev + cc]) + g.cf3 * __ldg(&v[2 * lev + cc]); };
      auto cu = [&](int cc) { return g.cf1 * __ldg(&u[cc]) + g.cf2 * __ldg(&u[lev + cc]) + g.cf3 * __ldg(&u[2 * lev + cc]); };
      const float h0 = __ldg(&ht[c]);
      w0 = msfty * 0.5f * g.rdy * ((__ldg(&ht[c + nx]) - h0) * cv(c + nx) + (h0 - __ldg(&ht[c - nx])) * cv(c)) +
           msftx * 0.5f * g.rdx * ((__ldg(&ht[c + 1]) - h0) * cu(c + 1) + (h0 - __ldg(&ht[c - 1])) * cu(c));
    }
    // --- sweep 2.  Step k: ww(k+1), theta(k), the phi right-hand side r(k),
    // and with it w's right-hand side at m = k - 1 and its elimination.
    struct Ops {
      float ww1n, t1n, p1n, pbn;                              // level k + 1
      float told, ft, vn, tn, v0, ts, ue, te, u0, tw;         // level k
      float ph, pt, w, wm, ww1;
      float c2, alt, rw, cq, a, al;                           // level m = k - 1
    };
    // E: a step near the column's ends; between them every condition on the
    // level holds
    auto load = [&](auto edge, int k, Ops& o) {
      constexpr bool E = decltype(edge)::value;
      const int p = k * lev + c, m = p - lev;
      o.wm = iteration == 1 ? 0.f : ww_m[p];
      o.ww1 = last ? __ldg(ww1 + p) : 0.f;
      o.ph = ph[p];
      if (!E || k < kend) {
        o.ww1n = !E || k + 1 < kend ? __ldg(ww1 + p + lev) : ww[p + lev];
        o.t1n = !E || k + 1 < kend ? __ldg(t1 + p + lev) : 0.f;
        o.told = t[p];
        o.ft = __ldg(ft + p);
        o.vn = __ldg(v + p + nx);
        o.tn = __ldg(t1 + p + nx);
        o.v0 = __ldg(v + p);
        o.ts = __ldg(t1 + p - nx);
        o.ue = __ldg(u + p + 1);
        o.te = __ldg(t1 + p + 1);
        o.u0 = __ldg(u + p);
        o.tw = __ldg(t1 + p - 1);
        o.p1n = __ldg(ph1 + p + lev);
        o.pbn = __ldg(phb + p + lev);
      }
      if (!E || k >= 1) {
        o.pt = __ldg(pht + p);
        o.w = w[p];
        o.c2 = __ldg(c2a + m);
        o.alt = __ldg(alt + m);
      }
      if (!E || k >= 2) {
        o.rw = __ldg(rw + m);
        o.cq = __ldg(cqw + m);
        o.a = __ldg(ca + m);
        o.al = __ldg(calpha + m);
      }
    };
    const float rw_top = __ldg(rw + kend * lev + c), a_top = __ldg(ca + kend * lev + c),
                al_top = __ldg(calpha + kend * lev + c);
    float scan = ww[c];              // the ww scan, ww1 not yet taken off
    float wwk = scan - __ldg(ww1 + c);
    ww[c] = wwk;
    float t1k = __ldg(t1 + c), p1k = __ldg(ph1 + c), pbk = __ldg(phb + c);
    float wdn = 0.f, swk = 0.f;      // wdtn(k), wdwn(k)
    float rm = 0.f, phm = 0.f, avm = 0.f, wm1 = 0.f;   // r, phi, t_2ave, w at k - 1
    float X = 0.f, Tq = 0.f;         // the pressure and buoyancy terms at m - 1
    float y = w0;
    auto step = [&](auto edge, int k, const Ops& o, Ops& n) {
      constexpr bool E = decltype(edge)::value;
      if (!E || k < kend) load(edge, k + 1, n);
      const int p = k * lev + c;
      const float rdk = pd[1][k], fk = pd[3][k], fpk = pd[4][k];
      float cc = o.wm + wwk;
      if (last) cc = divc(cc, fsub, r_nsub) + o.ww1;
      float wwn = 0.f, swn = 0.f, avk = 0.f;
      if (!E || k < kend) {
        float wup = 0.f;
        if (!E || k + 1 < kend) {
          scan = scan - divc(pd[0][k] * (dmdt + sy[k * kMarchTX] + mu_tend), msfty, r_msfty);
          wwn = scan - o.ww1n;
          ww[p + lev] = wwn;
          wup = wwn * (pd[3][k + 1] * o.t1n + pd[4][k + 1] * t1k);
        } else {
          wwn = o.ww1n;  // ww at the top level stays
        }
        float tt = o.told + msfty * dts * o.ft;
        const float hy = cy * (o.vn * (o.tn + t1k) - o.v0 * (t1k + o.ts));
        const float hx = cx * (o.ue * (o.te + t1k) - o.u0 * (t1k + o.tw));
        tt = tt - dts * msfty * (msftx * (hy + hx) + rdk * (wup - wdn));
        t[p] = tt;
        avk = 0.5f * (ep1 * tt + em1 * o.told);
        avk = (avk + muave * (float)T0) / (muts * ((float)T0 + t1k));
        t2a[p] = avk;
        swn = 0.5f * (wwn + wwk) * rdk * (o.p1n - p1k + o.pbn - pbk);
        wdn = wup;
        t1k = o.t1n;
        p1k = o.p1n;
        pbk = o.pbn;
      }
      ww_m[p] = cc;
      float r = 0.f;
      if (!E || k >= 1) {
        r = dts * (o.pt + cw * o.w);
        if (!E || k < kend) r = r - dts * (fk * swn + fpk * swk);
        r = o.ph + divc(msfty * r, mut, r_mut);
        const float rdm = pd[1][k - 1];
        const float X1 = divc(o.c2 * rdm, mut, r_mut) * (ep1 * (r - rm) + em1 * (o.ph - phm));
        const float T1 = o.c2 * o.alt * avm;
        if (!E || k >= 2) {
          const float rdn_m = pd[2][k - 1];
          const float wl = wm1 + dts * o.rw + msft_inv * o.cq * (cp * rdn_m * (X1 - X)) +
                           cq * msft_inv * (rdn_m * (T1 - Tq) - muave);
          y = (wl - o.a * y) * o.al;
          sy[(k - 1) * kMarchTX] = y;
        }
        if (E && k == kend) {
          const float cm = (float)(-0.5 * (double)dts * G);
          const float wl = o.w + dts * rw_top +
                           msft_inv * (divc(cm, mut, r_mut) * (rdm * rdm) * 2.0f * o.c2 *
                                           (ep1 * (r - rm) + em1 * (o.ph - phm)) -
                                       cq * (2.0f * rdm * o.c2 * o.alt * avm + muave));
          y = (wl - a_top * y) * al_top;
        }
        X = X1;
        Tq = T1;
        wm1 = o.w;
      }
      sr[k * kMarchTX] = r;
      rm = r;
      phm = o.ph;
      avm = avk;
      wwk = wwn;
      swk = swn;
    };
    {
      const std::true_type ends{};
      const std::false_type between{};
      Ops A, B;
      load(ends, 0, A);
      step(ends, 0, A, B);
      step(ends, 1, B, A);
      int k = 2;
      for (; k + 1 <= kend - 3; k += 2) {
        step(between, k, A, B);
        step(between, k + 1, B, A);
      }
      for (; k <= kend; k += 2) {
        step(ends, k, A, B);
        if (k < kend) step(ends, k + 1, B, A);
      }
    }
    // --- sweep 3: back substitution, damping, phi; calc_p_rho of each level
    struct Down { float gm, p1, pb, ws, alt, t1, c2, t, pm; };
    const float* __restrict__ wsave = s[WF_W_SAVE];
    auto load3 = [&](int k, Down& o) {
      const int p = k * lev + c;
      if (k >= 1) {
        o.p1 = __ldg(ph1 + p);
        o.pb = __ldg(phb + p);
        o.ws = __ldg(wsave + p);
      } else {
        o.ws = ph[p];  // phi(0) stays
      }
      if (k < kend) {
        o.gm = __ldg(cgamma + p);
        o.alt = __ldg(alt + p);
        o.t1 = __ldg(t1 + p);
        o.c2 = __ldg(c2a + p);
        o.t = t[p];
        o.pm = pm1[p];
      }
    };
    const float gf = (float)G;
    constexpr float r_g = 1.0f / (float)G, r_hd = 1.0f / 5000.0f;
    const float hdepth = 5000.0f;
    const float dampmag = (float)((double)dts * 0.2);
    const float hpi = (float)(0.5 * 3.14159265359);
    float hbot = 0.f, wn = 0.f, phn = 0.f;
    auto down = [&](int k, const Down& o, Down& n) {
      if (k >= 1) load3(k - 1, n);
      const int p = k * lev + c;
      float phk;
      if (k == 0) {
        w[c] = w0;
        phk = o.ws;
      } else {
        const float hk = divc(o.p1 + o.pb, gf, r_g);
        if (k == kend) {
          hbot = hk - hdepth;
          wn = y;
        } else {
          wn = sy[k * kMarchTX] - o.gm * wn;
        }
        float dwd = 0.f;
        if (hk >= hbot) {
          const float sn = sinf(divc(hpi * (hk - hbot), hdepth, r_hd));
          dwd = dampmag * (sn * sn);
        }
        const float num = wn - dwd * mut * o.ws;
        const float wk = dwd == 0.f ? num : num / (1.0f + dwd);  // x / 1 == x
        w[p] = wk;
        phk = sr[k * kMarchTX] + divc(msfty * 0.5f * dts * gf * ep1 * wk, muts, r_muts);
        ph[p] = phk;
      }
      if (k < kend) {
        const float alk = -r_muts * (o.alt * mu + pd[1][k] * (phn - phk));
        al[p] = alk;
        const float pnew = o.c2 * (o.alt * (o.t - mu * o.t1) / (muts * ((float)T0 + o.t1)) - alk);
        pp[p] = pnew + g.smdiv * (pnew - o.pm);
        pm1[p] = pnew;
      }
      phn = phk;
    };
    {
      Down A, B;
      load3(kend, A);
      for (int k = kend; k >= 0; k -= 2) {
        down(k, A, B);
        if (k >= 1) down(k - 1, B, A);
      }
    }
  } else if (spec) {
    const float mu = s[WF_MU][c] + dts * mu_tend;
    const float muts = s[WF_MUTS][c] + dts * mu_tend;
    s[WF_MU][c] = mu;
    s[WF_MUTS][c] = muts;
    const float r_muts = __frcp_rn(muts);
    const float mu_old = muts - dts * mu_tend;
    float phm = 0.f, altm = 0.f, t1m = 0.f, c2m = 0.f, tm = 0.f, pmm = 0.f;
    constexpr int B = 4;
    for (int kb = 0; kb < nz; kb += B) {
      float ov[B][11];
#pragma unroll
      for (int q = 0; q < B; ++q) {
        const int k = kb + q, p = k * lev + c;
        if (k >= nz) continue;
        ov[q][0] = ph[p];
        ov[q][1] = __ldg(pht + p);
        ov[q][2] = __ldg(ph1 + p);
        ov[q][3] = iteration == 1 ? 0.f : ww_m[p];
        ov[q][4] = ww[p];
        ov[q][5] = last ? __ldg(ww1 + p) : 0.f;
        if (k >= kend) continue;
        ov[q][6] = t[p] + dts * __ldg(ft + p);
        ov[q][7] = __ldg(alt + p);
        ov[q][8] = __ldg(t1 + p);
        ov[q][9] = __ldg(c2a + p);
        ov[q][10] = pm1[p];
      }
#pragma unroll
      for (int q = 0; q < B; ++q) {
        const int k = kb + q, p = k * lev + c;
        if (k >= nz) continue;
        float cc = ov[q][3] + ov[q][4];
        if (last) cc = divc(cc, fsub, r_nsub) + ov[q][5];
        ww_m[p] = cc;
        const float phk = divc(ov[q][0] * mu_old, muts, r_muts) + divc(dts * ov[q][1], muts, r_muts) +
                          ov[q][2] * (divc(mu_old, muts, r_muts) - 1.0f);
        ph[p] = phk;
        if (k < kend) t[p] = ov[q][6];
        if (k >= 1) {  // calc_p_rho of the level below
          const int pm = p - lev;
          const float alk = -r_muts * (altm * mu + pd[1][k - 1] * (phk - phm));
          al[pm] = alk;
          const float pnew = c2m * (altm * (tm - mu * t1m) / (muts * ((float)T0 + t1m)) - alk);
          pp[pm] = pnew + g.smdiv * (pnew - pmm);
          pm1[pm] = pnew;
        }
        phm = phk;
        tm = ov[q][6];
        altm = ov[q][7];
        t1m = ov[q][8];
        c2m = ov[q][9];
        pmm = ov[q][10];
      }
    }
  } else if (iteration == 1) {  // outside the mass columns the flux average only starts at zero
    for (int k = 0; k < nz; ++k) ww_m[k * lev + c] = 0.f;
  }
}

// The marching form takes one wave of at most 13 warps per SM whose length is
// the column's chain of levels (110 us per launch at 41 levels however few the
// columns), so it pays from about one and a half such waves on: at 400x400x41
// 397 us against 405 for the tiled form, at 320x320x61 374 against 411, at
// 512x512x61 828 against 1091; at 240x240x41 165 against 140.
static bool acoustic_col_marches(const Grid& g) {
  return kernel_form() == WRF_FORM_FAST &&
         2LL * (g.ide - g.ids) * (g.jde - g.jds) >= 3LL * 148 * 13 * kMarchTX;
}


__global__ void k_mu_uv_1(Grid g, S s) {
  WRF_COLUMN_INDEX(g, j, i);
  const int c = g.i2(j, i);
  const int jts = g.jds, jme = g.jde - 1, its = g.ids, ite = g.ide, ime = g.ide - 1, jte = g.jde;
  const float* muts = s[WF_MUTS];
  if (j >= jts && j < jme) {
    if (i >= its + 1 && i < ite - 1) s[WF_MUUS][c] = 0.5f * (muts[c] + muts[c - 1]);
    else if (i == its) s[WF_MUUS][c] = muts[c];
    else if (i == ite - 1) s[WF_MUUS][c] = muts[c - 1];
  }
  if (i >= its && i < ime) {
    if (j >= jts + 1 && j < jte - 1) s[WF_MUVS][c] = 0.5f * (muts[c] + muts[c - g.nx]);
    else if (j == jts) s[WF_MUVS][c] = muts[c];
    else if (j == jte - 1) s[WF_MUVS][c] = muts[c - g.nx];
  }
}

// operands first, then the stores (a store would hold back the later
// fields' loads)
__global__ void k_ssfinish(Grid g, S s, float dts, int nsub, int rk_step) {
  WRF_POINT_INDEX(g, k, j, i);
  const int nz = g.nz;
  const int jts = g.jds, jme = g.jde - 1, its = g.ids, ime = g.ide - 1, ieu = g.ide, jev = g.jde;
  const int c = g.i2(j, i);
  const size_t p = (size_t)k * g.ny * g.nx + c;
  const bool dv = k < nz - 1 && j >= jts && j < jev && i >= its && i < ime;
  const bool du = k < nz - 1 && j >= jts && j < jme && i >= its && i < ieu;
  const bool m3 = j >= jts && j < jme && i >= its && i < ime;
  float vv = 0.f, vs = 0.f, mfvx = 0.f, muv = 0.f, muvs = 1.f;
  if (dv) {
    vv = s[WF_V][p];
    vs = s[WF_V_SAVE][p];
    mfvx = s[WF_MSFVX][c];
    muv = s[WF_MUV][c];
    muvs = s[WF_MUVS][c];
  }
  float uu = 0.f, us = 0.f, mfuy = 0.f, muu = 0.f, muus = 1.f;
  if (du) {
    uu = s[WF_U][p];
    us = s[WF_U_SAVE][p];
    mfuy = s[WF_MSFUY][c];
    muu = s[WF_MUU][c];
    muus = s[WF_MUUS][c];
  }
  float mut = 0.f, muts = 1.f, mfty = 0.f, ww = 0.f, wsv = 0.f, phv = 0.f, phs = 0.f, wwv = 0.f, ww1 = 0.f;
  float tv = 0.f, ts = 0.f, hd = 0.f, muv0 = 0.f, mus0 = 0.f;
  if (m3) {
    mut = s[WF_MUT][c];
    muts = s[WF_MUTS][c];
    mfty = s[WF_MSFTY][c];
    ww = s[WF_W][p];
    wsv = s[WF_W_SAVE][p];
    phv = s[WF_PH][p];
    phs = s[WF_PH_SAVE][p];
    wwv = s[WF_WW][p];
    ww1 = s[WF_WW1][p];
    if (k < nz - 1) {
      tv = s[WF_T][p];
      ts = s[WF_T_SAVE][p];
      if (rk_step == 3) hd = s[WF_H_DIABATIC][p];
    }
    if (k == 0) {
      muv0 = s[WF_MU][c];
      mus0 = s[WF_MU_SAVE][c];
    }
  }
  if (dv) s[WF_V][p] = (mfvx * vv + vs * muv) / muvs;
  if (du) s[WF_U][p] = (mfuy * uu + us * muu) / muus;
  if (m3) {
    s[WF_W][p] = (mfty * ww + wsv * mut) / muts;
    s[WF_PH][p] = phv + phs;
    s[WF_WW][p] = wwv + ww1;
    if (k < nz - 1) {
      if (rk_step < 3)
        s[WF_T][p] = (tv + ts * mut) / muts;
      else
        s[WF_T][p] = (tv - (float)((double)dts * nsub) * mut * hd + ts * mut) / muts;
    }
    if (k == 0) s[WF_MU][c] = muv0 + mus0;
  }
}

int launch_small_step_prep(const Grid& g, const S& s, int rk_step, float dts, cudaStream_t st) {
  const dim3 b2(32, 8), b3(32, 4);
  k_ssp2d<<<col_grid(g, b2), b2, 0, st>>>(g, s, rk_step);
  k_ssp3d<<<point_grid(g, b3), b3, 0, st>>>(g, s, rk_step);
  k_p_rho0<<<point_grid(g, b3), b3, 0, st>>>(g, s);
  run_coef_w(g, s, dts, st);
  return 4;
}

// small_step_prep alone (the step's k_ssp2d and k_ssp3d)
int launch_ssp_only(const Grid& g, const S& s, int rk_step, cudaStream_t st) {
  const dim3 b2(32, 8), b3(32, 4);
  k_ssp2d<<<col_grid(g, b2), b2, 0, st>>>(g, s, rk_step);
  k_ssp3d<<<point_grid(g, b3), b3, 0, st>>>(g, s, rk_step);
  return 2;
}

int launch_coef_w(const Grid& g, const float* mut, const float* cqw, const float* c2a, const float* rdn,
                  const float* rdnw, float dts, float* a, float* alpha, float* gamma, cudaStream_t st) {
  S s{};
  s.f[WF_MUT] = const_cast<float*>(mut);
  s.f[WF_CQW] = const_cast<float*>(cqw);
  s.f[WF_C2A] = const_cast<float*>(c2a);
  s.f[WF_RDN] = const_cast<float*>(rdn);
  s.f[WF_RDNW] = const_cast<float*>(rdnw);
  s.f[WF_A] = a;
  s.f[WF_ALPHA] = alpha;
  s.f[WF_GAMMA] = gamma;
  run_coef_w(g, s, dts, st);
  return 1;
}

int launch_advance_uv(const Grid& g, const S& s, float dts, cudaStream_t st, bool expired) {
  if (kernel_form() == WRF_FORM_FAST && g.nx % 4 == 0 && g.nz >= 4) {
    UvTmaArgs a{};
    const char* err = nullptr;
    const int f[6] = {WF_ALT, WF_AL, WF_PB, WF_PHP, WF_PH, WF_P};
    CUtensorMap* m[6] = {&a.alt, &a.al, &a.pb, &a.php, &a.ph, &a.pp};
    bool ok = true;
    for (int e = 0; e < 6 && ok; ++e) ok = tma::encode_f32_4d(m[e], s[f[e]], g.nx, g.ny, g.nz, 1, kUvBW, kUvBH, &err);
    const int fo[kUvNO] = {WF_U, WF_RU_TEND, WF_V, WF_RV_TEND, WF_CQU, WF_CQV};
    for (int e = 0; e < kUvNO && ok; ++e)
      ok = tma::encode_f32_4d(&a.own[e], s[fo[e]], g.nx, g.ny, g.nz, 1, kUvOW, kUvOH, &err);
    if (ok) {
      const int bx = (g.ide + 1 - g.ids + kUvTX - 1) / kUvTX, by = (g.jde - g.jds + kUvTY - 1) / kUvTY;
      a.nchunk = level_chunks(g.nz - 1, bx * by, kUvKCH, 4);
      a.expired = expired;
      const dim3 gr(bx, by, a.nchunk);
      k_advance_uv_tma<<<gr, dim3(kUvTX, kUvTY), 0, st>>>(g, s, dts, a);
      return 1;
    }
  }
  if (expired) return 0;
  const dim3 b3(32, 4);
  dim3 gr = point_grid(g, b3);
  // two levels a thread while that leaves at most 12 blocks an SM (ten fit at a
  // time; the frame's return at once), where a thread's own chain is the time;
  // three from there on.  Two and three levels, us per launch with the operands
  // in L2 / in DRAM: 8.5 / 14.3 and 8.5 / 16.4 at 91x91x35 (8 blocks an SM), 9.0 /
  // 14.3 and 10.5 / 18.4 at 101x101x35 (11.9), 10.5 / 20.5 and 10.5 / 18.4 at
  // 107x107x35 (12.4), 11.2 / 20.5 and 10.5 / 18.4 at 91x91x61 (14), 11.8 / 20.5
  // and 10.5 / 18.4 at 121x121x35 (14.2), 12.6 / 20.5 and 10.5 / 18.4 at
  // 131x131x35 (19)
  const int ktf = g.nz - 1;
  const bool two = (long long)gr.x * gr.y * ((ktf + 1) / 2) <= 148 * 12;
  gr.z = two ? (ktf + 1) / 2 : (ktf + 2) / 3;
  if (two) k_advance_uv<2><<<gr, b3, 0, st>>>(g, s, dts);
  else k_advance_uv<3><<<gr, b3, 0, st>>>(g, s, dts);
  return 1;
}

int launch_acoustic_col(const Grid& g, const S& s, float dts, int iteration, int nsub, cudaStream_t st) {
  const int i0 = g.nx % 8 == 0 ? g.ids / 8 * 8 : g.ids;
  if (acoustic_col_marches(g)) {
    k_acoustic_march<<<dim3((g.ide - i0 + kMarchTX - 1) / kMarchTX, g.jde - g.jds), kMarchTX,
                       2 * (size_t)g.nz * kMarchTX * sizeof(float), st>>>(g, s, dts, iteration, nsub, i0);
    return 1;
  }
  const dim3 gc((g.ide - i0 + kColTX - 1) / kColTX, g.jde - g.jds);
  if (g.nz <= 2 * kColKT)
    k_acoustic_col<2><<<gc, kColTX * kColKT, 0, st>>>(g, s, dts, iteration, nsub, i0);
  else if (g.nz <= 3 * kColKT)
    k_acoustic_col<3><<<gc, kColTX * kColKT, 0, st>>>(g, s, dts, iteration, nsub, i0);
  else
    k_acoustic_col<4><<<gc, kColTX * kColKT, 0, st>>>(g, s, dts, iteration, nsub, i0);
  return 1;
}


int launch_small_step_finish(const Grid& g, const S& s, float dts, int nsub, int rk_step, cudaStream_t st) {
  const dim3 b2(32, 8), b3(32, 4);
  k_mu_uv_1<<<col_grid(g, b2), b2, 0, st>>>(g, s);
  k_ssfinish<<<point_grid(g, b3), b3, 0, st>>>(g, s, dts, nsub, rk_step);
  return 2;
}

}  // namespace wrf
