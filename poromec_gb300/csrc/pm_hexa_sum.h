// pm_hexa_sum.h -- the matrix-free hexa20 element passes by sum factorisation
// (included by pm_elements.cu inside its unnamed namespace).
//
// What bounds them.  These passes interpolate nodal values to the 64 points and
// sum point values back to the nodes: with 20 functions at 64 points that is
// 11,500 FP64 multiply-adds each way per vector field, and mapping all
// derivatives to physical coordinates 16,000 more, at 1.7 per clock and SM.  The
// points are a 4 x 4 x 4 product, and the serendipity functions are products of
// (1 - x) / 2, (1 + x) / 2 and 1 - x^2 of which at most one is quadratic: with the
// corners' values and, for each mid-side node, its value less the mean of its
// edge's ends as coefficients, one direction at a time (Orszag, "Spectral methods
// for problems in complex geometries", J. Comput. Phys. 37, 1980) takes 3,600, and
// only the gradients, not the functions, are mapped at a point.  The FP64 pipe is
// still what bounds them on many elements (79 % busy), the chain of sweeps on few.
// Less rounding too: fields and coordinates enter as differences in every direction,
// and one mid-side term is smaller than its node's value.  Errors against extended
// precision, rms by output, with the functions and now: isw 2's forces 2.7e-16 and
// 2.0e-16 on the 4^3 cube, 7.4e-16 and 2.6e-16 on the 18^3, the adjoint's gradients in
// log E 1.9e-16 and 2.3e-16, 5.2e-16 and 2.8e-16, in log k 3.3e-16 and 2.5e-16, 6.2e-16
// and 2.8e-16; jittered 8^3: forces 3.5e-16 and 2.6e-16, log E 2.8e-16 and 2.7e-16.
//
// One element per CTA of 192 threads: thread (point, direction) at the points,
// one output per thread in each sweep; FP64 instructions are spread over the four
// schedulers, since a warp's occupies one for 64 clocks.  Measured, before (every
// function mapped, 64 threads) and now: isw 2's forces of the 40^3 cube 8.74 and
// 2.83 ms, isw 4's 9.27 and 2.96, of the 2 x 2 x 40 column 0.43 and 0.03, 0.59 and
// 0.05 (colours overlapped); the adjoint's two passes of the 32^3 cube 7.75 and 3.01.
constexpr int kSfThreads = 192;

// index in the 3 x 3 x 3 grid (r + 3 s + 9 t) of each node, and the corners' in
// the 2 x 2 x 2 grid
__constant__ int cGrid27[20] = {26, 24, 18, 20, 8, 6, 0, 2, 25, 21, 19, 23, 7, 3, 1, 5,
                                17, 15, 9, 11};
__constant__ int cGrid8[8] = {7, 6, 4, 5, 3, 2, 0, 1};

struct SfLoads {  // isw 4 only
  const int32_t *eload, *eloadp, *load;
  const double* fload;
  int maxt;
};

enum SfOp { kSfResidual, kSfRhs4, kSfApply, kSfGrad };

template <SfOp OP>
struct SmSf {
  static constexpr bool GRAD = OP == kSfGrad, BODY = OP == kSfRhs4;
  static constexpr int NC = GRAD ? 6 : 3;  // vector components: u, or lam and u_n
  // linear fields: x, y, z, then the pressures the pass needs: the gradients of the
  // first NG are taken, the values of NVF
  static constexpr int NL = 3 + (GRAD ? 3 : OP == kSfRhs4 ? 2 : 1), NG = GRAD ? 5 : 4,
                       NVF = GRAD ? 2 : OP == kSfApply ? 0 : 1;
  double C[NC][27];          // coefficients, then the sums
  double A[2][NC][36];      // [value, derivative][c][zy x]
  double B[NC][3][48];      // [c][r, s, t][z yx]
  double lin[NL][8];
  double LB[NG][32];        // d/dr (z, y), d/ds (z, x), d/dt (y, x)
  double LV[NVF > 0 ? NVF : 1][32];  // value (z, yx)
  double JI[3][3][64];      // [x_j][xi_a]: dx_j / dxi_a, then det dxi_a / dx_j
  double rd[64], wq[64], w[64];  // 1 / det, the weight, weight times det
  double G[NC][3][64];      // physical gradients, then the natural fluxes
  double F[3][64];          // pressure flux
  double S0[64];            // value source of the pressure rows
  double body[BODY ? 64 : 1];
  double T2[2][32];         // pressure rows: sweeps back
  double LT[2][3][32];
  double out[68], out2[8], pf[BODY ? 68 : 1];
  double Q[4][3], Qd[4][3], Lw[4][2];
  double gsum[3][kSfThreads / 32];
  int nodes[20], mat;
  int iqm[7], iqh[7], any;
  int fail;
};

// A mid-side node's coefficient (edge e: four along r, four along s, four along
// t), in place.
__device__ __forceinline__ void sf_edge(double* c, int e) {
  const int d = e >> 2, a = 2 * (e & 1), b = 2 * ((e >> 1) & 1);
  const int sd = d == 0 ? 1 : d == 1 ? 3 : 9;
  const int m = sd + a * (d == 0 ? 3 : 1) + b * (d == 2 ? 3 : 9);
  c[m] -= 0.5 * (c[m - sd] + c[m + sd]);
}

// Transposed: what a node takes from the sums.
__device__ __forceinline__ double sf_fold(const double* c, int node) {
  const int g = cGrid27[node];
  if (node >= 8) return c[g];
  const int r = g % 3, s = (g / 3) % 3, t = g / 9;
  return c[g] - 0.5 * (c[1 + 3 * s + 9 * t] + c[r + 3 + 9 * t] + c[r + 3 * s + 9]);
}

// Face tractions (types 40, 41) and normal fluxes (43) of one element by one warp,
// into p: what does not depend on the point on every lane alike, a division of the
// rotation and a point of the 3 x 3 rule per lane, then an entry of p per lane over
// the points in order.  wt: 72 doubles of scratch.  One thread took 42 us of a launch.
__device__ bool hexa_face_loads(const ElemLaunch& L, const SfLoads& ld, const int* iqm,
                                const int* iqh, const double (*lin)[8], double* p, double* wt,
                                int lane) {
  bool fail = false;
  // (rotated in place a second time where a face has both loads, as the reference)
  auto rotate = [lane](double (&xf)[12]) {
    const double v1x = xf[3] - xf[0], v1y = xf[4] - xf[1], v1z = xf[5] - xf[2];
    double v2x = xf[6] - xf[0], v2y = xf[7] - xf[1], v2z = xf[8] - xf[2];
    const double v3x = v1y * v2z - v1z * v2y, v3y = v1z * v2x - v1x * v2z,
                 v3z = v1x * v2y - v1y * v2x;
    v2x = v1z * v3y - v1y * v3z;
    v2y = v1x * v3z - v1z * v3x;
    v2z = v1y * v3x - v1x * v3y;
    const int r = lane < 3 ? 0 : lane < 6 ? 1 : 2, c = lane - 3 * r;
    const double x = r == 0 ? v1x : r == 1 ? v2x : v3x, y = r == 0 ? v1y : r == 1 ? v2y : v3y,
                 z = r == 0 ? v1z : r == 1 ? v2z : v3z;
    const double n = sqrt(x * x + y * y + z * z);
    const double q = (c == 0 ? x : c == 1 ? y : z) / n;
    double R[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) R[k] = __shfl_sync(0xffffffffu, q, k);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      double* v = xf + 3 * i;
      const double a = R[0] * v[0] + R[1] * v[1] + R[2] * v[2];
      const double b = R[3] * v[0] + R[4] * v[1] + R[5] * v[2];
      const double d = R[6] * v[0] + R[7] * v[1] + R[8] * v[2];
      v[0] = a;
      v[1] = b;
      v[2] = d;
    }
  };
  const int ly = lane / 3, lx = lane - 3 * ly;
  // the point's weight times its determinant
  auto point = [&](const double (&xf)[12], double& r, double& s) {
    r = cPG3[lx];
    s = cPG3[ly];
    const double pr = 1 + r, ps = 1 + s, mr = 1 - r, ms = 1 - s;
    const double hx[4] = {ps * 0.25, -ps * 0.25, -ms * 0.25, ms * 0.25};
    const double hy[4] = {pr * 0.25, mr * 0.25, -mr * 0.25, -pr * 0.25};
    const double det = d_det2(hx, hy, xf, 4);
    if (!(det > 1.0e-14)) fail = true;
    return cWG3[lx] * cWG3[ly] * det;
  };
  for (int j = 0; j < 6; ++j) {
    if (!(iqm[j] > 0 || iqh[j] > 0)) continue;
    const int* fn = cHexaFace[j];
    double xf[12];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int k = 0; k < 3; ++k) xf[3 * i + k] = lin[k][cGrid8[fn[i] - 1]];
    const int cargm = iqm[j] != 0 ? ld.load[3 * (iqm[j] - 1)] : 0;
    const int cargh = iqh[j] != 0 ? ld.load[3 * (iqh[j] - 1)] : 0;
    double ff[3] = {0, 0, 0}, nc = 0, dd;
    const double mp[3] = {0, 0, 0};
    if (cargm == 40 || cargm == 41 || cargm == 42) {
      if (cargm == 41) {
        const double v1[3] = {xf[3] - xf[0], xf[4] - xf[1], xf[5] - xf[2]};
        const double v2[3] = {xf[6] - xf[0], xf[7] - xf[1], xf[8] - xf[2]};
        ff[0] = v2[1] * v1[2] - v2[2] * v1[1];
        ff[1] = v2[2] * v1[0] - v2[0] * v1[2];
        ff[2] = v2[0] * v1[1] - v2[1] * v1[0];
        const double tmp = 1.0 / sqrt(ff[0] * ff[0] + ff[1] * ff[1] + ff[2] * ff[2]);
        ff[0] *= tmp; ff[1] *= tmp; ff[2] *= tmp;
        if (j != 1) { ff[0] = -ff[0]; ff[1] = -ff[1]; ff[2] = -ff[2]; }
      }
      rotate(xf);
      if (cargm == 41 || cargm == 42) {
        d_tload(ld.load, ld.fload, ld.maxt, iqm[j], L.t, mp, L.gmod, nc, &dd);
        ff[0] *= nc; ff[1] *= nc; ff[2] *= nc;
      } else {
        d_tload(ld.load, ld.fload, ld.maxt, iqm[j], L.t, mp, L.gmod, dd, ff);
      }
      if (lane < 9) {
        double r, s;
        const double w = point(xf, r, s);
        const double pr = 1 + r, ps = 1 + s, mr = 1 - r, ms = 1 - s;
        double h[8];
        const double mrr = 1 - r * r, mss = 1 - s * s;
        h[4] = mrr * ps * 0.5; h[5] = mss * mr * 0.5; h[6] = mrr * ms * 0.5;
        h[7] = mss * pr * 0.5;
        h[0] = pr * ps * 0.25 - h[4] * 0.5 - h[7] * 0.5;
        h[1] = mr * ps * 0.25 - h[4] * 0.5 - h[5] * 0.5;
        h[2] = mr * ms * 0.25 - h[5] * 0.5 - h[6] * 0.5;
        h[3] = pr * ms * 0.25 - h[6] * 0.5 - h[7] * 0.5;
#pragma unroll
        for (int i = 0; i < 8; ++i) wt[8 * lane + i] = h[i] * w;
      }
      __syncwarp();
      if (lane < 24) {
        const int i = lane / 3, k = lane - 3 * i, e = 3 * fn[i] - 3 + k;
        const double f = k == 0 ? ff[0] : k == 1 ? ff[1] : ff[2];
        double acc = p[e];
#pragma unroll
        for (int q = 0; q < 9; ++q) acc -= f * wt[8 * q + i];
        p[e] = acc;
      }
      __syncwarp();
    }
    if (cargh == 43) {
      rotate(xf);
      d_tload(ld.load, ld.fload, ld.maxt, iqh[j], L.t, mp, L.gmod, nc, &dd);
      if (lane < 9) {
        double r, s;
        const double w = point(xf, r, s) * L.dt * nc;
        const double pr = 1 + r, ps = 1 + s, mr = 1 - r, ms = 1 - s;
        const double h[4] = {pr * ps * 0.25, mr * ps * 0.25, mr * ms * 0.25, pr * ms * 0.25};
#pragma unroll
        for (int i = 0; i < 4; ++i) wt[8 * lane + i] = h[i] * w;
      }
      __syncwarp();
      if (lane < 4) {
        const int e = 60 + fn[lane] - 1;
        double acc = p[e];
#pragma unroll
        for (int q = 0; q < 9; ++q) acc -= wt[8 * q + lane];
        p[e] = acc;
      }
      __syncwarp();
    }
  }
  return __any_sync(0xffffffffu, fail);
}

// OP kSfResidual: b -= K_e u_e (isw 2, rhs).  kSfRhs4: b -= p of isw 4 (internal
// force of the previous state, body force, Darcy gravity term, face loads).
// kSfApply: mu -= [Kuu lam_u ; Kpp_perm lam_p], nu -= Kpu lam_u.  kSfGrad: the
// contractions of launch_adjoint's mode 1.  a0: u (lam for the adjoint), a1: dp
// (u_n), a2: du.
template <SfOp OP>
__global__ void __launch_bounds__(kSfThreads, 5)
    k_hexa_sum(ElemLaunch L, const double* __restrict__ a0, const double* __restrict__ a1,
               const double* __restrict__ a2, SfLoads ld, double* __restrict__ o0,
               double* __restrict__ o1) {
  using Sm = SmSf<OP>;
  constexpr int NEN = 20, NV = 8, NC = Sm::NC, NL = Sm::NL;
  extern __shared__ __align__(16) unsigned char smem[];
  Sm& S = *reinterpret_cast<Sm*>(smem);
  const int tid = threadIdx.x, lane = tid & 31;
  colour_next();
  const int el = L.elems[blockIdx.x];
  const int32_t* ixe = L.ix + (size_t)(NEN + 1) * (el - 1);
  // ---- element data -----------------------------------------------------------
  if (tid < 80) {  // vector components and pressure of node tid / 4
    const int i = tid >> 2, q = tid & 3, n = ixe[i], n0 = ixe[0];
    if (q < 3) {
      // only gradients are taken of these: less node 1's value, what the sweeps
      // round is the field's variation over the element, not the field
      const size_t a = (size_t)kNdf * (n - 1) + q, r = (size_t)kNdf * (n0 - 1) + q;
      S.C[q][cGrid27[i]] = a0[a] - a0[r];
      if constexpr (Sm::GRAD) S.C[3 + q][cGrid27[i]] = a1[a] - a1[r];
      if (i < NV) S.lin[q][cGrid8[i]] = L.x[(size_t)3 * (n - 1) + q];
    } else {
      S.nodes[i] = n;
      if (i < NV) {
        const int k = cGrid8[i];
        S.lin[3][k] = a0[(size_t)kNdf * (n - 1) + 3];
        if constexpr (OP == kSfRhs4) S.lin[NL - 1][k] = a1[n - 1];
        if constexpr (Sm::GRAD) {
          S.lin[NL - 2][k] = a1[(size_t)kNdf * (n - 1) + 3];
          S.lin[NL - 1][k] = a2[(size_t)kNdf * (n - 1) + 3];
        }
      }
    }
  } else if (tid < 84) {  // the 1-D functions at the Gauss points
    const int g = tid - 80;
    const double x = cPG4[g];
    S.Q[g][0] = 0.5 * (1.0 - x);
    S.Q[g][1] = fma(-x, x, 1.0);
    S.Q[g][2] = 0.5 * (1.0 + x);
    S.Qd[g][0] = -0.5;
    S.Qd[g][1] = -2.0 * x;
    S.Qd[g][2] = 0.5;
    S.Lw[g][0] = S.Q[g][0];
    S.Lw[g][1] = S.Q[g][2];
  } else if (tid == 84) {
    S.mat = ixe[NEN];
    S.fail = 0;
    S.any = 0;
  } else if (tid >= 128 && tid < 128 + 4 * NC) {  // no function of a face's centre
    S.C[(tid - 128) >> 2][4 + 6 * (tid & 3)] = 0.0;
  } else if (tid >= 96 && tid < 96 + 4 * NC) {  // nor the line through two
    S.A[0][(tid - 96) >> 2][16 + (tid & 3)] = S.A[1][(tid - 96) >> 2][16 + (tid & 3)] = 0.0;
  }
  if constexpr (OP == kSfRhs4)
    for (int k = tid - 96; k >= 0 && k < 68; k += kSfThreads) S.pf[k] = 0.0;
  __syncthreads();
  if (OP == kSfRhs4 && tid < 7) {
    S.iqm[tid] = ld.eload ? ld.eload[(size_t)7 * (el - 1) + tid] : 0;
    S.iqh[tid] = ld.eloadp ? ld.eloadp[(size_t)7 * (el - 1) + tid] : 0;
    if (S.iqm[tid] > 0 || S.iqh[tid] > 0) S.any = 1;
  }
  if (tid >= 32 && tid < 32 + 12 * NC) sf_edge(S.C[(tid - 32) / 12], (tid - 32) % 12);
  // ---- linear fields, two directions --------------------------------------------
  // (every derivative from the differences of the corners, then interpolated: what is
  // rounded is the field's variation, not the field)
  constexpr int NG = Sm::NG;
  for (int k = tid; k < 32 * (NG + Sm::NVF); k += kSfThreads) {  // (nearly one kind per warp)
    if (k < 16 * NG) {
      const bool dr = k < 8 * NG;
      const int m = dr ? k : k - 8 * NG, f = m >> 3, o = m & 7;
      const double* c = S.lin[f] + 4 * (o >> 2);
      const double* wx = S.Lw[o & 3];
      if (dr)  // d/dr at (z, y)
        S.LB[f][o] = 0.5 * ((c[1] - c[0]) * wx[0] + (c[3] - c[2]) * wx[1]);
      else  // d/ds at (z, x)
        S.LB[f][8 + o] = 0.5 * ((c[2] - c[0]) * wx[0] + (c[3] - c[1]) * wx[1]);
    } else {
      const int m = k - 16 * NG, o = m & 15;
      const double *wx = S.Lw[o & 3], *wy = S.Lw[o >> 2];
      if (m < 16 * NG) {  // d/dt at (y, x)
        const double* c = S.lin[m >> 4];
        S.LB[m >> 4][16 + o] = 0.5 * (((c[4] - c[0]) * wx[0] + (c[5] - c[1]) * wx[1]) * wy[0] +
                                      ((c[6] - c[2]) * wx[0] + (c[7] - c[3]) * wx[1]) * wy[1]);
      } else {  // value at (z, y, x): of the last field, the pass with two also of the first
        const int z = ((m - 16 * NG) >> 4) & 1, v = (m - 16 * NG) >> 5;
        const double* c = S.lin[Sm::NVF == 2 && v == 0 ? 3 : NL - 1] + 4 * z;
        S.LV[v][16 * z + o] =
            (c[0] * wx[0] + c[1] * wx[1]) * wy[0] + (c[2] * wx[0] + c[3] * wx[1]) * wy[1];
      }
    }
  }
  __syncthreads();
  // ---- vector fields: r, then s -----------------------------------------------
  for (int k = tid; k < NC * 32; k += kSfThreads) {
    const int c = k >> 5, l = (k >> 2) & 7, zy = l + (l > 3), x = k & 3;
    const double* v = S.C[c] + 3 * zy;
    S.A[0][c][zy * 4 + x] = v[0] * S.Q[x][0] + v[2] * S.Q[x][2] + v[1] * S.Q[x][1];
    S.A[1][c][zy * 4 + x] = 0.5 * (v[2] - v[0]) + v[1] * S.Qd[x][1];
  }
  // the Jacobian meanwhile: thread (point, coordinate)
  const int g = tid & 63, j = tid >> 6, yx = g & 15, zg = g >> 4;
  const double l0 = S.Lw[zg][0], l1 = S.Lw[zg][1];
  auto grad_lin = [&](int f, double (&n)[3]) {
    const double* b = S.LB[f];
    n[0] = b[yx >> 2] * l0 + b[4 + (yx >> 2)] * l1;
    n[1] = b[8 + (yx & 3)] * l0 + b[12 + (yx & 3)] * l1;
    n[2] = b[16 + yx];
  };
  auto value_lin = [&](int v) { return S.LV[v][yx] * l0 + S.LV[v][16 + yx] * l1; };
  {
    double n[3];
    grad_lin(j, n);
#pragma unroll
    for (int a = 0; a < 3; ++a) S.JI[j][a][g] = n[a];
  }
  __syncthreads();
  for (int k = tid; k < NC * 48; k += kSfThreads) {
    const int c = k / 48, o = k % 48, z = o >> 4, y = (o >> 2) & 3, x = o & 3;
    double br = 0, bs = 0, bt = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double av = S.A[0][c][(3 * z + i) * 4 + x], ad = S.A[1][c][(3 * z + i) * 4 + x];
      br += ad * S.Q[y][i];
      bs += av * S.Qd[y][i];
      bt += av * S.Q[y][i];
    }
    S.B[c][0][o] = br;
    S.B[c][1][o] = bs;
    S.B[c][2][o] = bt;
  }
  // column j of the adjugate; the first two warps also form the determinant
  double ji[3];
  {
    const int j1 = j == 2 ? 0 : j + 1, j2 = j == 0 ? 2 : j - 1;
    double m[3][3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      m[a][0] = S.JI[j][a][g];
      m[a][1] = S.JI[j1][a][g];
      m[a][2] = S.JI[j2][a][g];
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const int p = (a + 1) % 3, q = (a + 2) % 3;
      ji[a] = m[p][1] * m[q][2] - m[p][2] * m[q][1];
    }
    if (j == 0) {
      const double det = m[0][0] * ji[0] + m[1][0] * ji[1] + m[2][0] * ji[2];
      if (!(det > 1.0e-14)) S.fail = 1;
      const double wq = cWG4[g & 3] * cWG4[(g >> 2) & 3] * cWG4[zg];
      S.rd[g] = 1.0 / det;
      S.wq[g] = wq;
      S.w[g] = wq * det;
    }
  }
  __syncthreads();
#pragma unroll
  for (int a = 0; a < 3; ++a) S.JI[j][a][g] = ji[a];
  // natural gradients of component j at the point
  double h[NC / 3][3];
#pragma unroll
  for (int v = 0; v < NC / 3; ++v) {
    const int c = 3 * v + j;
    h[v][0] = h[v][1] = h[v][2] = 0.0;
#pragma unroll
    for (int z = 0; z < 3; ++z) {
      h[v][0] += S.B[c][0][16 * z + yx] * S.Q[zg][z];
      h[v][1] += S.B[c][1][16 * z + yx] * S.Q[zg][z];
      h[v][2] += S.B[c][2][16 * z + yx] * S.Qd[zg][z];
    }
  }
  __syncthreads();
  if (S.fail) {
    if (tid == 0) atomicOr(L.err, 1);
    colour_wait();
    return;
  }
  const double rd = S.rd[g], wq = S.wq[g];
#pragma unroll
  for (int v = 0; v < NC / 3; ++v)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double t = h[v][0] * S.JI[k][0][g] + h[v][1] * S.JI[k][1][g] +
                       h[v][2] * S.JI[k][2][g];
      S.G[3 * v + j][k][g] = Sm::GRAD ? t : rd * t;  // (the contraction scales its sum)
    }
  // physical pressure gradient, component j
  const MatConst mc = L.mat[S.mat - 1];
  const double gj = j == 0 ? L.g0 : j == 1 ? L.g1 : L.g2;
  const double dtk = mc.perm * L.dt;
  double gp;
  {
    double n[3];
    grad_lin(3, n);
    gp = n[0] * ji[0] + n[1] * ji[1] + n[2] * ji[2];  // times det
  }
  // (times the weight alone: det goes into the adjugate that maps it back)
  double gk = 0.0;
  if constexpr (OP == kSfRhs4) {
    S.F[j][g] = wq * dtk * (mc.fluid_d * gj - rd * gp);
  } else if constexpr (OP != kSfGrad) {
    S.F[j][g] = wq * dtk * (rd * gp);
  } else {
    double n[3];
    grad_lin(4, n);
    gk = wq * dtk * gp *
         (rd * (n[0] * ji[0] + n[1] * ji[1] + n[2] * ji[2]) - mc.fluid_d * gj);
  }
  __syncthreads();
  if constexpr (OP == kSfGrad) {
    // row j of the contraction of lam's strain with u_n's stress
    const int j1 = j == 2 ? 0 : j + 1, j2 = j == 0 ? 2 : j - 1;
    const double s =
        (S.G[3 + j][j][g] + mc.b * S.G[3 + j1][j1][g] + mc.b * S.G[3 + j2][j2][g]) * mc.a;
    const double shl = S.G[j][j1][g] + S.G[j1][j][g];
    const double shu = S.G[3 + j][j1][g] + S.G[3 + j1][j][g];
    double v[3] = {-wq * rd * (S.G[j][j][g] * s + mc.c * mc.a * (shl * shu)), gk,
                   j == 0 ? -S.w[g] * mc.imod_biot * value_lin(0) * value_lin(1) : 0.0};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      double x = v[k];
      for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      if (lane == 0) S.gsum[k][tid >> 5] = x;
    }
    __syncthreads();
    colour_wait();
    if (tid < 3) {
      double t = 0.0;
      for (int i = 0; i < kSfThreads / 32; ++i) t += S.gsum[tid][i];
      o0[(size_t)3 * (el - 1) + tid] += t;
    }
    return;
  } else {
    // row j of the weight times the stress, and the sources of the pressure rows
    double q[3];
    {
      const int j1 = j == 2 ? 0 : j + 1, j2 = j == 0 ? 2 : j - 1;
      const double e0 = S.G[j][j][g], e1 = S.G[j1][j1][g], e2 = S.G[j2][j2][g];
      double sn = (e0 + mc.b * e1 + mc.b * e2) * mc.a;
      if constexpr (OP == kSfResidual) {
        const double pg = value_lin(0);
        sn -= mc.coef_biot * pg;
        if (j == 0) S.S0[g] = S.w[g] * (mc.coef_biot * (e0 + e1 + e2) + mc.imod_biot * pg);
      } else if constexpr (OP == kSfRhs4) {
        sn -= mc.coef_biot * value_lin(0);
        if (j == 0) S.body[g] = S.w[g] * mc.pm_d;
      } else if (j == 0) {
        S.S0[g] = S.w[g] * mc.coef_biot * (e0 + e1 + e2);
      }
      const double ca = mc.c * mc.a;
      double st[3];
#pragma unroll
      for (int k = 0; k < 3; ++k)
        st[k] = wq * (k == j ? sn : ca * (S.G[j][k][g] + S.G[k][j][g]));
#pragma unroll
      for (int a = 0; a < 3; ++a)
        q[a] = st[0] * S.JI[0][a][g] + st[1] * S.JI[1][a][g] + st[2] * S.JI[2][a][g];
    }
    // natural pressure flux, component j
    const double fa = S.F[0][g] * S.JI[0][j][g] + S.F[1][g] * S.JI[1][j][g] +
                      S.F[2][g] * S.JI[2][j][g];
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 3; ++a) S.G[j][a][g] = q[a];
    S.F[j][g] = fa;
    __syncthreads();
    // ---- back: t ----------------------------------------------------------------
    const double gl[3] = {L.g0, L.g1, L.g2};
    if (tid < 144) {
      const int c = tid / 48, o = tid % 48, z = o >> 4, p = o & 15;
      double br = 0, bs = 0, bt = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        br += S.G[c][0][16 * k + p] * S.Q[k][z];
        bs += S.G[c][1][16 * k + p] * S.Q[k][z];
        bt += S.G[c][2][16 * k + p] * S.Qd[k][z];
        if constexpr (OP == kSfRhs4) bt -= S.body[16 * k + p] * gl[c] * S.Q[k][z];
      }
      S.B[c][0][o] = br;
      S.B[c][1][o] = bs;
      S.B[c][2][o] = bt;
    } else if (tid >= 160) {  // pressure rows: (z, yx)
      const int o = tid - 160, z = o >> 4, p = o & 15;
      const double dz = z ? 0.5 : -0.5;
      double tr = 0, ts = 0, tv = 0, t2 = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        tr += S.F[0][16 * k + p] * S.Lw[k][z];
        ts += S.F[1][16 * k + p] * S.Lw[k][z];
        tv += S.F[2][16 * k + p] * dz;
        if (OP == kSfResidual) tv += S.S0[16 * k + p] * S.Lw[k][z];
        if (OP == kSfApply) t2 += S.S0[16 * k + p] * S.Lw[k][z];
      }
      S.LT[0][0][o] = tr;
      S.LT[0][1][o] = ts;
      S.LT[0][2][o] = tv;
      if (OP == kSfApply) S.LT[1][2][o] = t2;
    }
    __syncthreads();
    // ---- back: s ----------------------------------------------------------------
    if constexpr (OP == kSfRhs4)
      if (S.any && tid >= 128 && tid < 160) {  // (G is read)
        if (hexa_face_loads(L, ld, S.iqm, S.iqh, S.lin, S.pf, &S.G[0][0][0], lane) &&
            lane == 0)
          S.fail = 1;
      }
    if (tid < 96) {
      const int c = tid >> 5, l = (tid >> 2) & 7, zy = l + (l > 3), x = tid & 3;
      const int z = zy / 3, k = zy % 3;
      double v = 0, d = 0;
#pragma unroll
      for (int y = 0; y < 4; ++y) {
        const int o = 16 * z + 4 * y + x;
        v += S.B[c][1][o] * S.Qd[y][k] + S.B[c][2][o] * S.Q[y][k];
        d += S.B[c][0][o] * S.Q[y][k];
      }
      S.A[0][c][zy * 4 + x] = v;
      S.A[1][c][zy * 4 + x] = d;
    } else if (tid >= 160 && tid < 176) {
      const int o = tid - 160, z = o >> 3, k = (o >> 2) & 1, x = o & 3;
      const double dy = k ? 0.5 : -0.5;
      double v = 0, d = 0, v2 = 0;
#pragma unroll
      for (int y = 0; y < 4; ++y) {
        const int p = 16 * z + 4 * y + x;
        v += S.LT[0][1][p] * dy + S.LT[0][2][p] * S.Lw[y][k];
        d += S.LT[0][0][p] * S.Lw[y][k];
        if (OP == kSfApply) v2 += S.LT[1][2][p] * S.Lw[y][k];
      }
      S.T2[0][o] = v;
      S.T2[0][16 + o] = d;
      if (OP == kSfApply) S.T2[1][o] = v2;
    }
    __syncthreads();
    // ---- back: r ----------------------------------------------------------------
    if (tid < 60) {
      const int c = tid / 20, i = cGrid27[tid % 20], zy = i / 3, k = i % 3;
      double v = 0;
#pragma unroll
      for (int x = 0; x < 4; ++x)
        v += S.A[0][c][zy * 4 + x] * S.Q[x][k] + S.A[1][c][zy * 4 + x] * S.Qd[x][k];
      S.C[c][i] = v;
    } else if (tid >= 160 && tid < 168) {
      const int i = tid - 160, zy = i >> 1, k = i & 1;
      const double dx = k ? 0.5 : -0.5;
      double v = 0, v2 = 0;
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        v += S.T2[0][zy * 4 + x] * S.Lw[x][k] + S.T2[0][16 + zy * 4 + x] * dx;
        if (OP == kSfApply) v2 += S.T2[1][zy * 4 + x] * S.Lw[x][k];
      }
      S.out[60 + i] = v;
      if (OP == kSfApply) S.out2[i] = v2;
    }
    __syncthreads();
    colour_wait();
    if (OP == kSfRhs4 && S.fail) {
      if (tid == 0) atomicOr(L.err, 1);
      return;
    }
    if (tid < 60) {
      double acc = sf_fold(S.C[tid % 3], tid / 3);
      if constexpr (OP == kSfRhs4) acc += S.pf[tid];
      const int e = eq_of(L, S.nodes[tid / 3], tid % 3);
      if (e > 0) o0[e - 1] -= acc;
    } else if (tid < 68) {
      const int l = tid - 60, i = cGrid8[l];
      const int e = eq_of(L, S.nodes[l], 3);
      if (e > 0) {
        if constexpr (OP == kSfRhs4) o0[e - 1] -= S.out[60 + i] + S.pf[tid];
        else o0[e - 1] += S.out[60 + i];
        if (OP == kSfApply) o1[e - 1] += S.out2[i];
      }
    }
  }
}

// isw 3 (MODE 3) and the porosity change (MODE 7) at the 8 vertices (see k_vertex_tetra):
// there the derivative along a direction is that of the edge's three nodes, and the
// Jacobian's row half the edge.  A warp per element, thread (vertex, coordinate); the
// latency of one element bounds it.  The 20 functions' derivatives by a thread per
// vertex took 33 us a launch on the 2 x 2 x 40 column.
constexpr int kHvWarps = 4;
struct SmHv {
  double c[3][27];  // displacements on the 3 x 3 x 3 grid
  double l[4][8];   // coordinates, pressure
  double J[3][3][8];
  double G[3][3][8];
};
struct SmHvs {
  SmHv warp[kHvWarps];
};

template <int MODE>
__global__ void __launch_bounds__(32 * kHvWarps)
    k_hexa_vertex(ElemLaunch L, const double* __restrict__ u, const double* __restrict__ dp,
                  double* __restrict__ tx, double* __restrict__ txb,
                  double* __restrict__ flux) {
  constexpr int NEN = 20;
  extern __shared__ __align__(16) unsigned char smem[];
  SmHv& S = reinterpret_cast<SmHvs*>(smem)->warp[threadIdx.x >> 5];
  colour_next();
  const int lane = threadIdx.x & 31;
  const int ie = blockIdx.x * kHvWarps + (threadIdx.x >> 5);
  if (ie >= L.nelem) {
    colour_wait();
    return;
  }
  const int32_t* ixe = L.ix + (size_t)(NEN + 1) * (L.elems[ie] - 1);
  for (int k = lane; k < 3 * NEN; k += 32)
    S.c[k % 3][cGrid27[k / 3]] = u[(size_t)kNdf * (ixe[k / 3] - 1) + k % 3];
  {
    const int n = ixe[lane >> 2] - 1, q = lane & 3;
    S.l[q][cGrid8[lane >> 2]] = q < 3 ? L.x[(size_t)3 * n + q] : u[(size_t)kNdf * n + 3];
  }
  const MatConst mc = L.mat[ixe[NEN] - 1];
  __syncwarp();
  // vertex i at corner g of the grid (bit a: side of direction a), coordinate j;
  // lanes 24..31 repeat coordinate 2
  const int i = lane & 7, j = min(lane >> 3, 2), g = cGrid8[i];
  const int no = ixe[i] - 1;
  double h[3], hp[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int st = a == 0 ? 1 : a == 1 ? 3 : 9, up = (g >> a) & 1;
    const int o = 2 * ((g & 1) + 3 * ((g >> 1) & 1) + 9 * (g >> 2));
    const double* c = S.c[j];
    const double own = c[o], mid = c[up ? o - st : o + st], opp = c[up ? o - 2 * st : o + 2 * st];
    const double d = 2.0 * (own - mid) - 0.5 * (own - opp);
    h[a] = up ? d : -d;
    const int lo = g & ~(1 << a), hi = lo | (1 << a);
    S.J[j][a][i] = 0.5 * (S.l[j][hi] - S.l[j][lo]);
    hp[a] = 0.5 * (S.l[3][hi] - S.l[3][lo]);
  }
  __syncwarp();
  const int j1 = j == 2 ? 0 : j + 1, j2 = j == 0 ? 2 : j - 1;
  double ji[3], det = 0.0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int p = (a + 1) % 3, q = (a + 2) % 3;
    ji[a] = S.J[j1][p][i] * S.J[j2][q][i] - S.J[j2][p][i] * S.J[j1][q][i];
    det += S.J[j][a][i] * ji[a];
  }
  if (__any_sync(0xffffffffu, !(det > 1.0e-14))) {
    if (lane == 0) atomicOr(L.err, 1);
    colour_wait();
    return;
  }
  const double rd = 1.0 / det;
  if constexpr (MODE == 7) {
    // tx is the porosity change accumulator here
    const double e = rd * (h[0] * ji[0] + h[1] * ji[1] + h[2] * ji[2]);
    const double e1 = __shfl_sync(0xffffffffu, e, i + 8), e2 = __shfl_sync(0xffffffffu, e, i + 16);
    colour_wait();
    if (lane < 8) tx[no] += mc.coef_biot * (e + e1 + e2) + mc.imod_biot * S.l[3][g];
  } else {
    __syncwarp();
    // (lanes 24..31 write what lanes 16..23 do)
#pragma unroll
    for (int a = 0; a < 3; ++a) S.J[j][a][i] = ji[a];
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 3; ++k)
      S.G[j][k][i] =
          rd * (h[0] * S.J[k][0][i] + h[1] * S.J[k][1][i] + h[2] * S.J[k][2][i]);
    const double gj = j == 0 ? L.g0 : j == 1 ? L.g1 : L.g2;
    const double f =
        mc.perm * (mc.fluid_d * gj - rd * (hp[0] * ji[0] + hp[1] * ji[1] + hp[2] * ji[2]));
    __syncwarp();
    const double sn = (S.G[j][j][i] + mc.b * S.G[j1][j1][i] + mc.b * S.G[j2][j2][i]) * mc.a -
                      mc.coef_biot * dp[no];
    const double sh = (S.G[j][j1][i] + S.G[j1][j][i]) * mc.c * mc.a;
    colour_wait();
    if (lane < 24) {  // components xx yy zz xy yz zx
      double* T6 = tx + (size_t)6 * no;
      double* B6 = txb + (size_t)6 * no;
      T6[j] += sn;
      B6[j] += sn + mc.coef_biot * S.l[3][g];
      T6[3 + j] += sh;
      B6[3 + j] += sh;
      flux[(size_t)3 * no + j] += f;
    }
  }
}
