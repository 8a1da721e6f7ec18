// pm_hexa_mma.h -- hexa20 element matrices on the FP16 tensor pipe, as accurate as
// FP64 sums (included by pm_elements.cu inside its unnamed namespace).
//
// What bounds it.  All the matrix needs from the 64 points are the products
//   P(r, c) = sum_g X_r(g) X_c(g)
// of 92 rows X: sqrt(w) dN_i/dx_k (60), sqrt(w) Np_l (8) and
// sqrt(w) dNp_l/dx_k (24).  With DFMA that contraction is most of the element
// (117,000 clocks of an SM per element, at 1.7 DFMA per clock), and FP64 tensor
// instructions are no faster here.  mma.sync with FP16 operands and FP32 sums
// does 1,017 multiply-adds per clock and SM (measured; int8 252).
//
// Split.  Each X is a 54-bit integer q (every value within a factor 2 of its row's
// largest is held exactly, smaller ones to 2^-54 of it), cut into
// 7 balanced base-256 digits (Ozaki, Ogita, Oishi and Rump, "Error-free
// transformations of matrix multiplication", Numer. Algorithms 59, 2012).
// Digits are exact in FP16, their products are at most 2^14, and the sums
// of all pairs s + t = d over 64 points stay below 2^23: exact in FP32.  The
// 34 pairs with s + t <= 7 are kept; the dropped ones are 2^-59 of the largest
// product, the final 64-bit integer's last place 2^-54 to 2^-56.  (Without s + t = 7
// the entries' error against 64 bits was 1.6 times that of the DFMA sums.)
//
// Error.  Every row has its own exponent, so the error of P(r, c) is relative to
// sqrt(P(r, r) P(c, c)) whatever the element's shape: at most 1.4e-16 of it, where
// FP64 sums have up to 1.3e-15, on cubes, jittered elements and thicknesses that
// taper from 1 to 1e-1 .. 1e-6 between opposite corners.  (With one exponent for all
// derivatives of a direction, and a last place of 2^-50 to 2^-52, it was 1.4e-14 at
// 1e-2 and 7e-12 at 1e-4.)
//
// Per element: 256 threads (geometry: 4 threads per point, then 28 tiles of
// 16 x 8 over 8 warps, then a node pair per thread), two elements per SM.
// Measured (assembly with the fused product, 40^3 cube, 64,000 elements): 10.1 ms
// against 28.0 ms with DFMA sums (64 threads per element); a launch of 20
// elements (2 x 2 x 40 column) 32 us against 184 us.  FP64 pipe 48 % busy: the
// geometry, the blocks and the panel adds; the rest is the phases' latency with
// two elements per SM: 97 KB of digits each, and 128 registers a thread, either of
// which alone keeps a third out.
constexpr int kHxThreads = 256;
constexpr int kHxRows = 96;     // 0..59 u, 60..67 Np, 68..71 zero, 72 + 8 k + l grad Np
constexpr int kHxStride = 72;   // halves per digit row of 64 points: no bank conflicts
constexpr int kHxDig = 7;
constexpr int kHxSum = 8;       // digit pairs kept: s + t < kHxSum
constexpr int kHxPs = 69;       // doubles per row of P
constexpr int kHxBad = 1 << 14; // exponent of a row with a value that is not finite
constexpr int kHxSlots = 28;    // product slots per row: 20 nodes, 8 vertices

struct SmHx {
  union {
    unsigned short dig[kHxDig][kHxRows][kHxStride];
    struct {
      double P[64][kHxPs];         // rows 0..63, columns >= the row's block
      double mass[4][4];           // Np 4..7
      double grad[3][8][8];        // per direction
      double C[68][kHxSlots];      // K_e u_e, one slot per block
      double Cs[68][4];
    } r;
  };
  double J[64][9];                 // dx_j/dr_a, then sqrt(w) times its inverse
  double sw[64];
  double xv[8][3];
  double ul[68];
  int nodes[20], mat;
  int eq[20][kNdf], e0[20], W[20];
  int64_t off[20];
  int em[kHxRows];                 // largest exponent of each row
  int fail;
};

__device__ __forceinline__ int hx_exp(double v) { return (__double2hiint(v) >> 20) & 0x7ff; }

// The 7 digits of v (exponent em at the top) as FP16 numbers, most significant
// first, into d[0 .. 6] planes apart: m 2^1 >> (em - e), signed, rounded.
__device__ __forceinline__ void hx_digits(double v, int em, unsigned short* d) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  int e = (int)(b >> 52) & 0x7ff;
  unsigned long long m = b & 0xfffffffffffffull;
  if (e) m |= 0x10000000000000ull;
  else e = 1;
  const int sh = min(em - e, 60);
  m <<= 1;
  if (sh > 0) m = (m + (1ull << (sh - 1))) >> sh;
  // biased bytes: q + 0x80..80, carries included
  const unsigned long long neg = (long long)b < 0 ? ~0ull : 0ull;
  const unsigned long long t = (m ^ neg) - neg + 0x0080808080808080ull;
  const unsigned lo = (unsigned)t, hi = (unsigned)(t >> 32);
  // byte y -> FP16 1024 + y, less 1152
  const __half2 bias = __half2half2(__ushort_as_half(0x6480));
  auto two = [&](unsigned w, unsigned sel) {
    unsigned h = __byte_perm(w, 0x64646464u, sel);
    const __half2 r = __hsub2(*reinterpret_cast<__half2*>(&h), bias);
    return *reinterpret_cast<const unsigned*>(&r);
  };
  constexpr int plane = kHxRows * kHxStride;
  const unsigned h65 = two(hi, 0x4142), h43 = two(hi, 0x4340), l32 = two(lo, 0x4243),
                 l10 = two(lo, 0x4041);
  d[0 * plane] = (unsigned short)h65;          // byte 6
  d[1 * plane] = (unsigned short)(h65 >> 16);  // byte 5
  d[2 * plane] = (unsigned short)h43;          // byte 4
  d[3 * plane] = (unsigned short)l32;          // byte 3
  d[4 * plane] = (unsigned short)(l32 >> 16);  // byte 2
  d[5 * plane] = (unsigned short)l10;          // byte 1
  d[6 * plane] = (unsigned short)(l10 >> 16);  // byte 0
}

__device__ __forceinline__ void hx_ldsm(unsigned (&r)[4], const unsigned short* p) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a));
}

// Rows ra .. ra + 15 times rows rb .. rb + 7 over the 64 points: the lane's
// four entries (row g, g, g + 8, g + 8 with g = lane / 4; column 2 (lane % 4),
// + 1, ...) as integers below 2^62 in units of 2^52 of q q.
__device__ __forceinline__ void hx_tile(const SmHx& S, int ra, int rb, int lane,
                                        long long (&out)[4]) {
  float acc[kHxSum][4];
#pragma unroll
  for (int d = 0; d < kHxSum; ++d)
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[d][k] = 0.f;
#pragma unroll 1
  for (int kk = 0; kk < 64; kk += 32) {
    unsigned b[kHxDig][4];
#pragma unroll
    for (int s = 0; s < kHxDig; ++s)
      hx_ldsm(b[s], &S.dig[s][rb + (lane & 7)][kk + (lane >> 3) * 8]);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
      for (int s = 0; s < kHxDig; ++s) {
        unsigned a[4];
        hx_ldsm(a, &S.dig[s][ra + (lane & 15)][kk + 16 * h + (lane >> 4) * 8]);
#pragma unroll
        for (int t = 0; t < kHxDig && t + s < kHxSum; ++t)
          asm volatile(
              "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3},"
              "{%4,%5,%6,%7},{%8,%9},{%0,%1,%2,%3};"
              : "+f"(acc[s + t][0]), "+f"(acc[s + t][1]), "+f"(acc[s + t][2]), "+f"(acc[s + t][3])
              : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[t][2 * h]),
                "r"(b[t][2 * h + 1]));
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    // weights 16 256^(5 - d), d = 6 and 7 rounded to the last place
    const long long hi = ((long long)__float2int_rn(acc[0][k]) << 16) +
                         ((long long)__float2int_rn(acc[1][k]) << 8) +
                         __float2int_rn(acc[2][k]);
    const long long lo = ((long long)__float2int_rn(acc[3][k]) << 16) +
                         ((long long)__float2int_rn(acc[4][k]) << 8) +
                         __float2int_rn(acc[5][k]);
    const int tail = __float2int_rn(acc[6][k]) + ((__float2int_rn(acc[7][k]) + 128) >> 8);
    out[k] = (((hi << 24) + lo) << 4) + ((tail + 8) >> 4);
  }
}

// An integer of hx_tile as the sum it stands for, v 2^(52 + ea + eb - 2 * 1076):
// one conversion, the power of two added to the exponent field; NaN for a bad row.
__device__ __forceinline__ double hx_value(long long v, int ea, int eb) {
  const int e = ea + eb - 2100;
  double d = double(v);  // 0 or 2^0 .. 2^62
  if (abs(e) < 900) {
    const int hi = __double2hiint(d);
    return v == 0 ? d : __hiloint2double(hi + (e << 20), __double2loint(d));
  }
  if (max(ea, eb) >= kHxBad) return __longlong_as_double(0x7ff8000000000000ll);
  const int e1 = max(-1022, min(1023, e)), e2 = max(-1022, min(1023, e - e1));
  return d * __longlong_as_double((long long)(e1 + 1023) << 52) *
         __longlong_as_double((long long)(e2 + 1023) << 52);
}

// Element matrix into the panels; with RHS also b -= K_e u_e from the same
// blocks (p = s.u, the product the reference forms in lku for isw 2 with
// rhs).  The product is deterministic: every block writes its share of a row
// into a slot of its own (row r of the element vector: slot j for node j's u
// columns, slot 20 + l for vertex l's p column) and each row sums its slots in
// order.
template <bool RHS>
__global__ void __launch_bounds__(kHxThreads, 2)
    k_assemble_hexa(ElemLaunch L, double* __restrict__ val, const double* __restrict__ u,
                    double* __restrict__ bvec) {
  constexpr int NEN = 20, NV = 8;
  extern __shared__ __align__(16) unsigned char smem[];
  SmHx& S = *reinterpret_cast<SmHx*>(smem);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  colour_next();
  const int el = L.elems[blockIdx.x];
  const int32_t* ixe = L.ix + (size_t)(NEN + 1) * (el - 1);
  // ---- element data ---------------------------------------------------------
  if (tid <= NEN) {
    const int n = ixe[tid];
    if (tid < NEN) {
      S.nodes[tid] = n;
      int e0 = 0x7fffffff;
      for (int q = 0; q < kNdf; ++q) {
        const int e = eq_of(L, n, q);
        S.eq[tid][q] = e;
        if (e > 0 && e < e0) e0 = e;
      }
      S.e0[tid] = e0;
      S.off[tid] = L.node_val_off[n - 1];
      S.W[tid] = L.node_W[n - 1];
    } else {
      S.mat = n;
    }
  }
  if (tid >= 32 && tid < 32 + 3 * NV) {
    const int k = tid - 32;
    S.xv[k / 3][k % 3] = L.x[(size_t)3 * (ixe[k / 3] - 1) + k % 3];
  }
  if (tid >= 64 && tid < 64 + kHxRows) S.em[tid - 64] = 1;
  if (tid == 255) S.fail = 0;
  // rows 68..71 are read with the row tiles around them
  for (int k = tid; k < kHxDig * 4 * 32; k += kHxThreads) {
    const int s = k >> 7, r = (k >> 5) & 3, c = k & 31;
    *reinterpret_cast<unsigned*>(&S.dig[s][68 + r][2 * c]) = 0u;
  }
  if (RHS && tid >= 128 && tid < 128 + 68) {
    const int k = tid - 128;
    const int n = ixe[k < 3 * NEN ? k / 3 : k - 3 * NEN], q = k < 3 * NEN ? k % 3 : 3;
    S.ul[k] = u[(size_t)kNdf * (n - 1) + q];
  }
  __syncthreads();
  // ---- geometry of the points -------------------------------------------------
  const int gq = tid & 63, part = tid >> 6;
  const double* tb = gShapeHexa + gq;
  auto tab = [tb](int row) { return __ldg(tb + row * kHexaGp); };
  if (part < 3) {  // column part of the Jacobian
    double a0 = 0, a1 = 0, a2 = 0;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const double xk = S.xv[k][part];
      a0 += tab(kTabH8 + 8 + k) * xk;
      a1 += tab(kTabH8 + 16 + k) * xk;
      a2 += tab(kTabH8 + 24 + k) * xk;
    }
    S.J[gq][part] = a0;
    S.J[gq][3 + part] = a1;
    S.J[gq][6 + part] = a2;
  }
  __syncthreads();
  if (part == 0) {
    double* Jp = S.J[gq];
    const double J00 = Jp[0], J01 = Jp[1], J02 = Jp[2], J10 = Jp[3], J11 = Jp[4], J12 = Jp[5],
                 J20 = Jp[6], J21 = Jp[7], J22 = Jp[8];
    const double det = J00 * J11 * J22 + J01 * J12 * J20 + J02 * J10 * J21 - J20 * J11 * J02 -
                       J10 * J01 * J22 - J00 * J21 * J12;
    if (!(det > 1.0e-14)) {
      S.fail = 1;
    } else {
      const int lz = gq >> 4, ly = (gq >> 2) & 3, lx = gq & 3;
      const double sw = sqrt(cWG4[lx] * cWG4[ly] * cWG4[lz] * det);
      const double f = (1.0 / det) * sw;
      S.sw[gq] = sw;
      Jp[0] = (J11 * J22 - J12 * J21) * f;
      Jp[3] = -(J10 * J22 - J12 * J20) * f;
      Jp[6] = (J10 * J21 - J11 * J20) * f;
      Jp[1] = -(J01 * J22 - J02 * J21) * f;
      Jp[4] = (J00 * J22 - J02 * J20) * f;
      Jp[7] = -(J00 * J21 - J01 * J20) * f;
      Jp[2] = (J01 * J12 - J02 * J11) * f;
      Jp[5] = -(J00 * J12 - J02 * J10) * f;
      Jp[8] = (J00 * J11 - J01 * J10) * f;
    }
  }
  __syncthreads();
  if (S.fail) {
    if (tid == 0) atomicOr(L.err, 1);
    colour_wait();
    return;
  }
  {
    // 5 nodes and 2 vertices of one point per thread
    double v[7][3], np[2];
    {
      double Ji[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) Ji[k] = S.J[gq][k];
#pragma unroll
      for (int k = 0; k < 7; ++k) {
        const int i = part * 5 + k, l = part * 2 + k - 5;
        const double tr = k < 5 ? tab(kTabH20D + i) : tab(kTabH8 + 8 + l);
        const double ts = k < 5 ? tab(kTabH20D + 20 + i) : tab(kTabH8 + 16 + l);
        const double tt = k < 5 ? tab(kTabH20D + 40 + i) : tab(kTabH8 + 24 + l);
#pragma unroll
        for (int j = 0; j < 3; ++j)
          v[k][j] = Ji[3 * j] * tr + Ji[3 * j + 1] * ts + Ji[3 * j + 2] * tt;
      }
    }
    const double sw = S.sw[gq];
    np[0] = tab(kTabH8 + part * 2) * sw;
    np[1] = tab(kTabH8 + part * 2 + 1) * sw;
    auto row_of = [part](int k, int j) {
      return k < 5 ? 3 * (part * 5 + k) + j : 72 + 8 * j + part * 2 + k - 5;
    };
    // lane 3 k + j keeps the warp's largest exponent of row (k, j), lanes 21 and 22 of Np
    int mine = 0;
#pragma unroll
    for (int k = 0; k < 23; ++k) {
      const int e = __reduce_max_sync(0xffffffffu, hx_exp(k < 21 ? v[k / 3][k % 3] : np[k - 21]));
      mine = lane == k ? e : mine;
    }
    if (lane < 23)
      atomicMax(&S.em[lane < 21 ? row_of(lane / 3, lane % 3) : 60 + part * 2 + lane - 21],
                mine == 0x7ff ? kHxBad : mine);
    __syncthreads();
    // (all read before the first digit is stored: the compiler keeps their order)
    int em[23];
#pragma unroll
    for (int k = 0; k < 23; ++k)
      em[k] = S.em[k < 21 ? row_of(k / 3, k % 3) : 60 + part * 2 + k - 21];
#pragma unroll
    for (int k = 0; k < 23; ++k) {
      const int row = k < 21 ? row_of(k / 3, k % 3) : 60 + part * 2 + k - 21;
      hx_digits(k < 21 ? v[k / 3][k % 3] : np[k - 21], em[k], &S.dig[0][row][gq]);
    }
  }
  __syncthreads();
  // ---- the products -------------------------------------------------------------
  // tiles 0..23: (16 I, 8 J), J >= 2 I, J <= 8; 24: Np 4..7; 25..27: grad Np
  constexpr int kTiles = 28, kPer = (kTiles + 7) / 8;
  long long res[kPer][4];
  int er[kPer][2], ec[kPer][2];  // their rows' and columns' exponents
  auto where = [](int t, int& ra, int& rb) {
    if (t < 9) { ra = 0; rb = 8 * t; }
    else if (t < 16) { ra = 16; rb = 8 * (t - 7); }
    else if (t < 21) { ra = 32; rb = 8 * (t - 12); }
    else if (t < 24) { ra = 48; rb = 8 * (t - 15); }
    else if (t == 24) { ra = 64; rb = 64; }
    else { ra = t == 25 ? 64 : 80; rb = 72 + 8 * (t - 25); }
  };
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const int t = wid + 8 * q;
    if (t < kTiles) {
      int ra, rb;
      where(t, ra, rb);
      hx_tile(S, ra, rb, lane, res[q]);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        er[q][k] = S.em[ra + (lane >> 2) + 8 * k];
        ec[q][k] = S.em[rb + 2 * (lane & 3) + k];
      }
    }
  }
  __syncthreads();  // the digits are read: their space takes the sums
  {
    auto& R = S.r;
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      const int t = wid + 8 * q;
      if (t >= kTiles) continue;
      int ra, rb;
      where(t, ra, rb);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int row = ra + (lane >> 2) + 8 * (k >> 1), col = rb + 2 * (lane & 3) + (k & 1);
        const double d = hx_value(res[q][k], er[q][k >> 1], ec[q][k & 1]);
        if (t < 24) {
          if (col < 68) R.P[row][col] = d;
        } else if (t == 24) {
          if (row < 68 && col < 68) R.mass[row - 64][col - 64] = d;
        } else {
          const int l = row - (72 + 8 * (t - 25));
          if (l >= 0 && l < 8) R.grad[t - 25][l][col - rb] = d;
        }
      }
    }
  }
  __syncthreads();
  colour_wait();
  // ---- blocks of the element matrix ---------------------------------------------
  const MatConst mc = L.mat[S.mat - 1];
  const int32_t* slot = L.slot + (size_t)NEN * NEN * blockIdx.x;
  const double* ul = S.ul;
  auto& R = S.r;
  constexpr int NUU = NEN * (NEN + 1) / 2, NPU = NV * NEN, NPP = NV * (NV + 1) / 2;
  for (int task = tid; task < NUU + NPU + NPP; task += kHxThreads) {
    if (task < NUU) {
      // Kuu: node pair (i >= j)
      int i = int((sqrtf(8.0f * task + 1.0f) - 1.0f) * 0.5f);
      while ((i + 1) * (i + 2) / 2 <= task) ++i;
      while (i * (i + 1) / 2 > task) --i;
      const int j = task - i * (i + 1) / 2;
      double P[3][3];
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int l = 0; l < 3; ++l) {
          const int r = 3 * i + k, c = 3 * j + l;
          P[k][l] = R.P[min(r, c)][max(r, c)];
        }
      const double a = mc.a, b = mc.b, c = mc.c;
      const double tr = P[0][0] + P[1][1] + P[2][2];
      double K[3][3];
      // (explicit roundings: the same panels with and without RHS)
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int l = 0; l < 3; ++l)
          K[k][l] = __dmul_rn(a, (k == l) ? fma(c, tr - P[k][k], P[k][k])
                                          : fma(b, P[k][l], __dmul_rn(c, P[l][k])));
      if (RHS) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          R.C[3 * i + k][j] =
              K[k][0] * ul[3 * j] + K[k][1] * ul[3 * j + 1] + K[k][2] * ul[3 * j + 2];
          if (i != j)
            R.C[3 * j + k][i] =
                K[0][k] * ul[3 * i] + K[1][k] * ul[3 * i + 1] + K[2][k] * ul[3 * i + 2];
        }
      }
      // the panel entries, read together (one latency, not one per entry):
      // (k, l) in node i's rows and, for i != j, transposed in node j's
      const int sij = slot[i * NEN + j] - S.e0[j], sji = slot[j * NEN + i] - S.e0[i];
      double* pi[3][3];
      double* pj[3][3];
      double vi[3][3], vj[3][3];
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int l = 0; l < 3; ++l) {
          const int er = S.eq[i][k], ec = S.eq[j][l];
          const bool on = er != 0 && ec != 0;
          pi[k][l] = on ? val + S.off[i] + (int64_t)(er - S.e0[i]) * S.W[i] + sij + ec : nullptr;
          pj[k][l] = on && i != j
                         ? val + S.off[j] + (int64_t)(ec - S.e0[j]) * S.W[j] + sji + er
                         : nullptr;
          vi[k][l] = pi[k][l] ? *pi[k][l] : 0.0;
          vj[k][l] = pj[k][l] ? *pj[k][l] : 0.0;
        }
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int l = 0; l < 3; ++l) {
          if (pi[k][l]) *pi[k][l] = __dadd_rn(vi[k][l], K[k][l]);
          if (pj[k][l]) *pj[k][l] = __dadd_rn(vj[k][l], K[k][l]);
        }
    } else if (task < NUU + NPU) {
      // Kpu / Kup: vertex l, node j
      const int l = (task - NUU) / NEN, j = (task - NUU) % NEN;
      double Kv[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) Kv[k] = __dmul_rn(-mc.coef_biot, R.P[3 * j + k][60 + l]);
      if (RHS) {
        const double pl = ul[3 * NEN + l];
        R.C[3 * NEN + l][j] =
            Kv[0] * ul[3 * j] + Kv[1] * ul[3 * j + 1] + Kv[2] * ul[3 * j + 2];
#pragma unroll
        for (int k = 0; k < 3; ++k) R.C[3 * j + k][NEN + l] = Kv[k] * pl;
      }
      const int er = S.eq[l][3];
      if (er == 0) continue;
      double* rowl =
          val + S.off[l] + (int64_t)(er - S.e0[l]) * S.W[l] + slot[l * NEN + j] - S.e0[j];
      double* colj = val + S.off[j] + slot[j * NEN + l] - S.e0[l] + er;
      double vl[3], vj[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const int ec = S.eq[j][k];
        vl[k] = ec ? rowl[ec] : 0.0;
        vj[k] = ec ? colj[(int64_t)(ec - S.e0[j]) * S.W[j]] : 0.0;
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const int ec = S.eq[j][k];
        if (ec == 0) continue;
        rowl[ec] = __dadd_rn(vl[k], Kv[k]);
        colj[(int64_t)(ec - S.e0[j]) * S.W[j]] = __dadd_rn(vj[k], Kv[k]);
      }
    } else {
      // Kpp: vertex pair (l >= m)
      const int pr = task - NUU - NPU;
      int l = 0;
      while ((l + 1) * (l + 2) / 2 <= pr) ++l;
      const int m = pr - l * (l + 1) / 2;
      const double am = m < 4 ? R.P[60 + m][60 + l] : R.mass[m - 4][l - 4];
      const double ak = R.grad[0][l][m] + R.grad[1][l][m] + R.grad[2][l][m];
      const double acc = fma(mc.imod_biot, am, __dmul_rn(mc.perm * L.dt, ak));
      if (RHS) {
        R.C[3 * NEN + l][NEN + m] = -acc * ul[3 * NEN + m];
        if (l != m) R.C[3 * NEN + m][NEN + l] = -acc * ul[3 * NEN + l];
      }
      const int er = S.eq[l][3], ec = S.eq[m][3];
      if (er == 0 || ec == 0) continue;
      val[S.off[l] + (int64_t)(er - S.e0[l]) * S.W[l] + slot[l * NEN + m] - S.e0[m] + ec] += -acc;
      if (l != m)
        val[S.off[m] + (int64_t)(ec - S.e0[m]) * S.W[m] + slot[m * NEN + l] - S.e0[l] + er] +=
            -acc;
    }
  }
  if (RHS) {
    __syncthreads();
    for (int k = tid; k < 4 * 68; k += kHxThreads) {
      const int r = k >> 2, q = (k & 3) * (kHxSlots / 4);
      double s = 0.0;
#pragma unroll
      for (int i = 0; i < kHxSlots / 4; ++i) s += R.C[r][q + i];
      R.Cs[r][k & 3] = s;
    }
    __syncthreads();
    if (tid < 68) {
      const int e = tid < 3 * NEN ? S.eq[tid / 3][tid % 3] : S.eq[tid - 3 * NEN][3];
      if (e > 0) bvec[e - 1] -= (R.Cs[tid][0] + R.Cs[tid][1]) + (R.Cs[tid][2] + R.Cs[tid][3]);
    }
  }
}
