// Apply on uniform lattices with constant coefficients as a sum of line
// products (the vmult of heat_diffuse_operator.cpp:179-197 and
// advection_diffusion_operator.cpp:238-272 on an axis-aligned box).  Included
// by operator_kernels.cu after apply_warp.cuh.
//
// On such a lattice every term of the operator, integrated by the tensor
// quadrature, is a product of matrices along x, y and z that are block-banded
// sums of (P+1)^2 element matrices:
//   A u = Mz [My X1 + Y2 Mx] u + Z2 [My Mx] u
// with M mass, X1 = c_m M + c_d K + c_v u_x A, Y2 = c_d K + c_v u_y A, Z2 alike
// (K stiffness, A advection of a constant velocity).  The vortex and the
// rotation are products along the axes too:
//   vortex    + Mz [My(cos) X(sin A) - Y(sin A) Mx(cos)] u
//   rotation  + Mz(z) [My Ax] u - Az [My Mx(x)] u        (times c_v w)
// so a DoF costs 7 (P+1)^2 / P multiply-adds (Q2 32, Q4 44) where the cell-wise
// sum factorisation took 150 for Q2, every DoF is computed by one thread, no
// cell colouring is needed and dst is written once.
//
// Layout and schedule: a warp owns a strip of the lattice -- up to 60 columns
// along x and one y-unit, a unit being a vertex and the P-1 nodes after it --
// and marches along z, without any block barrier.
//  1. lane = two columns: loads the 2P+1 rows of the y-unit (coalesced along x;
//     the next planes' while these are computed), applies the y matrices in
//     registers, stores the results as pairs in the warp's shared memory;
//  2. lane = two (x-unit, row) slots: applies the x matrices to the slot's 2P+1
//     pairs, then adds the plane to its z accumulators, element by element: a
//     layer's lower planes are complete when its last plane has been added,
//     and that plane opens the next layer's accumulators;
//  3. a finished layer goes through shared memory to coalesced stores.
// Element matrices are kernel parameters (constant-bank operands); a lane applies
// each to two columns or slots of up to two planes.  A vertex adds the last row of
// the element before it and the first row of its own; at the ends of an axis
// the missing one reads zeros.
// A chunk of layers that starts above the bottom first adds the layer below it.
//
// Bound: instruction issue and the FP64 pipe (53 % busy in FP64 at 128^3 Q2; 12
// warps per SM), no longer memory passes: DRAM moves src and dst once (230 MB
// read + write at 17 M DoFs against 780 MB of the cell-per-thread apply in eight
// colours that served Q1/Q2 before).  Measured on a B200, applies back to back:
//   128^3 Q2 vortex, FP64       272 -> 170 us      16^3 Q2 heat, FP64  22.8 -> 7.2 us
//   45 x 39 x 52 Q3 heat, FP64   69 -> 37 us
#pragma once

// Strip of degree P: x-units such that its columns with the halo fit the 64
// column slots of a warp.  Shared-memory rows hold the P node classes of a row
// apart by `half` pairs, strides chosen so that the accesses of consecutive
// columns (stores) and of consecutive units (loads) meet different banks.
template <int P, typename Real>
struct BandShape {
  static constexpr bool f64 = sizeof(Real) == 8;
  static constexpr int nxu = 63 / P - 1;
  // warps of a CTA: independent strips, adjacent in y.  8 share more rows in the
  // L1, 4 pack the registers better where a lane needs more than 80 (FP64 128^3
  // Q2 heat: 141 us with 8, 117 us with 4; 256^3 Q1: 106 and 127 us)
  static constexpr int warps = (f64 ? P >= 2 : P >= 3) ? 4 : 8;
  static constexpr int batch = P == 2 ? 2 : 1;  // planes at a time
  static constexpr int half = P == 1 ? 64 : P == 2 ? (f64 ? 36 : 40) : P == 3 ? 27 : (f64 ? 18 : 20);
  static constexpr int row = P == 1 ? 64 : P == 2 ? 2 * half : P == 3 ? 84 : (f64 ? 78 : 94);
  static constexpr int plane = P * row;  // pairs of one plane array
  static constexpr int orow = 64;        // staged output row
  static constexpr int oplane = P * orow;
  // a warp's shared memory in pairs: the plane arrays (NB each), the staged
  // layer, and (vortex) its y matrices and its lanes' x matrices
  static constexpr int warp_pairs(bool vortex)
  {
    return batch * (vortex ? 2 : 1) * plane + (P + 1) * oplane / 2 + (vortex ? (P + 1) * (P + 1) * (1 + 32 * (P == 1 ? 2 : 1)) : 0);
  }
  static_assert(half >= nxu + 2 && row >= P * half, "a row holds its classes");
  static_assert((nxu + 1) * P + 1 <= 64 && nxu * P <= 64, "two columns and two slots per lane");
};

template <typename Real>
struct Pair;
template <>
struct Pair<double> {
  using type = double2;
};
template <>
struct Pair<float> {
  using type = float2;
};

enum { BAND_PLAIN = 0, BAND_VORTEX = 1, BAND_ROTATION = 2 };

template <int P, typename Real>
struct BandP {
  static constexpr int n2 = (P + 1) * (P + 1);
  const Real *src;
  Real *dst;
  // Dirichlet DoFs read as 0 and (w) not written: as whole box faces (bit 2 d +
  // side), or as bytes, or none
  const uint8_t *dmask, *wmask;
  int faces, wfaces;
  int add;               // adds to dst (constrained DoFs keep their value) instead of storing (0 there)
  long NX, NY, NZ;
  int nc[3];
  int nxu;               // x-units of a strip
  int ntx, nty;          // strips along x, CTAs along y
  int warps;             // warps per CTA
  int zlo, zhi, len;     // layers of the launch, layers per chunk
  const Real *trig;      // vortex: sin, cos of pi x, pi y at the Gauss coordinates
  int trig_stride;
  Real cv;               // vortex: c_vel; rotation: c_vel w
  Real ox, oz, hx, hy, hz;  // origin and cell sizes
  // element matrices (test row, trial column)
  Real My[n2], Y2[n2], X1[n2], Mx[n2], Mz[n2], Z2[n2];
  Real A[n2], Mi[n2];    // rotation: advection; mass weighted by the cell coordinate
};

// values at a 32-bit byte offset (the launcher checks that vectors are < 4 GiB)
template <typename Real>
__device__ __forceinline__ Real at_offset(const Real *base, unsigned off)
{
  return __ldg(reinterpret_cast<const Real *>(reinterpret_cast<const char *>(base) + off));
}

template <int P, typename Real, int VK>
__global__ void __launch_bounds__(BandShape<P, Real>::warps * 32) band_apply_kernel(const BandP<P, Real> p)
{
  using BS = BandShape<P, Real>;
  using Real2 = typename Pair<Real>::type;
  constexpr int n = P + 1, n2 = n * n, PB = BS::batch;
  constexpr bool VOR = VK == BAND_VORTEX, ROT = VK == BAND_ROTATION;
  constexpr int NB = VOR ? 2 : 1;  // pair arrays per plane
  static_assert(!VOR || P <= 2, "the vortex serves degrees 1 and 2");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  Real2 *const pairs = reinterpret_cast<Real2 *>(smem_raw) + warp * BS::warp_pairs(VOR);  // [PB][NB][plane]
  Real *const outs = reinterpret_cast<Real *>(pairs + PB * NB * BS::plane);               // [n][P][orow]
  Real2 *const ymat = reinterpret_cast<Real2 *>(outs + n * BS::oplane);                   // vortex: [n2]
  Real2 *const xmat = ymat + n2;                                                          // vortex: [slot unit][n2][32]

  unsigned b = blockIdx.x;
  const int tx = (int)(b % (unsigned)p.ntx);
  b /= (unsigned)p.ntx;
  const int ty = (int)(b % (unsigned)p.nty), chunk = (int)(b / (unsigned)p.nty);
  const int xb = tx * p.nxu, yu = ty * p.warps + warp;
  const int z0 = p.zlo + chunk * p.len, z1 = min(p.zhi, z0 + p.len);
  if (z0 >= z1 || yu > p.nc[1]) return;  // whole warps; no block barrier follows

  // the strip's y-unit: rows present, rows on constrained faces
  const bool ylo = yu > 0, yhi = yu < p.nc[1];
  const bool zero_hi0 = (yu == 0 && (p.faces & 4)) || (yu == p.nc[1] && (p.faces & 8));
  const bool zero_lo0 = yu == 1 && (p.faces & 4), zero_hiP = yu == p.nc[1] - 1 && (p.faces & 8);
  const bool inner = ylo && yhi && !zero_lo0 && !zero_hiP && !p.dmask;
  const bool winner = ylo && yhi && !p.wmask && !p.add;
  const Real fyl = ylo ? Real(1) : Real(0), fyr = yhi ? Real(1) : Real(0);
  const unsigned rowb = (unsigned)p.NX * sizeof(Real), planeb = (unsigned)p.NY * rowb;

  // phase 1: the lane's columns
  bool cin[2], cok[2];  // inside the lattice; and not on a constrained face
  unsigned cat[2];      // byte offset of row 0 of the unit in its plane
  int cput[2];
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const int col = lane + 32 * c, X = (xb - 1) * P + col;
    cin[c] = col < (p.nxu + 1) * P + 1 && X >= 0 && X < (int)p.NX;
    cok[c] = cin[c] && !(X == 0 && (p.faces & 1)) && !(X == (int)p.NX - 1 && (p.faces & 2));
    cat[c] = (unsigned)(yu * P) * rowb + (unsigned)X * (unsigned)sizeof(Real);
    cput[c] = (col % P) * BS::half + col / P;
  }

  // phase 2: the lane's (x-unit, row) slots
  int sget[2], sout[2], sxu[2];
  bool sok[2];
  Real fl[2], fr[2];
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const int idx = s * 32 + lane;
    const int row = P == 2 ? s : idx / p.nxu, xl = P == 2 ? lane : idx - row * p.nxu;
    sxu[s] = xb + xl;
    sok[s] = row < P && xl < p.nxu && sxu[s] <= p.nc[0];
    sget[s] = sok[s] ? row * BS::row + xl : 0;  // class 0 of the unit before: index xl, own: xl + 1
    sout[s] = row * BS::orow + xl * P;
    fl[s] = sok[s] && sxu[s] > 0 ? Real(1) : Real(0);
    fr[s] = sok[s] && sxu[s] < p.nc[0] ? Real(1) : Real(0);
  }

  // vortex: element matrices of the y-unit and of the lane's x-units, rows 0..P-1
  // of the own element and row P of the one before (zero where it is missing)
  if constexpr (VOR) {
    const Tables<Real> &T = tab<Real>(P);
    auto entry = [&](const Real *sn, const Real *cs, int e, int ne, int i, int r, Real h, Real sign) {
      const int el = i < P ? e : e - 1;
      const bool ok = el >= 0 && el < ne;
      Real a = 0, m = 0;
#pragma unroll
      for (int q = 0; q < n; ++q) {
        const Real sq = ok ? sn[el * n + q] : Real(0), cq = ok ? cs[el * n + q] : Real(0);
        a += T.w[q] * sq * T.S[q * n + i] * T.D[q * n + r];
        m += T.w[q] * cq * T.S[q * n + i] * T.S[q * n + r];
      }
      Real2 v;
      v.x = h * m;                // mass weighted by the cosine
      v.y = sign * p.cv * a;      // advection weighted by the sine
      return v;
    };
    const Real *tr = p.trig;
    const int st = p.trig_stride;
#pragma unroll
    for (int i = 0; i < n; ++i)
#pragma unroll
      for (int r = 0; r < n; ++r) {
        const Real2 y = entry(tr + 2 * st, tr + 3 * st, yu, p.nc[1], i, r, p.hy, Real(-1));
        if (lane == 0) ymat[i * n + r] = y;
#pragma unroll
        for (int s = 0; s < (P == 1 ? 2 : 1); ++s)
          xmat[(s * n2 + i * n + r) * 32 + lane] = entry(tr, tr + st, sok[s] ? sxu[s] : -2, p.nc[0], i, r, p.hx, Real(1));
      }
    __syncwarp();
  }

  // rows of the unit (lo: of the unit before) in the lane's columns; columns
  // outside the strip's lattice part stay zero
  Real lo[PB][2][P], hi[PB][2][n];
#pragma unroll
  for (int k = 0; k < PB; ++k)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
#pragma unroll
      for (int r = 0; r < P; ++r) lo[k][c][r] = Real(0);
#pragma unroll
      for (int r = 0; r < n; ++r) hi[k][c][r] = Real(0);
    }
  auto load = [&](int k, int Z) {
    const unsigned zo = (unsigned)Z * planeb;
    const bool ez = (Z == 0 && (p.faces & 16)) || (Z == (int)p.NZ - 1 && (p.faces & 32));
    if (inner && !ez) {
#pragma unroll
      for (int c = 0; c < 2; ++c)
        if (cok[c]) {
          const unsigned o = zo + cat[c];
#pragma unroll
          for (int r = 0; r < P; ++r) lo[k][c][r] = at_offset(p.src, o - (unsigned)(P - r) * rowb);
#pragma unroll
          for (int r = 0; r < n; ++r) hi[k][c][r] = at_offset(p.src, o + (unsigned)r * rowb);
        }
      return;
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const unsigned o = zo + cat[c];
      const bool ok = cok[c] && !ez;
#pragma unroll
      for (int r = 0; r < P; ++r)
        lo[k][c][r] = ok && ylo && !(r == 0 && zero_lo0) ? at_offset(p.src, o - (unsigned)(P - r) * rowb) : Real(0);
#pragma unroll
      for (int r = 0; r < n; ++r)
        hi[k][c][r] = ok && (r == 0 ? !zero_hi0 : yhi) && !(r == P && zero_hiP) ? at_offset(p.src, o + (unsigned)r * rowb)
                                                                                 : Real(0);
      if (p.dmask && ok) {
        const uint8_t *m = p.dmask + o / (unsigned)sizeof(Real);
#pragma unroll
        for (int r = 0; r < P; ++r)
          if (ylo && *(m - (long)(P - r) * p.NX)) lo[k][c][r] = Real(0);
#pragma unroll
        for (int r = 0; r < n; ++r)
          if ((r == 0 || yhi) && m[(long)r * p.NX]) hi[k][c][r] = Real(0);
      }
    }
  };

  // y matrices (Ma, Mb) of the first NP loaded planes
  auto y_sweep = [&](auto np) {
    constexpr int NP = decltype(np)::value;
    auto rows_of = [&](auto mat, int array) {
#pragma unroll
      for (int i = 0; i < P; ++i) {
        Real2 v[NP][2];
#pragma unroll
        for (int k = 0; k < NP; ++k)
#pragma unroll
          for (int c = 0; c < 2; ++c) v[k][c].x = v[k][c].y = Real(0);
#pragma unroll
        for (int e = 0; e < (i == 0 ? 2 : 1); ++e)  // the own element, then (vertex) the one before
#pragma unroll
          for (int r = 0; r < n; ++r) {
            const Real2 m = mat(e == 0 ? i : P, r);
#pragma unroll
            for (int k = 0; k < NP; ++k)
#pragma unroll
              for (int c = 0; c < 2; ++c) {
                const Real u = e == 0 ? (r == 0 ? fyr * hi[k][c][0] : hi[k][c][r])
                                      : (r == P ? fyl * hi[k][c][0] : lo[k][c][r < P ? r : 0]);
                v[k][c].x += m.x * u;
                v[k][c].y += m.y * u;
              }
          }
#pragma unroll
        for (int k = 0; k < NP; ++k)
#pragma unroll
          for (int c = 0; c < 2; ++c) pairs[(k * NB + array) * BS::plane + i * BS::row + cput[c]] = v[k][c];
      }
    };
    rows_of(
        [&](int i, int r) {
          Real2 m;
          m.x = p.My[i * n + r];
          m.y = p.Y2[i * n + r];
          return m;
        },
        0);
    if constexpr (VOR) rows_of([&](int i, int r) { return ymat[i * n + r]; }, 1);
  };

  Real acc[2][n][P];  // z accumulators of the slots' P columns
#pragma unroll
  for (int s = 0; s < 2; ++s)
#pragma unroll
    for (int k = 0; k < n; ++k)
#pragma unroll
      for (int i = 0; i < P; ++i) acc[s][k][i] = Real(0);

  // x matrices of plane array slot k, then plane `zk` of layer iz into the
  // accumulators (zk = 0: opens the layer)
  auto add_plane = [&](int s, int zk, const Real (&W)[P], const Real (&V)[P], const Real (&W2)[P], const Real (&V2)[P],
                       int iz) {
#pragma unroll
    for (int i = 0; i < P; ++i) {
      Real w = W[i];
      if constexpr (ROT) w += (p.oz + iz * p.hz) * W2[i];
#pragma unroll
      for (int kk = 0; kk < n; ++kk) {
        acc[s][kk][i] += p.Mz[kk * n + zk] * w + p.Z2[kk * n + zk] * V[i];
        if constexpr (ROT) acc[s][kk][i] += (p.hz * p.hz) * p.Mi[kk * n + zk] * W2[i] + p.A[kk * n + zk] * V2[i];
      }
    }
  };
  auto x_sweep = [&](int k, int zk, int iz, bool stage) {
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      if (P >= 3) asm volatile("" ::: "memory");  // one slot's pairs in registers at a time
      const Real2 *g = pairs + k * NB * BS::plane + sget[s];
      Real W[P], V[P], W2[P], V2[P];
      Real2 q[2 * P + 1];  // columns -P..P of the unit
#pragma unroll
      for (int r = 0; r < P; ++r) q[r] = g[r * BS::half];
#pragma unroll
      for (int r = 0; r < P; ++r) q[P + r] = g[r * BS::half + 1];
      q[2 * P] = g[2];
#pragma unroll
      for (int i = 0; i < P; ++i) {
        Real w = 0, v = 0, w2 = 0, v2 = 0;
#pragma unroll
        for (int e = 0; e < (i == 0 ? 2 : 1); ++e)
#pragma unroll
          for (int r = 0; r < n; ++r) {
            const int t = e == 0 ? i : P;
            Real a = q[e == 0 ? P + r : r].x, c = q[e == 0 ? P + r : r].y;
            if (e == 0 && r == 0) a *= fr[s], c *= fr[s];
            if (e == 1 && r == P) a *= fl[s], c *= fl[s];
            w += p.X1[t * n + r] * a + p.Mx[t * n + r] * c;
            v += p.Mx[t * n + r] * a;
            if constexpr (ROT) {
              w2 += p.A[t * n + r] * a;
              v2 += ((p.ox + (sxu[s] - e) * p.hx) * p.Mx[t * n + r] + p.hx * p.hx * p.Mi[t * n + r]) * a;
            }
          }
        W[i] = w;
        V[i] = v;
        W2[i] = V2[i] = Real(0);
        if constexpr (ROT) {
          W2[i] = p.cv * w2;
          V2[i] = -p.cv * v2;
        }
      }
      if constexpr (VOR) {
        g += BS::plane;
#pragma unroll
        for (int r = 0; r < P; ++r) q[r] = g[r * BS::half];
#pragma unroll
        for (int r = 0; r < P; ++r) q[P + r] = g[r * BS::half + 1];
        q[2 * P] = g[2];
        const Real2 *xm = xmat + (P == 1 ? s : 0) * n2 * 32 + lane;
#pragma unroll
        for (int i = 0; i < n; ++i)  // row P: of the element before, to the vertex
#pragma unroll
          for (int r = 0; r < n; ++r) {
            const Real2 m = xm[(i * n + r) * 32], c = q[i < P ? P + r : r];
            W[i < P ? i : 0] += m.y * c.x + m.x * c.y;
          }
      }
      if (zk == 0) {
        add_plane(s, 0, W, V, W2, V2, iz);
      } else {
        add_plane(s, zk, W, V, W2, V2, iz);
        if (zk == P) {
          if (stage && sok[s]) {
#pragma unroll
            for (int kk = 0; kk < n; ++kk)
#pragma unroll
              for (int i = 0; i < P; ++i) outs[kk * BS::oplane + sout[s] + i] = acc[s][kk][i];
          }
#pragma unroll
          for (int i = 0; i < P; ++i) {
            acc[s][0][i] = acc[s][P][i];
#pragma unroll
            for (int kk = 1; kk < n; ++kk) acc[s][kk][i] = Real(0);
          }
          add_plane(s, 0, W, V, W2, V2, iz + 1);
        }
      }
    }
  };

  int iz = z0 > 0 ? z0 - 1 : 0;
  load(0, iz * P);
  y_sweep(std::integral_constant<int, 1>{});  // the first layer's lower plane
  __syncwarp();
#pragma unroll
  for (int k = 0; k < PB; ++k) load(k, iz * P + 1 + k);
  x_sweep(0, 0, iz, false);
  for (; iz < z1; ++iz) {
    const bool out = iz >= z0;
#pragma unroll
    for (int k0 = 1; k0 <= P; k0 += PB) {
      __syncwarp();  // the plane arrays have been read
      y_sweep(std::integral_constant<int, PB>{});
      __syncwarp();
      if (k0 + PB <= P || iz + 1 < z1) {
#pragma unroll
        for (int k = 0; k < PB; ++k) load(k, iz * P + k0 + PB + k);
      }
#pragma unroll
      for (int k = 0; k < PB; ++k) x_sweep(k, k0 + k, iz, out);
    }
    if (out) {
      __syncwarp();
      const bool top = iz + 1 == p.nc[2];  // the top layer of the mesh closes its last plane too
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int oc = lane + 32 * c, X = xb * P + oc;
        if (oc >= p.nxu * P || X >= (int)p.NX) continue;
        const unsigned o0 = (unsigned)(iz * P) * planeb + (unsigned)(yu * P) * rowb + (unsigned)X * (unsigned)sizeof(Real);
        const bool ex = (X == 0 && (p.wfaces & 1)) || (X == (int)p.NX - 1 && (p.wfaces & 2));
        const bool zfree = !(iz == 0 && (p.wfaces & 16)) && !top;
        if (winner && zfree && !ex) {  // nothing constrained
#pragma unroll
          for (int k = 0; k < P; ++k) {
            unsigned o = o0 + (unsigned)k * planeb;
#pragma unroll
            for (int i = 0; i < P; ++i, o += rowb)
              *reinterpret_cast<Real *>(reinterpret_cast<char *>(p.dst) + o) = outs[k * BS::oplane + i * BS::orow + oc];
          }
          continue;
        }
        for (int k = 0; k < n; ++k) {
          if (k == P && !top) break;
          const int Z = iz * P + k;
          const bool ez = (Z == 0 && (p.wfaces & 16)) || (Z == (int)p.NZ - 1 && (p.wfaces & 32));
          for (int i = 0; i < P; ++i) {
            if (i > 0 && !yhi) break;  // past the last vertex row
            const unsigned o = o0 + (unsigned)k * planeb + (unsigned)i * rowb;
            bool masked = ex || ez || (i == 0 && ((yu == 0 && (p.wfaces & 4)) || (yu == p.nc[1] && (p.wfaces & 8))));
            if (p.wmask) masked = p.wmask[o / (unsigned)sizeof(Real)] != 0;
            const Real v = outs[k * BS::oplane + i * BS::orow + oc];
            Real *d = reinterpret_cast<Real *>(reinterpret_cast<char *>(p.dst) + o);
            if (p.add) *d += masked ? Real(0) : v;
            else *d = masked ? Real(0) : v;
          }
        }
      }
      // staged again after at least one more __syncwarp
    }
  }
}

// Diagonal of the same operator: sums of products of the line matrices' diagonals (a
// vertex has the last entry of the element before it and the first of its own).
// Thread = column (X, Y) of the flattened lattice over a chunk of planes: its x and y
// factors are formed once, a plane is two products.  Bound by the one store per DoF
// where the chip is full, below that by the factors' quadrature (vortex).  A block per
// row, with the planes in 16 chunks and factors in local memory (parameters captured by
// value), took 5.6 ms on 4x4000x4 Q2 cells with the vortex and 401 us at 64^3; the
// cells' element diagonals 89 and 236; this 8 and 10.
template <int P, typename Real, int VK>
__global__ void __launch_bounds__(128) band_diag_kernel(const __grid_constant__ BandP<P, Real> p, int zlen)
{
  constexpr int n = P + 1;
  const Tables<Real> &T = tab<Real>(P);
  const unsigned col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= (unsigned)(p.NX * p.NY)) return;
  // a line node: its own element e and node i there; and whether that element and the
  // one before (node P) exist
  struct At {
    int e, i;
    bool own, before;
    __device__ At(int at, int ne) : e(at / P), i(at - at / P * P), own(at / P < ne), before(at / P * P == at && at > 0) {}
  };
  const At x((int)(col % (unsigned)p.NX), p.nc[0]), y((int)(col / (unsigned)p.NX), p.nc[1]);
  auto sum = [](const At &a, auto &&f) -> Real { return (a.own ? f(a.e, a.i) : Real(0)) + (a.before ? f(a.e - 1, P) : Real(0)); };
  auto line = [&](const Real *M, const At &a) { return sum(a, [&](int, int i) { return M[i * (n + 1)]; }); };
  const Real mx = line(p.Mx, x), my = line(p.My, y);
  Real w = my * line(p.X1, x) + line(p.Y2, y) * mx;  // times Mz
  const Real v = my * mx;                            // times Z2
  Real w2 = 0, v2 = 0;                               // rotation: times Mz(z) and Az
  if constexpr (VK == BAND_VORTEX) {
    // mass and advection weighted by a function at the Gauss points
    auto mass = [&](const Real *f, Real h, const At &a) {
      return sum(a, [&](int e, int i) {
        Real s = 0;
#pragma unroll
        for (int q = 0; q < n; ++q) s += T.w[q] * f[e * n + q] * T.S[q * n + i] * T.S[q * n + i];
        return h * s;
      });
    };
    auto adv = [&](const Real *f, const At &a) {
      return sum(a, [&](int e, int i) {
        Real s = 0;
#pragma unroll
        for (int q = 0; q < n; ++q) s += T.w[q] * f[e * n + q] * T.S[q * n + i] * T.D[q * n + i];
        return s;
      });
    };
    const Real *tr = p.trig;
    const int st = p.trig_stride;
    w += p.cv * (mass(tr + 3 * st, p.hy, y) * adv(tr, x) - adv(tr + 2 * st, y) * mass(tr + st, p.hx, x));
  }
  if constexpr (VK == BAND_ROTATION) {
    w2 = p.cv * my * line(p.A, x);
    v2 = -p.cv * my *
         sum(x, [&](int e, int i) { return (p.ox + e * p.hx) * p.Mx[i * (n + 1)] + p.hx * p.hx * p.Mi[i * (n + 1)]; });
  }
  const int z0 = blockIdx.y * zlen, z1 = min((int)p.NZ, z0 + zlen);
  Real *d = p.dst + (long)z0 * (p.NX * p.NY) + col;
  for (int Z = z0; Z < z1; ++Z, d += p.NX * p.NY) {
    const At z(Z, p.nc[2]);
    Real s = line(p.Mz, z) * w + line(p.Z2, z) * v;
    if constexpr (VK == BAND_ROTATION)
      s += sum(z, [&](int e, int i) { return (p.oz + e * p.hz) * p.Mz[i * (n + 1)] + p.hz * p.hz * p.Mi[i * (n + 1)]; }) * w2 +
           line(p.A, z) * v2;
    *d = s;
  }
}
