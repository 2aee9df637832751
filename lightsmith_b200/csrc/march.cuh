// The in-place H and E updates: one thread per (y, z) node, marching along x.
//
// update_h_node / update_e_node (yee.cuh) per node and half step issue most of their instructions on finding the
// node: region tests per component, CPML slab tests and psi indices per component and axis, 64-bit addresses. Here
// a thread keeps its (y, z) for a segment of x planes, so all of that but the x axis's part is worked out once per
// segment: the region mask, the neighbours' offsets (0 where there is none: such a difference is masked), the y and
// z slabs' psi pointers and profile values. Along x everything is uniform across the CTA. The components that the
// x neighbour shares are carried from plane to plane in registers (H: E_y, E_z of plane i + 1; E: H_y, H_z of plane
// i - 1), and all of a plane's loads are issued before its arithmetic. Threads run along the flat (y, z) plane, so
// rows of any length and parity fill whole warps and every access is coalesced. The arithmetic per value and its
// order are update_h_node's and update_e_node's. Measured on B200 in float32 against one node per thread with those
// functions (k_update_nodes; H and E kernels together, between events): 129^3 54 against 62 us, 201 x 215 x 199 207
// against 229, 123 x 139 x 3 5.7 against 16. Bound by the latency of a plane's loads (long scoreboard 9 to 10 of the
// stalls an issue, issue active 47 %) at 32 warps an SM. Which grids take it: Engine::marches (lsfdtd.cu).
#pragma once

#include "yee.cuh"

namespace lsfdtd {

// short CTAs leave a smaller last wave: passes at 128 and 256 threads (us): 49^3 714 725, 129^3 7011 7341,
// 201 x 215 x 199 3895 3977
constexpr int kMarchThreads = 128;
// CTAs per SM that the kernel's registers are held to. Each plane of a thread is one round trip of its loads, so the
// warps in flight set the rate (129^3 in FP32: 54 us a step at 32 warps an SM, 64 registers; 85 at 16 without a cap, 60
// at 40, 80 at 48, where values spill). Wider values, whole steps, us: float64 (spills 48 to 92 bytes a thread at 6) 97
// x 89 x 101 49.2 at 4 CTAs, 44.5 at 5, 48.5 at 6, 52.6 at 7, 60 at 8; 100 x 96 x 100 39.7, 42.4, 40.3; 400 x 400 x 3
// 29.4, 30.7, 27.4; complex float32 (no spills up to 6) 32 x 32 x 200 27.1, 28.3, 28.8, at 8 29.5; 62 x 62 x 200 44.0,
// 42.6, 45.1, at 8 42.4; complex float64 (28 to 44 bytes at 4) 32 x 32 x 200 32.8 at 2 CTAs, 33.0 at 3, 31.9 at 4, 35.8
// at 5. Grids past L2 of these types take k_update_nodes (Engine::marches)
template <typename F>
__host__ __device__ constexpr int march_ctas() {
  return sizeof(F) == 4 ? 8 : (sizeof(F) == 8 ? 6 : 4);
}

// the slab of axis d (0: low, 1: high, -1: none) that holds coordinate u; the two components with a psi along d
// have the same slabs. One at most: grids whose two slabs of an axis share nodes take k_update_nodes (yee.cuh)
template <int FLD, typename F>
__device__ __forceinline__ int march_side(const PmlAxis<F>& p, int d, int u) {
  if (!p.on) return -1;
  const int c = d == 0 ? 1 : 0;
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const int st = p.start[FLD][c][s];
    if (u >= st && u < st + p.len[FLD][c][s]) return s;
  }
  return -1;
}

// a thread's CPML terms along axis d (1 or 2): psi pointers of the two components at plane i0, their step per plane
// and the profile values at the thread's coordinate
template <typename F>
struct MarchSlab {
  using R = typename real_of<F>::type;
  int on;
  F* psi[2];      // components (d + 1) % 3 and (d + 2) % 3
  unsigned step;  // elements from one x plane to the next
  R b, c, k;
};

template <int FLD, int D, typename F>
__device__ __forceinline__ MarchSlab<F> march_slab(const YeeArgs<F>& g, int i0, int j, int k) {
  using R = typename real_of<F>::type;
  MarchSlab<F> m;
  const PmlAxis<F>& p = g.pml[D];
  const int u = D == 1 ? j : k;
  const int s = march_side<FLD>(p, D, u);
  m.on = s >= 0;
  m.psi[0] = m.psi[1] = nullptr;
  m.step = 0;
  m.b = m.c = m.k = R(0);
  if (!m.on) return m;
  const int c0 = (D + 1) % 3, c1 = (D + 2) % 3;
  const int off = u - p.start[FLD][c0][s], len = p.len[FLD][c0][s];
  const int x[3] = {i0, j, k};
  const long long q = psi_index(x, g.n, D, off, len);
  m.psi[0] = p.psi[FLD][c0][s] + q;
  m.psi[1] = p.psi[FLD][c1][s] + q;
  m.step = (unsigned)(D == 1 ? len * g.n[2] : g.n[1] * len);
  m.b = p.b[FLD][u];
  m.c = p.c[FLD][u];
  if (p.k[FLD]) m.k = p.k[FLD][u];
  return m;
}

// v += the CPML term of component c along axis d (apply_cpml's arithmetic), the node's psi given and returned
template <int FLD, int C, int D, int UNI, typename F>
__device__ __forceinline__ F march_term(F& v, const YeeArgs<F>& g, F psi, F der, typename real_of<F>::type scale,
                                        typename real_of<F>::type b, typename real_of<F>::type cc,
                                        typename real_of<F>::type kk) {
  using R = typename real_of<F>::type;
  constexpr bool minus = (D == (C + 1) % 3) == (FLD == 1);
  R s = UNI ? scale : scale / g.pml[D].div;
  if (minus) s = -s;
  psi = psi * b;
  if (g.pml[D].k[FLD]) v += (s * kk) * der;
  psi += der * (s * cc);
  v += psi;
  return psi;
}

// One half step of field FLD (1: H from E, 0: E from H) over x planes [blockIdx.y seg, + seg)
template <typename F, int FLD, int UNI>
__global__ void __launch_bounds__(kMarchThreads, march_ctas<F>())
    k_march(const __grid_constant__ YeeArgs<F> g, int seg, long long* bump) {
  using R = typename real_of<F>::type;
  const unsigned n1 = g.n[1], n2 = g.n[2], plane = n1 * n2;
  const unsigned q = blockIdx.x * kMarchThreads + threadIdx.x;
  if (q >= plane) return;  // (threads past the plane touch no memory)
  const int j = (int)(q / n2), k = (int)(q - (unsigned)j * n2);
  const int i0 = (int)blockIdx.y * seg, i1 = min(g.n[0], i0 + seg);
  // bit c: component c is stepped at this (y, z); along x: the planes [xlo, xhi) of H_x or E_x and of the others
  unsigned yz = 0;
  int xlo[2], xhi[2];
  {
    int x[3] = {0, j, k};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      bool in = true;
#pragma unroll
      for (int a = 1; a < 3; ++a) {
        const int per = g.periodic[a], mir = g.mirror[a], n = g.n[a];
        int lo, hi;
        if (FLD == 1) {
          lo = per ? 1 : 0;
          hi = per ? n - 1 : (a == c ? n : n - 1);
          if (mir) lo = (mir < 0 && a == c) ? 2 : 1;
        } else {
          lo = (per || a != c) ? 1 : 0;
          hi = n - 1;
          if (mir) lo = (mir < 0 && a != c) ? 2 : 1;
        }
        in = in && x[a] >= lo && x[a] < hi;
      }
      yz |= (in ? 1u : 0u) << c;
    }
    const int per = g.periodic[0], mir = g.mirror[0], n = g.n[0];
    if (FLD == 1) {
      xlo[0] = mir ? (mir < 0 ? 2 : 1) : (per ? 1 : 0);
      xhi[0] = per ? n - 1 : n;
      xlo[1] = mir || per ? 1 : 0;
      xhi[1] = n - 1;
    } else {
      xlo[0] = mir || per ? 1 : 0;
      xlo[1] = mir < 0 ? 2 : 1;
      xhi[0] = xhi[1] = n - 1;
    }
  }
  const MarchSlab<F> sy = march_slab<FLD, 1>(g, i0, j, k), sz = march_slab<FLD, 2>(g, i0, j, k);
  // neighbour offsets: +1 for H, -1 for E
  const unsigned oy = FLD == 1 ? ((unsigned)j + 1 < n1 ? n2 : 0u) : (j > 0 ? n2 : 0u);
  const unsigned oz = FLD == 1 ? ((unsigned)k + 1 < n2 ? 1u : 0u) : (k > 0 ? 1u : 0u);
  const size_t base = (size_t)i0 * plane;
  F *const t0 = (FLD == 1 ? g.H[0] : g.E[0]) + base, *const t1 = (FLD == 1 ? g.H[1] : g.E[1]) + base,
           *const t2 = (FLD == 1 ? g.H[2] : g.E[2]) + base;
  const F *const f0 = (FLD == 1 ? g.E[0] : g.H[0]) + base, *const f1 = (FLD == 1 ? g.E[1] : g.H[1]) + base,
                *const f2 = (FLD == 1 ? g.E[2] : g.H[2]) + base;
  const R *const cb0 = g.cbE[0] + base, *const cb1 = g.cbE[1] + base, *const cb2 = g.cbE[2] + base;
  const bool iso = FLD == 1 || (g.cbE[1] == g.cbE[0] && g.cbE[2] == g.cbE[0]);
  dependent_wait();  // everything above reads parameters and the CPML profiles
  // the step before left its count to this one (its readers have ended, this step's come after this kernel)
  if (bump && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *bump += 1;
  unsigned p = q;  // the node, from plane i0
  F c1, c2;        // FLD 1: E_y, E_z of this plane; FLD 0: H_y, H_z of the plane before
  if (FLD == 1) {
    c1 = f1[p];
    c2 = f2[p];
  } else {
    c1 = i0 > 0 ? *(f1 + p - plane) : zero<F>();
    c2 = i0 > 0 ? *(f2 + p - plane) : zero<F>();
  }
  unsigned ps_y = 0, ps_z = 0;
#pragma unroll 1
  for (int i = i0; i < i1; ++i, p += plane, ps_y += sy.step, ps_z += sz.step) {
    unsigned m = yz;
    if (i < xlo[0] || i >= xhi[0]) m &= 6u;
    if (i < xlo[1] || i >= xhi[1]) m &= 1u;
    const int sx = march_side<FLD>(g.pml[0], 0, i);
    // every load of the plane before its arithmetic
    const F v0 = f0[p];
    F v1, v2, x1, x2;  // the differentiated field's y and z components at the node, and one plane along x
    if (FLD == 1) {
      v1 = c1;
      v2 = c2;
      const unsigned pn = p + (i + 1 < g.n[0] ? plane : 0u);
      x1 = f1[pn];
      x2 = f2[pn];
    } else {
      v1 = f1[p];
      v2 = f2[p];
      x1 = c1;
      x2 = c2;
    }
    const unsigned py = FLD == 1 ? p + oy : p - oy, pz = FLD == 1 ? p + oz : p - oz;
    const F y0 = f0[py], y2 = f2[py], z0 = f0[pz], z1 = f1[pz];
    F h0 = t0[p], h1 = t1[p], h2 = t2[p];
    R w0 = g.cH, w1 = g.cH, w2 = g.cH;
    if (FLD == 0) {
      w0 = cb0[p];
      w1 = iso ? w0 : cb1[p];
      w2 = iso ? w0 : cb2[p];
    }
    F psx[2], psy[2], psz[2];  // per axis, its two components in cyclic order: x: 1, 2; y: 2, 0; z: 0, 1
    size_t qx = 0;
    R bx = R(0), cx = R(0), kx = R(0);
    if (sx >= 0) {
      const PmlAxis<F>& px = g.pml[0];
      qx = (size_t)(i - px.start[FLD][1][sx]) * plane + q;
      psx[0] = px.psi[FLD][1][sx][qx];
      psx[1] = px.psi[FLD][2][sx][qx];
      bx = px.b[FLD][i];
      cx = px.c[FLD][i];
      if (px.k[FLD]) kx = px.k[FLD][i];
    }
    if (sy.on) {
      psy[0] = sy.psi[0][ps_y];
      psy[1] = sy.psi[1][ps_y];
    }
    if (sz.on) {
      psz[0] = sz.psi[0][ps_z];
      psz[1] = sz.psi[1][ps_z];
    }
    // (a, b) per component: H_c -= cH (dE_{d2}/dd1 - dE_{d1}/dd2), E_c += cbE (dH_{d2}/dd1 - dH_{d1}/dd2)
    const F a0 = FLD == 1 ? y2 - v2 : v2 - y2, b0 = FLD == 1 ? z1 - v1 : v1 - z1;
    const F a1 = FLD == 1 ? z0 - v0 : v0 - z0, b1 = FLD == 1 ? x2 - v2 : v2 - x2;
    const F a2 = FLD == 1 ? x1 - v1 : v1 - x1, b2 = FLD == 1 ? y0 - v0 : v0 - y0;
    const F r0 = UNI ? a0 - b0 : a0 * g.inv_d[1] - b0 * g.inv_d[2];
    const F r1 = UNI ? a1 - b1 : a1 * g.inv_d[2] - b1 * g.inv_d[0];
    const F r2 = UNI ? a2 - b2 : a2 * g.inv_d[0] - b2 * g.inv_d[1];
    if (FLD == 1) {
      h0 = h0 - r0 * w0;
      h1 = h1 - r1 * w1;
      h2 = h2 - r2 * w2;
    } else {
      h0 = h0 + r0 * w0;
      h1 = h1 + r1 * w1;
      h2 = h2 + r2 * w2;
    }
    if (sx >= 0) {
      psx[0] = march_term<FLD, 1, 0, UNI>(h1, g, psx[0], b1, w1, bx, cx, kx);
      psx[1] = march_term<FLD, 2, 0, UNI>(h2, g, psx[1], a2, w2, bx, cx, kx);
      F* const o = g.pml[0].psi[FLD][1][sx];
      F* const o2 = g.pml[0].psi[FLD][2][sx];
      if (m & 2u) o[qx] = psx[0];
      if (m & 4u) o2[qx] = psx[1];
    }
    if (sy.on) {
      psy[0] = march_term<FLD, 2, 1, UNI>(h2, g, psy[0], b2, w2, sy.b, sy.c, sy.k);
      psy[1] = march_term<FLD, 0, 1, UNI>(h0, g, psy[1], a0, w0, sy.b, sy.c, sy.k);
      if (m & 4u) sy.psi[0][ps_y] = psy[0];
      if (m & 1u) sy.psi[1][ps_y] = psy[1];
    }
    if (sz.on) {
      psz[0] = march_term<FLD, 0, 2, UNI>(h0, g, psz[0], b0, w0, sz.b, sz.c, sz.k);
      psz[1] = march_term<FLD, 1, 2, UNI>(h1, g, psz[1], a1, w1, sz.b, sz.c, sz.k);
      if (m & 1u) sz.psi[0][ps_z] = psz[0];
      if (m & 2u) sz.psi[1][ps_z] = psz[1];
    }
    if (m & 1u) t0[p] = h0;
    if (m & 2u) t1[p] = h1;
    if (m & 4u) t2[p] = h2;
    c1 = FLD == 1 ? x1 : v1;
    c2 = FLD == 1 ? x2 : v2;
  }
}

}  // namespace lsfdtd
