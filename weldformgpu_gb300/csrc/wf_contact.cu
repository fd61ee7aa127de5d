// wf_contact.cu — contact of the SPH solid with rigid triangle meshes.
//
// Free-surface tagging (Domain_d::CalculateSurface, src/cuda/Geometry.cu:26-88),
// the contact neighbour list (CalcContactNb, src/cuda/Contact.cu:29-62), the
// penalty force with friction (CalcContactForcesWang, Contact.cu:134-321), the
// rigid mesh motion (MeshUpdateKernel, src/cuda/Mesh.cu:24-29, 222-276) and the
// rigid centroid particles (UpdateContactParticles, Contact.cu:85-112).
//
// Compiled with -fmad=false: the FP64 arithmetic follows the reference's
// operation order (vector_math.h: a / s is a * (1.0 / s), dot sums left to
// right, length = sqrt(dot)), so the plain form matches the oracle bit for bit.
// 1 to 32 lanes per particle (surface, list, force; wf_lanes64.cuh), one thread
// per node (mesh motion) or element (element geometry and rigid particle).
#include <algorithm>

#include "wf_common.cuh"
#include "wf_integrate.cuh"
#include "wf_lanes64.cuh"
#include "wf_nsearch.cuh"

namespace {

struct V3 {
  double x, y, z;
};
__device__ __forceinline__ V3 mk(double x, double y, double z) { return V3{x, y, z}; }
__device__ __forceinline__ V3 mk(const double4& a) { return V3{a.x, a.y, a.z}; }
__device__ __forceinline__ V3 operator+(V3 a, V3 b) { return mk(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ V3 operator-(V3 a, V3 b) { return mk(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ V3 scale(V3 a, double s) { return mk(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ V3 divide(V3 a, double s) { return scale(a, 1.0 / s); }
__device__ __forceinline__ double dot(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ double len(V3 a) { return sqrt(dot(a, a)); }
__device__ __forceinline__ V3 cross(V3 a, V3 b) {
  return mk(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ double4 d4(V3 a, double w = 0.0) { return make_double4(a.x, a.y, a.z, w); }

// the mesh whose element centroids include the particle of original id `orig`
__device__ __forceinline__ int mesh_of(const StepParams& P, int32_t orig) {
  for (int m = 0; m < P.ncsid; m++)
    if (orig >= P.mesh[m].first && orig < P.mesh[m].first + P.mesh[m].ne) return m;
  return -1;
}

// CalculateSurface: normal = N / (M n') sum m_j (x_i - x_j) over the n'
// neighbours that are not rigid particles of the first mesh; |normal| >= 0.25 h
// with n' <= 46 tags the particle as free surface unless its zone is protected.
// Other threads may turn a neighbour's id into the free-surface id meanwhile;
// that id is never a mesh zone id, so the test on ID[j] does not change.
// Several lanes share a particle as in the pair passes (5.4k particles: 37 us
// with one thread each, 17 us so).
template <int kG>
__global__ void __launch_bounds__(kG == 1 ? 64 : 32) k_surface(StepParams P, Fields F,
                                                               const int32_t* __restrict__ nb,
                                                               const int32_t* __restrict__ cnt) {
  __shared__ double sh[kG == 1 ? 1 : 32 * 3];
  int g;
  const int64_t i0 = slot64<kG>(g);
  const bool solid = i0 < P.n && F.perm[i0] < P.n_solid;
  if (kG == 1 && !solid) return;
  const int64_t i = solid ? i0 : 0;
  const V3 xi = mk(F.xm[i]);
  V3 nrm = mk(0.0, 0.0, 0.0);
  int corr = 0;
  const int c = solid ? cnt[i] : 0;
  if constexpr (kG == 1) {
    for (int k = 0; k < c; k++) {
      const int j = __ldg(nb + nb_at(P.npad, i, k));
      const double4 xj = F.xm[j];
      const V3 xij = xi - mk(xj);
      if (F.id[j] != P.csid[0]) {
        nrm = nrm + scale(xij, xj.w);
        corr++;
      }
    }
  } else {
    const int rounds = warp_rounds<kG>(c);
    double acc[2] = {0.0, 0.0};
    for (int b = 0; b < rounds; b++) {
      double t[3] = {0.0, 0.0, 0.0};
      if (kG * b + g < c) {
        const int j = __ldg(nb + nb_at(P.npad, i, kG * b + g));
        const double4 xj = F.xm[j];
        const V3 xij = scale(xi - mk(xj), xj.w);
        if (F.id[j] != P.csid[0]) {
          t[0] = xij.x; t[1] = xij.y; t[2] = xij.z;
          corr++;
        }
      }
      add_in_order<kG, 3>(sh, t, g, acc, c - kG * b);
    }
#pragma unroll
    for (int k = kG / 2; k > 0; k /= 2) corr += __shfl_xor_sync(0xffffffffu, corr, k);
    nrm = mk(__shfl_sync(0xffffffffu, acc[0], 0, kG), __shfl_sync(0xffffffffu, acc[0], 1, kG),
             __shfl_sync(0xffffffffu, acc[0], 2, kG));
    if (!solid || g != 0) return;
  }
  nrm = scale(nrm, (double)P.n / (P.totmass * (double)corr));
  F.nrm[i] = d4(nrm);
  if (len(nrm) >= 0.25 * P.h && corr <= 46 && !F.nw[i]) F.id[i] = P.id_free_surf;
}

// CalcContactNb: rigid neighbours within 2h of a free-surface particle, in
// neighbour order, once per mesh whose zone id matches; at most WF_CONT_NB
// (the reference writes past its 20 slots).  Column-major: cnb[k * npad + i].
// The distance is computed of rigid neighbours only, the lanes of a particle
// append in list order (5.4k particles 47 us with one thread each and all
// distances, 36 without, 12 so).
template <int kG>
__global__ void __launch_bounds__(kG == 1 ? 64 : 32) k_contact_nb(StepParams P, Fields F,
                                                                  const int32_t* __restrict__ nb,
                                                                  const int32_t* __restrict__ cnt) {
  int g;
  const int64_t i0 = slot64<kG>(g);
  const bool solid = i0 < P.n && F.perm[i0] < P.n_solid;
  const int64_t i = solid ? i0 : 0;
  int cc = 0;
  const int c = solid && F.id[i] == P.id_free_surf ? cnt[i] : 0;
  const V3 xi = mk(F.xm[i]);
  const int rounds = warp_rounds<kG>(c);
  for (int b = 0; b < rounds; b++) {
    int j = 0, meshes = 0;
    if (kG * b + g < c) {
      j = __ldg(nb + nb_at(P.npad, i, kG * b + g));
      const int32_t idj = F.id[j];
      for (int mc = 0; mc < P.ncsid; mc++) meshes += idj == P.csid[mc];
      if (meshes && !(len(xi - mk(F.xm[j])) < 2. * P.h)) meshes = 0;
    }
    int upto = meshes;                                   // of the lanes up to this one
#pragma unroll
    for (int k = 1; k < kG; k *= 2) {
      const int v = __shfl_up_sync(0xffffffffu, upto, k, kG);
      if (g >= k) upto += v;
    }
    for (int q = cc + upto - meshes; q < cc + upto && q < WF_CONT_NB; q++)
      P.cnb[(int64_t)q * P.npad + i] = j;
    cc += __shfl_sync(0xffffffffu, upto, kG - 1, kG);
  }
  if (solid && g == 0) P.ccnt[i] = cc < WF_CONT_NB ? cc : WF_CONT_NB;
}

// CalcContactForcesWang: for each contact neighbour j (the centroid particle of
// element e), the predicted position x + v dt + a dt^2 / 2 is tested against
// the element's plane and, projected on it, against the triangle's edges; a
// hit adds the penalty force 0.4 kij (h - dist) n, kij = 2 m / dt^2, with
// static or dynamic friction.  contforce keeps the last contact's force; the
// acceleration accumulates all of them, and later contacts see the earlier
// ones through the predicted position.  Mixed form: the acceleration comes
// from and returns to the FP32 array.
//
// Eight lanes share a particle in domains that do not fill the GPU (lanes64):
// they test eight contacts in a row against the acceleration so far, the first
// that hits applies its force, and the contacts behind it are tested anew.  A
// hit is rare, so the chain of contacts (each some 100 operations at 19 cycles)
// shrinks by up to 8: 5.4k particles 44 -> 15 us.
struct ContactHit {
  V3 x_pred, n;
  double dist;
  int j;
};
__device__ __forceinline__ bool contact_test(const StepParams& P, const Fields& F, int64_t i, int k,
                                             V3 xi, V3 vi, V3 a, ContactHit& H) {
  const double dt = P.dt, h = P.h;
  const int j = P.cnb[(int64_t)k * P.npad + i];
  const int32_t oj = F.perm[j];
  const int mid = mesh_of(P, oj);
  const MeshDev& M = P.mesh[mid];
  const int e = oj - M.first;
  const V3 x_pred = (xi + scale(vi, dt)) + divide(scale(scale(a, dt), dt), 2.);
  const V3 n = mk(M.normal[e]);
  const double dist = dot(n, x_pred) - M.pplane[e];
  H = ContactHit{x_pred, n, dist, j};
  if (!(dist < h)) return false;
  const V3 Qj = xi - scale(n, dist);
  for (int l = 0; l < 3; l++) {
    const int nx = l + 1 > 2 ? 0 : l + 1;
    const V3 pl = mk(M.node[M.elnode[3 * e + l]]);
    const V3 pn = mk(M.node[M.elnode[3 * e + nx]]);
    if (dot(cross(pn - pl, Qj - pl), n) < 0.0) return false;
  }
  return true;
}
// the force of one contact: cf becomes its force, a gains it
__device__ __forceinline__ void contact_apply(const StepParams& P, const Fields& F,
                                              const ContactHit& H, V3 xi, double mi, V3& a,
                                              V3& cf) {
  const double dt = P.dt, delta = P.h - H.dist;
  const double kij = 2.0 * mi / (dt * dt);
  cf = scale(H.n, 0.4 * kij * delta);
  a = a + divide(cf, mi);
  if (P.mu_s > 0.) {
    const V3 du = (H.x_pred - xi) - scale(mk(F.vd[H.j]), dt);
    const V3 dtg = du - scale(H.n, dot(du, H.n));
    const V3 ft = scale(dtg, kij);
    if (len(ft) < P.mu_s * len(cf)) {
      a = a - divide(ft, mi);
    } else {
      const V3 fd = divide(scale(ft, P.mu_d * len(cf)), len(ft));
      cf = cf - fd;
      a = a - divide(fd, mi);
    }
  }
}

template <int kG>
__global__ void __launch_bounds__(kG == 1 ? 64 : 32) k_contact_force(StepParams P, Fields F,
                                                                     float4* a32) {
  constexpr unsigned kAll = 0xffffffffu;
  int g;
  const int64_t i0 = slot64<kG>(g);
  const bool solid = i0 < P.n && F.perm[i0] < P.n_solid;
  const int64_t i = solid ? i0 : 0;
  const int cc = solid ? P.ccnt[i] : 0;
  V3 cf = mk(0.0, 0.0, 0.0);
  if (__any_sync(kAll, cc > 0)) {
    const double4 x4 = F.xm[i];
    const V3 xi = mk(x4), vi = mk(F.vd[i]);
    V3 a = a32 ? mk(a32[i].x, a32[i].y, a32[i].z) : mk(F.a[i]);
    const int base = (threadIdx.x & 31) - g;             // the group's first lane
    for (int pos = 0; __any_sync(kAll, pos < cc);) {
      ContactHit H;
      const bool hit = pos + g < cc && contact_test(P, F, i, pos + g, xi, vi, a, H);
      const unsigned m = (__ballot_sync(kAll, hit) >> base) & ((1u << kG) - 1u);
      const int first = m ? __ffs(m) - 1 : 0;
      if (hit && g == first) contact_apply(P, F, H, xi, x4.w, a, cf);
      a = mk(__shfl_sync(kAll, a.x, first, kG), __shfl_sync(kAll, a.y, first, kG),
             __shfl_sync(kAll, a.z, first, kG));
      cf = mk(__shfl_sync(kAll, cf.x, first, kG), __shfl_sync(kAll, cf.y, first, kG),
              __shfl_sync(kAll, cf.z, first, kG));
      pos += m ? first + 1 : kG;
    }
    if (cc > 0 && g == 0) {
      if (a32) a32[i] = make_float4((float)a.x, (float)a.y, (float)a.z, 0.f);
      else F.a[i] = d4(a);
    }
  }
  if (solid && g == 0) F.cf[i] = d4(cf);
}

// Closest point of triangle abc to p (Ericson, Real-Time Collision Detection,
// 5.1.5: Voronoi regions of the vertices, edges and face).
__device__ V3 closest_on_tri(V3 p, V3 a, V3 b, V3 c) {
  const V3 ab = b - a, ac = c - a, ap = p - a;
  const double d1 = dot(ab, ap), d2 = dot(ac, ap);
  if (d1 <= 0.0 && d2 <= 0.0) return a;
  const V3 bp = p - b;
  const double d3 = dot(ab, bp), d4 = dot(ac, bp);
  if (d3 >= 0.0 && d4 <= d3) return b;
  const double vc = d1 * d4 - d3 * d2;
  if (vc <= 0.0 && d1 >= 0.0 && d3 <= 0.0) return a + scale(ab, d1 / (d1 - d3));
  const V3 cp = p - c;
  const double d5 = dot(ab, cp), d6 = dot(ac, cp);
  if (d6 >= 0.0 && d5 <= d6) return c;
  const double vb = d5 * d2 - d1 * d6;
  if (vb <= 0.0 && d2 >= 0.0 && d6 <= 0.0) return a + scale(ac, d2 / (d2 - d6));
  const double va = d3 * d6 - d5 * d4;
  if (va <= 0.0 && (d4 - d3) >= 0.0 && (d5 - d6) >= 0.0)
    return b + scale(c - b, (d4 - d3) / ((d4 - d3) + (d5 - d6)));
  const double denom = 1.0 / (va + vb + vc);
  return (a + scale(ab, vb * denom)) + scale(ac, vc * denom);
}

// The same closest-point rule in FP32 on tool-relative coordinates; returns
// the squared distance.  Used only to choose which triangles the FP64 rule
// evaluates (the FP64 pipe runs at 1/64 of the FP32 rate on this GPU).
__device__ __forceinline__ float3 f3sub(float3 a, float3 b) {
  return make_float3(a.x - b.x, a.y - b.y, a.z - b.z);
}
__device__ __forceinline__ float f3dot(float3 a, float3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ float3 f3axpy(float3 a, float3 d, float t) {
  return make_float3(a.x + d.x * t, a.y + d.y * t, a.z + d.z * t);
}
__device__ float closest_sq32(float3 p, float3 a, float3 b, float3 c) {
  const float3 ab = f3sub(b, a), ac = f3sub(c, a), ap = f3sub(p, a);
  const float d1 = f3dot(ab, ap), d2 = f3dot(ac, ap);
  float3 q;
  const float3 bp = f3sub(p, b), cp = f3sub(p, c);
  const float d3 = f3dot(ab, bp), d4 = f3dot(ac, bp);
  const float d5 = f3dot(ab, cp), d6 = f3dot(ac, cp);
  const float vc = d1 * d4 - d3 * d2, vb = d5 * d2 - d1 * d6, va = d3 * d6 - d5 * d4;
  if (d1 <= 0.f && d2 <= 0.f) q = a;
  else if (d3 >= 0.f && d4 <= d3) q = b;
  else if (vc <= 0.f && d1 >= 0.f && d3 <= 0.f) q = f3axpy(a, ab, d1 / (d1 - d3));
  else if (d6 >= 0.f && d5 <= d6) q = c;
  else if (vb <= 0.f && d2 >= 0.f && d6 <= 0.f) q = f3axpy(a, ac, d2 / (d2 - d6));
  else if (va <= 0.f && (d4 - d3) >= 0.f && (d5 - d6) >= 0.f)
    q = f3axpy(b, f3sub(c, b), (d4 - d3) / ((d4 - d3) + (d5 - d6)));
  else {
    const float den = 1.f / (va + vb + vc);
    q = f3axpy(f3axpy(a, ab, vb * den), ac, vc * den);
  }
  const float3 dq = f3sub(p, q);
  return f3dot(dq, dq);
}

__device__ __forceinline__ float3 rel32(const float4* r, int q) {
  const float4 v = r[q];
  return make_float3(v.x, v.y, v.z);
}

// Bins of a rotating tool, rebuilt every step from the current nodes: every
// triangle goes into each cell that its bounding box (relative to node 0)
// widened by the margin touches, with its vertices relative to node 0 in
// FP32.  Count, exclusive scan (cstart), fill; the order within a cell depends
// on the atomics, which the search's explicit tie rule makes irrelevant.
__device__ __forceinline__ void tri_cells(const MeshDev& M, int e, V3 rv[3], int r0[3], int r1[3]) {
  const int32_t* en = M.elnode + 3 * e;
  const V3 n0 = mk(M.node[0]);
  for (int k = 0; k < 3; k++) rv[k] = mk(M.node[en[k]]) - n0;
  const double lo[3] = {fmin(fmin(rv[0].x, rv[1].x), rv[2].x), fmin(fmin(rv[0].y, rv[1].y), rv[2].y),
                        fmin(fmin(rv[0].z, rv[1].z), rv[2].z)};
  const double hi[3] = {fmax(fmax(rv[0].x, rv[1].x), rv[2].x), fmax(fmax(rv[0].y, rv[1].y), rv[2].y),
                        fmax(fmax(rv[0].z, rv[1].z), rv[2].z)};
  for (int k = 0; k < 3; k++) {
    const double a = floor((lo[k] - M.margin - M.grel[k]) * M.inv_cs);
    const double b = floor((hi[k] + M.margin - M.grel[k]) * M.inv_cs);
    // clamped in double before the conversion (NaN gives an empty range)
    r0[k] = (int)fmin(fmax(a, 0.0), (double)M.dims[k]);
    r1[k] = (int)fmax(fmin(b, (double)(M.dims[k] - 1)), -1.0);
  }
}
__global__ void k_bins_count(MeshDev M) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= M.ne) return;
  V3 rv[3];
  int r0[3], r1[3];
  tri_cells(M, e, rv, r0, r1);
  uint32_t* cnt = reinterpret_cast<uint32_t*>(M.cstart);
  for (int z = r0[2]; z <= r1[2]; z++)
    for (int y = r0[1]; y <= r1[1]; y++)
      for (int x = r0[0]; x <= r1[0]; x++)
        atomicAdd(cnt + ((int64_t)z * M.dims[1] + y) * M.dims[0] + x, 1u);
}
__global__ void k_bins_fill(MeshDev M) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= M.ne) return;
  V3 rv[3];
  int r0[3], r1[3];
  tri_cells(M, e, rv, r0, r1);
  for (int z = r0[2]; z <= r1[2]; z++)
    for (int y = r0[1]; y <= r1[1]; y++)
      for (int x = r0[0]; x <= r1[0]; x++) {
        const uint32_t pos = atomicAdd(M.cursor + ((int64_t)z * M.dims[1] + y) * M.dims[0] + x, 1u);
        if ((int64_t)pos >= M.cap) continue;   // bounded by construction (cap)
        float4* v = M.cvert + 3 * (int64_t)pos;
        v[0] = make_float4((float)rv[0].x, (float)rv[0].y, (float)rv[0].z, __int_as_float(e));
        v[1] = make_float4((float)rv[1].x, (float)rv[1].y, (float)rv[1].z, 0.f);
        v[2] = make_float4((float)rv[2].x, (float)rv[2].y, (float)rv[2].z, 0.f);
      }
}

// The force, frictional heat and acceleration of law 1 from the nearest surface
// point bq (triangle be of mesh bm, squared distance best; bm < 0: none).
__device__ __forceinline__ void law1_force(const StepParams& P, const Fields& F, int64_t i,
                                           const double4& x4, float4* a32, double best, int bm,
                                           int be, V3 bq) {
  const V3 xi = mk(x4);
  V3 f = mk(0.0, 0.0, 0.0);
  double qf = 0.0;
  int cnt = 0;
  if (bm >= 0) {
    const MeshDev& M = P.mesh[bm];
    // contact normal: from the nearest surface point to the particle (the
    // face normal inside a face, continuous across edges and vertices); the
    // face normal and its signed gap for a centre behind the face
    const V3 dv = xi - bq;
    const double dist = sqrt(best);
    const double gf = dot(dv, mk(M.normal[be]));
    V3 n;
    double g;
    if (gf >= 0.0 && dist > 0.0) {
      n = divide(dv, dist);
      g = dist;
    } else {
      n = mk(M.normal[be]);
      g = gf;
    }
    const double delta = 0.5 * P.c_dx - g;
    if (delta > 0.0) {
      const double fn = P.c_kappa * P.Kbulk * P.c_dx * delta;
      f = scale(n, fn);
      // relative to the tool surface at the nearest point: m_v + m_w x q
      const V3 vtool = mk(M.mv[0], M.mv[1], M.mv[2]) + cross(mk(M.mw[0], M.mw[1], M.mw[2]), bq);
      const V3 vrel = mk(F.vd[i]) - vtool;
      const V3 vt = vrel - scale(n, dot(vrel, n));
      const double vtl = len(vt);
      if (P.mu_s > 0.0) {
        const double s = P.mu_s * fn / (vtl > P.c_vreg ? vtl : P.c_vreg);
        f = f - scale(vt, s);
        qf = P.c_eta * s * vtl * vtl;
      }
      V3 a;
      if (a32) {
        const float4 af = a32[i];
        a = mk(af.x, af.y, af.z);
      } else {
        a = mk(F.a[i]);
      }
      a = a + divide(f, x4.w);
      if (a32) a32[i] = make_float4((float)a.x, (float)a.y, (float)a.z, 0.f);
      else F.a[i] = d4(a);
      cnt = 1;
    }
  }
  F.cf[i] = d4(f);
  F.qf[i] = qf;
  P.ccnt[i] = cnt;
}

// Contact law 1 (the 2M-particle contact workload; no reference
// counterpart).  A solid particle looks up its cell in each tool's triangle
// bins (built once in the tool's frame; the frame moves with node 0) and takes
// the nearest triangle whose closest point q lies within h (ties: first mesh,
// lowest triangle index), searched in FP32 and decided in FP64.  With the gap
// g = |x - q| along n = (x - q)/g (the face normal and the signed gap for a
// centre behind the face) and the penetration delta = dx/2 - g > 0 the normal
// force is
// kappa K dx delta (pressure kappa K / dx on the face dx^2); friction is
// Coulomb, regularised below v_reg: F_t = -mu F_n v_t / max(|v_t|, v_reg);
// eta of the frictional power heats the particle.  Mixed form: the
// acceleration comes from and returns to the FP32 array.
__device__ void law1_one(const StepParams& P, const Fields& F, int64_t i, float4* a32) {
  const double4 x4 = F.xm[i];
  const V3 xi = mk(x4);
  // Pass 1, FP32: the smallest squared distance over the candidate triangles,
  // in coordinates relative to each tool's node 0 (each bin entry carries its
  // triangle's FP32 vertices, so the loads of successive entries overlap).
  float m32 = P.hf * P.hf, tol = 0.f;
  unsigned n32 = 0, n64 = 0;
  for (int m = 0; m < P.ncsid; m++) {
    const MeshDev& M = P.mesh[m];
    const int cell = tool_cell(M, xi.x, xi.y, xi.z);
    if (cell < 0) continue;
    tol = fmaxf(tol, M.tol32);
    const double4 n0 = M.node[0];
    const float3 pr = make_float3((float)(xi.x - n0.x), (float)(xi.y - n0.y), (float)(xi.z - n0.z));
    const int t0 = M.cstart[cell], t1 = M.cstart[cell + 1];
    n32 += (unsigned)(t1 - t0);
#pragma unroll 4
    for (int t = t0; t < t1; t++) {
      const float4* v = M.cvert + 3 * (int64_t)t;
      m32 = fminf(m32, closest_sq32(pr, rel32(v, 0), rel32(v, 1), rel32(v, 2)));
    }
  }
  // Pass 2, FP64: the triangles within tol (in distance) of that minimum, in
  // the order and with the tie rule of a scan of every triangle.  tol is far
  // above the FP32 distance error, so the FP64 minimum is always among them.
  // Candidates are collected first (FP32) and evaluated together: inside the
  // scan, lanes pass the filter at different entries and a warp would run the
  // FP64 test once per such entry.  A lane with more than kCand candidates
  // (never seen on tessellated tools) scans again in FP64.
  constexpr int kCand = 8;
  const float lim = sqrtf(m32) + tol;
  const float thr = lim * lim;
  int cand[kCand];
  int ncand = 0;
  for (int m = 0; m < P.ncsid; m++) {
    const MeshDev& M = P.mesh[m];
    const int cell = tool_cell(M, xi.x, xi.y, xi.z);
    if (cell < 0) continue;
    const double4 n0 = M.node[0];
    const float3 pr = make_float3((float)(xi.x - n0.x), (float)(xi.y - n0.y), (float)(xi.z - n0.z));
    const int t1 = M.cstart[cell + 1];
#pragma unroll 4
    for (int t = M.cstart[cell]; t < t1; t++) {
      const float4* v = M.cvert + 3 * (int64_t)t;
      const float4 v0 = v[0];
      if (closest_sq32(pr, make_float3(v0.x, v0.y, v0.z), rel32(v, 1), rel32(v, 2)) > thr)
        continue;
      if (ncand < kCand) cand[ncand] = (m << 24) | __float_as_int(v0.w);
      ncand++;
    }
  }
  double best = P.h * P.h;
  int bm = -1, be = -1;
  V3 bq = mk(0.0, 0.0, 0.0);
  auto consider = [&](int m, int e) {
    const MeshDev& M = P.mesh[m];
    const int32_t* en = M.elnode + 3 * e;
    const V3 q = closest_on_tri(xi, mk(M.node[en[0]]), mk(M.node[en[1]]), mk(M.node[en[2]]));
    const V3 dv = xi - q;
    const double d2 = dot(dv, dv);
    if (d2 < best || (d2 == best && bm == m && e < be)) {
      best = d2; bm = m; be = e; bq = q;
    }
  };
  if (ncand <= kCand) {
    for (int k = 0; k < ncand; k++) consider(cand[k] >> 24, cand[k] & 0xffffff);
    n64 += (unsigned)ncand;
  } else {
    for (int m = 0; m < P.ncsid; m++) {
      const MeshDev& M = P.mesh[m];
      const int cell = tool_cell(M, xi.x, xi.y, xi.z);
      if (cell < 0) continue;
      const double4 n0 = M.node[0];
      const float3 pr = make_float3((float)(xi.x - n0.x), (float)(xi.y - n0.y), (float)(xi.z - n0.z));
      for (int t = M.cstart[cell]; t < M.cstart[cell + 1]; t++) {
        const float4* v = M.cvert + 3 * (int64_t)t;
        const float4 v0 = v[0];
        if (closest_sq32(pr, make_float3(v0.x, v0.y, v0.z), rel32(v, 1), rel32(v, 2)) > thr)
          continue;
        consider(m, __float_as_int(v0.w));
        n64++;
      }
    }
  }
  {
    const unsigned mask = __activemask();
    const unsigned s32 = __reduce_add_sync(mask, n32), s64 = __reduce_add_sync(mask, n64);
    if ((int)(threadIdx.x & 31) == __ffs(mask) - 1 && s32) {
      atomicAdd(P.cstat, (unsigned long long)s32);
      atomicAdd(P.cstat + 1, (unsigned long long)s64);
    }
  }
  law1_force(P, F, i, x4, a32, best, bm, be, bq);
}

__global__ void __launch_bounds__(128) k_contact_law1(StepParams P, Fields F, float4* a32) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= P.n || F.perm[i] >= P.n_solid) return;
  // most particles are nowhere near a tool and skip all FP64 work; the mixed
  // form keeps an FP32 position mirror
  float px, py, pz;
  if (a32) {
    const float4 p = F.pv[i].p;
    px = p.x; py = p.y; pz = p.z;
  } else {
    const double4 p = F.xm[i];
    px = (float)p.x; py = (float)p.y; pz = (float)p.z;
  }
  if (!law1_near(P, px, py, pz)) {
    F.cf[i] = make_double4(0.0, 0.0, 0.0, 0.0);
    F.qf[i] = 0.0;
    P.ccnt[i] = 0;
    return;
  }
  law1_one(P, F, i, a32);
}

// The slots listed by the fused acceleration pass (those whose cell of a tool's
// bins is not empty): contact, then integration.  kLaw1Lanes lanes per slot
// share its triangles: the search is a chain of loads and FP64 operations, and
// a thread per slot of the widened box, most of them with empty cells, walked
// its few dozen triangles twice and its FP64 candidates one after the other
// (60 us a step with 500k particles and 10,304 triangles, now 34; a warp per
// slot repeats the FP64 work on 32 lanes: 342).  The smallest FP32 distance
// and the smallest (FP64 distance, mesh, triangle) do not depend on the order,
// so the choice is that of law1_one's scan.
constexpr int kLaw1Lanes = 4;
__global__ void __launch_bounds__(64) k_contact_law1_list(StepParams P, Fields F,
                                                          const double4* __restrict__ vd2,
                                                          float4* a32) {
  const int lane = threadIdx.x & (kLaw1Lanes - 1);
  const int slots = gridDim.x * blockDim.x / kLaw1Lanes;
  const int count = *P.near_count;
  const int first = (blockIdx.x * blockDim.x + threadIdx.x) / kLaw1Lanes;
  const unsigned group = ((1u << kLaw1Lanes) - 1u) << ((threadIdx.x & 31) & ~(kLaw1Lanes - 1));
  unsigned n32 = 0, n64 = 0;                  // this lane's triangle tests
  for (int w = first; w < count; w += slots) {
    const int64_t i = P.near_list[w];
    const double4 x4 = F.xm[i];
    const V3 xi = mk(x4);
    // FP32: the smallest squared distance
    float m32 = P.hf * P.hf, tol = 0.f;
    for (int m = 0; m < P.ncsid; m++) {
      const MeshDev& M = P.mesh[m];
      const int cell = tool_cell(M, xi.x, xi.y, xi.z);
      if (cell < 0) continue;
      tol = fmaxf(tol, M.tol32);
      const double4 n0 = M.node[0];
      const float3 pr = make_float3((float)(xi.x - n0.x), (float)(xi.y - n0.y), (float)(xi.z - n0.z));
      const int t1 = M.cstart[cell + 1];
#pragma unroll 4
      for (int t = M.cstart[cell] + lane; t < t1; t += kLaw1Lanes) {
        const float4* v = M.cvert + 3 * (int64_t)t;
        m32 = fminf(m32, closest_sq32(pr, rel32(v, 0), rel32(v, 1), rel32(v, 2)));
        n32++;
      }
    }
#pragma unroll
    for (int o = kLaw1Lanes / 2; o > 0; o >>= 1)
      m32 = fminf(m32, __shfl_xor_sync(group, m32, o));
    // FP64: the triangles within tol of it, with the scan's tie rule; a lane
    // collects its candidates first, so that the lanes evaluate them together
    const float lim = sqrtf(m32) + tol;
    const float thr = lim * lim;
    double best = P.h * P.h;
    int bm = -1, be = -1;
    V3 bq = mk(0.0, 0.0, 0.0);
    auto consider = [&](int m, int e) {
      const MeshDev& M = P.mesh[m];
      const int32_t* en = M.elnode + 3 * e;
      const V3 q = closest_on_tri(xi, mk(M.node[en[0]]), mk(M.node[en[1]]), mk(M.node[en[2]]));
      const V3 dv = xi - q;
      const double d2 = dot(dv, dv);
      n64++;
      if (d2 < best || (d2 == best && bm == m && e < be)) {
        best = d2; bm = m; be = e; bq = q;
      }
    };
    for (int m = 0; m < P.ncsid; m++) {
      const MeshDev& M = P.mesh[m];
      const int cell = tool_cell(M, xi.x, xi.y, xi.z);
      if (cell < 0) continue;
      const double4 n0 = M.node[0];
      const float3 pr = make_float3((float)(xi.x - n0.x), (float)(xi.y - n0.y), (float)(xi.z - n0.z));
      const int t1 = M.cstart[cell + 1];
      int cand = -1;
#pragma unroll 4
      for (int t = M.cstart[cell] + lane; t < t1; t += kLaw1Lanes) {
        const float4* v = M.cvert + 3 * (int64_t)t;
        const float4 v0 = v[0];
        if (closest_sq32(pr, make_float3(v0.x, v0.y, v0.z), rel32(v, 1), rel32(v, 2)) > thr)
          continue;
        const int e = __float_as_int(v0.w);
        if (cand < 0) cand = e;
        else consider(m, e);                   // a lane's second: rare
      }
      if (cand >= 0) consider(m, cand);
    }
    // the group's smallest (distance, mesh, triangle); lanes without one hold h^2 and -1
#pragma unroll
    for (int o = kLaw1Lanes / 2; o > 0; o >>= 1) {
      const double d1 = __shfl_xor_sync(group, best, o);
      const int m1 = __shfl_xor_sync(group, bm, o), e1 = __shfl_xor_sync(group, be, o);
      const V3 q1 = mk(__shfl_xor_sync(group, bq.x, o), __shfl_xor_sync(group, bq.y, o),
                       __shfl_xor_sync(group, bq.z, o));
      if (d1 < best || (d1 == best && (m1 < bm || (m1 == bm && e1 < be)))) {
        best = d1; bm = m1; be = e1; bq = q1;
      }
    }
    if (lane == 0) {
      law1_force(P, F, i, x4, a32, best, bm, be, bq);
      integrate_mixed_one(P, F, vd2, i, a32[i]);
    }
  }
  __syncwarp();
  n32 = __reduce_add_sync(0xffffffffu, n32);
  n64 = __reduce_add_sync(0xffffffffu, n64);
  if ((threadIdx.x & 31) == 0 && n32) {
    atomicAdd(P.cstat, (unsigned long long)n32);
    atomicAdd(P.cstat + 1, (unsigned long long)n64);
  }
}

// Does a particle carry a mesh's zone id without adding exact zeros?  It does
// add them if it is rigid (the pair passes of the mixed form skip its own sums,
// as the filter does), without mass, and with a density and a velocity that
// FP32 holds: 0 / 0 or 0 times infinity would not be zero.
__global__ void __launch_bounds__(256) k_zone_mass(StepParams P, Fields F, int* flag) {
  bool any = false;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < P.n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t id = F.id[i];
    bool zone = false;
    for (int m = 0; m < P.ncsid; m++) zone |= id == P.csid[m];
    if (!zone) continue;
    const double4 v = F.vd[i];
    const float rho = (float)v.w;
    any |= F.perm[i] < P.n_solid || F.xm[i].w != 0.0 || !(rho > 0.0f) || !isfinite(rho) ||
           !isfinite((float)v.x) || !isfinite((float)v.y) || !isfinite((float)v.z);
  }
  if (any) *flag = 1;
}

__global__ void k_mesh_move(MeshDev M, double dt) {
  mesh_move_one(M, dt, blockIdx.x * blockDim.x + threadIdx.x);
}

// CalcCentroids, CalcNormals and UpdatePlaneCoeff of one element from the
// moved nodes; the plane coefficient reads node[elnode[3e] + nfar] with
// nfar = 2, the index CalcSpheres leaves (Mesh.cu:205-231).  Then
// UpdateContactParticles: the element's rigid particle takes the mean node
// velocity, zero acceleration and the element normal.  `plane`: only the plane
// coefficient.
__global__ void k_mesh_elems(StepParams P, Fields F, MeshDev M, int plane, int mixed) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= M.ne) return;
  if (plane) {
    M.pplane[e] = dot(mk(M.node[M.elnode[3 * e] + 2]), mk(M.normal[e]));
    return;
  }
  const int e0 = M.elnode[3 * e], e1 = M.elnode[3 * e + 1], e2 = M.elnode[3 * e + 2];
  const V3 n0 = mk(M.node[e0]), n1 = mk(M.node[e1]), n2 = mk(M.node[e2]);
  M.centroid[e] = d4(divide((n0 + n1) + n2, 3.));
  const V3 w = cross(n1 - n0, n2 - n0);
  const V3 normal = divide(w, len(w));
  M.normal[e] = d4(normal);
  M.pplane[e] = dot(mk(M.node[e0 + 2]), normal);
  const int32_t s = P.inv[M.first + e];
  const V3 vv = ((mk(0.0, 0.0, 0.0) + mk(M.node_v[e0])) + mk(M.node_v[e1])) + mk(M.node_v[e2]);
  const V3 v = divide(vv, 3.);
  const double rho = F.vd[s].w;
  F.vd[s] = d4(v, rho);
  F.a[s] = make_double4(0.0, 0.0, 0.0, 0.0);
  F.nrm[s] = d4(normal);
  if (mixed) {
    float4& m = F.pv[s].v;
    m.x = (float)v.x; m.y = (float)v.y; m.z = (float)v.z;
  }
}

inline int blocks_for(int64_t n, int t) { return (int)((n + t - 1) / t); }

}  // namespace

int launch_contact_stage(const StepParams& P, const Fields& F, const NbBuffers& N, bool list,
                         float4* a32, cudaStream_t s) {
  if (P.contact_law == 1) {
    int launches = 0;
    for (int m = 0; m < P.ncsid; m++) {   // rotating tools: bins from the current nodes
      const MeshDev& M = P.mesh[m];
      if (!M.rot) continue;
      const int64_t ncell = (int64_t)M.dims[0] * M.dims[1] * M.dims[2];
      cudaMemsetAsync(M.cstart, 0, sizeof(uint32_t) * (ncell + 1), s);
      k_bins_count<<<blocks_for(M.ne, 128), 128, 0, s>>>(M);
      launches +=
          2 + device_exclusive_scan(reinterpret_cast<uint32_t*>(M.cstart), ncell + 1, M.scan_tmp, s);
      cudaMemcpyAsync(M.cursor, M.cstart, sizeof(uint32_t) * ncell, cudaMemcpyDeviceToDevice, s);
      k_bins_fill<<<blocks_for(M.ne, 128), 128, 0, s>>>(M);
    }
    if (P.near_count) return launches;
    k_contact_law1<<<blocks_for(P.n, 128), 128, 0, s>>>(P, F, a32);
    return launches + 1;
  }
  const int lanes = lanes64(P.n), grid = blocks_for(P.n * lanes, lanes == 1 ? 64 : 32);
  if (lanes == 32) k_surface<32><<<grid, 32, 0, s>>>(P, F, N.nb, N.cnt);
  else if (lanes == 16) k_surface<16><<<grid, 32, 0, s>>>(P, F, N.nb, N.cnt);
  else if (lanes == 8) k_surface<8><<<grid, 32, 0, s>>>(P, F, N.nb, N.cnt);
  else k_surface<1><<<grid, 64, 0, s>>>(P, F, N.nb, N.cnt);
  if (lanes > 1) {
    const int grid8 = blocks_for(P.n * 8, 32);
    if (list) k_contact_nb<8><<<grid8, 32, 0, s>>>(P, F, N.nb, N.cnt);
    k_contact_force<8><<<grid8, 32, 0, s>>>(P, F, a32);
  } else {
    if (list) k_contact_nb<1><<<grid, 64, 0, s>>>(P, F, N.nb, N.cnt);
    k_contact_force<1><<<grid, 64, 0, s>>>(P, F, a32);
  }
  return list ? 3 : 2;
}

void launch_contact_law1_list(const StepParams& P, const Fields& F, const double4* vd2,
                              float4* a32, cudaStream_t s) {
  // a few thousand slots in practice (16 a block); a larger list loops
  k_contact_law1_list<<<std::min(blocks_for(P.n * kLaw1Lanes, 64), 912), 64, 0, s>>>(P, F, vd2,
                                                                                     a32);
}
void launch_zone_mass(const StepParams& P, const Fields& F, int* flag, cudaStream_t s) {
  k_zone_mass<<<std::min(blocks_for(P.n, 256), 1024), 256, 0, s>>>(P, F, flag);
}

void launch_mesh_update(const StepParams& P, const Fields& F, int mixed, bool moved,
                        cudaStream_t s) {
  for (int m = 0; m < P.ncsid && !moved; m++)
    k_mesh_move<<<blocks_for(P.mesh[m].nn, 128), 128, 0, s>>>(P.mesh[m], P.dt);
  for (int m = 0; m < P.ncsid; m++)
    k_mesh_elems<<<blocks_for(P.mesh[m].ne, 64), 64, 0, s>>>(P, F, P.mesh[m], 0, mixed);
}

void launch_mesh_plane(const StepParams& P, const Fields& F, cudaStream_t s) {
  for (int m = 0; m < P.ncsid; m++)
    k_mesh_elems<<<blocks_for(P.mesh[m].ne, 64), 64, 0, s>>>(P, F, P.mesh[m], 1, 0);
}
