// separable.cuh -- the densities and the field projection of a basis whose functions
// are products of a z part and a radial part.
//
// The oscillator functions of the reference (hfbtho_solver.f90:3463-3671) on its
// Gauss-Hermite x Gauss-Laguerre mesh, r = (ih, il), are
//   phi_0(a) = s R(il) Z(ih)        phi_1(a) = s R'(il) Z(ih)      (d/dr)
//   phi_3(a) = s R(il) Z'(ih)       (d/dz)
//   phi_2(a) = lambda y(il) phi_0   (Lambda / r, one lambda per block and spin)
//   phi_4(a) = (V(ih, il) - e_a) phi_0   (Laplacian of an oscillator function)
// with one Z per n_z and one R per (n_r, |Lambda|).  Every density and every projection
// (pnfam_hamiltonian_blas.f90:124-711, :1107-1167, :1212-1260) is a sum over pairs of
// states and mesh points of products of two of these, so the sums can be taken one
// direction at a time:
//   density     G[u](il)   = sum over the pairs (a, b) of unit u of R_a R_b rho_ab
//               C(q, q')   = sum over the units of Z Z' G           -> 28 densities
//   projection  H[u](il)   = sum over ih of Z Z' mf(q, q')(ih, il)
//               h_ab       = 2 sum over il of R_a R_b H[u]
// where a unit u = (spin class, n_z, n_z') collects the element pairs of every block
// with these z functions.  Per matrix element this costs the mesh points of one
// direction instead of the whole mesh, and the sums over the blocks come before the
// other direction is expanded: about 0.15 GFLOP per point at N_sh = 16 (20 x 20 mesh)
// against 3.5 GFLOP of the sums over the whole mesh.  Measured there, per point, FP64
// (nine points): densities 0.14 ms against 2.2 ms, projection 0.18 against 2.7 ms; FP32
// (40 points): 23 and 18 us against 39 and 41 us of the pair-tensor GEMMs, whose operand
// (12 GB) is not needed; errors against FP64 2e-7 instead of 8e-6.
//
// The factors are recovered from the basis functions that the caller passes
// (sep_factors) and every value of the products is compared with them (k_sep_check);
// a basis that is not of this form keeps the general kernels.
#pragma once
#include <math.h>

#include <algorithm>
#include <vector>

#ifdef __CUDACC__
#define SEP_HD __host__ __device__ __forceinline__
#else
#define SEP_HD inline
#endif

namespace pnfam {

// ---------------------------------------------------------------------------
// factors
// ---------------------------------------------------------------------------
struct SepBasis {
  int ngh = 0, ngl = 0, nzf = 0, nrow = 0;
  std::vector<double> z;      // [nzf][2][ngh]   Z, Z'
  std::vector<double> r;      // [nrow][ngl][2]  R, R'
  std::vector<double> v;      // [nghl]
  std::vector<double> y;      // [ngl]
  std::vector<double> e;      // [dqp]
  std::vector<double> lam, sgn;   // [2 nb] per (block, spin)
  std::vector<int> zi, ri;    // [dqp] z function and radial row of a state
};

// largest relative deviation that the factor form may have from the basis functions:
// the products differ from stored functions by a few roundings (1e-15 measured for the
// reference's functions)
constexpr double SEP_TOL = 2e-13;

// component q of state a at (ih, il) from the factors
SEP_HD double sep_value(int q, const double* z, const double* r, double v, double y, double e, double lam, double sgn,
                        int ih, int il, int ngh, int zi, int ri, int ngl) {
  const double Z = z[(zi * 2) * ngh + ih], Zd = z[(zi * 2 + 1) * ngh + ih];
  const double R = r[(ri * ngl + il) * 2], Rd = r[(ri * ngl + il) * 2 + 1];
  switch (q) {
    case 0: return sgn * R * Z;
    case 1: return sgn * Rd * Z;
    case 2: return lam * y * (sgn * R * Z);
    case 3: return sgn * R * Zd;
    default: return (v - e) * (sgn * R * Z);
  }
}

// the factors of phi [5][dqp][nghl] for a mesh of ngh points along z; false when the
// functions are plainly not of the product form (sep_value still has to be compared)
inline bool sep_factors(int nb, const int* db, const int* st, const int* nup, int dqp, int nghl, int ngh,
                        const double* phi, SepBasis& B) {
  const int ngl = nghl / ngh;
  const size_t ps = (size_t)dqp * nghl;
  B = SepBasis();
  B.ngh = ngh; B.ngl = ngl;
  B.zi.assign(dqp, 0); B.ri.assign(dqp, 0); B.e.assign(dqp, 0.0);
  B.lam.assign(2 * nb, 0.0); B.sgn.assign(2 * nb, 1.0);
  B.v.assign(nghl, 0.0); B.y.assign(ngl, 0.0);
  std::vector<int> zstar;               // ih of the largest |Z| of each z function
  std::vector<double> ztop;             // and Z there
  std::vector<std::vector<double>> lseg(2 * nb);
  std::vector<double> row(ngl * 2), wbest(ngl);
  for (int i = 0; i < nb; ++i)
    for (int s = 0; s < 2; ++s) {
      const int lo = st[i] + (s ? nup[i] : 0), hi = s ? st[i] + db[i] : st[i] + nup[i];
      std::vector<double> c(ngl, 0.0);
      std::fill(wbest.begin(), wbest.end(), 0.0);
      bool first = true;
      for (int a = lo; a < hi; ++a) {
        const double* f = phi + (size_t)a * nghl;
        int m = 0;
        for (int k = 1; k < nghl; ++k)
          if (fabs(f[k]) > fabs(f[m])) m = k;
        const double top = fabs(f[m]);
        if (!(top > 0.0) || !std::isfinite(top)) return false;
        const int ls = m / ngh, hs = m % ngh;
        const double* p = f + (size_t)ls * ngh;   // the state along z at its largest point
        int c0 = -1;
        for (int k = 0; k < B.nzf && c0 < 0; ++k) {
          const double q = p[zstar[k]] / ztop[k];
          double d = 0.0;
          for (int h = 0; h < ngh; ++h) d = fmax(d, fabs(p[h] - q * B.z[(size_t)(2 * k) * ngh + h]));
          if (d <= SEP_TOL * top) c0 = k;
        }
        if (c0 < 0) {
          if (B.nzf >= 256) return false;   // not a product basis of any size in use
          // scaled so that the state's radial function is a row that is there already,
          // if there is one: every (n_r, |Lambda|) then has one row for all n_z
          double scale = 1.0;
          for (int k = 0; k < B.nrow; ++k) {
            const double *rk = &B.r[(size_t)k * ngl * 2], sg = B.sgn[2 * i + s];
            if (rk[2 * ls] == 0.0) continue;
            const double al = f[(size_t)ls * ngh + hs] / (sg * rk[2 * ls]);
            double d0 = 0.0, d1 = 0.0, dtop = 0.0;
            for (int l = 0; l < ngl; ++l) {
              const double fd = phi[ps + (size_t)a * nghl + (size_t)l * ngh + hs];
              d0 = fmax(d0, fabs(f[(size_t)l * ngh + hs] - al * sg * rk[2 * l]));
              d1 = fmax(d1, fabs(fd - al * sg * rk[2 * l + 1]));
              dtop = fmax(dtop, fabs(fd));
            }
            if (d0 <= SEP_TOL * top && d1 <= SEP_TOL * dtop) { scale = al; break; }
          }
          c0 = B.nzf++;
          zstar.push_back(hs);
          ztop.push_back(scale);
          for (int h = 0; h < ngh; ++h) B.z.push_back(scale * (p[h] / p[hs]));
          const double* g = phi + 3 * ps + (size_t)a * nghl + (size_t)ls * ngh;
          for (int h = 0; h < ngh; ++h) B.z.push_back(scale * (g[h] / p[hs]));
        }
        B.zi[a] = c0;
        double rtop = 0.0, dtop = 0.0;
        for (int l = 0; l < ngl; ++l) {
          row[2 * l] = f[(size_t)l * ngh + zstar[c0]] / ztop[c0];
          row[2 * l + 1] = phi[ps + (size_t)a * nghl + (size_t)l * ngh + zstar[c0]] / ztop[c0];
          rtop = fmax(rtop, fabs(row[2 * l]));
          dtop = fmax(dtop, fabs(row[2 * l + 1]));
          const double g2 = phi[2 * ps + (size_t)a * nghl + (size_t)l * ngh + zstar[c0]];
          if (fabs(row[2 * l]) > wbest[l]) { wbest[l] = fabs(row[2 * l]); c[l] = g2 / ztop[c0] / row[2 * l]; }
        }
        auto find = [&](double sg) {
          for (int k = 0; k < B.nrow; ++k) {
            double d0 = 0.0, d1 = 0.0;
            for (int l = 0; l < ngl; ++l) {
              d0 = fmax(d0, fabs(row[2 * l] - sg * B.r[((size_t)k * ngl + l) * 2]));
              d1 = fmax(d1, fabs(row[2 * l + 1] - sg * B.r[((size_t)k * ngl + l) * 2 + 1]));
              if (d0 > SEP_TOL * rtop) break;
            }
            if (d0 <= SEP_TOL * rtop && d1 <= SEP_TOL * dtop) return k;
          }
          return -1;
        };
        int k = first || B.sgn[2 * i + s] > 0 ? find(1.0) : find(-1.0);
        if (first && k < 0 && (k = find(-1.0)) >= 0) B.sgn[2 * i + s] = -1.0;
        if (k < 0) {
          if (B.nrow >= 4096) return false;
          k = B.nrow++;
          for (double x : row) B.r.push_back(B.sgn[2 * i + s] * x);
        }
        B.ri[a] = k;
        first = false;
      }
      lseg[2 * i + s] = c;
    }
  // lambda per segment: multiples of one y(il), that of the segment with the largest
  int ref = -1;
  double big = 0.0;
  for (int k = 0; k < 2 * nb; ++k) {
    double n = 0.0;
    for (double x : lseg[k]) n += x * x;
    if (n > big) { big = n; ref = k; }
  }
  if (ref >= 0) {
    B.y = lseg[ref];
    for (int k = 0; k < 2 * nb; ++k) {
      double d = 0.0;
      for (int l = 0; l < ngl && !lseg[k].empty(); ++l) d += lseg[k][l] * B.y[l];
      B.lam[k] = d / big;
    }
  }
  // V and e: phi_4 / phi_0 = V - e_a, each taken where the state is large
  std::vector<double> w(nghl, 0.0);
  for (int pass = 0; pass < 2; ++pass)
    for (int a = 0; a < dqp; ++a) {
      const double *f = phi + (size_t)a * nghl, *g = phi + 4 * ps + (size_t)a * nghl;
      double top = 0.0, s0 = 0.0, s1 = 0.0;
      for (int k = 0; k < nghl; ++k) top = fmax(top, fabs(f[k]));
      for (int k = 0; k < nghl; ++k) {
        const double x = fabs(f[k]);
        if (x < 1e-2 * top || w[k] == 0.0) continue;
        s0 += x * w[k];
        s1 += x * w[k] * (B.v[k] - g[k] / f[k]);
      }
      if (s0 > 0.0) B.e[a] = s1 / s0;
      if (pass == 0)
        for (int k = 0; k < nghl; ++k)
          if (fabs(f[k]) > w[k]) { w[k] = fabs(f[k]); B.v[k] = g[k] / f[k] + B.e[a]; }
    }
  return true;
}

// mesh points along z: the divisor of nghl for which the largest states are products
inline int sep_mesh(int dqp, int nghl, const double* phi) {
  for (int ngh = 2; ngh <= nghl / 2; ++ngh) {
    if (nghl % ngh) continue;
    const int ngl = nghl / ngh;
    bool ok = true;
    for (int a = 0; a < dqp && ok; a += std::max(1, dqp / 16)) {
      const double* f = phi + (size_t)a * nghl;
      int m = 0;
      for (int k = 1; k < nghl; ++k)
        if (fabs(f[k]) > fabs(f[m])) m = k;
      const int ls = m / ngh, hs = m % ngh;
      if (f[m] == 0.0) { ok = false; break; }
      for (int l = 0; l < ngl && ok; ++l)
        for (int h = 0; h < ngh && ok; ++h) {
          const double want = f[(size_t)l * ngh + hs] * (f[(size_t)ls * ngh + h] / f[m]);
          ok = fabs(f[(size_t)l * ngh + h] - want) <= SEP_TOL * fabs(f[m]);
        }
    }
    if (ok) return ngh;
  }
  return 0;
}

// ---------------------------------------------------------------------------
// units of one block structure
// ---------------------------------------------------------------------------
struct SepUnit { int cls, nz, nzp, ent0, nent; };   // spin class 2 (s_a < 0) + (s_b < 0)
// one (block, spin) x (block, spin) part of a unit: ng radial rows of its row states,
// ngp of its column states, the elements in the order (column state, row state)
struct SepEnt { int ng, ngp, row0, rowp0, el0, seg, segp; };

enum { SEP_GC = 5, SEP_STAGE = 512 };   // column states per projection item; elements staged at a time

struct SepItem {        // one row state against up to SEP_GC column states of a unit
  int seg, segp, ja, row, n;
  int jb[SEP_GC], rowp[SEP_GC], off[SEP_GC];
};
struct SepWarp { int unit, item0, nitem, nmax; };   // 32 items of one unit (nmax: their largest n)

struct SepStruct {
  std::vector<SepUnit> units;      // by (class, n_z', n_z)
  std::vector<SepEnt> ents;
  std::vector<int> rows, offs, ubeg, order;   // ubeg [4][nzf + 1]: first unit of (class, n_z'); order: largest first
  std::vector<SepItem> items;
  std::vector<SepWarp> warps;
};

// cols, offs_: the block structure; items: also the projection's items.  false when a
// part of a unit does not fit the staging buffer
inline bool sep_structure(const SepBasis& B, int nb, const int* db, const int* st, const int* nup, const int* cols,
                          const long long* boff, bool project, SepStruct& S) {
  S = SepStruct();
  const int nzf = B.nzf;
  struct Part { int i, s, j, t; };
  std::vector<Part> parts[4];
  for (int i = 0; i < nb; ++i) {
    const int j = cols[i];
    if (j < 0) continue;
    for (int s = 0; s < 2; ++s)
      for (int t = 0; t < 2; ++t) parts[2 * s + t].push_back({i, s, j, t});
  }
  // states of each (block, spin) by z function
  std::vector<std::vector<std::vector<int>>> byz(2 * nb, std::vector<std::vector<int>>(nzf));
  for (int i = 0; i < nb; ++i)
    for (int a = st[i]; a < st[i] + db[i]; ++a) byz[2 * i + (a - st[i] >= nup[i])][B.zi[a]].push_back(a);
  for (int c = 0; c < 4; ++c)
    for (int zp = 0; zp < nzf; ++zp) {
      S.ubeg.push_back((int)S.units.size());
      for (int z = 0; z < nzf; ++z) {
        SepUnit u{c, z, zp, (int)S.ents.size(), 0};
        const int item0 = (int)S.items.size();
        for (const Part& p : parts[c]) {
          const std::vector<int>&A = byz[2 * p.i + p.s][z], &C = byz[2 * p.j + p.t][zp];
          if (A.empty() || C.empty()) continue;
          SepEnt en{(int)A.size(), (int)C.size(), (int)S.rows.size(), 0, (int)S.offs.size(), 2 * p.i + p.s,
                    2 * p.j + p.t};
          if ((long long)en.ng * en.ngp > SEP_STAGE) return false;
          for (int a : A) S.rows.push_back(B.ri[a]);
          en.rowp0 = (int)S.rows.size();
          for (int b : C) S.rows.push_back(B.ri[b]);
          auto off = [&](int a, int b) {
            return (int)(boff[p.i] + (a - st[p.i]) + (long long)(b - st[p.j]) * db[p.i]);
          };
          for (int b : C)
            for (int a : A) S.offs.push_back(off(a, b));
          if (project) {
            // columns in nearly equal groups of at most SEP_GC
            const int nc = ((int)C.size() + SEP_GC - 1) / SEP_GC;
            for (int k = 0; k < nc; ++k) {
              const int b0 = (int)C.size() * k / nc, b1 = (int)C.size() * (k + 1) / nc;
              for (int a : A) {
                SepItem it{};
                it.seg = en.seg; it.segp = en.segp; it.ja = a; it.row = B.ri[a]; it.n = b1 - b0;
                for (int b = b0; b < b1; ++b) {
                  it.jb[b - b0] = C[b]; it.rowp[b - b0] = B.ri[C[b]]; it.off[b - b0] = off(a, C[b]);
                }
                S.items.push_back(it);
              }
            }
          }
          S.ents.push_back(en);
        }
        u.nent = (int)S.ents.size() - u.ent0;
        if (!u.nent) continue;
        if (project) {
          // items of one size next to each other, so that a warp's lanes run the same loop
          std::stable_sort(S.items.begin() + item0, S.items.end(),
                           [](const SepItem& x, const SepItem& y) { return x.n > y.n; });
          for (int k = item0; k < (int)S.items.size(); k += 32)
            S.warps.push_back({(int)S.units.size(), k, std::min(32, (int)S.items.size() - k), S.items[k].n});
        }
        S.units.push_back(u);
      }
      if (zp == nzf - 1) S.ubeg.push_back((int)S.units.size());
    }
  auto work = [&](const SepUnit& u) {
    long long n = 0;
    for (int k = u.ent0; k < u.ent0 + u.nent; ++k) n += (long long)S.ents[k].ng * S.ents[k].ngp;
    return n;
  };
  std::vector<long long> w;
  for (const SepUnit& u : S.units) { S.order.push_back((int)w.size()); w.push_back(work(u)); }
  std::stable_sort(S.order.begin(), S.order.end(), [&](int x, int y) { return w[x] > w[y]; });
  std::stable_sort(S.warps.begin(), S.warps.end(), [](const SepWarp& x, const SepWarp& y) { return x.nmax > y.nmax; });
  return true;
}

// sums of a unit at one radial point that the density keeps (lambda factors per part):
// products of the row side's and the column side's radial functions
enum { SG_RR = 0, SG_DR, SG_RD, SG_DD, SG_ARR, SG_BRR, SG_ABRR, SG_BDR, SG_ARD, SG_N };
// the projection's unit fields: the same nine, then the (0, 4) and (4, 0) field
enum { SH_L = SG_N, SH_N };

}  // namespace pnfam

#ifdef __CUDACC__
namespace pnfam {

template <class T> struct Vec2;
template <> struct Vec2<float> { using t = float2; };
template <> struct Vec2<double> { using t = double2; };

struct SepStructDev {
  const SepUnit* units;
  const SepEnt* ents;
  const int *rows, *offs, *ubeg, *order;
  const SepItem* items;
  const SepWarp* warps;
  int nu, nwarp;
};

template <class T>
struct SepDev {
  int ngh, ngl, nzf, nghl;
  const typename Vec2<T>::t* r;   // [nrow][ngl] (R, R')
  const T *z, *v, *y, *e, *lam, *sgn;
  SepStructDev f, k[2], d[2];     // F; pairing densities (X^T, Y^T); pairing fields (X, Y)
  // unit sums of one point: per call the F units [ngl][nu][SH_N][2 planes], then per
  // call the pairing units [ngl][nu][2 planes]
  long long gstride, gpair[2];
  T* g;                           // [P][gstride]
  // the points of a launch: a list, or (list null) all P with their flags
  const int *list, *act;
  int n;
};

template <class T>
__device__ __forceinline__ int sep_point(const SepDev<T>& S, int i) {
  if (i >= S.n) return -1;
  if (S.list) return S.list[i];
  return S.act[i] ? i : -1;
}

// every basis function against its factors: *bad = 1 where one is off by more than
// SEP_TOL of the state's largest value of the component.  grid (dqp), 128 threads
__global__ void __launch_bounds__(128) k_sep_check(const double* __restrict__ phi, int dqp, int nghl, int ngh,
                                                   const double* __restrict__ z, const double* __restrict__ r,
                                                   const double* __restrict__ v, const double* __restrict__ y,
                                                   const double* __restrict__ e, const double* __restrict__ lam,
                                                   const double* __restrict__ sgn, const int* __restrict__ zi,
                                                   const int* __restrict__ ri, const int* __restrict__ seg,
                                                   int* __restrict__ bad) {
  const int a = blockIdx.x, ngl = nghl / ngh, sg = seg[a];
  __shared__ double sh[4];
  for (int q = 0; q < 5; ++q) {
    const double* f = phi + ((long long)q * dqp + a) * nghl;
    double top = 0.0;
    for (int k = threadIdx.x; k < nghl; k += 128) top = fmax(top, fabs(f[k]));
    for (int o = 16; o > 0; o >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = top;
    __syncthreads();
    top = fmax(fmax(sh[0], sh[1]), fmax(sh[2], sh[3]));
    for (int k = threadIdx.x; k < nghl; k += 128) {
      const int ih = k % ngh, il = k / ngh;
      const double w = sep_value(q, z, r, v[k], y[il], e[a], lam[sg], sgn[sg], ih, il, ngh, zi[a], ri[a], ngl);
      if (!(fabs(f[k] - w) <= SEP_TOL * top)) atomicExch(bad, 1);   // a NaN too
    }
  }
}

// ---------------------------------------------------------------------------
// densities 1: the radial sums of every unit.  A CTA takes one unit and NPT points; a
// thread one radial point and one column (point, call, plane).  The unit's elements are
// gathered into shared memory and every part is summed over its row states, then over
// its column states.  FP64: bound by the FP64 pipe (2 DFMA per element, radial point
// and column); FP32: by shared-memory and L1 loads.
// grid (units of F, X^T and Y^T; point groups)
// ---------------------------------------------------------------------------
template <class T, int KT, bool NORMAL>
__device__ __forceinline__ void sep_tile(const typename Vec2<T>::t* __restrict__ r, const int* __restrict__ rows,
                                         const int* __restrict__ rowsp, int ng, const T* s, int ld, int ir, int ngl,
                                         T (&o)[4]) {
  T t0[KT], t1[KT];
#pragma unroll
  for (int k = 0; k < KT; ++k) t0[k] = t1[k] = T(0);
#pragma unroll 3
  for (int g = 0; g < ng; ++g) {
    const typename Vec2<T>::t ra = r[rows[g] * ngl + ir];
#pragma unroll
    for (int k = 0; k < KT; ++k) {
      const T x = s[(k * ng + g) * ld];
      t0[k] = fma(ra.x, x, t0[k]);
      if (NORMAL) t1[k] = fma(ra.y, x, t1[k]);
    }
  }
#pragma unroll
  for (int k = 0; k < KT; ++k) {
    const typename Vec2<T>::t rb = r[rowsp[k] * ngl + ir];
    o[0] = fma(rb.x, t0[k], o[0]);
    if (NORMAL) {
      o[1] = fma(rb.x, t1[k], o[1]);
      o[2] = fma(rb.y, t0[k], o[2]);
      o[3] = fma(rb.y, t1[k], o[3]);
    }
  }
}

template <class T, int NPT, bool NORMAL>
__device__ __forceinline__ void sep_radial_unit(const SepDev<T>& S, const SepStructDev& X, int ui, int call,
                                                const T* __restrict__ rsp, long long nxy, T* sx) {
  constexpr int NC = (NORMAL ? 4 : 2) * NPT;   // columns: (point, call, plane) or (point, plane)
  const SepUnit u = X.units[ui];
  const int ngl = S.ngl;
  const SepEnt* en = X.ents + u.ent0;
  for (int t0 = 0; t0 < ngl * NC; t0 += blockDim.x) {
    const int t = t0 + threadIdx.x, ir = t % ngl, col = t / ngl;
    const bool live = t < ngl * NC;
    T acc[SG_N];
#pragma unroll
    for (int k = 0; k < SG_N; ++k) acc[k] = T(0);
    for (int e0 = 0; e0 < u.nent;) {
      // the parts that fit the staging buffer together
      int e1 = e0, nel = 0;
      while (e1 < u.nent && nel + en[e1].ng * en[e1].ngp <= SEP_STAGE) { nel += en[e1].ng * en[e1].ngp; ++e1; }
      const int el0 = en[e0].el0;
      __syncthreads();
      for (int c = 0; c < NC; ++c) {
        const int p = sep_point(S, blockIdx.y * NPT + (NORMAL ? c >> 2 : c >> 1));
        if (p < 0) {
          for (int k = threadIdx.x; k < nel; k += blockDim.x) sx[k * NC + c] = T(0);
          continue;
        }
        const int quad = NORMAL ? ((c >> 1) & 1 ? 3 : 0) : (call ? 2 : 1);
        const T* src = rsp + ((long long)p * 2 + (c & 1)) * 4 * nxy + (long long)quad * nxy;
        for (int k = threadIdx.x; k < nel; k += blockDim.x) sx[k * NC + c] = src[X.offs[el0 + k]];
      }
      __syncthreads();
      if (live) {
        for (int e = e0; e < e1; ++e) {
          const SepEnt q = en[e];
          const int *ra = X.rows + q.row0, *rb = X.rows + q.rowp0;
          const T* s = sx + (q.el0 - el0) * NC + col;
          T o[4] = {T(0), T(0), T(0), T(0)};
          int k = 0;
          if (sizeof(T) == 4)
            for (; k + 4 <= q.ngp; k += 4) sep_tile<T, 4, NORMAL>(S.r, ra, rb + k, q.ng, s + k * q.ng * NC, NC, ir, ngl, o);
          for (; k + 2 <= q.ngp; k += 2) sep_tile<T, 2, NORMAL>(S.r, ra, rb + k, q.ng, s + k * q.ng * NC, NC, ir, ngl, o);
          if (k < q.ngp) sep_tile<T, 1, NORMAL>(S.r, ra, rb + k, q.ng, s + k * q.ng * NC, NC, ir, ngl, o);
          const T sg = S.sgn[q.seg] * S.sgn[q.segp];
          acc[SG_RR] = fma(sg, o[0], acc[SG_RR]);
          if (NORMAL) {
            const T la = S.lam[q.seg] * sg, lb = S.lam[q.segp];
            acc[SG_DR] = fma(sg, o[1], acc[SG_DR]);
            acc[SG_RD] = fma(sg, o[2], acc[SG_RD]);
            acc[SG_DD] = fma(sg, o[3], acc[SG_DD]);
            acc[SG_ARR] = fma(la, o[0], acc[SG_ARR]);
            acc[SG_BRR] = fma(lb * sg, o[0], acc[SG_BRR]);
            acc[SG_ABRR] = fma(la * lb, o[0], acc[SG_ABRR]);
            acc[SG_BDR] = fma(lb * sg, o[1], acc[SG_BDR]);
            acc[SG_ARD] = fma(la, o[2], acc[SG_ARD]);
          }
        }
      }
      e0 = e1;
    }
    if (!live) continue;
    const int p = sep_point(S, blockIdx.y * NPT + (NORMAL ? col >> 2 : col >> 1));
    if (p < 0) continue;
    T* g = S.g + p * S.gstride;
    if (NORMAL) {
      const T y = S.y[ir];
      g += ((long long)(((col >> 1) & 1) * ngl + ir) * X.nu + ui) * (2 * SH_N) + (col & 1);
      g[2 * SG_RR] = acc[SG_RR];
      g[2 * SG_DR] = acc[SG_DR];
      g[2 * SG_RD] = acc[SG_RD];
      g[2 * SG_DD] = acc[SG_DD];
      g[2 * SG_ARR] = y * acc[SG_ARR];
      g[2 * SG_BRR] = y * acc[SG_BRR];
      g[2 * SG_ABRR] = y * y * acc[SG_ABRR];
      g[2 * SG_BDR] = y * acc[SG_BDR];
      g[2 * SG_ARD] = y * acc[SG_ARD];
    } else {
      g[S.gpair[call] + ((long long)ir * X.nu + ui) * 2 + (col & 1)] = acc[SG_RR];
    }
  }
}

template <class T, int NPT>
__global__ void __launch_bounds__(256) k_sep_radial(const __grid_constant__ SepDev<T> S, const T* __restrict__ rsp,
                                                    long long nxy) {
  __shared__ __align__(16) T sx[SEP_STAGE * 4 * NPT];
  if (NPT == 1 && sep_point(S, blockIdx.y) < 0) return;
  int b = blockIdx.x;
  if (b < S.f.nu) { sep_radial_unit<T, NPT, true>(S, S.f, S.f.order[b], 0, rsp, nxy, sx); return; }
  b -= S.f.nu;
  if (b < S.k[0].nu) sep_radial_unit<T, NPT, false>(S, S.k[0], S.k[0].order[b], 0, rsp, nxy, sx);
  else sep_radial_unit<T, NPT, false>(S, S.k[1], S.k[1].order[b - S.k[0].nu], 1, rsp, nxy, sx);
}

// ---------------------------------------------------------------------------
// densities 2: the z sums of one radial point, call and class, folded into the class's
// share of the 28 densities: dpart [P][2 calls][4 classes][2 ND][nghl].  A thread takes
// one z point and every ng-th n_z' (ng groups of ngh threads).
// grid (ngl, 2 calls x 4 classes, points), ngh * ng threads
// ---------------------------------------------------------------------------
template <class T>
__host__ __device__ inline size_t sep_dens_smem(int ngh, int ng) { return (size_t)ng * 34 * ngh * sizeof(T); }

template <class T>
__global__ void __launch_bounds__(256) k_sep_density(const __grid_constant__ SepDev<T> S, int ng,
                                                     T* __restrict__ dpart) {
  const int p = sep_point(S, blockIdx.z);
  if (p < 0) return;
  const int ir = blockIdx.x, call = blockIdx.y >> 2, cls = blockIdx.y & 3;
  const int ngh = S.ngh, nzf = S.nzf;
  extern __shared__ __align__(16) unsigned char smraw[];
  T* red = reinterpret_cast<T*>(smraw);   // [ng][34][ngh]
  const int ih = threadIdx.x % ngh, grp = threadIdx.x / ngh;
  // C(q, q') at q * 4 + q', (re, im); then the pairing sum
  T C[17][2];
#pragma unroll
  for (int k = 0; k < 17; ++k) C[k][0] = C[k][1] = T(0);
  using V2 = typename Vec2<T>::t;
  const T* gp = S.g + p * S.gstride;
  for (int zp = grp; zp < nzf; zp += ng) {
    const T Zp = S.z[(2 * zp) * ngh + ih], Zdp = S.z[(2 * zp + 1) * ngh + ih];
    {
      const V2* g = reinterpret_cast<const V2*>(gp) + (long long)(call * S.ngl + ir) * S.f.nu * SH_N;
      T A[SG_N][2], D[3][2];
#pragma unroll
      for (int k = 0; k < SG_N; ++k) A[k][0] = A[k][1] = T(0);
#pragma unroll
      for (int k = 0; k < 3; ++k) D[k][0] = D[k][1] = T(0);
      const int u0 = S.f.ubeg[cls * (nzf + 1) + zp], u1 = S.f.ubeg[cls * (nzf + 1) + zp + 1];
#pragma unroll 2
      for (int u = u0; u < u1; ++u) {
        const int nz = S.f.units[u].nz;
        const T Z = S.z[(2 * nz) * ngh + ih], Zd = S.z[(2 * nz + 1) * ngh + ih];
        V2 x[SG_N];
#pragma unroll
        for (int k = 0; k < SG_N; ++k) x[k] = g[(long long)u * SH_N + k];
#pragma unroll
        for (int k = 0; k < SG_N; ++k) { A[k][0] = fma(Z, x[k].x, A[k][0]); A[k][1] = fma(Z, x[k].y, A[k][1]); }
        D[0][0] = fma(Zd, x[SG_RR].x, D[0][0]); D[0][1] = fma(Zd, x[SG_RR].y, D[0][1]);
        D[1][0] = fma(Zd, x[SG_RD].x, D[1][0]); D[1][1] = fma(Zd, x[SG_RD].y, D[1][1]);
        D[2][0] = fma(Zd, x[SG_BRR].x, D[2][0]); D[2][1] = fma(Zd, x[SG_BRR].y, D[2][1]);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        C[0][i] = fma(Zp, A[SG_RR][i], C[0][i]); C[1][i] = fma(Zp, A[SG_RD][i], C[1][i]);
        C[2][i] = fma(Zp, A[SG_BRR][i], C[2][i]); C[3][i] = fma(Zdp, A[SG_RR][i], C[3][i]);
        C[4][i] = fma(Zp, A[SG_DR][i], C[4][i]); C[5][i] = fma(Zp, A[SG_DD][i], C[5][i]);
        C[6][i] = fma(Zp, A[SG_BDR][i], C[6][i]); C[7][i] = fma(Zdp, A[SG_DR][i], C[7][i]);
        C[8][i] = fma(Zp, A[SG_ARR][i], C[8][i]); C[9][i] = fma(Zp, A[SG_ARD][i], C[9][i]);
        C[10][i] = fma(Zp, A[SG_ABRR][i], C[10][i]); C[11][i] = fma(Zdp, A[SG_ARR][i], C[11][i]);
        C[12][i] = fma(Zp, D[0][i], C[12][i]); C[13][i] = fma(Zp, D[1][i], C[13][i]);
        C[14][i] = fma(Zp, D[2][i], C[14][i]); C[15][i] = fma(Zdp, D[0][i], C[15][i]);
      }
    }
    {
      const SepStructDev& X = S.k[call];
      const V2* g = reinterpret_cast<const V2*>(gp + S.gpair[call]) + (long long)ir * X.nu;
      T a0 = T(0), a1 = T(0);
      const int u0 = X.ubeg[cls * (nzf + 1) + zp], u1 = X.ubeg[cls * (nzf + 1) + zp + 1];
#pragma unroll 4
      for (int u = u0; u < u1; ++u) {
        const T Z = S.z[(2 * X.units[u].nz) * ngh + ih];
        const V2 x = g[u];
        a0 = fma(Z, x.x, a0); a1 = fma(Z, x.y, a1);
      }
      C[16][0] = fma(Zp, a0, C[16][0]); C[16][1] = fma(Zp, a1, C[16][1]);
    }
  }
#pragma unroll
  for (int k = 0; k < 17; ++k) {
    red[(grp * 34 + 2 * k) * ngh + ih] = C[k][0];
    red[(grp * 34 + 2 * k + 1) * ngh + ih] = C[k][1];
  }
  __syncthreads();
  for (int k = threadIdx.x; k < 34 * ngh; k += blockDim.x) {
    T s = red[k];
    for (int g = 1; g < ng; ++g) s += red[g * 34 * ngh + k];
    red[k] = s;
  }
  __syncthreads();
  if (grp) return;
  T Cr[16], Ci[16], acc[2 * ND];
#pragma unroll
  for (int k = 0; k < 16; ++k) { Cr[k] = red[(2 * k) * ngh + ih]; Ci[k] = red[(2 * k + 1) * ngh + ih]; }
#pragma unroll
  for (int k = 0; k < 2 * ND; ++k) acc[k] = T(0);
  const T sb = (cls & 1) ? T(-1) : T(1), sig = -sb;
  const T xr = T(2) * red[32 * ngh + ih], xi = T(2) * red[33 * ngh + ih];
  if ((cls >> 1) == (cls & 1)) {
    fold_same(acc, Cr, Ci, sb);
    accC(acc, D_SBR, sig * xr, sig * xi);
    accC(acc, D_SBP, xi, -xr);
  } else {
    fold_opp(acc, Cr, Ci, sig);
    accC(acc, D_RB, -sb * xr, -sb * xi);
    accC(acc, D_SBZ, xr, xi);
  }
  T* out = dpart + (((long long)p * 2 + call) * 4 + cls) * (2 * ND) * S.nghl + ir * ngh + ih;
#pragma unroll
  for (int k = 0; k < 2 * ND; ++k) out[(long long)k * S.nghl] = acc[k];
}

// ---------------------------------------------------------------------------
// projection 1: the unit fields of one radial point, call and class, from the field
// tensor mf [P][2 calls][NMF][2 planes][nghl].  For SEP_ZC column functions at a time
// the field is combined with Z' and Z'' into the 13 factors of Z and Z' of the row side
// (shared memory), then a thread sums one unit and plane over the z points.
// grid (ngl, 2 calls x 4 classes, points), 128 threads
// ---------------------------------------------------------------------------
enum { SEP_ZC = 8, SEP_NX = 13 };
template <class T>
__host__ __device__ inline size_t sep_field_smem(int ngh) {
  return (size_t)(18 * 2 + 1 + SEP_ZC * SEP_NX * 2) * ngh * sizeof(T);
}

template <class T>
__global__ void __launch_bounds__(128) k_sep_field(const __grid_constant__ SepDev<T> S, const T* __restrict__ mf) {
  const int p = sep_point(S, blockIdx.z);
  if (p < 0) return;
  const int ir = blockIdx.x, call = blockIdx.y >> 2, cls = blockIdx.y & 3;
  const int ngh = S.ngh, nzf = S.nzf;
  const int sa = (cls & 2) ? -1 : 1, sb = (cls & 1) ? -1 : 1;
  extern __shared__ __align__(16) unsigned char smraw[];
  T* sm = reinterpret_cast<T*>(smraw);     // [16 (q, q') + (0, 4) + pairing][2][ngh]
  T* sv = sm + 18 * 2 * ngh;               // [ngh]
  T* sx = sv + ngh;                        // [SEP_ZC][SEP_NX][2][ngh]
  const T* mp = mf + ((long long)p * 2 + call) * NMF * 2 * S.nghl + ir * ngh;
  for (int k = threadIdx.x; k < 36 * ngh; k += blockDim.x) {
    const int ih = k % ngh, pl = (k / ngh) & 1, c = k / (2 * ngh);
    const int slot = c < 16 ? mfslot(c >> 2, c & 3, sa, sb) : c == 16 ? mfslot(0, 4, sa, sb) : 100 + cls;
    sm[k] = mp[((long long)slot * 2 + pl) * S.nghl + ih];
  }
  for (int k = threadIdx.x; k < ngh; k += blockDim.x) sv[k] = S.v[ir * ngh + k];
  T* gp = S.g + p * S.gstride;
  const T y = S.y[ir];
  __syncthreads();
  for (int z0 = 0; z0 < nzf; z0 += SEP_ZC) {
    const int z1 = min(nzf, z0 + SEP_ZC);
    for (int k = threadIdx.x; k < (z1 - z0) * 2 * ngh; k += blockDim.x) {
      const int ih = k % ngh, pl = (k / ngh) & 1, c = k / (2 * ngh);
      const T Zp = S.z[(2 * (z0 + c)) * ngh + ih], Zdp = S.z[(2 * (z0 + c) + 1) * ngh + ih];
      T* x = sx + ((long long)c * SEP_NX * 2 + pl) * ngh + ih;
#define MF_(q, qp) sm[(((q) * 4 + (qp)) * 2 + pl) * ngh + ih]
      const T m04 = sm[(16 * 2 + pl) * ngh + ih];
      x[0 * 2 * ngh] = fma(Zp, fma(T(2) * sv[ih], m04, MF_(0, 0)), Zdp * MF_(0, 3));
      x[1 * 2 * ngh] = fma(Zp, MF_(1, 0), Zdp * MF_(1, 3));
      x[2 * 2 * ngh] = Zp * MF_(0, 1);
      x[3 * 2 * ngh] = Zp * MF_(1, 1);
      x[4 * 2 * ngh] = fma(Zp, MF_(2, 0), Zdp * MF_(2, 3));
      x[5 * 2 * ngh] = Zp * MF_(0, 2);
      x[6 * 2 * ngh] = Zp * MF_(2, 2);
      x[7 * 2 * ngh] = Zp * MF_(1, 2);
      x[8 * 2 * ngh] = Zp * MF_(2, 1);
      x[9 * 2 * ngh] = Zp * m04;
      x[10 * 2 * ngh] = fma(Zp, MF_(3, 0), Zdp * MF_(3, 3));
      x[11 * 2 * ngh] = Zp * MF_(3, 1);
      x[12 * 2 * ngh] = Zp * MF_(3, 2);
#undef MF_
    }
    __syncthreads();
    {
      const int u0 = S.f.ubeg[cls * (nzf + 1) + z0], u1 = S.f.ubeg[cls * (nzf + 1) + z1];
      for (int k = threadIdx.x; k < 2 * (u1 - u0); k += blockDim.x) {
        const int pl = k & 1, u = u0 + (k >> 1);
        const SepUnit U = S.f.units[u];
        const T* x = sx + ((long long)(U.nzp - z0) * SEP_NX * 2 + pl) * ngh;
        const T *Z = S.z + (2 * U.nz) * ngh, *Zd = Z + ngh;
        T h[SH_N];
#pragma unroll
        for (int i = 0; i < SH_N; ++i) h[i] = T(0);
#pragma unroll 2
        for (int ih = 0; ih < ngh; ++ih) {
          const T a = Z[ih], b = Zd[ih];
#pragma unroll
          for (int i = 0; i < SH_N; ++i) h[i] = fma(a, x[i * 2 * ngh + ih], h[i]);
          h[SG_RR] = fma(b, x[10 * 2 * ngh + ih], h[SG_RR]);
          h[SG_RD] = fma(b, x[11 * 2 * ngh + ih], h[SG_RD]);
          h[SG_BRR] = fma(b, x[12 * 2 * ngh + ih], h[SG_BRR]);
        }
        h[SG_ARR] *= y; h[SG_BRR] *= y; h[SG_ABRR] *= y * y; h[SG_BDR] *= y; h[SG_ARD] *= y;
        T* g = gp + ((long long)(call * S.ngl + ir) * S.f.nu + u) * (2 * SH_N) + pl;
#pragma unroll
        for (int i = 0; i < SH_N; ++i) g[2 * i] = h[i];
      }
    }
    {
      const SepStructDev& X = S.d[call];
      const int u0 = X.ubeg[cls * (nzf + 1) + z0], u1 = X.ubeg[cls * (nzf + 1) + z1];
      for (int k = threadIdx.x; k < 2 * (u1 - u0); k += blockDim.x) {
        const int pl = k & 1, u = u0 + (k >> 1);
        const SepUnit U = X.units[u];
        const T *Z = S.z + (2 * U.nz) * ngh, *Zp = S.z + (2 * U.nzp) * ngh, *m = sm + (17 * 2 + pl) * ngh;
        T h = T(0);
        for (int ih = 0; ih < ngh; ++ih) h = fma(Z[ih] * Zp[ih], m[ih], h);
        gp[S.gpair[call] + ((long long)ir * X.nu + u) * 2 + pl] = h;
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// projection 2: the radial sums, hsp [P][2 planes][4 quadrants][nxy].  A warp takes 32
// items of one unit, so that the unit's fields are read once for all lanes; a lane
// combines them with its row state (5 products per column of Re, Im and the two calls)
// and sums SEP_GC column states.
// grid (ceil(warps of F, X and Y / 4), points), 128 threads
// ---------------------------------------------------------------------------
template <class T>
__device__ __forceinline__ void sep_project_normal(const SepDev<T>& S, const SepWarp& W, int p, T* __restrict__ hsp,
                                                   long long nxy, int call) {
  using V2 = typename Vec2<T>::t;
  const int lane = threadIdx.x & 31, ngl = S.ngl;
  const SepItem& it = S.f.items[W.item0 + min(lane, W.nitem - 1)];
  const T la = S.lam[it.seg], lb = S.lam[it.segp], lab = la * lb;
  const V2* ra = S.r + it.row * ngl;
  int rp[SEP_GC];
#pragma unroll
  for (int k = 0; k < SEP_GC; ++k) rp[k] = it.rowp[k < it.n ? k : 0] * ngl;
  T acc[SEP_GC][2], lap[SEP_GC][2];
#pragma unroll
  for (int k = 0; k < SEP_GC; ++k) { acc[k][0] = acc[k][1] = lap[k][0] = lap[k][1] = T(0); }
  const V2* g = reinterpret_cast<const V2*>(S.g + p * S.gstride) + ((long long)call * ngl * S.f.nu + W.unit) * SH_N;
  const long long gs = (long long)S.f.nu * SH_N;
  for (int ir = 0; ir < ngl; ++ir, g += gs) {
    V2 h[SH_N];
#pragma unroll
    for (int i = 0; i < SH_N; ++i) h[i] = g[i];
    const V2 a = ra[ir];
    T vr[2], vd[2], vl[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
#define H_(k) (i ? h[k].y : h[k].x)
      const T rr = fma(lab, H_(SG_ABRR), fma(lb, H_(SG_BRR), fma(la, H_(SG_ARR), H_(SG_RR))));
      const T dr = fma(lb, H_(SG_BDR), H_(SG_DR));
      const T rd = fma(la, H_(SG_ARD), H_(SG_RD));
      vr[i] = fma(a.x, rr, a.y * dr);
      vd[i] = fma(a.x, rd, a.y * H_(SG_DD));
      vl[i] = a.x * H_(SH_L);
#undef H_
    }
#pragma unroll
    for (int k = 0; k < SEP_GC; ++k) {
      if (k >= W.nmax) break;
      const V2 b = S.r[rp[k] + ir];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        acc[k][i] = fma(b.x, vr[i], fma(b.y, vd[i], acc[k][i]));
        lap[k][i] = fma(b.x, vl[i], lap[k][i]);
      }
    }
  }
  if (lane >= W.nitem) return;
  const T s = T(2) * S.sgn[it.seg] * S.sgn[it.segp], ea = S.e[it.ja];
  T* out = hsp + (long long)p * 8 * nxy + (call ? 3 * nxy : 0);
#pragma unroll
  for (int k = 0; k < SEP_GC; ++k) {
    if (k >= it.n) break;
    const T ee = ea + S.e[it.jb[k]];
#pragma unroll
    for (int i = 0; i < 2; ++i) out[(long long)i * 4 * nxy + it.off[k]] = s * fma(-ee, lap[k][i], acc[k][i]);
  }
}

template <class T>
__device__ __forceinline__ void sep_project_pair(const SepDev<T>& S, const SepWarp& W, int call, int p,
                                                 T* __restrict__ hsp, long long nxy) {
  using V2 = typename Vec2<T>::t;
  const SepStructDev& X = S.d[call];
  const int lane = threadIdx.x & 31, ngl = S.ngl;
  const SepItem& it = X.items[W.item0 + min(lane, W.nitem - 1)];
  const V2* ra = S.r + it.row * ngl;
  int rp[SEP_GC];
#pragma unroll
  for (int k = 0; k < SEP_GC; ++k) rp[k] = it.rowp[k < it.n ? k : 0] * ngl;
  T acc[SEP_GC][2];
#pragma unroll
  for (int k = 0; k < SEP_GC; ++k) acc[k][0] = acc[k][1] = T(0);
  const V2* g = reinterpret_cast<const V2*>(S.g + p * S.gstride + S.gpair[call]) + W.unit;
#pragma unroll 2
  for (int ir = 0; ir < ngl; ++ir) {
    const V2 h = g[(long long)ir * X.nu];
    const T a = ra[ir].x, v0 = a * h.x, v1 = a * h.y;
#pragma unroll
    for (int k = 0; k < SEP_GC; ++k) {
      if (k >= W.nmax) break;
      const T b = S.r[rp[k] + ir].x;
      acc[k][0] = fma(b, v0, acc[k][0]);
      acc[k][1] = fma(b, v1, acc[k][1]);
    }
  }
  if (lane >= W.nitem) return;
  const T s = T(2) * S.sgn[it.seg] * S.sgn[it.segp];
  T* out = hsp + (long long)p * 8 * nxy + (call ? 2 : 1) * nxy;
#pragma unroll
  for (int k = 0; k < SEP_GC; ++k) {
    if (k >= it.n) break;
    out[it.off[k]] = s * acc[k][0];
    out[4 * nxy + it.off[k]] = s * acc[k][1];
  }
}

template <class T>
__global__ void __launch_bounds__(128) k_sep_project(const __grid_constant__ SepDev<T> S, T* __restrict__ hsp,
                                                     long long nxy) {
  const int p = sep_point(S, blockIdx.y);
  if (p < 0) return;
  int w = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (w < 2 * S.f.nwarp) { sep_project_normal<T>(S, S.f.warps[w >> 1], p, hsp, nxy, w & 1); return; }
  w -= 2 * S.f.nwarp;
  if (w < S.d[0].nwarp) { sep_project_pair<T>(S, S.d[0].warps[w], 0, p, hsp, nxy); return; }
  w -= S.d[0].nwarp;
  if (w < S.d[1].nwarp) sep_project_pair<T>(S, S.d[1].warps[w], 1, p, hsp, nxy);
}

}  // namespace pnfam
#endif
