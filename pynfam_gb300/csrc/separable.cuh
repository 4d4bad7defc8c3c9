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
// (nine points): densities 0.13 ms against 1.8 ms, projection 0.19 against 1.8 ms; FP32
// (24 points): 16 and 17 us (radial sums 264, z sums 111, unit fields 104, projection 298 us
// a launch) against 39 and 41 us of the pair-tensor GEMMs (40 points), whose operand (12 GB)
// is not needed; errors against FP64 2e-7 instead of 8e-6.
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
// functions are plainly not of the product form (sep_value still has to be compared).
// Blocks nb / 2 ... are the time-reversed partners of the first half: their states are tried
// with the factors of the partner's (same functions, spins exchanged) before a search, and
// the others' searches look at one value before they compare whole functions; the values are
// those of the full search. Host time,
// Grace: 0.12 ms at N_sh = 6 and 1.6 at 16 (0.33 and 4.3 with a full search for every state)
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
  std::vector<double> row(ngl * 2), wbest(ngl), tops(dqp, 0.0);
  std::vector<int> peer(dqp, -1);       // the state whose factors a state was found to share
  for (int i = 0; i < nb; ++i)
    for (int s = 0; s < 2; ++s) {
      const int lo = st[i] + (s ? nup[i] : 0), hi = s ? st[i] + db[i] : st[i] + nup[i];
      const int ip = i - nb / 2;        // partner block, if it came before
      int po = -1;                      // its states of the other spin
      if (ip >= 0 && nb % 2 == 0 && db[ip] == db[i] && nup[ip] == db[i] - nup[i]) po = st[ip] + (s ? 0 : nup[ip]);
      std::vector<double> c(ngl, 0.0);
      std::fill(wbest.begin(), wbest.end(), 0.0);
      bool first = true;
      // the state's radial function with the z function c0 divided out, its largest values
      double rtop = 0.0, dtop = 0.0;
      int rmax = 0;
      auto radial = [&](const double* f, int c0) {
        const double* fd = f + ps;
        rtop = dtop = 0.0;
        for (int l = 0; l < ngl; ++l) {
          row[2 * l] = f[(size_t)l * ngh + zstar[c0]] / ztop[c0];
          row[2 * l + 1] = fd[(size_t)l * ngh + zstar[c0]] / ztop[c0];
          if (fabs(row[2 * l]) > rtop) { rtop = fabs(row[2 * l]); rmax = l; }
          if (fabs(row[2 * l + 1]) > dtop) dtop = fabs(row[2 * l + 1]);
        }
      };
      auto same_z = [&](const double* p, int k, double top) {
        const double q = p[zstar[k]] / ztop[k], *z = &B.z[(size_t)(2 * k) * ngh];
        for (int h = 0; h < ngh; ++h)
          if (fabs(p[h] - q * z[h]) > SEP_TOL * top) return false;
        return true;
      };
      auto same_row = [&](int k, double sg) {
        const double* r = &B.r[(size_t)k * ngl * 2];
        if (fabs(row[2 * rmax] - sg * r[2 * rmax]) > SEP_TOL * rtop) return false;
        for (int l = 0; l < ngl; ++l)
          if (fabs(row[2 * l] - sg * r[2 * l]) > SEP_TOL * rtop || fabs(row[2 * l + 1] - sg * r[2 * l + 1]) > SEP_TOL * dtop)
            return false;
        return true;
      };
      auto find = [&](double sg) {
        for (int k = 0; k < B.nrow; ++k)
          if (same_row(k, sg)) return k;
        return -1;
      };
      for (int a = lo; a < hi; ++a) {
        const double* f = phi + (size_t)a * nghl;
        int c0 = -1, k = -1;
        if (po >= 0) {
          const int b = po + a - lo, zb = B.zi[b];
          radial(f, zb);
          const double* p = f + (size_t)rmax * ngh;
          if (rtop > 0.0 && std::isfinite(rtop) && same_z(p, zb, fabs(p[zstar[zb]]))) {
            if (same_row(B.ri[b], B.sgn[2 * i + s])) k = B.ri[b];
            else if (first && same_row(B.ri[b], -1.0)) { k = B.ri[b]; B.sgn[2 * i + s] = -1.0; }
          }
          if (k >= 0) { c0 = zb; peer[a] = b; }
        }
        if (k < 0) {
          double m4[4] = {0.0, 0.0, 0.0, 0.0};   // four chains
          int q = 0;
          for (; q + 4 <= nghl; q += 4)
            for (int u = 0; u < 4; ++u) { const double x = fabs(f[q + u]); m4[u] = x > m4[u] ? x : m4[u]; }
          for (; q < nghl; ++q) { const double x = fabs(f[q]); m4[0] = x > m4[0] ? x : m4[0]; }
          const double top = std::max(std::max(m4[0], m4[1]), std::max(m4[2], m4[3]));
          if (!(top > 0.0) || !std::isfinite(top)) return false;
          tops[a] = top;
          int m = 0;
          while (fabs(f[m]) != top) ++m;
          const int ls = m / ngh, hs = m % ngh;
          const double* p = f + (size_t)ls * ngh;   // the state along z at its largest point
          for (int z = 0; z < B.nzf && c0 < 0; ++z)
            if (same_z(p, z, top)) c0 = z;
          if (c0 < 0) {
            if (B.nzf >= 256) return false;   // not a product basis of any size in use
            // scaled so that the state's radial function is a row that is there already,
            // if there is one: every (n_r, |Lambda|) then has one row for all n_z
            double scale = 1.0;
            for (int z = 0; z < B.nrow; ++z) {
              const double *rk = &B.r[(size_t)z * ngl * 2], sg = B.sgn[2 * i + s];
              if (rk[2 * ls] == 0.0) continue;
              const double al = f[(size_t)ls * ngh + hs] / (sg * rk[2 * ls]);
              double d0 = 0.0, d1 = 0.0, dt = 0.0;
              for (int l = 0; l < ngl; ++l) {
                const double fd = phi[ps + (size_t)a * nghl + (size_t)l * ngh + hs];
                d0 = fmax(d0, fabs(f[(size_t)l * ngh + hs] - al * sg * rk[2 * l]));
                d1 = fmax(d1, fabs(fd - al * sg * rk[2 * l + 1]));
                dt = fmax(dt, fabs(fd));
              }
              if (d0 <= SEP_TOL * top && d1 <= SEP_TOL * dt) { scale = al; break; }
            }
            c0 = B.nzf++;
            zstar.push_back(hs);
            ztop.push_back(scale);
            for (int h = 0; h < ngh; ++h) B.z.push_back(scale * (p[h] / p[hs]));
            const double* g = phi + 3 * ps + (size_t)a * nghl + (size_t)ls * ngh;
            for (int h = 0; h < ngh; ++h) B.z.push_back(scale * (g[h] / p[hs]));
          }
          radial(f, c0);
          k = first || B.sgn[2 * i + s] > 0 ? find(1.0) : find(-1.0);
          if (first && k < 0 && (k = find(-1.0)) >= 0) B.sgn[2 * i + s] = -1.0;
          if (k < 0) {
            if (B.nrow >= 4096) return false;
            k = B.nrow++;
            for (double x : row) B.r.push_back(B.sgn[2 * i + s] * x);
          }
        }
        B.zi[a] = c0;
        B.ri[a] = k;
        first = false;
        for (int l = 0; l < ngl; ++l)
          if (fabs(row[2 * l]) > wbest[l]) {
            wbest[l] = fabs(row[2 * l]);
            c[l] = phi[2 * ps + (size_t)a * nghl + (size_t)l * ngh + zstar[c0]] / ztop[c0] / row[2 * l];
          }
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
      if (peer[a] >= 0) { B.e[a] = B.e[peer[a]]; continue; }
      const double *f = phi + (size_t)a * nghl, *g = phi + 4 * ps + (size_t)a * nghl;
      double s0 = 0.0, s1 = 0.0;
      for (int k = 0; k < nghl; ++k) {
        const double x = fabs(f[k]);
        if (x < 1e-2 * tops[a] || w[k] == 0.0) continue;
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

// column states per projection item; elements, parts and rows staged at a time
enum { SEP_GC = 5, SEP_STAGE = 256, SEP_STAGE_E = 64, SEP_STAGE_R = SEP_STAGE + SEP_STAGE_E };

struct SepItem {        // one row state against up to SEP_GC column states of a unit
  int seg, segp, ja, row, n;
  int jb[SEP_GC], rowp[SEP_GC], off[SEP_GC];
};
// the same as columns of integers, so that the lanes of a warp read them side by side:
// [SI_N][items]
enum { SI_SEG = 0, SI_SEGP, SI_JA, SI_ROW, SI_CNT, SI_JB, SI_ROWP = SI_JB + SEP_GC, SI_OFF = SI_ROWP + SEP_GC,
       SI_N = SI_OFF + SEP_GC };
inline std::vector<int> sep_item_columns(const std::vector<SepItem>& it) {
  const size_t n = it.size();
  std::vector<int> v(SI_N * n);
  for (size_t k = 0; k < n; ++k) {
    const SepItem& i = it[k];
    const int head[5] = {i.seg, i.segp, i.ja, i.row, i.n};
    for (int j = 0; j < 5; ++j) v[j * n + k] = head[j];
    for (int j = 0; j < SEP_GC; ++j) {   // absent column states repeat the first
      const int q = j < i.n ? j : 0;
      v[(SI_JB + j) * n + k] = i.jb[q];
      v[(SI_ROWP + j) * n + k] = i.rowp[q];
      v[(SI_OFF + j) * n + k] = i.off[q];
    }
  }
  return v;
}
struct SepWarp { int unit, item0, nitem, nmax; };   // up to 32 / SPL items of one unit (nmax: their largest n)
enum { SEP_SPL = 4 };   // lanes that share an item where the kernel splits its radial points

struct SepStruct {
  std::vector<SepUnit> units;      // by (class, n_z', n_z)
  std::vector<SepEnt> ents;
  std::vector<int> rows, offs, ubeg, order;   // ubeg [4][nzf + 1]: first unit of (class, n_z'); order: largest first
  std::vector<SepItem> items;
  std::vector<SepWarp> warps[2];   // 32 items, 32 / SEP_SPL items
  int umax = 0;                    // most units of one (class, n_z')
};

// cols, boff: the block structure; project: also the projection's items.  false when a
// part of a unit does not fit the staging buffer.  The five structures of an operator with
// their item columns: 0.19 ms at N_sh = 6, 4.3 at 16 on one Grace core
inline bool sep_structure(const SepBasis& B, int nb, const int* db, const int* st, const int* nup, const int* cols,
                          const long long* boff, bool project, SepStruct& S) {
  S = SepStruct();
  const int nzf = B.nzf;
  // states of each (block, spin) by z function: byz[first[seg * nzf + z] ...]
  std::vector<int> first(2 * nb * nzf + 1, 0), byz, at;
  for (int i = 0; i < nb; ++i)
    for (int a = 0; a < db[i]; ++a) ++first[(2 * i + (a >= nup[i])) * nzf + B.zi[st[i] + a] + 1];
  for (size_t k = 1; k < first.size(); ++k) first[k] += first[k - 1];
  byz.resize(first.back());
  at.assign(first.begin(), first.end() - 1);
  for (int i = 0; i < nb; ++i)
    for (int a = 0; a < db[i]; ++a) byz[at[(2 * i + (a >= nup[i])) * nzf + B.zi[st[i] + a]]++] = st[i] + a;
  auto count = [&](int seg, int z) { return first[seg * nzf + z + 1] - first[seg * nzf + z]; };
  long long nel = 0;
  for (int i = 0; i < nb; ++i)
    if (cols[i] >= 0) nel += (long long)db[i] * db[cols[i]];
  S.offs.reserve(nel);
  if (project) S.items.reserve(nel / 2);
  struct Part { int i, seg, j, segp; };
  std::vector<Part> parts[4], live;   // of a class; those with column states of a z function
  for (int i = 0; i < nb; ++i) {
    const int j = cols[i];
    if (j < 0) continue;
    for (int s = 0; s < 2; ++s)
      for (int t = 0; t < 2; ++t) parts[2 * s + t].push_back({i, 2 * i + s, j, 2 * j + t});
  }
  for (int c = 0; c < 4; ++c)
    for (int zp = 0; zp < nzf; ++zp) {
      S.ubeg.push_back((int)S.units.size());
      live.clear();
      for (const Part& p : parts[c])
        if (count(p.segp, zp)) live.push_back(p);
      for (int z = 0; z < nzf; ++z) {
        SepUnit u{c, z, zp, (int)S.ents.size(), 0};
        const int item0 = (int)S.items.size();
        for (const Part& p : live) {
          const int na = count(p.seg, z), nc = count(p.segp, zp);
          if (!na) continue;
          const int *A = &byz[first[p.seg * nzf + z]], *C = &byz[first[p.segp * nzf + zp]];
          if ((long long)na * nc > SEP_STAGE) return false;
          SepEnt en{na, nc, (int)S.rows.size(), (int)S.rows.size() + na, (int)S.offs.size(), p.seg, p.segp};
          for (int a = 0; a < na; ++a) S.rows.push_back(B.ri[A[a]]);
          for (int b = 0; b < nc; ++b) S.rows.push_back(B.ri[C[b]]);
          for (int b = 0; b < nc; ++b)
            for (int a = 0; a < na; ++a)
              S.offs.push_back((int)(boff[p.i] + (A[a] - st[p.i]) + (long long)(C[b] - st[p.j]) * db[p.i]));
          S.ents.push_back(en);
        }
        u.nent = (int)S.ents.size() - u.ent0;
        if (!u.nent) continue;
        if (project) {
          // a part's columns in nearly equal groups of at most SEP_GC; items of one size next
          // to each other, so that a warp's lanes run the same loop
          for (int n = SEP_GC; n > 0; --n)
            for (int e = u.ent0; e < u.ent0 + u.nent; ++e) {
              const SepEnt& en = S.ents[e];
              const int ng = (en.ngp + SEP_GC - 1) / SEP_GC;
              if (en.ngp / ng != n && (en.ngp + ng - 1) / ng != n) continue;
              const int *A = &byz[first[en.seg * nzf + z]], *C = &byz[first[en.segp * nzf + zp]];
              for (int k = 0; k < ng; ++k) {
                const int b0 = en.ngp * k / ng;
                if (en.ngp * (k + 1) / ng - b0 != n) continue;
                for (int a = 0; a < en.ng; ++a) {
                  S.items.emplace_back();
                  SepItem& it = S.items.back();
                  it.seg = en.seg; it.segp = en.segp; it.ja = A[a]; it.row = S.rows[en.row0 + a]; it.n = n;
                  for (int b = 0; b < n; ++b) {
                    it.jb[b] = C[b0 + b]; it.rowp[b] = S.rows[en.rowp0 + b0 + b];
                    it.off[b] = S.offs[en.el0 + (b0 + b) * en.ng + a];
                  }
                }
              }
            }
          for (int h = 0; h < 2; ++h) {
            const int n = h ? 32 / SEP_SPL : 32;
            for (int k = item0; k < (int)S.items.size(); k += n)
              S.warps[h].push_back({(int)S.units.size(), k, std::min(n, (int)S.items.size() - k), S.items[k].n});
          }
        }
        S.units.push_back(u);
      }
      S.umax = std::max(S.umax, (int)S.units.size() - S.ubeg.back());
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
  for (auto& w : S.warps)
    std::stable_sort(w.begin(), w.end(), [](const SepWarp& x, const SepWarp& y) { return x.nmax > y.nmax; });
  return true;
}

// sums of a unit at one radial point that the density keeps (lambda factors per part):
// products of the row side's and the column side's radial functions
enum { SG_RR = 0, SG_DR, SG_RD, SG_DD, SG_ARR, SG_BRR, SG_ABRR, SG_BDR, SG_ARD, SG_N };
// the projection's unit fields: the same nine, then the (0, 4) and (4, 0) field
enum { SH_L = SG_N, SH_N };

// values of one point's unit sums, for nu units of the structures F, X^T, Y^T, X and Y:
// per call the F units [ngl][nu][SH_N][2 planes], then per call, from gpair[call] on, the
// pairing units [ngl][nu][2 planes] (densities and fields in the same place).  A multiple of
// 4, so that every point's sums start on 16 bytes in FP32 too: k_sep_project reads the F
// units 16 bytes at a time
inline long long sep_sums(long long ngl, const long long nu[5], long long gpair[2]) {
  gpair[0] = 2 * ngl * nu[0] * 2 * SH_N;
  gpair[1] = gpair[0] + 2 * ngl * std::max(nu[1], nu[3]);
  const long long n = gpair[1] + 2 * ngl * std::max(nu[2], nu[4]);
  return (n + 3) / 4 * 4;
}

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
  const int* items;                // [SI_N][nitem]
  const SepWarp* warps[2];
  int nitem, umax, nu, nwarp[2];   // umax: most units of one (class, n_z')
};

template <class T>
struct SepDev {
  int ngh, ngl, nzf, nghl, nrow;
  const typename Vec2<T>::t *r, *rt;   // (R, R') as [nrow][ngl] and as [ngl][nrow]
  const T *z, *v, *y, *e, *lam, *sgn;
  SepStructDev f, k[2], d[2];     // F; pairing densities (X^T, Y^T); pairing fields (X, Y)
  long long gstride, gpair[2];    // of one point's unit sums (sep_sums)
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
// thread one radial point and CT columns of (point, call, plane).  The unit's elements
// are gathered into shared memory (all columns of an element by one thread, so that
// 4 NPT loads are in flight) and every part is summed over its row states, then over its
// column states.  FP64 is bound by the FP64 pipe (about 3.7 DFMA per element, radial
// point and column at N_sh = 16, where a part has 14 elements): one column per thread,
// two points where they fill the last warp (160 threads at 20 radial points, not 80 of
// 96).  FP32 is bound by shared-memory and L1 reads: a thread takes Re and Im, so that a
// radial function is read once for both and the elements as pairs, and four points share
// a CTA.
// grid (units of F, X^T and Y^T; point groups)
// ---------------------------------------------------------------------------
template <class T, int KT, int CT, bool NORMAL>
__device__ __forceinline__ void sep_tile(const typename Vec2<T>::t* __restrict__ r, const int* __restrict__ rows,
                                         const int* __restrict__ rowsp, int ng, const T* s, int ld, int ir, T (&o)[4][CT]) {
  T t0[KT][CT], t1[KT][CT];
#pragma unroll
  for (int k = 0; k < KT; ++k)
#pragma unroll
    for (int c = 0; c < CT; ++c) t0[k][c] = t1[k][c] = T(0);
#pragma unroll 2
  for (int g = 0; g < ng; ++g) {
    const typename Vec2<T>::t ra = r[rows[g] + ir];
#pragma unroll
    for (int k = 0; k < KT; ++k) {
      T x[CT];
      if constexpr (CT == 2) {
        const typename Vec2<T>::t v = *reinterpret_cast<const typename Vec2<T>::t*>(s + (k * ng + g) * ld);
        x[0] = v.x; x[1] = v.y;
      } else {
        x[0] = s[(k * ng + g) * ld];
      }
#pragma unroll
      for (int c = 0; c < CT; ++c) {
        t0[k][c] = fma(ra.x, x[c], t0[k][c]);
        if (NORMAL) t1[k][c] = fma(ra.y, x[c], t1[k][c]);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < KT; ++k) {
    const typename Vec2<T>::t rb = r[rowsp[k] + ir];
#pragma unroll
    for (int c = 0; c < CT; ++c) {
      o[0][c] = fma(rb.x, t0[k][c], o[0][c]);
      if (NORMAL) {
        o[1][c] = fma(rb.x, t1[k][c], o[1][c]);
        o[2][c] = fma(rb.y, t0[k][c], o[2][c]);
        o[3][c] = fma(rb.y, t1[k][c], o[3][c]);
      }
    }
  }
}

template <class T, int NPT, int CT, bool NORMAL>
__device__ __forceinline__ void sep_radial_unit(const SepDev<T>& S, const SepStructDev& X, int ui, int call,
                                                const T* __restrict__ rsp, long long nxy, T* sx, SepEnt* sent,
                                                int* srow) {
  constexpr int NP1 = NORMAL ? 4 : 2, NC = NP1 * NPT;   // columns of a point (call, plane) or (plane), of the CTA
  constexpr int NN = NORMAL ? SG_N : 1;
  const SepUnit u = X.units[ui];
  const int ngl = S.ngl;
  const SepEnt* en = X.ents + u.ent0;
  const int nthr = ngl * (NC / CT);
  for (int t0 = 0; t0 < nthr; t0 += blockDim.x) {
    const int t = t0 + threadIdx.x, ir = t % ngl, col = t / ngl * CT;
    const bool live = t < nthr;
    T acc[NN][CT];
#pragma unroll
    for (int k = 0; k < NN; ++k)
#pragma unroll
      for (int c = 0; c < CT; ++c) acc[k][c] = T(0);
    for (int e0 = 0; e0 < u.nent;) {
      // the parts that fit the staging buffers together (a part of n x n' elements has
      // n + n' <= n n' + 1 rows)
      int e1 = e0, nel = 0, nrow = 0;
      while (e1 < u.nent && e1 < e0 + SEP_STAGE_E) {
        const int n = en[e1].ng * en[e1].ngp;
        if (nel + n > SEP_STAGE) break;
        nel += n;
        nrow += en[e1].ng + en[e1].ngp;
        ++e1;
      }
      const int el0 = en[e0].el0, row0 = en[e0].row0;
      __syncthreads();
      for (int k = threadIdx.x; k < nrow; k += blockDim.x) srow[k] = X.rows[row0 + k] * ngl;
      for (int k = threadIdx.x; k < e1 - e0; k += blockDim.x) sent[k] = en[e0 + k];
      for (int k = threadIdx.x; k < nel; k += blockDim.x) {
        const long long off = X.offs[el0 + k];
        T v[NC];
#pragma unroll
        for (int i = 0; i < NPT; ++i) {
          const int p = sep_point(S, blockIdx.y * NPT + i);
          const T* src = rsp + (long long)max(p, 0) * 8 * nxy + off;
#pragma unroll
          for (int c = 0; c < NP1; ++c) {
            const int quad = NORMAL ? (c >= 2 ? 3 : 0) : (call ? 2 : 1);
            v[NP1 * i + c] = p < 0 ? T(0) : src[((c & 1) * 4 + quad) * nxy];
          }
        }
#pragma unroll
        for (int c = 0; c < NC; c += 2) {
          typename Vec2<T>::t w;
          w.x = v[c]; w.y = v[c + 1];
          *reinterpret_cast<typename Vec2<T>::t*>(sx + k * NC + c) = w;
        }
      }
      __syncthreads();
      if (live) {
        for (int e = e0; e < e1; ++e) {
          const SepEnt q = sent[e - e0];
          const int *ra = srow + (q.row0 - row0), *rb = srow + (q.rowp0 - row0);
          const T* s = sx + (q.el0 - el0) * NC + col;
          T o[4][CT];
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int c = 0; c < CT; ++c) o[i][c] = T(0);
          int k = 0;
          if (sizeof(T) == 4)
            for (; k + 4 <= q.ngp; k += 4)
              sep_tile<T, 4, CT, NORMAL>(S.r, ra, rb + k, q.ng, s + k * q.ng * NC, NC, ir, o);
          for (; k + 2 <= q.ngp; k += 2)
            sep_tile<T, 2, CT, NORMAL>(S.r, ra, rb + k, q.ng, s + k * q.ng * NC, NC, ir, o);
          if (k < q.ngp) sep_tile<T, 1, CT, NORMAL>(S.r, ra, rb + k, q.ng, s + k * q.ng * NC, NC, ir, o);
          const T sg = S.sgn[q.seg] * S.sgn[q.segp], la = S.lam[q.seg] * sg, lb = S.lam[q.segp];
#pragma unroll
          for (int c = 0; c < CT; ++c) {
            acc[SG_RR][c] = fma(sg, o[0][c], acc[SG_RR][c]);
            if constexpr (NORMAL) {
              acc[SG_DR][c] = fma(sg, o[1][c], acc[SG_DR][c]);
              acc[SG_RD][c] = fma(sg, o[2][c], acc[SG_RD][c]);
              acc[SG_DD][c] = fma(sg, o[3][c], acc[SG_DD][c]);
              acc[SG_ARR][c] = fma(la, o[0][c], acc[SG_ARR][c]);
              acc[SG_BRR][c] = fma(lb * sg, o[0][c], acc[SG_BRR][c]);
              acc[SG_ABRR][c] = fma(la * lb, o[0][c], acc[SG_ABRR][c]);
              acc[SG_BDR][c] = fma(lb * sg, o[1][c], acc[SG_BDR][c]);
              acc[SG_ARD][c] = fma(la, o[2][c], acc[SG_ARD][c]);
            }
          }
        }
      }
      e0 = e1;
    }
    if (!live) continue;
    const int p = sep_point(S, blockIdx.y * NPT + col / NP1);
    if (p < 0) continue;
    T* g = S.g + p * S.gstride;
    if constexpr (NORMAL) {
      const T y = S.y[ir];
      g += ((long long)(((col >> 1) & 1) * ngl + ir) * X.nu + ui) * (2 * SH_N) + (col & 1);
#pragma unroll
      for (int c = 0; c < CT; ++c) {
        g[2 * SG_RR + c] = acc[SG_RR][c];
        g[2 * SG_DR + c] = acc[SG_DR][c];
        g[2 * SG_RD + c] = acc[SG_RD][c];
        g[2 * SG_DD + c] = acc[SG_DD][c];
        g[2 * SG_ARR + c] = y * acc[SG_ARR][c];
        g[2 * SG_BRR + c] = y * acc[SG_BRR][c];
        g[2 * SG_ABRR + c] = y * y * acc[SG_ABRR][c];
        g[2 * SG_BDR + c] = y * acc[SG_BDR][c];
        g[2 * SG_ARD + c] = y * acc[SG_ARD][c];
      }
    } else {
      g += S.gpair[call] + ((long long)ir * X.nu + ui) * 2 + (col & 1);
#pragma unroll
      for (int c = 0; c < CT; ++c) g[c] = acc[0][c];
    }
  }
}

template <class T, int NPT>
__global__ void __launch_bounds__(192, sizeof(T) == 4 ? 5 : 1) k_sep_radial(const __grid_constant__ SepDev<T> S, const T* __restrict__ rsp,
                                                    long long nxy) {
  constexpr int CT = sizeof(T) == 4 ? 2 : 1;
  __shared__ __align__(16) T sx[SEP_STAGE * 4 * NPT];
  __shared__ SepEnt sent[SEP_STAGE_E];
  __shared__ int srow[SEP_STAGE_R];
  if (NPT == 1 && sep_point(S, blockIdx.y) < 0) return;
  int b = blockIdx.x;
  if (b < S.f.nu) { sep_radial_unit<T, NPT, CT, true>(S, S.f, S.f.order[b], 0, rsp, nxy, sx, sent, srow); return; }
  b -= S.f.nu;
  if (b < S.k[0].nu) sep_radial_unit<T, NPT, CT, false>(S, S.k[0], S.k[0].order[b], 0, rsp, nxy, sx, sent, srow);
  else sep_radial_unit<T, NPT, CT, false>(S, S.k[1], S.k[1].order[b - S.k[0].nu], 1, rsp, nxy, sx, sent, srow);
}

// ---------------------------------------------------------------------------
// densities 2: the z sums of one radial point, call and class, folded into the class's
// share of the 28 densities: dpart [P][2 calls][4 classes][2 ND][nghl].  A thread takes
// one z point and every ng-th n_z' (ng groups of ngh threads); the unit sums of ng n_z'
// at a time are staged in shared memory (read from L2 as they are used they stalled 75 %
// of the issue slots in FP32).
// grid (ngl, 2 calls x 4 classes, points), ngh * ng threads
// ---------------------------------------------------------------------------
template <class T>
__host__ __device__ inline size_t sep_dens_smem(int ngh, int ng, int nzf) {
  const size_t stage = (size_t)ng * nzf * (SH_N + 1) * 2, red = (size_t)ng * 34 * ngh;
  return ((stage > red ? stage : red) + (size_t)nzf * 2 * ngh) * sizeof(T) + (size_t)2 * ng * nzf * sizeof(int);
}

template <class T>
__global__ void __launch_bounds__(256) k_sep_density(const __grid_constant__ SepDev<T> S, int ng,
                                                     T* __restrict__ dpart) {
  const int p = sep_point(S, blockIdx.z);
  if (p < 0) return;
  const int ir = blockIdx.x, call = blockIdx.y >> 2, cls = blockIdx.y & 3;
  const int ngh = S.ngh, nzf = S.nzf;
  using V2 = typename Vec2<T>::t;
  extern __shared__ __align__(16) unsigned char smraw[];
  T* sz = reinterpret_cast<T*>(smraw);      // [nzf][2][ngh]
  T* red = sz + (size_t)nzf * 2 * ngh;      // [ng][34][ngh], after the sums
  V2* sg = reinterpret_cast<V2*>(red);      // [units of ng n_z'][SH_N]
  V2* sk = sg + (size_t)ng * nzf * SH_N;    // [pairing units of ng n_z']
  const size_t nred = (size_t)ng * 34 * ngh, nst = (size_t)ng * nzf * (SH_N + 1) * 2;
  int* snz = reinterpret_cast<int*>(red + (nst > nred ? nst : nred));   // n_z of the staged units
  int* snk = snz + ng * nzf;
  const int ih = threadIdx.x % ngh, grp = threadIdx.x / ngh;
  const SepStructDev& X = S.k[call];
  const T* gp = S.g + p * S.gstride;
  const V2* gf = reinterpret_cast<const V2*>(gp) + (long long)(call * S.ngl + ir) * S.f.nu * SH_N;
  const V2* gk = reinterpret_cast<const V2*>(gp + S.gpair[call]) + (long long)ir * X.nu;
  // C(q, q') at q * 4 + q', (re, im); then the pairing sum
  T C[17][2];
#pragma unroll
  for (int k = 0; k < 17; ++k) C[k][0] = C[k][1] = T(0);
  for (int i = threadIdx.x; i < nzf * 2 * ngh; i += blockDim.x) sz[i] = S.z[i];
  for (int z0 = 0; z0 < nzf; z0 += ng) {
    const int z1 = min(nzf, z0 + ng), zp = z0 + grp;
    const int f0 = S.f.ubeg[cls * (nzf + 1) + z0], f1 = S.f.ubeg[cls * (nzf + 1) + z1];
    const int k0 = X.ubeg[cls * (nzf + 1) + z0], k1 = X.ubeg[cls * (nzf + 1) + z1];
    __syncthreads();
    for (int i = threadIdx.x; i < (f1 - f0) * SH_N; i += blockDim.x)
      if (i % SH_N < SG_N) sg[i] = gf[(long long)f0 * SH_N + i];
    for (int i = threadIdx.x; i < k1 - k0; i += blockDim.x) { sk[i] = gk[k0 + i]; snk[i] = X.units[k0 + i].nz; }
    for (int i = threadIdx.x; i < f1 - f0; i += blockDim.x) snz[i] = S.f.units[f0 + i].nz;
    __syncthreads();
    if (zp >= z1) continue;
    const T Zp = sz[(2 * zp) * ngh + ih], Zdp = sz[(2 * zp + 1) * ngh + ih];
    {
      T A[SG_N][2], D[3][2];
#pragma unroll
      for (int k = 0; k < SG_N; ++k) A[k][0] = A[k][1] = T(0);
#pragma unroll
      for (int k = 0; k < 3; ++k) D[k][0] = D[k][1] = T(0);
      const int u0 = S.f.ubeg[cls * (nzf + 1) + zp], u1 = S.f.ubeg[cls * (nzf + 1) + zp + 1];
#pragma unroll 2
      for (int u = u0; u < u1; ++u) {
        const int nz = snz[u - f0];
        const T Z = sz[(2 * nz) * ngh + ih], Zd = sz[(2 * nz + 1) * ngh + ih];
        const V2* x = sg + (u - f0) * SH_N;
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
      T a0 = T(0), a1 = T(0);
      const int u0 = X.ubeg[cls * (nzf + 1) + zp], u1 = X.ubeg[cls * (nzf + 1) + zp + 1];
#pragma unroll 4
      for (int u = u0; u < u1; ++u) {
        const T Z = sz[(2 * snk[u - k0]) * ngh + ih];
        const V2 x = sk[u - k0];
        a0 = fma(Z, x.x, a0); a1 = fma(Z, x.y, a1);
      }
      C[16][0] = fma(Zp, a0, C[16][0]); C[16][1] = fma(Zp, a1, C[16][1]);
    }
  }
  __syncthreads();
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
// projection 1: the mean field of one class and the unit fields of one radial point and
// call.  The class's 18 field components at the CTA's mesh points (k_meanfield computes
// the same 104 of all classes) are dealt to the threads, so that the FP64 pipe works on
// them in all CTAs and nothing of the field tensor goes through memory; then, for zc
// column functions at a time, the field is combined with Z' and Z'' into the 13 factors
// of Z and Z' of the row side (shared memory) and a thread sums two units over the z
// points, reading each factor once.
// grid (ngl, 2 calls x 4 classes, points), SEP_FTHR threads
// ---------------------------------------------------------------------------
// component c (q * 4 + q', 16: (0, 4), 17: pairing) of the field of class cls from the
// densities d (pnfam_hamiltonian_blas.f90:775-1094, 1201-1208, as in k_meanfield; s: the
// sign that changes between the two classes of same or of opposite spins)
template <class T>
__device__ __forceinline__ cplxT<T> sep_meanfield(int c, int cls, const T* d, int ld, const T* sc, T crho, T cs,
                                                  T cpair, T cspair) {
  using Z = cplxT<T>;
  auto D = [&](int k) { return cmk<T>(d[(2 * k) * ld], d[(2 * k + 1) * ld]); };
  auto add = [](Z a, Z b) { return cadd<T>(a, b); };
  auto sub = [](Z a, Z b) { return cmk<T>(a.r - b.r, a.i - b.i); };
  auto mul = [](T a, Z b) { return csc<T>(a, b); };
  auto im = [](Z a) { return cmk<T>(-a.i, a.r); };   // i a
  const T cdrho = sc[0], ctau = sc[1], ctj0 = sc[2], ctj1 = sc[3], ctj2 = sc[4], crdj = sc[5];
  const T cds = sc[6], ct = sc[7], cj = sc[8], cgs = sc[9], cf = sc[10], csdj = sc[11];
  const bool same = (cls >> 1) == (cls & 1);
  const T s = (cls & 2) ? T(-1) : T(1), h5 = T(0.5);
  const T e = (c == 4 || c == 8 || c == 12) ? T(-1) : T(1);   // (q', q) of (0, q): antisymmetric parts change sign
  const T t3 = T(1) / T(3);
  if (c == 17) {
    const Z rb = D(D_RB), sz = D(D_SBZ), sr = D(D_SBR), sp = im(D(D_SBP));
    switch (cls) {
      case 0: return mul(cspair, sub(sr, sp));
      case 1: return sub(mul(cpair, rb), mul(cspair, sz));
      case 2: return sub(mul(-cpair, rb), mul(cspair, sz));
      default: return mul(-cspair, add(sr, sp));
    }
  }
  if (same) {
    switch (c) {
      case 0:
        return add(add(mul(T(2) * crho, D(D_RHO)), mul(ctau, D(D_TAU))),
                   mul(s, add(add(mul(T(2) * cs, D(D_SZ)), mul(ct, D(D_TZ))), mul(cf, D(D_FZ)))));
      case 1: case 4: {
        const Z a = add(mul(-crdj, sub(D(D_TJPZ), D(D_TJZP))), mul(-s * csdj, D(D_JP)));
        const Z t1 = mul(ctj1, sub(D(D_TJZR), D(D_TJRZ))), t2 = mul(ctj2, add(D(D_TJRZ), D(D_TJZR)));
        return add(a, mul(e, sub(mul(s, im(sub(t1, mul(h5, t2)))), im(mul(cj, D(D_JR))))));
      }
      case 2: case 8: {
        const Z t1 = mul(ctj1, sub(D(D_TJPZ), D(D_TJZP))), t2 = mul(ctj2, add(D(D_TJPZ), D(D_TJZP)));
        const Z a = add(mul(cj, D(D_JP)), mul(s, add(t1, mul(h5, t2))));
        return add(a, mul(e, sub(im(mul(s * csdj, D(D_JR))), im(mul(crdj, sub(D(D_TJZR), D(D_TJRZ)))))));
      }
      case 3: case 12: {
        const Z a = add(mul(-crdj, sub(D(D_TJRP), D(D_TJPR))), mul(s * T(2) * cgs, D(D_GS)));
        const Z rr = D(D_TJRR), pp = D(D_TJPP), zz = D(D_TJZZ), rp = add(rr, pp);
        const Z t = sub(mul(ctj0, add(rp, zz)), mul(ctj2 * t3, sub(rp, mul(T(2), zz))));
        return sub(a, mul(e, im(add(mul(s, t), mul(cj, D(D_JZ))))));
      }
      case 16: return add(mul(T(2) * cdrho, D(D_RHO)), mul(s * T(2) * cds, D(D_SZ)));
      case 6: case 9: return add(mul(csdj, D(D_SZ)), mul(s * crdj, D(D_RHO)));
      case 7: return add(mul(s * h5 * cf, D(D_SR)), im(mul(csdj, D(D_SP))));
      case 13: return sub(mul(s * h5 * cf, D(D_SR)), im(mul(csdj, D(D_SP))));
      case 11: return sub(mul(-csdj, D(D_SR)), im(mul(s * h5 * cf, D(D_SP))));
      case 14: return add(mul(-csdj, D(D_SR)), im(mul(s * h5 * cf, D(D_SP))));
      default: {   // (1, 1), (2, 2), (3, 3)
        const Z a = add(mul(T(4) * cdrho + ctau, D(D_RHO)), mul(s * (T(4) * cds + ct), D(D_SZ)));
        return c == 15 ? add(a, mul(s * cf, D(D_SZ))) : a;
      }
    }
  }
  switch (c) {
    case 0:
      return sub(add(add(mul(T(2) * cs, D(D_SR)), mul(ct, D(D_TR))), mul(cf, D(D_FR))),
                 im(mul(s, add(add(mul(T(2) * cs, D(D_SP)), mul(ct, D(D_TP))), mul(cf, D(D_FP))))));
    case 1: case 4: case 2: case 8: {
      const Z g = sub(mul(T(2) * cgs, D(D_GS)), im(mul(s * csdj, D(D_JZ))));
      const Z rr = D(D_TJRR), pp = D(D_TJPP), zz = D(D_TJZZ), rp = D(D_TJRP), pr = D(D_TJPR);
      const Z a1 = mul(-ctj1, sub(rp, pr)), a2 = im(mul(-ctj0, add(add(rr, pp), zz))), a3 = mul(-h5 * ctj2, add(rp, pr));
      if (c == 1 || c == 4) {
        const Z a4 = im(mul(ctj2 * t3, add(mul(T(-2), rr), add(pp, zz))));
        return add(g, mul(e, add(mul(s, add(a1, a3)), add(a2, a4))));
      }
      const Z a5 = im(mul(ctj2 * t3, add(add(rr, mul(T(-2), pp)), zz)));
      return add(mul(s, add(mul(e, g), add(a2, a5))), sub(a1, a3));
    }
    case 3: case 12: {
      const Z f = add(mul(csdj, D(D_JP)), im(mul(s * csdj, D(D_JR))));
      const Z t1a = mul(ctj1, sub(D(D_TJZR), D(D_TJRZ))), t2a = mul(ctj2, add(D(D_TJRZ), D(D_TJZR)));
      const Z t1b = mul(ctj1, sub(D(D_TJPZ), D(D_TJZP))), t2b = mul(ctj2, add(D(D_TJPZ), D(D_TJZP)));
      return add(f, mul(e, sub(mul(s, sub(t1b, mul(h5, t2b))), im(add(t1a, mul(h5, t2a))))));
    }
    case 16: return sub(mul(T(2) * cds, D(D_SR)), im(mul(s * T(2) * cds, D(D_SP))));
    case 6: case 9: {
      const Z a = add(im(mul(h5 * cf, D(D_SP))), mul(s * h5 * cf, D(D_SR)));
      return c == 6 ? a : mul(T(-1), a);
    }
    case 7: return add(mul(h5 * cf, D(D_SZ)), mul(s * crdj, D(D_RHO)));
    case 13: return sub(mul(h5 * cf, D(D_SZ)), mul(s * crdj, D(D_RHO)));
    case 11: return sub(mul(-s * h5 * cf, D(D_SZ)), mul(crdj, D(D_RHO)));
    case 14: return sub(mul(s * h5 * cf, D(D_SZ)), mul(crdj, D(D_RHO)));
    default: {   // (1, 1), (2, 2), (3, 3)
      const T k = ct + T(4) * cds;
      const Z a = sub(mul(k, D(D_SR)), im(mul(s * k, D(D_SP))));
      return c == 5 ? add(a, mul(cf, D(D_SR))) : c == 10 ? sub(a, im(mul(s * cf, D(D_SP)))) : a;
    }
  }
}

enum { SEP_ZC = 8, SEP_NX = 13, SEP_FTHR = 128 };
template <class T>
__host__ __device__ inline size_t sep_field_smem(int ngh, int zc) {
  const int x = zc * SEP_NX * 2;   // the densities (2 ND) share this space
  return (size_t)(18 * 2 + 5 + (x > 2 * ND ? x : 2 * ND)) * ngh * sizeof(T);
}
// column functions per round: the number with the fewest passes of the CTA over its unit
// sums, a round's factors and barriers counted as a third of a pass.  Up to SEP_ZC, where
// the space was judged to fit, and beyond while seven CTAs (FP32; four in FP64) fit on an SM.
// N_sh = 8 has 9 z functions (two rounds at 8, 40 sums of the threads in the second idle),
// N_sh = 16 17 (8, 8, 1: five passes; 7, 7, 3: three).  FP32, 16 points at N_sh = 8: 60 ->
// 52 us, 24 at N_sh = 16 121 -> 107 us; FP64, 9 points at N_sh = 16 443 -> 404 us
template <class T>
inline int sep_field_zc(int ngh, int nzf, int umax) {
  const int half = (umax + 1) / 2;
  int best = 1;
  long long bcost = -1;
  for (int zc = 1; zc <= 16 && zc <= nzf; ++zc) {
    if (zc > SEP_ZC && sep_field_smem<T>(ngh, zc) > (sizeof(T) == 4 ? 31 : 55) * (size_t)1024) break;
    long long cost = 0;
    for (int z0 = 0; z0 < nzf; z0 += zc)
      cost += 3LL * ((std::min(zc, nzf - z0) * half * 2 + SEP_FTHR - 1) / SEP_FTHR) + 1;
    if (bcost < 0 || cost < bcost) { bcost = cost; best = zc; }
  }
  return best;
}

template <class T>
__device__ __forceinline__ T sep_to(double x) {
  if constexpr (sizeof(T) == 4) return f32_of(x);
  else return x;
}

// dpart: the classes' shares of the densities, as k_sep_density leaves them
template <class T>
__global__ void __launch_bounds__(SEP_FTHR) k_sep_field(const __grid_constant__ SepDev<T> S,
                                                        const __grid_constant__ DevBasisT<T> B, int zc,
                                                        const T* __restrict__ dpart) {
  const int p = sep_point(S, blockIdx.z);
  if (p < 0) return;
  const int ir = blockIdx.x, call = blockIdx.y >> 2, cls = blockIdx.y & 3;
  const int ngh = S.ngh, nzf = S.nzf;
  extern __shared__ __align__(16) unsigned char smraw[];
  T* sm = reinterpret_cast<T*>(smraw);     // [16 (q, q') + (0, 4) + pairing][2][ngh]
  T* sv = sm + 18 * 2 * ngh;               // [ngh]
  T* sc4 = sv + ngh;                       // [crho, cs, cpair, cspair][ngh]
  T* sx = sc4 + 4 * ngh;                   // [zc][SEP_NX][2][ngh]
  __shared__ T ssc[12];
  {
    const T* dp = dpart + ((long long)p * 2 + call) * 4 * (2 * ND) * S.nghl + ir * ngh;
    for (int k = threadIdx.x; k < 2 * ND * ngh; k += blockDim.x) {
      const T* q = dp + (long long)(k / ngh) * S.nghl + k % ngh;
      const long long ld = (long long)(2 * ND) * S.nghl;
      sx[k] = ((q[0] + q[ld]) + (q[2 * ld] + q[3 * ld])) * sep_to<T>(B.wdcori[ir * ngh + k % ngh]);
    }
    // the couplings are FP64: converted once per CTA (and not by the FP64 pipe, which spent
    // 32 us of 108 on it when every component converted what it used): 24 points at N_sh = 16
    // 107 -> 103.5 us, 16 at N_sh = 8 52 -> 48 us, FP64 9 points at N_sh = 16 404 -> 375 us
    for (int k = threadIdx.x; k < ngh; k += blockDim.x) {
      const int r = ir * ngh + k;
      sv[k] = S.v[r];
      sc4[k] = sep_to<T>(B.crho[r]);
      sc4[ngh + k] = sep_to<T>(B.cs[r]);
      sc4[2 * ngh + k] = sep_to<T>(B.cpair[r]);
      sc4[3 * ngh + k] = sep_to<T>(B.cspair[r]);
    }
    if (threadIdx.x < 12) ssc[threadIdx.x] = sep_to<T>(B.sc[threadIdx.x]);
    __syncthreads();
    // a warp takes one component at a time: the components' formulas differ
    const int nh = (ngh + 31) / 32 * 32;
    for (int k = threadIdx.x; k < 18 * nh; k += blockDim.x) {
      const int ih = k % nh, c = k / nh;
      if (ih >= ngh) continue;
      const cplxT<T> f = sep_meanfield<T>(c, cls, sx + ih, ngh, ssc, sc4[ih], sc4[ngh + ih], sc4[2 * ngh + ih],
                                          sc4[3 * ngh + ih]);
      sm[(2 * c) * ngh + ih] = f.r;
      sm[(2 * c + 1) * ngh + ih] = f.i;
    }
  }
  T* gp = S.g + p * S.gstride;
  const T y = S.y[ir];
  __syncthreads();
  for (int z0 = 0; z0 < nzf; z0 += zc) {
    const int z1 = min(nzf, z0 + zc);
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
    // a thread takes the units (n_z', n_z) and (n_z', next n_z) of one plane
    const int half = (S.f.umax + 1) / 2;
    for (int k = threadIdx.x; k < (z1 - z0) * half * 2; k += blockDim.x) {
      const int pl = k & 1, c = (k >> 1) / half, j = (k >> 1) % half;
      const int ub = S.f.ubeg[cls * (nzf + 1) + z0 + c], ue = S.f.ubeg[cls * (nzf + 1) + z0 + c + 1];
      const int u = ub + 2 * j;
      if (u >= ue) continue;
      const bool two = u + 1 < ue;
      const T* x = sx + ((long long)c * SEP_NX * 2 + pl) * ngh;
      const T *Z0 = S.z + (2 * S.f.units[u].nz) * ngh, *Z1 = S.z + (2 * S.f.units[two ? u + 1 : u].nz) * ngh;
      T h[2][SH_N];
#pragma unroll
      for (int i = 0; i < SH_N; ++i) h[0][i] = h[1][i] = T(0);
      for (int ih = 0; ih < ngh; ++ih) {
        const T a0 = Z0[ih], b0 = Z0[ngh + ih], a1 = Z1[ih], b1 = Z1[ngh + ih];
#pragma unroll
        for (int i = 0; i < SEP_NX; ++i) {
          const T v = x[i * 2 * ngh + ih];
          const int o = i < SH_N ? i : i == 10 ? SG_RR : i == 11 ? SG_RD : SG_BRR;
          h[0][o] = fma(i < SH_N ? a0 : b0, v, h[0][o]);
          if (two) h[1][o] = fma(i < SH_N ? a1 : b1, v, h[1][o]);
        }
      }
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        if (w && !two) break;
        h[w][SG_ARR] *= y; h[w][SG_BRR] *= y; h[w][SG_ABRR] *= y * y; h[w][SG_BDR] *= y; h[w][SG_ARD] *= y;
        T* g = gp + ((long long)(call * S.ngl + ir) * S.f.nu + u + w) * (2 * SH_N) + pl;
#pragma unroll
        for (int i = 0; i < SH_N; ++i) g[2 * i] = h[w][i];
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
// projection 2: the radial sums, hsp [P][2 planes][4 quadrants][nxy].  A warp takes 32 /
// SPL items of one unit and call and first brings the unit's fields at all radial points
// into shared memory (80 or 160 consecutive bytes per point, where reading them as they
// are used is one load per value); a lane combines them with its row state (10 products
// per column of Re and Im) and sums SEP_GC column states, over every SPL-th radial point.
// SPL = 1 on large bases in FP32, where a unit's items fill warps; SPL = 4 in FP64, which
// is bound by its pipe and so by lanes without an item (units have 9 items at N_sh = 6,
// 52 at N_sh = 16), and on small bases, bound by the chain of a lane.  CTAs of eight
// warps also keep the radial functions in shared memory (STAGE; not when few warps make
// one-warp CTAs).
// grid (warps of F x 2 calls, X and Y, over the warps of a CTA; points)
// ---------------------------------------------------------------------------
template <class T>
__host__ __device__ inline size_t sep_project_smem(int ngl, int nrow, int nwarp, bool stage) {
  return ((size_t)nwarp * ngl * SH_N + (stage ? (size_t)ngl * nrow : 0)) * 2 * sizeof(T);
}

template <class T, int SPL>
__device__ __forceinline__ void sep_project_normal(const SepDev<T>& S, const SepWarp& W, int p, T* __restrict__ hsp,
                                                   long long nxy, int call, const typename Vec2<T>::t* rt,
                                                   typename Vec2<T>::t* sh) {
  using V2 = typename Vec2<T>::t;
  const int lane = threadIdx.x & 31, li = lane / SPL, part = lane % SPL, ngl = S.ngl;
  {
    const V2* g = reinterpret_cast<const V2*>(S.g + p * S.gstride) +
                  ((long long)call * ngl * S.f.nu + W.unit) * SH_N;
    const long long gs = (long long)S.f.nu * SH_N;
    if constexpr (sizeof(T) == 4) {   // 16 bytes at a time: SH_N pairs are five of them
      for (int k = lane; k < ngl * (SH_N / 2); k += 32)
        reinterpret_cast<float4*>(sh)[k] =
            reinterpret_cast<const float4*>(g + (long long)(k / (SH_N / 2)) * gs)[k % (SH_N / 2)];
    } else {
      for (int k = lane; k < ngl * SH_N; k += 32) sh[k] = g[(long long)(k / SH_N) * gs + k % SH_N];
    }
  }
  const int* it = S.f.items + W.item0 + min(li, W.nitem - 1);
  const long long ni = S.f.nitem;
  const int seg = it[SI_SEG * ni], segp = it[SI_SEGP * ni], row = it[SI_ROW * ni];
  const T la = S.lam[seg], lb = S.lam[segp], lab = la * lb;
  int rp[SEP_GC];
#pragma unroll
  for (int k = 0; k < SEP_GC; ++k) rp[k] = it[(SI_ROWP + k) * ni];
  T acc[SEP_GC][2], lap[SEP_GC][2];
#pragma unroll
  for (int k = 0; k < SEP_GC; ++k) acc[k][0] = acc[k][1] = lap[k][0] = lap[k][1] = T(0);
  const int nmax = W.nmax;
  __syncwarp();
#pragma unroll 2
  for (int ir = part; ir < ngl; ir += SPL) {
    const V2 *r = rt + ir * S.nrow, *h = sh + ir * SH_N;
    const V2 a = r[row];
    T vr[2], vd[2], vl[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
#define H_(k) (c ? h[k].y : h[k].x)
      const T rr = fma(lab, H_(SG_ABRR), fma(lb, H_(SG_BRR), fma(la, H_(SG_ARR), H_(SG_RR))));
      const T dr = fma(lb, H_(SG_BDR), H_(SG_DR));
      const T rd = fma(la, H_(SG_ARD), H_(SG_RD));
      vr[c] = fma(a.x, rr, a.y * dr);
      vd[c] = fma(a.x, rd, a.y * H_(SG_DD));
      vl[c] = a.x * H_(SH_L);
#undef H_
    }
#pragma unroll
    for (int k = 0; k < SEP_GC; ++k) {
      if (k >= nmax) break;
      const V2 b = r[rp[k]];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        acc[k][c] = fma(b.x, vr[c], fma(b.y, vd[c], acc[k][c]));
        lap[k][c] = fma(b.x, vl[c], lap[k][c]);
      }
    }
  }
  const T s = T(2) * S.sgn[seg] * S.sgn[segp], ea = S.e[it[SI_JA * ni]];
  const int cnt = it[SI_CNT * ni];
  T* out = hsp + (long long)p * 8 * nxy + (call ? 3 * nxy : 0);
#pragma unroll
  for (int k = 0; k < SEP_GC; ++k) {
    if (k >= nmax) break;
    const bool mine = part == 0 && li < W.nitem && k < cnt;
    const T ee = ea + S.e[it[(SI_JB + k) * ni]];
    const int off = it[(SI_OFF + k) * ni];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      T x = acc[k][c], y = lap[k][c];
#pragma unroll
      for (int o = 1; o < SPL; o *= 2) {
        x += __shfl_xor_sync(0xffffffffu, x, o);
        y += __shfl_xor_sync(0xffffffffu, y, o);
      }
      if (mine) out[c * 4 * nxy + off] = s * fma(-ee, y, x);
    }
  }
}

template <class T, int SPL>
__device__ __forceinline__ void sep_project_pair(const SepDev<T>& S, const SepWarp& W, int call, int p,
                                                 T* __restrict__ hsp, long long nxy,
                                                 const typename Vec2<T>::t* rt, typename Vec2<T>::t* sh) {
  using V2 = typename Vec2<T>::t;
  const SepStructDev& X = S.d[call];
  const int lane = threadIdx.x & 31, li = lane / SPL, part = lane % SPL, ngl = S.ngl;
  {
    const V2* g = reinterpret_cast<const V2*>(S.g + p * S.gstride + S.gpair[call]) + W.unit;
    for (int k = lane; k < ngl; k += 32) sh[k] = g[(long long)k * X.nu];
  }
  const int* it = X.items + W.item0 + min(li, W.nitem - 1);
  const long long ni = X.nitem;
  const int seg = it[SI_SEG * ni], segp = it[SI_SEGP * ni], row = it[SI_ROW * ni];
  int rp[SEP_GC];
#pragma unroll
  for (int k = 0; k < SEP_GC; ++k) rp[k] = it[(SI_ROWP + k) * ni];
  T acc[SEP_GC][2];
#pragma unroll
  for (int k = 0; k < SEP_GC; ++k) acc[k][0] = acc[k][1] = T(0);
  const int nmax = W.nmax;
  __syncwarp();
#pragma unroll 2
  for (int ir = part; ir < ngl; ir += SPL) {
    const V2* r = rt + ir * S.nrow;
    const V2 h = sh[ir];
    const T a = r[row].x, v0 = a * h.x, v1 = a * h.y;
#pragma unroll
    for (int k = 0; k < SEP_GC; ++k) {
      if (k >= nmax) break;
      const T b = r[rp[k]].x;
      acc[k][0] = fma(b, v0, acc[k][0]);
      acc[k][1] = fma(b, v1, acc[k][1]);
    }
  }
  const T s = T(2) * S.sgn[seg] * S.sgn[segp];
  const int cnt = it[SI_CNT * ni];
  T* out = hsp + (long long)p * 8 * nxy + (call ? 2 : 1) * nxy;
#pragma unroll
  for (int k = 0; k < SEP_GC; ++k) {
    if (k >= nmax) break;
    const bool mine = part == 0 && li < W.nitem && k < cnt;
    const int off = it[(SI_OFF + k) * ni];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      T v = acc[k][c];
#pragma unroll
      for (int o = 1; o < SPL; o *= 2) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (mine) out[c * 4 * nxy + off] = s * v;
    }
  }
}

template <class T, int SPL, bool STAGE>
__global__ void __launch_bounds__(256) k_sep_project(const __grid_constant__ SepDev<T> S, T* __restrict__ hsp,
                                                     long long nxy) {
  using V2 = typename Vec2<T>::t;
  constexpr int H = SPL > 1;
  const int p = sep_point(S, blockIdx.y);
  if (p < 0) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  V2* sh = reinterpret_cast<V2*>(smraw) + (size_t)(threadIdx.x >> 5) * S.ngl * SH_N;
  const V2* rt = S.rt;
  if (STAGE) {
    V2* sr = reinterpret_cast<V2*>(smraw) + (size_t)(blockDim.x >> 5) * S.ngl * SH_N;
    for (int k = threadIdx.x; k < S.ngl * S.nrow; k += blockDim.x) sr[k] = rt[k];
    rt = sr;
    __syncthreads();
  }
  int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int nf = S.f.nwarp[H] * 2;
  if (w < nf) { sep_project_normal<T, SPL>(S, S.f.warps[H][w >> 1], p, hsp, nxy, w & 1, rt, sh); return; }
  w -= nf;
  if (w < S.d[0].nwarp[H]) { sep_project_pair<T, SPL>(S, S.d[0].warps[H][w], 0, p, hsp, nxy, rt, sh); return; }
  w -= S.d[0].nwarp[H];
  if (w < S.d[1].nwarp[H]) sep_project_pair<T, SPL>(S, S.d[1].warps[H][w], 1, p, hsp, nxy, rt, sh);
}

}  // namespace pnfam
#endif
