// The tables of csrc/separable.cuh on the host: the factors of a basis, and one real
// density and one field projection summed through a structure's units, in the order of
// the kernels (their index arithmetic is that of the tables).
#include "../pynfam_gb300/csrc/separable.cuh"

using namespace pnfam;

// out_c [4 classes][16][nghl]: C(q, q'); fields m [4][17][nghl] ((q, q'), then (0, 4));
// out_h [elements].  Returns the mesh points along z, 0 when the basis is not accepted.
extern "C" int sep_host_check(int nb, const int* db, const int* nup, int nghl, const double* phi, const int* cols,
                              const double* rho, const double* m, double* out_c, double* out_h) {
  std::vector<int> st(nb);
  int dqp = 0;
  for (int i = 0; i < nb; ++i) { st[i] = dqp; dqp += db[i]; }
  const int ngh = sep_mesh(dqp, nghl, phi);
  SepBasis B;
  if (!ngh || !sep_factors(nb, db, st.data(), nup, dqp, nghl, ngh, phi, B)) return 0;
  const int ngl = B.ngl;
  for (int i = 0; i < nb; ++i)
    for (int a = st[i]; a < st[i] + db[i]; ++a) {
      const int sg = 2 * i + (a >= st[i] + nup[i]);
      for (int q = 0; q < 5; ++q) {
        const double* f = phi + ((size_t)q * dqp + a) * nghl;
        double top = 0.0;
        for (int k = 0; k < nghl; ++k) top = fmax(top, fabs(f[k]));
        for (int k = 0; k < nghl; ++k) {
          const double w = sep_value(q, B.z.data(), B.r.data(), B.v[k], B.y[k / ngh], B.e[a], B.lam[sg], B.sgn[sg],
                                     k % ngh, k / ngh, ngh, B.zi[a], B.ri[a], ngl);
          if (!(fabs(f[k] - w) <= SEP_TOL * top)) return 0;
        }
      }
    }
  std::vector<long long> off(nb, -1);
  long long nxy = 0;
  for (int i = 0; i < nb; ++i)
    if (cols[i] >= 0) { off[i] = nxy; nxy += (long long)db[i] * db[cols[i]]; }
  SepStruct S;
  if (!sep_structure(B, nb, db, st.data(), nup, cols, off.data(), true, S)) return 0;
  auto R = [&](int row, int il) { return &B.r[((size_t)row * ngl + il) * 2]; };
  auto Z = [&](int z, int d, int ih) { return B.z[(size_t)(2 * z + d) * ngh + ih]; };
  // units in their launch order, both directions
  for (int ui : S.order) {
    const SepUnit& u = S.units[ui];
    if (ui < S.ubeg[u.cls * (B.nzf + 1) + u.nzp] || ui >= S.ubeg[u.cls * (B.nzf + 1) + u.nzp + 1]) return 0;
    for (int il = 0; il < ngl; ++il) {
      double g[SG_N] = {0};
      for (int e = u.ent0; e < u.ent0 + u.nent; ++e) {
        const SepEnt& q = S.ents[e];
        double o[4] = {0};
        for (int k = 0; k < q.ngp; ++k)
          for (int j = 0; j < q.ng; ++j) {
            const double *a = R(S.rows[q.row0 + j], il), *b = R(S.rows[q.rowp0 + k], il);
            const double x = rho[S.offs[q.el0 + k * q.ng + j]];
            o[0] += a[0] * b[0] * x; o[1] += a[1] * b[0] * x; o[2] += a[0] * b[1] * x; o[3] += a[1] * b[1] * x;
          }
        const double sg = B.sgn[q.seg] * B.sgn[q.segp], la = B.lam[q.seg] * B.y[il], lb = B.lam[q.segp] * B.y[il];
        g[SG_RR] += sg * o[0]; g[SG_DR] += sg * o[1]; g[SG_RD] += sg * o[2]; g[SG_DD] += sg * o[3];
        g[SG_ARR] += sg * la * o[0]; g[SG_BRR] += sg * lb * o[0]; g[SG_ABRR] += sg * la * lb * o[0];
        g[SG_BDR] += sg * lb * o[1]; g[SG_ARD] += sg * la * o[2];
      }
      const int zz[16] = {SG_RR, SG_RD, SG_BRR, SG_RR, SG_DR, SG_DD, SG_BDR, SG_DR,
                          SG_ARR, SG_ARD, SG_ABRR, SG_ARR, SG_RR, SG_RD, SG_BRR, SG_RR};
      for (int ih = 0; ih < ngh; ++ih)
        for (int c = 0; c < 16; ++c)
          out_c[((size_t)u.cls * 16 + c) * nghl + il * ngh + ih] +=
              Z(u.nz, c / 4 == 3, ih) * Z(u.nzp, c % 4 == 3, ih) * g[zz[c]];
    }
  }
  // both groupings hold the same items
  std::vector<int> seen(S.items.size(), 0);
  for (const SepWarp& w : S.warps[1])
    for (int k = w.item0; k < w.item0 + w.nitem; ++k) seen[k] += w.nitem <= 32 / SEP_SPL && S.items[k].n <= w.nmax;
  for (int k : seen)
    if (k != 1) return 0;
  for (const SepWarp& w : S.warps[0]) {
    const SepUnit& u = S.units[w.unit];
    for (int k = w.item0; k < w.item0 + w.nitem; ++k) {
      const SepItem& it = S.items[k];
      if (it.n > w.nmax || it.n > SEP_GC) return 0;
      for (int b = 0; b < it.n; ++b) {
        double h = 0.0;
        for (int il = 0; il < ngl; ++il) {
          const double la = B.lam[it.seg] * B.y[il], lb = B.lam[it.segp] * B.y[il];
          const double *r = R(it.row, il), *p = R(it.rowp[b], il);
          for (int ih = 0; ih < ngh; ++ih) {
            const double fa[4] = {r[0] * Z(u.nz, 0, ih), r[1] * Z(u.nz, 0, ih), la * r[0] * Z(u.nz, 0, ih),
                                  r[0] * Z(u.nz, 1, ih)};
            const double fb[4] = {p[0] * Z(u.nzp, 0, ih), p[1] * Z(u.nzp, 0, ih), lb * p[0] * Z(u.nzp, 0, ih),
                                  p[0] * Z(u.nzp, 1, ih)};
            const double* f = m + (size_t)u.cls * 17 * nghl + il * ngh + ih;
            for (int c = 0; c < 16; ++c) h += fa[c / 4] * fb[c % 4] * f[(size_t)c * nghl];
            h += fa[0] * fb[0] * f[(size_t)16 * nghl] * (2 * B.v[il * ngh + ih] - B.e[it.ja] - B.e[it.jb[b]]);
          }
        }
        out_h[it.off[b]] += 2 * B.sgn[it.seg] * B.sgn[it.segp] * h;
      }
    }
  }
  return ngh;
}
