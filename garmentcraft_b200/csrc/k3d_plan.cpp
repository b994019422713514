// Pattern of the block operator and the tiles of the tiled PCG (host).
#include "k3d_plan.h"

#include <algorithm>
#include <cmath>

namespace k3d {

void spalten(const Elemente& E, Spalten& S) {
  S.anf.assign(E.n + 1, 0);
  S.sp.clear();
  S.sp.reserve(E.n * 14);
  std::vector<uint32_t> wer(E.n, 0xffffffffu);
  for (size_t i = 0; i < E.n; ++i) {
    const size_t a0 = S.sp.size();
    auto nimm = [&](uint32_t j) {
      if (wer[j] == uint32_t(i)) return;
      wer[j] = uint32_t(i);
      S.sp.push_back(j);
    };
    nimm(uint32_t(i));
    for (uint32_t e = E.off_t[i]; e < E.off_t[i + 1]; ++e)
      for (int b = 0; b < 3; ++b) nimm(E.m_p[3 * size_t(E.ent_t[e] / 3) + b]);
    for (uint32_t e = E.off_b[i]; e < E.off_b[i + 1]; ++e)
      for (int b = 0; b < 4; ++b) nimm(E.b_p[4 * size_t(E.ent_b[e] / 4) + b]);
    for (uint32_t e = E.off_s[i]; e < E.off_s[i + 1]; ++e) {
      nimm(E.s_p[E.ent_s[e] / 2].x);
      nimm(E.s_p[E.ent_s[e] / 2].y);
    }
    std::sort(S.sp.begin() + std::ptrdiff_t(a0), S.sp.end());
    S.anf[i + 1] = uint32_t(S.sp.size());
  }
}

namespace {

// Bytes of streamed slabs that are asked to stay in L2 where there are more of
// them. Measured, thousand cycles an iteration with 100 (no rule), 64, 40, 24,
// 16 and 8 MB: 160 k points, FP32 blocks (65 MB streamed) 49.6, 49.3, 47.9,
// 42.1, 42.9, 45.0; 160 k, FP64 (146 MB) 94.8, -, 77.9, 74.0, 72.5, 72.0;
// 205 k of a garment, FP32 blocks -, 62.2, 54.7, 52.1, 52.2, 52.5; 90 k, FP64
// (81 MB) 48.2, -, 43.4, 43.3, 44.0, 41.3; up to 55 MB no difference.
constexpr size_t kKachelL2 = size_t(24) << 20;

// Splits the points idx[lo, hi) into nb parts of whole slices (the last one
// may be ragged), in the order of the bisection, across the longest side of
// their box; ties by point, so the parts are the same everywhere.
void teile(std::vector<uint32_t>& idx, size_t lo, size_t hi, int nb, const double* x, std::vector<size_t>& anf) {
  if (nb == 1) {
    anf.push_back(hi);
    return;
  }
  double mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
  auto wert = [&](uint32_t i, int a) {
    const double v = x[3 * size_t(i) + a];
    return std::isfinite(v) ? v : 0.0;
  };
  for (size_t q = lo; q < hi; ++q)
    for (int a = 0; a < 3; ++a) {
      const double v = wert(idx[q], a);
      mn[a] = std::min(mn[a], v);
      mx[a] = std::max(mx[a], v);
    }
  int achse = 0;
  for (int a = 1; a < 3; ++a)
    if (mx[a] - mn[a] > mx[achse] - mn[achse]) achse = a;
  const int nl = nb / 2;
  const size_t sl = (hi - lo + 31) / 32;
  size_t links = (sl * size_t(nl) + size_t(nb) / 2) / size_t(nb);
  links = std::max<size_t>(links, size_t(nl));
  links = std::min<size_t>(links, sl - size_t(nb - nl));
  const size_t m = lo + 32 * links;
  std::nth_element(idx.begin() + std::ptrdiff_t(lo), idx.begin() + std::ptrdiff_t(m), idx.begin() + std::ptrdiff_t(hi),
                   [&](uint32_t a, uint32_t b) {
                     const double u = wert(a, achse), v = wert(b, achse);
                     return u < v || (u == v && a < b);
                   });
  teile(idx, lo, m, nl, x, anf);
  teile(idx, m, hi, nb - nl, x, anf);
}

}  // namespace

bool kachelplan(const Spalten& S, const double* x, const std::vector<int64_t>& io, const std::vector<int>& nblk,
                size_t rsize, bool federn, size_t smem, size_t kopf, Kachelplan& P) {
  const size_t n = S.anf.size() - 1;
  if (n == 0 || smem == 0 || n >= (size_t(1) << 31)) return false;
  P = Kachelplan{};
  const int ng = int(nblk.size());
  P.nblk.assign(size_t(ng), 0);
  std::vector<uint32_t> idx(n), von(n);
  P.pos.assign(n, 0);
  P.q = 1;
  uint32_t worte = 0;
  const size_t warps = kachel_warps(rsize);
  auto kachel = [&](const uint32_t* i, size_t m) {  // one tile of the points i[0, m), positions in this order
    KachelBlk B{};
    B.row0 = uint32_t(P.row.size());
    B.rows = uint32_t(m);
    for (size_t q = 0; q < m; ++q) {
      P.pos[i[q]] = uint32_t(P.row.size());
      von[i[q]] = uint32_t(P.blk.size());
      P.row.push_back(i[q]);
    }
    const size_t ns = (m + 31) / 32;
    P.row.resize(size_t(B.row0) + 32 * ns, 0xffffffffu);
    P.q = std::max(P.q, int((ns + 15) / 16));
    P.blk.push_back(B);
  };
  for (int k = 0; k < ng; ++k) {
    const size_t lo = size_t(io[k]), hi = size_t(io[k + 1]), m = hi - lo, nb = size_t(nblk[k]);
    const size_t erst = P.blk.size(), ns = (m + 31) / 32;
    if (m == 0 || nb < 1) return false;
    for (size_t i = lo; i < hi; ++i) idx[i] = uint32_t(i);
    bool einzeln = false;
    if (ng > 1 || (m <= kKachelNatur && !federn)) {
      einzeln = m <= 512 * nb && ns <= 512 && ns <= nb * warps;
      if (einzeln) {
        for (size_t s = 0; s < ns; s += warps)
          kachel(&idx[lo + 32 * s], std::min<size_t>(32 * warps, m - 32 * s));
      } else {
        std::vector<uint32_t> r;
        for (size_t b = 0; b < nb && 512 * b < m; ++b) {
          r.clear();
          for (size_t c = b; 512 * c < m; c += nb)
            for (size_t i = 512 * c; i < std::min(m, 512 * (c + 1)); ++i) r.push_back(uint32_t(lo + i));
          kachel(r.data(), r.size());
        }
      }
    } else {
      std::vector<size_t> anf(1, lo);
      teile(idx, lo, hi, int(std::min(nb, federn ? (ns + 1) / 2 : ns)), x, anf);
      for (size_t b = 0; b + 1 < anf.size(); ++b) {  // within a tile the points keep their natural order
        std::sort(idx.begin() + std::ptrdiff_t(anf[b]), idx.begin() + std::ptrdiff_t(anf[b + 1]));
        kachel(&idx[anf[b]], anf[b + 1] - anf[b]);
      }
    }
    P.nblk[k] = int(P.blk.size() - erst);
    const uint32_t w0 = worte;
    for (size_t b = erst; b < P.blk.size(); ++b) {
      P.blk[b].wort0 = worte;
      worte += einzeln ? (P.blk[b].rows + 31) / 32 : 1;
    }
    for (size_t b = erst; b < P.blk.size(); ++b) {
      P.blk[b].gruppe0 = w0;
      P.blk[b].worte = worte - w0;
      P.blk[b].einzeln = einzeln ? 1u : 0u;
    }
  }
  P.blocks = int(P.blk.size());
  if (P.blocks > kKachelBloecke || P.q > kKachelZeilen || worte > uint32_t(kKachelWorte)) return false;
  // halos
  std::vector<uint32_t> in(n, 0xffffffffu);  // the tile whose halo holds the point (last seen)
  std::vector<uint32_t> halo;
  for (int b = 0; b < P.blocks; ++b) {
    KachelBlk& B = P.blk[b];
    halo.clear();
    for (uint32_t r = 0; r < B.rows; ++r) {
      const uint32_t i = P.row[B.row0 + r];
      for (uint32_t e = S.anf[i]; e < S.anf[i + 1]; ++e) {
        const uint32_t j = S.sp[e];
        if (von[j] == uint32_t(b) || in[j] == uint32_t(b)) continue;
        in[j] = uint32_t(b);
        halo.push_back(j);
      }
    }
    std::sort(halo.begin(), halo.end());
    B.halo0 = uint32_t(P.halo.size());
    B.halos = uint32_t(halo.size());
    P.halo.insert(P.halo.end(), halo.begin(), halo.end());
  }
  // slabs: a slice is as wide as its widest row. What a warp's share of the
  // shared memory behind the tile does not hold is streamed: whole grips of
  // the first ranks, evenly over the warp's slices (warp, warp + 16, ...)
  P.slice.assign(P.row.size() / 32, make_uint4(0u, 0u, 0u, 0u));
  const size_t satz = kachel_satz(rsize), griff = size_t(kachel_griff(rsize, P.q));
  for (KachelBlk& B : P.blk) {
    const size_t ns = (size_t(B.rows) + 31) / 32, s0 = B.row0 / 32, nw = std::min<size_t>(ns, 16);
    const size_t ts = 32 * ns + B.halos;
    if (ts > 65535) return false;
    const size_t vorn = kopf + kachel_tile(rsize, ns, B.halos, kachel_ap(rsize, P.q), federn);
    if (vorn >= smem) return false;
    const size_t platz = (smem - vorn) / (nw * satz);
    std::vector<uint32_t> breit(ns, 0);
    size_t most = 0;
    for (size_t w = 0; w < nw; ++w) {
      size_t m = 0;
      for (size_t s = w; s < ns; s += 16) {
        for (size_t l = 0; l < 32; ++l) {
          const uint32_t i = P.row[32 * (s0 + s) + l];
          if (i != 0xffffffffu) breit[s] = std::max(breit[s], S.breit(i));
        }
        m += breit[s];
      }
      most = std::max(most, m);
    }
    B.platz = uint32_t(platz);
    B.stufen = 0;
    // the ring's depth: what a warp reads ahead against what it keeps. Two
    // stages (three of one slab) serve where most of the slabs stay; one more
    // where most are streamed
    if (most > platz) {
      size_t rest = 0;
      for (size_t w = 0; w < nw; ++w) {
        size_t r = 0;
        for (size_t s = w; s < ns; s += 16) r += breit[s] % griff;
        rest = std::max(rest, r);
      }
      B.stufen = uint32_t((griff == 1 ? 3 : 2) + (most >= 2 * platz ? 1 : 0));
      while (B.stufen > 2 && B.stufen * griff + rest > platz) --B.stufen;
    }
    const size_t fest = platz < B.stufen * griff ? 0 : platz - B.stufen * griff;
    for (size_t w = 0; w < nw; ++w) {
      size_t m = 0, rest = 0;
      for (size_t s = w; s < ns; s += 16) {
        m += breit[s];
        rest += breit[s] % griff;
      }
      if (B.stufen && (platz < B.stufen * griff || rest > fest)) return false;
      size_t strom = 0;  // slabs streamed so far
      const size_t soll = B.stufen && m > fest ? m - fest : 0;
      size_t vor = 0;    // slabs of the slices before
      for (size_t s = w; s < ns; s += 16) {
        vor += breit[s];
        // up to here at least soll * vor / m of the slabs, in whole grips
        const size_t ziel = m ? (soll * vor + m - 1) / m : 0;
        size_t k = ziel > strom ? (ziel - strom + griff - 1) / griff * griff : 0;
        if (k > breit[s]) k = breit[s] / griff * griff;
        P.slice[s0 + s].y = uint32_t(k);
        P.slice[s0 + s].w = breit[s] - uint32_t(k);
        strom += k;
      }
      for (size_t s = w; strom < soll && s < ns; s += 16)  // what the rounding down left
        while (strom < soll && P.slice[s0 + s].w >= griff) {
          P.slice[s0 + s].y += uint32_t(griff);
          P.slice[s0 + s].w -= uint32_t(griff);
          strom += griff;
        }
      if (strom < soll) return false;
      for (size_t s = w; s < ns; s += 16) {
        P.slice[s0 + s].x = uint32_t(P.slabs);
        P.slabs += P.slice[s0 + s].y;
      }
      for (size_t s = w; s < ns; s += 16) {
        P.slice[s0 + s].z = uint32_t(P.slabs);
        P.slabs += P.slice[s0 + s].w;
      }
    }
  }
  if (P.slabs * 32 >= (size_t(1) << 32)) return false;
  // What an iteration streams comes round again in the same order, so where the
  // L2 cannot keep it all each slab is evicted before its next turn. A part is
  // then asked to stay and the rest to leave first.
  {
    size_t alle = 0;
    for (const uint4& s : P.slice) alle += s.y;
    const double anteil = alle * satz > kKachelL2 ? double(kKachelL2) / double(alle * satz) : 1.0;
    for (KachelBlk& B : P.blk) {
      const size_t ns = (size_t(B.rows) + 31) / 32;
      size_t m = 0;
      for (size_t s = 0; s < ns; s += 16) m += P.slice[B.row0 / 32 + s].y;
      B.bleibt = anteil < 1.0 ? uint32_t(anteil * double(m)) : 0xffffffffu;
    }
  }
  // columns
  P.col.assign(P.slabs * 32, 0xffffffffu);
  P.lc.assign(P.slabs * 32, 0);
  std::vector<uint32_t> lokal(n);
  for (int b = 0; b < P.blocks; ++b) {
    const KachelBlk& B = P.blk[b];
    const size_t ns = (size_t(B.rows) + 31) / 32;
    for (uint32_t r = 0; r < B.rows; ++r) lokal[P.row[B.row0 + r]] = r;
    for (uint32_t h = 0; h < B.halos; ++h) lokal[P.halo[B.halo0 + h]] = uint32_t(32 * ns + h);
    for (uint32_t r = 0; r < B.rows; ++r) {
      const uint32_t i = P.row[B.row0 + r];
      const uint4 sl = P.slice[(B.row0 + r) / 32];
      for (uint32_t k = 0; k < sl.y + sl.w; ++k) {
        const size_t q = size_t(k < sl.y ? sl.x + k : sl.z + (k - sl.y)) * 32 + (r & 31u);
        if (k < S.breit(i)) {
          const uint32_t j = S.sp[S.anf[i] + k];
          P.col[q] = j | (j == i ? 0x80000000u : 0u);
          P.lc[q] = uint16_t(lokal[j]);
        } else {
          P.lc[q] = uint16_t(r);
        }
      }
    }
  }
  for (uint32_t j : P.halo) P.row[P.pos[j]] |= 0x80000000u;
  return true;
}

}  // namespace k3d
