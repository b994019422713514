// Host side of the block operator: the pattern of A, the tiles of the tiled
// PCG and the blocks' contribution lists (internal to the library).
#pragma once
#include <cstdint>
#include <vector>

#include "k3d_step.h"

namespace k3d {

// The elements of a scene and each point's element corners (element order):
// ent_t holds 3 t + corner, ent_b 4 b + corner, ent_s 2 s + end.
struct Elemente {
  size_t n = 0;
  const uint32_t* m_p = nullptr;  // 3 points per membrane
  const uint32_t* b_p = nullptr;  // 4 per hinge
  const uint4* s_p = nullptr;     // 2 per spring (x, y)
  size_t nt = 0, nb = 0, ns = 0;
  const uint32_t *off_t = nullptr, *ent_t = nullptr, *off_b = nullptr, *ent_b = nullptr, *off_s = nullptr,
                 *ent_s = nullptr;
};

// 3x3-block pattern of A: per point its sorted columns (its own among them).
struct Spalten {
  std::vector<uint32_t> anf, sp;  // starts (n + 1), columns
  uint32_t breit(size_t i) const { return anf[i + 1] - anf[i]; }
};
void spalten(const Elemente& E, Spalten& S);

// Contribution lists of the blocks, block (row i, rank k) at slot(i, k) of
// `slots`: per block its element contributions in a fixed order (membranes,
// then bends, then springs, each in element order, then by corner pair). Code:
// type << 30 | a << 28 | b << 26 | id.
template <typename Slot>
void beitraege(const Elemente& E, const Spalten& S, size_t slots, Slot&& slot, std::vector<uint32_t>& off,
               std::vector<uint32_t>& ctr) {
  off.assign(slots + 1, 0);
  std::vector<uint32_t> rang(E.n), wo(E.n, 0xffffffffu);
  std::vector<uint32_t> cur;
  auto reihe = [&](size_t i, auto&& f) {  // f(rank, code) over row i's contributions
    const uint32_t a0 = S.anf[i], m = S.breit(i);
    for (uint32_t k = 0; k < m; ++k) rang[S.sp[a0 + k]] = k;
    for (uint32_t e = E.off_t[i]; e < E.off_t[i + 1]; ++e) {
      const uint32_t c = E.ent_t[e], t = c / 3, a = c % 3;
      for (uint32_t b = 0; b < 3; ++b) f(rang[E.m_p[3 * size_t(t) + b]], (0u << 30) | (a << 28) | (b << 26) | t);
    }
    for (uint32_t e = E.off_b[i]; e < E.off_b[i + 1]; ++e) {
      const uint32_t c = E.ent_b[e], t = c / 4, a = c % 4;
      for (uint32_t b = 0; b < 4; ++b) f(rang[E.b_p[4 * size_t(t) + b]], (1u << 30) | (a << 28) | (b << 26) | t);
    }
    for (uint32_t e = E.off_s[i]; e < E.off_s[i + 1]; ++e) {
      const uint32_t c = E.ent_s[e], t = c / 2, a = c % 2;
      const uint32_t ij[2] = {E.s_p[t].x, E.s_p[t].y};
      for (uint32_t b = 0; b < 2; ++b) f(rang[ij[b]], (2u << 30) | (a << 28) | (b << 26) | t);
    }
  };
  for (size_t i = 0; i < E.n; ++i) reihe(i, [&](uint32_t k, uint32_t) { off[slot(i, k) + 1]++; });
  for (size_t q = 0; q < slots; ++q) off[q + 1] += off[q];
  ctr.assign(off[slots], 0);
  for (size_t i = 0; i < E.n; ++i) {
    const uint32_t m = S.breit(i);
    cur.assign(m, 0);
    reihe(i, [&](uint32_t k, uint32_t code) { ctr[off[slot(i, k)] + cur[k]++] = code; });
  }
}

// The tiles of the tiled PCG.
struct Kachelplan {
  int blocks = 0, q = 0;
  std::vector<KachelBlk> blk;
  std::vector<int> nblk;           // tiles per group
  std::vector<uint32_t> row, pos;  // per position its point (all ones: padding); per point its position
  std::vector<uint32_t> halo;
  std::vector<uint4> slice;        // as StepArgs::ka_slice
  size_t slabs = 0;
  std::vector<uint32_t> col;       // per slab lane, as StepArgs::col in slab form
  std::vector<uint16_t> lc;
  size_t slot(size_t i, uint32_t k) const {  // the lane of block (point i, rank k)
    const uint4 s = slice[pos[i] >> 5];
    return (size_t(k < s.y ? s.x + k : s.z + (k - s.y))) * 32 + (pos[i] & 31u);
  }
};
// Tiles for the groups of points [io[k], io[k + 1]) on at most nblk[k] CTAs
// each. False where a tile does not fit: more than kKachelZeilen rows a
// thread, local columns beyond 16 bits, or no room in `smem` bytes (`kopf` of
// them the header) for the least ring and the slabs that are left over beside
// it. On a B200's 148 CTAs a regular sheet (13 blocks a row) so fits up to some
// 227 k points with FP32 blocks, where the two slabs of a grip leave the odd one of
// every slice over, and beyond 266 k with FP64 blocks.
//
// A group of up to kKachelNatur points, and every instance of a batch, keeps
// the rows and sums of the launch over ELL rows (CTA b, thread t: the rows
// b * 512 + t + k * nblk * 512 of the group), so its results are that
// launch's bit for bit: small meshes' halos are small in any order. Where one
// row a thread suffices and the CTAs allow, kachel_warps of its warps share a
// CTA and each posts its own sum. Larger groups are cut into compact tiles by
// recursive bisection of the positions x (3 per point). With self-collision
// (`federn`) every group is, into tiles of 64 points at least: the springs'
// rows are spread over the CTAs' threads, and more CTAs take them in fewer turns
// (3 k points with 2.8 k rows: 22 k cycles an iteration on 16 CTAs, 16 k on 48).
constexpr size_t kKachelNatur = 16384;  // 512 warps, one posted word a thread
bool kachelplan(const Spalten& S, const double* x, const std::vector<int64_t>& io, const std::vector<int>& nblk,
                size_t rsize, bool federn, size_t smem, size_t kopf, Kachelplan& P);

}  // namespace k3d
