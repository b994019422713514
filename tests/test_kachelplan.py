"""The tiles of the tiled PCG as the host plans them (kachelplan, run on the CPU):
every block in one lane of one slab, every column where its tile holds it, what is
streamed and what stays within the shared memory of a CTA; and the plans that are
refused, whose scenes take the launch over ELL rows."""
import os
import struct
import subprocess

import numpy as np
import pytest

from garmentcraft_b200 import synth
from garmentcraft_b200.implizit import build_scene

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "garmentcraft_b200", "csrc")
SMEM, KOPF = 232448, 9856  # a CTA's shared memory on the B200, the kernel's header

PROBE = r"""
#include <cstdio>
#include <cstdlib>
#include "k3d_plan.h"
using namespace k3d;
template <typename T> static std::vector<T> lies(size_t n) {
  std::vector<T> v(n);
  if (std::fread(v.data(), sizeof(T), n, stdin) != n) std::abort();
  return v;
}
template <typename T> static void gib(const std::vector<T>& v) {
  const uint64_t n = v.size();
  std::fwrite(&n, 8, 1, stdout);
  std::fwrite(v.data(), sizeof(T), v.size(), stdout);
}
int main() {
  const auto k = lies<int64_t>(9);  // points, membranes, hinges, groups, bytes a value, self-collision, smem, header, 0
  const size_t n = size_t(k[0]);
  const auto x = lies<double>(3 * n);
  const auto m = lies<uint32_t>(3 * size_t(k[1])), b = lies<uint32_t>(4 * size_t(k[2]));
  const auto io = lies<int64_t>(size_t(k[3]) + 1);
  const auto nb = lies<int32_t>(size_t(k[3]));
  auto liste = [&](const std::vector<uint32_t>& p, std::vector<uint32_t>& off, std::vector<uint32_t>& ent) {
    off.assign(n + 1, 0);
    for (uint32_t i : p) ++off[i + 1];
    for (size_t i = 0; i < n; ++i) off[i + 1] += off[i];
    ent.resize(p.size());
    auto f = off;
    for (size_t q = 0; q < p.size(); ++q) ent[f[p[q]]++] = uint32_t(q);
  };
  std::vector<uint32_t> ot, et, ob, eb, os(n + 1, 0);
  liste(m, ot, et);
  liste(b, ob, eb);
  Elemente E;
  E.n = n;
  E.m_p = m.data(), E.b_p = b.data();
  E.nt = size_t(k[1]), E.nb = size_t(k[2]);
  E.off_t = ot.data(), E.ent_t = et.data(), E.off_b = ob.data(), E.ent_b = eb.data(), E.off_s = os.data();
  Spalten S;
  spalten(E, S);
  Kachelplan P;
  const bool ok = kachelplan(S, x.data(), io, std::vector<int>(nb.begin(), nb.end()), size_t(k[4]), k[5] != 0,
                             size_t(k[6]), size_t(k[7]), P);
  gib(std::vector<int64_t>{ok, P.q, P.blocks, int64_t(P.slabs), kachel_griff(size_t(k[4]), P.q ? P.q : 1),
                           int64_t(ok ? kachel_ap(size_t(k[4]), P.q) : 0)});
  if (!ok) return 0;
  gib(S.anf), gib(S.sp), gib(P.row), gib(P.pos), gib(P.halo);
  std::vector<uint32_t> blk, sl;
  std::vector<int64_t> vorn;
  for (const KachelBlk& B : P.blk) {
    for (uint32_t q : {B.row0, B.rows, B.halo0, B.halos, B.platz, B.stufen, B.wort0, B.gruppe0, B.worte, B.einzeln})
      blk.push_back(q);
    vorn.push_back(int64_t(size_t(k[7]) + kachel_tile(size_t(k[4]), (B.rows + 31) / 32, B.halos,
                                                      kachel_ap(size_t(k[4]), P.q), k[5] != 0)));
  }
  for (const uint4& q : P.slice)
    for (uint32_t w : {q.x, q.y, q.z, q.w}) sl.push_back(w);
  gib(blk), gib(vorn), gib(sl), gib(P.col), gib(P.lc), gib(P.nblk);
  return 0;
}
"""


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    src, exe = d / "probe.cpp", d / "probe"
    src.write_text(PROBE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=address,undefined", "-include", "math.h", "-I", CSRC,
                    "-I/usr/local/cuda/include", str(src), os.path.join(CSRC, "k3d_plan.cpp"), "-o", str(exe)],
                   check=True)
    return str(exe)


def gitter(n):
    """A regular sheet's points, membranes and hinges without a scene build."""
    i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    x = np.stack([i.ravel() / n, j.ravel() / n, np.zeros(n * n)], axis=1)
    a = (i[:-1, :-1] * n + j[:-1, :-1]).ravel()
    m = np.concatenate([np.stack([a, a + n, a + n + 1], 1), np.stack([a, a + n + 1, a + 1], 1)])
    h = [np.stack([a, a + n + 1, a + n, a + 1], 1)]
    b = (i[:-2, 1:-1] * n + j[:-2, 1:-1]).ravel()
    h.append(np.stack([b + n, b + n + 1, b, b + 2 * n + 1], 1) if len(b) else np.zeros((0, 4), int))
    c = (i[1:-1, :-2] * n + j[1:-1, :-2]).ravel()
    h.append(np.stack([c + 1, c + n + 1, c, c + n + 2], 1) if len(c) else np.zeros((0, 4), int))
    return x, m.astype(np.uint32), np.concatenate(h).astype(np.uint32)


def plan(probe, x, m, b, io, nblk, rsize, federn=False, smem=SMEM):
    kopf = struct.pack("9q", len(x), len(m), len(b), len(nblk), rsize, int(federn), smem, KOPF, 0)
    ein = kopf + np.ascontiguousarray(x, dtype=np.float64).tobytes() + m.tobytes() + b.tobytes() + np.asarray(
        io, dtype=np.int64).tobytes() + np.asarray(nblk, dtype=np.int32).tobytes()
    r = subprocess.run([probe], input=ein, capture_output=True)
    assert r.returncode == 0, r.stderr.decode()
    aus, p = [], 0

    def nimm(dt):
        nonlocal p
        k = struct.unpack_from("Q", r.stdout, p)[0]
        a = np.frombuffer(r.stdout, dtype=dt, count=k, offset=p + 8)
        p += 8 + a.nbytes
        return a
    ok, q, blocks, slabs, griff, ap = nimm(np.int64)
    if not ok:
        return None
    P = dict(q=int(q), blocks=int(blocks), slabs=int(slabs), griff=int(griff))
    for k, dt in (("anf", np.uint32), ("sp", np.uint32), ("row", np.uint32), ("pos", np.uint32), ("halo", np.uint32),
                  ("blk", np.uint32), ("vorn", np.int64), ("slice", np.uint32), ("col", np.uint32), ("lc", np.uint16),
                  ("nblk", np.int32)):
        P[k] = nimm(dt)
    P["blk"], P["slice"] = P["blk"].reshape(-1, 10).astype(np.int64), P["slice"].reshape(-1, 4).astype(np.int64)
    return P


def pruefe(P, n, rsize, smem=SMEM):
    satz = 288 * rsize + 64
    row, sl = P["row"], P["slice"]
    echt = row != 0xffffffff
    pt = row & np.uint32(0x7fffffff)
    assert np.array_equal(np.sort(pt[echt]), np.arange(n))  # every point in one position
    assert np.array_equal(P["pos"][pt[echt]], np.flatnonzero(echt))
    im_halo = np.zeros(n, dtype=bool)
    im_halo[P["halo"]] = True
    assert np.array_equal((row[echt] >> 31) == 1, im_halo[pt[echt]])
    breit = np.diff(P["anf"].astype(np.int64))
    belegt = np.zeros(P["slabs"], dtype=int)
    worte = 0
    for B, vorn in zip(P["blk"], P["vorn"]):
        row0, rows, halo0, halos, platz, stufen, wort0, gruppe0, anzahl, einzeln = (int(v) for v in B)
        ns = (rows + 31) // 32
        assert row0 % 32 == 0 and 0 < ns <= 16 * P["q"] and (P["q"] == 1 or P["blk"][:, 1].max() > 512 * (P["q"] - 1))
        nw = min(ns, 16)
        assert vorn + nw * platz * satz <= smem
        assert wort0 == worte and gruppe0 <= wort0 < gruppe0 + anzahl
        worte += ns if einzeln else 1
        tile = np.concatenate([pt[row0:row0 + 32 * ns], P["halo"][halo0:halo0 + halos]])
        eigen = set(pt[row0:row0 + rows].tolist())
        assert not eigen & set(P["halo"][halo0:halo0 + halos].tolist())
        for w in range(nw):
            s = [row0 // 32 + k for k in range(w, ns, 16)]
            y, f = sl[s, 1], sl[s, 3]
            assert (y % P["griff"] == 0).all()
            # a warp's streamed slabs lie one after another, and its resident ones
            assert (sl[s, 0] == sl[s[0], 0] + np.concatenate([[0], np.cumsum(y)[:-1]])).all()
            assert (sl[s, 2] == sl[s[0], 2] + np.concatenate([[0], np.cumsum(f)[:-1]])).all()
            if y.sum():
                assert stufen >= 2 and stufen * P["griff"] + f.sum() <= platz and stufen <= 4
            else:
                assert f.sum() <= platz
            for k in s:
                r = np.arange(32 * k, min(32 * k + 32, row0 + rows))
                i = pt[r].astype(np.int64)
                assert sl[k, 1] + sl[k, 3] == breit[i].max()
                for rang in range(int(sl[k, 1] + sl[k, 3])):
                    slab = int(sl[k, 0] + rang if rang < sl[k, 1] else sl[k, 2] + rang - sl[k, 1])
                    belegt[slab] += 1
                    da = rang < breit[i]
                    lane = slab * 32 + (r - 32 * k)
                    j = P["sp"][P["anf"][i[da]] + np.uint32(rang)]
                    c = P["col"][lane]
                    assert (c[~da] == 0xffffffff).all() and np.array_equal(c[da] & np.uint32(0x7fffffff), j)
                    assert np.array_equal((c[da] >> 31) == 1, j == i[da])
                    assert np.array_equal(tile[P["lc"][lane[da]]], j)  # the tile holds the column there
                    assert (P["lc"][slab * 32:slab * 32 + 32] < len(tile)).all()
    assert (belegt == 1).all()


def io1(n):
    return [0, n * n]


# (side, CTAs, bytes a value, self-collision, rows a thread, streamed): below a slice, one ragged
# slice, the last natural and the first compact size, rings, two to four rows a thread, one CTA
@pytest.mark.parametrize("n, nb, rsize, federn, q, strom", [
    (2, 148, 8, False, 1, False), (5, 148, 4, False, 1, False), (33, 148, 8, False, 1, False),
    (128, 148, 8, False, 1, False), (129, 148, 8, False, 1, False), (129, 148, 4, False, 1, False),
    (190, 148, 8, False, 1, True), (257, 148, 4, False, 1, True), (300, 148, 8, False, 2, True),
    (300, 148, 4, False, 2, True), (400, 148, 8, False, 3, True), (400, 148, 4, False, 3, True),
    (41, 1, 8, False, 4, True), (41, 2, 4, False, 2, True), (41, 7, 8, False, 1, True),
    (30, 48, 8, True, 1, False), (56, 148, 4, True, 1, False), (453, 148, 4, True, 3, True)])
def test_plan(probe, n, nb, rsize, federn, q, strom):
    x, m, b = gitter(n)
    P = plan(probe, x, m, b, io1(n), [nb], rsize, federn)
    assert P is not None and P["q"] == q and P["blocks"] <= nb
    assert (P["slice"][:, 1].sum() > 0) == strom
    pruefe(P, n * n, rsize)


@pytest.mark.parametrize("rsize", [4, 8])
def test_stapel(probe, rsize):
    teile, io = [gitter(k) for k in (3, 9, 40, 95, 17)], [0]
    x = np.concatenate([t[0] for t in teile])
    for t in teile:
        io.append(io[-1] + len(t[0]))
    m = np.concatenate([t[1] + np.uint32(o) for t, o in zip(teile, io)])
    b = np.concatenate([t[2] + np.uint32(o) for t, o in zip(teile, io)])
    P = plan(probe, x, m, b, io, [1, 1, 12, 130, 4], rsize)
    assert P is not None
    pruefe(P, len(x), rsize)
    for k in range(5):  # no tile crosses two instances
        for B in P["blk"][int(P["nblk"][:k].sum()):int(P["nblk"][:k + 1].sum())]:
            p = P["row"][B[0]:B[0] + B[1]] & np.uint32(0x7fffffff)
            assert (p >= io[k]).all() and (p < io[k + 1]).all()


def test_zwei_lagen(probe):
    # the scene builder's own element order, two pieces
    s = build_scene(synth.zwei_lagen(groesse_m=0.2, kante_mm=5.0))
    m, b = np.ascontiguousarray(s.membran_punkte, np.uint32), np.ascontiguousarray(s.biegung_punkte, np.uint32)
    P = plan(probe, s.x, m, b, [0, s.n], [148], 8, True)
    assert P is not None
    pruefe(P, s.n, 8)


# FP32 blocks end near 227 k points of a regular sheet: a two-slab grip leaves the
# odd slab of each slice of 13 over, which has to stay, beside two stages
@pytest.mark.parametrize("n, nb, rsize, passt", [
    (475, 148, 4, True), (480, 148, 4, False), (516, 148, 8, True), (41, 1, 4, False), (300, 3, 8, False)])
def test_grenze(probe, n, nb, rsize, passt):
    x, m, b = gitter(n)
    P = plan(probe, x, m, b, io1(n), [nb], rsize)
    assert (P is not None) == passt
    assert plan(probe, x, m, b, io1(n), [nb], rsize, smem=KOPF) is None  # no room at all
