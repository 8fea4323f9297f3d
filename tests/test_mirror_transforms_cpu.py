"""When W is taken through the mirror-symmetric transforms (green-mbpt_b200/csrc/w_transforms.h, compiled as host code):
every synthetic grid qualifies, also with the round-off that another solution of its least-squares problem carries; a
grid without the symmetry does not, nor one whose asymmetry cancels in the composed transform."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from gb200 import grids

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HARNESS = r'''
#include <cstdio>
#include "w_transforms.h"
int main() {
  int dims[2];
  if (std::fread(dims, sizeof(int), 2, stdin) != 2) return 2;
  const int nts = dims[0], nw = dims[1];
  std::vector<std::complex<double>> F((size_t)nw * (nts / 2)), B((size_t)nts * nw);
  if (std::fread(F.data(), 16, F.size(), stdin) != F.size() || std::fread(B.data(), 16, B.size(), stdin) != B.size()) return 2;
  const gb200::MirrorTransforms m = gb200::mirror_transforms(F.data(), B.data(), nts, nw);
  std::printf("%d %d %.17g %.17g\n", (int)m.ok, m.nu, m.change, m.bound);
  if (!m.ok) return 0;
  for (auto* v : {&m.fwd, &m.half, &m.full})
    for (auto z : *v) std::printf("%.17g %.17g\n", z.real(), z.imag());
  return 0;
}
'''


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not installed")
    d = tmp_path_factory.mktemp("mirror")
    src, exe = d / "h.cpp", d / "h"
    src.write_text(HARNESS)
    r = subprocess.run([cxx, "-std=c++17", "-O2", "-Wall", "-Werror", "-I", os.path.join(ROOT, "green-mbpt_b200", "csrc"),
                        str(src), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return str(exe)


def fold(Tnt):
    nth = Tnt.shape[1] // 2
    return Tnt[:, :nth] + Tnt[:, ::-1][:, :nth]


def decide(harness, F, B):
    nts, nw = B.shape
    data = np.array([nts, nw], dtype=np.int32).tobytes() + np.ascontiguousarray(F, dtype=complex).tobytes() + \
        np.ascontiguousarray(B, dtype=complex).tobytes()
    r = subprocess.run([harness], input=data, capture_output=True)
    assert r.returncode == 0
    lines = r.stdout.decode().splitlines()
    ok, nu, change, bound = lines[0].split()
    z = np.array([[float(x) for x in ln.split()] for ln in lines[1:]]).reshape(-1, 2) @ np.array([1, 1j]) if int(ok) else None
    return bool(int(ok)), int(nu), float(change), float(bound), z


def chebyshev(beta, nts):
    return grids.ChebyshevGrid(beta, nts, nts, nts, candidates=max(512, (nts - 2) ** 2 // 8))


def apply(B, F, P):
    """W = B (1 - F P)^-1 F P"""
    x = np.tensordot(F, P, 1)
    return np.tensordot(B, np.linalg.solve(np.eye(P.shape[-1]) - x, x), 1)


@pytest.mark.parametrize("beta,nts", [(10.0, 14), (20.0, 24), (50.0, 34), (100.0, 60), (100.0, 80), (200.0, 118), (200.0, 120)])
def test_synthetic_grids_qualify_and_keep_W(harness, beta, nts):
    g = chebyshev(beta, nts)
    F, B = fold(g.Tnt_b), g.Ttn_b
    nth = nts // 2
    ok, nu, change, bound, z = decide(harness, F, B)
    assert ok and nu == (g.nw_b + 1) // 2  # Omega = 0 and the +-Omega pairs
    assert change < 2.0 ** -39 / 5  # well clear of the limit
    fwd, half, full = np.split(z, [nu * nth, 2 * nu * nth])
    fwd, half, full = fwd.reshape(nu, nth), half.reshape(nth, nu), full.reshape(nts, nu)
    # W of a polarization of pairs of levels, through the solve of each frequency, in both forms: the change stays within
    # the bound, and below what rounding P0 to the unit of five slices, 2^-39 of its largest element, does to W
    rng = np.random.default_rng(1)
    e, v = rng.uniform(0.02, 4.0, 100), rng.standard_normal((100, 12)) + 1j * rng.standard_normal((100, 12))
    tau = g.tau[:nth]
    P = -np.einsum("tp,pi,pj->tij", np.exp(-np.outer(tau, e)) + np.exp(-np.outer(beta - tau, e)), v, v.conj()) / 100
    W, Wm, Wf = apply(B, F, P), apply(half, fwd, P), apply(full, fwd, P)
    Wm = np.concatenate([Wm, Wm[::-1]])
    top = max(np.abs(Wm - W).max(), np.abs(Wf - W).max())
    assert top <= bound * nth * np.abs(B @ F).max() * np.abs(P).max()  # nth terms of at most the largest element each
    five = apply(B, F, P + 2.0 ** -39 * np.abs(P).max() * rng.uniform(-0.5, 0.5, P.shape))
    assert top <= np.abs(five - W).max()


@pytest.mark.parametrize("beta,nts", [(50.0, 34), (100.0, 80), (200.0, 118), (200.0, 120)])
def test_other_solvers_of_the_same_grid_decide_alike(harness, beta, nts):
    """The backward transform is a least-squares solution: solved another way (QR, SVD, frequencies in another order) its
    digits differ by more than its mirror asymmetry, and the decision must not."""
    g = chebyshev(beta, nts)
    F = fold(g.Tnt_b)
    L = nts - 2
    Mb = grids.chebyshev_fourier(g.wsample_b, L, beta)
    Q, R = np.linalg.qr(Mb)
    p = np.random.default_rng(2).permutation(len(Mb))
    inverses = [np.linalg.solve(R, Q.conj().T), np.linalg.pinv(Mb), np.linalg.pinv(Mb[p])[:, np.argsort(p)]]
    for inv in inverses:
        B = g.T_tau @ inv
        assert np.abs(B - g.Ttn_b).max() < 1e-9 * np.abs(B).max()
        ok, nu, change, _, _ = decide(harness, F, B)
        assert ok and nu == (g.nw_b + 1) // 2 and change < 2.0 ** -39 / 4


def test_grids_without_the_symmetry_do_not_qualify(harness):
    g = chebyshev(50.0, 34)
    F, B = fold(g.Tnt_b), g.Ttn_b.copy()
    B[20:] *= 1 + 1e-9  # a thousand times the unit of five slices
    assert not decide(harness, F, B)[0]
    B = g.Ttn_b.copy()
    B[3] += 1e-3 * np.abs(B).max()
    assert not decide(harness, F, B)[0]
    # an asymmetry of B that the folded forward transform cannot reach: the composed transform is symmetric, W is not
    null = np.linalg.svd(F)[0][:, -1].conj()  # F [35][17]: null @ F = 0
    assert np.abs(null @ F).max() < 1e-12
    B = g.Ttn_b.copy()
    B[2] += 1e-7 * null
    ok, _, change, bound, _ = decide(harness, F, B)
    assert not ok and (bound > 2.0 ** -30 or change > 2.0 ** -39)
    # frequencies that nearly coincide are not merged where that would show
    F2 = F.copy()
    F2[1] += 1e-10 * np.abs(F).max()
    ok, nu, _, _, _ = decide(harness, F2, g.Ttn_b)
    assert nu == 19 and not ok
    for bad in (np.nan, np.inf):
        B = g.Ttn_b.copy()
        B[5, 5] = bad
        assert not decide(harness, F, B)[0]
        F2 = F.copy()
        F2[4, 4] = bad
        assert not decide(harness, F2, g.Ttn_b)[0]


def test_sampled_ir_grid_does_not_qualify(harness):
    import _gw_golden
    g = _gw_golden.grid()
    ok, nu, change, _, _ = decide(harness, fold(g.Tnt_b), g.Ttn_b)
    assert not ok and nu == g.Ttn_b.shape[1] and change > 0.1
