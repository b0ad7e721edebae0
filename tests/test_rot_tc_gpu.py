"""The tcgen05 tensor-core rotation (three bf16 parts per value) against an FP64 reference product
and against the cuBLAS FP32 rotation, alone and inside apply_noise.  GPU only.

Tolerance: the split keeps FP32-level accuracy; max |R - R64| / max |R64| <= 5e-6.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
cuda = torch.device("cuda", 0)


@pytest.fixture(scope="module")
def K():
    from minkasi_gb300 import kernels
    return kernels


def rel(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.abs(a - b).max() / np.abs(b).max())


@pytest.mark.parametrize("ndet", [32, 64, 128, 256])
@pytest.mark.parametrize("ncol", [128, 1000, 4097])
def test_tc_rotation_matches_fp64(K, ndet, ncol):
    rng = np.random.default_rng(ndet * 7 + ncol)
    A = rng.standard_normal((ndet, ndet)).astype(np.float32)
    X = rng.standard_normal((ndet, ncol)).astype(np.float32)
    ref = A.astype(np.float64) @ X.astype(np.float64)
    plan = K.NoisePlan(ndet, ncol, torch.float32)
    At, Xt = torch.from_numpy(A).to(cuda), torch.from_numpy(X).to(cuda)
    R2 = plan.rotate(At, Xt, rot_mode=2).cpu().numpy()
    assert plan.status() == 0
    R1 = plan.rotate(At, Xt, rot_mode=1).cpu().numpy()
    assert rel(R1, ref) < 5e-6
    assert rel(R2, ref) < 5e-6


@pytest.mark.parametrize("ndet", [32, 64, 128, 256])
@pytest.mark.parametrize("ncol", [2, 127, 129, 255, 257, 40_001])
def test_tc_rotation_tile_edges_and_nonfinite(K, ndet, ncol):
    """Around the tiles of 128 samples and the items of two tiles, more items
    than CTAs, entries over the FP32 range, and NaN / infinity in one sample
    each (all of its outputs become NaN, every other sample stays).  Bound per
    sample: each output is accumulated in 6 ndet / 16 <= 96 steps, each off by
    at most 2^-23 of a partial sum (taken as at most twice the largest
    output): 2.3e-5."""
    rng = np.random.default_rng(ndet + ncol)
    A = rng.standard_normal((ndet, ndet)).astype(np.float32)
    X = (rng.standard_normal((ndet, ncol)) * 10.0 ** rng.integers(-20, 20, size=ncol)[None, :]).astype(np.float32)
    ref = A.astype(np.float64) @ X.astype(np.float64)
    plan = K.NoisePlan(ndet, ncol, torch.float32)
    At = torch.from_numpy(A).to(cuda)
    R = plan.rotate(At, torch.from_numpy(X).to(cuda), rot_mode=2).cpu().numpy()
    assert (np.abs(R - ref).max(0) <= 2.3e-5 * np.abs(ref).max(0)).all()
    X[ndet // 3, 0], X[ndet // 2, ncol - 1] = np.nan, np.inf
    R2 = plan.rotate(At, torch.from_numpy(X).to(cuda), rot_mode=2).cpu().numpy()
    assert np.isnan(R2[:, 0]).all() and np.isnan(R2[:, ncol - 1]).all()
    assert np.array_equal(R2[:, 1:ncol - 1], R[:, 1:ncol - 1])
    assert plan.status() == 0


@pytest.mark.parametrize("ncol", [19_456, 19_457, 19_584, 19_585])
def test_tc_rotation_around_one_tile_per_sm(K, ncol):
    """256 detectors: 152 tiles of 128 samples (one tile per item on 152 SMs), a
    ragged 153rd, 153 and a ragged 154th (two tiles per item, the last one half
    empty or ragged), at the bound of test_tc_rotation_tile_edges_and_nonfinite."""
    rng = np.random.default_rng(ncol)
    A = rng.standard_normal((256, 256)).astype(np.float32)
    X = rng.standard_normal((256, ncol)).astype(np.float32)
    ref = A.astype(np.float64) @ X.astype(np.float64)
    plan = K.NoisePlan(256, ncol, torch.float32)
    R = plan.rotate(torch.from_numpy(A).to(cuda), torch.from_numpy(X).to(cuda), rot_mode=2).cpu().numpy()
    assert (np.abs(R - ref).max(0) <= 2.3e-5 * np.abs(ref).max(0)).all()
    assert plan.status() == 0


def test_noise_group_of_more_tiles_than_its_tods(K):
    """Three 256-detector TODs of one tile per item each, two as a group: as
    each TOD's own filter gives, bit for bit."""
    g = torch.Generator(device="cuda").manual_seed(4)
    r = lambda *s: torch.randn(s, generator=g, device=cuda)
    ns = [9001, 300, 12_001]
    plans = [K.NoisePlan(256, n, torch.float32) for n in ns]
    ops = [(r(256, 256), r(256, 256), r(256, n).abs()) for n in ns]
    data = [r(256, n) for n in ns]
    want = [p.apply(*o, d, rot_mode=2) for p, o, d in zip(plans, ops, data)]
    grp = K.NoiseGroup(plans, ops, data)
    grp.apply()
    assert grp.status() == 0
    assert all(torch.equal(a, b) for a, b in zip(data, want))


def test_tc_apply_noise_matches_golden(K, gold):
    g = gold("noise.npz")
    x = g["x"]
    # pad the 10-detector fixture into a 32-detector block (identity elsewhere)
    nd = 32
    v = np.eye(nd)
    vT = np.eye(nd)
    w = np.zeros((nd, x.shape[1]))
    xx = np.zeros((nd, x.shape[1]))
    v[:10, :10], vT[:10, :10], w[:10], xx[:10] = g["v"], g["vT"], g["mywt"], x
    plan = K.NoisePlan(nd, x.shape[1], torch.float32)
    f = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).to(cuda)
    dd = plan.apply(f(v), f(vT), f(w), f(xx), rot_mode=2).cpu().numpy()
    assert plan.status() == 0
    assert rel(dd[:10], g["dd"]) < 2e-5


@pytest.mark.parametrize("dct", ["0", "1"])
def test_noise_group_equals_per_tod_filter(monkeypatch, dct):
    """The one-call filter over all TODs (rotations of all TODs with one
    detector count in one tensor-core launch, in place) gives bit for bit
    what the per-TOD apply_noise gives, on TODs of 32 and 64 detectors with
    untruncated lengths (so some run Bluestein's algorithm), with the
    four-step FFT and with cuFFT plans."""
    from dataclasses import replace
    from minkasi_gb300 import synth
    from minkasi_gb300.engine import MapmakingOperator
    monkeypatch.setenv("MINKASI_GB300_DCT", dct)
    cfg = replace(synth.CONFIGS["tiny"], ntod=5, ndet_choices=(32, 64), nsamp_range=(3000, 9000),
                  truncate=False)
    tv, m = synth.make_todvec(cfg)
    op = MapmakingOperator(tv, m, torch.float32, tod2map="atomic", rot_mode=2)
    if dct == "0":
        assert set(op.dct_engines.values()) <= {0, 2} and 2 in op.dct_engines.values()
    else:
        assert set(op.dct_engines.values()) == {1}
    grp = op._noise_group()
    assert grp is not None
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(op.tmp.shape, generator=g, dtype=torch.float32, device="cuda")
    op.tmp.copy_(x)
    op.noise_all()
    grouped = op.tmp.clone()
    assert grp.status() == 0
    op.tmp.copy_(x)
    for (v, vT, w), view, dims in zip(op.ops, op.views(op.tmp), op.dims):
        op.plans[dims].apply(v, vT, w, view, out=view, rot_mode=2)
    assert torch.equal(grouped, op.tmp)


def test_rotations_that_time_out_are_nan(K, tmp_path):
    """The rotations built with a limit of no tries on every wait between their
    roles, so that each block stops at its first one: the error word is set and
    every output is NaN (FP64 in slices; FP32 with the mirrored extension, one
    tile and two per item); nothing is left in flight: the library's own
    kernels run on afterwards."""
    import ctypes
    import os
    import subprocess
    from minkasi_gb300 import build
    objs = []
    for f in ("mk_ozaki", "mk_rot_tc", "mk_common"):
        objs.append((f, subprocess.Popen(
            [build._nvcc(), "-O1", "-std=c++17", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", *build.ARCH,
             "-DMK_ROLE_SPIN_LIMIT=0", "-c", os.path.join(build.CSRC, f + ".cu"), "-o", f + ".o"], cwd=tmp_path)))
    assert all(p.wait() == 0 for _, p in objs)
    subprocess.run([build._nvcc(), "-shared", *build.ARCH, "-o", "quick.so", *[f + ".o" for f, _ in objs]],
                   cwd=tmp_path, check=True)
    h = ctypes.CDLL(str(tmp_path / "quick.so"))
    g = torch.Generator(device="cuda").manual_seed(1)
    vp, i64 = ctypes.c_void_p, ctypes.c_int64
    ws = torch.empty(128 << 20, dtype=torch.uint8, device=cuda)
    rot64 = h._ZN2mk16ozaki_rotate_f64EPKdS1_lPdlllPvmPiP11CUstream_st
    rot64.argtypes = [vp, vp, i64, vp, i64, i64, i64, vp, ctypes.c_size_t, vp, vp]
    rot32 = h._ZN2mk10rot_tc_f32EPKfS1_lPflllPvPiP11CUstream_stlli
    rot32.argtypes = [vp, vp, i64, vp, i64, i64, i64, vp, vp, vp, i64, i64, ctypes.c_int]
    # 40: two detector blocks; 3001: a ragged last tile; 256 x 20,001: two tiles per item
    for nd, n, dt in ((40, 3001, torch.float64), (64, 3001, torch.float32), (256, 20_001, torch.float32)):
        err = torch.zeros(1, dtype=torch.int32, device=cuda)
        A, X = (torch.randn(s, generator=g, dtype=dt, device=cuda) for s in ((nd, nd), (nd, n)))
        N = n if dt == torch.float64 else 2 * (n - 1)
        R = torch.zeros((nd, N), dtype=dt, device=cuda)
        args = [A.data_ptr(), X.data_ptr(), n, R.data_ptr(), N, nd, n, ws.data_ptr()]
        if dt == torch.float64:
            assert rot64(*args, ws.numel(), err.data_ptr(), K._stream()) == 0
        else:
            assert rot32(*args, err.data_ptr(), K._stream(), N, 1, 0) == 0
        assert err.item() == 1 and R.isnan().all()
        plan = K.NoisePlan(nd, n, dt)
        assert plan.rotate(A, X, rot_mode=4 if dt == torch.float64 else 2).isfinite().all() and plan.status() == 0


def test_solvers_raise_on_a_reported_timeout(K, monkeypatch):
    """run_pcg, run_pcg_mixed (both modes) and the generic solver end with an
    error where a plan's or the group's status word says that a wait timed out."""
    import minkasi_gb300 as mk
    from minkasi_gb300 import synth
    monkeypatch.setenv("MINKASI_GB300_TOD2MAP", "atomic")
    tv, m = synth.make_todvec(synth.CONFIGS["tiny"])
    tv.rot_mode = 4
    b = mk.Mapset()
    b.add_map(m)
    tv.make_rhs(b, do_clear=True)
    x0 = b.copy()
    x0.clear()
    solve = [lambda: mk.run_pcg(b, x0, tv, maxiter=2, verbose=False),
             lambda: mk.run_pcg_mixed(b, x0, tv, max_iter=2, replace_every=2),
             lambda: mk.run_pcg_mixed(b, x0, tv, max_iter=2, mode="refine", max_outer=1),
             lambda: mk.run_pcg(b, x0, tv, mask=None, maxiter=1, verbose=False, precon=mk.null_precon())]
    tv.engine(m, torch.float32).rot_mode = 2  # (where the group or the plans would report)
    tv.engine(m, torch.float32)._group = False
    monkeypatch.setattr(K.NoisePlan, "apply", _cublas_apply(K))
    for f in solve[:3]:
        f()
    monkeypatch.setattr(K.NoisePlan, "status", lambda self: 1)
    for f in solve:
        with pytest.raises(RuntimeError, match="timed-out"):
            f()


def _cublas_apply(K):
    apply = K.NoisePlan.apply

    def run(self, *a, rot_mode=0, **k):
        return apply(self, *a, rot_mode=1, **k)
    return run
