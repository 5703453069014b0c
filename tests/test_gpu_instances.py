"""Which compiled instance of the fused forward kernels a call runs, and its values.

Grids too small to fill the chip share each column's g-points between CTAs (the split kernels); the
tests with a few dozen columns run those.  Here grids wide enough to run unsplit cover the
instances that larger calls use: chunk counts up to 8, 10, 12 and 16, sparse and dense tables,
with and without aerosols.  Instance, grid and block are read from the
profiler (<chunk length, dense, threads, CTAs per SM>); a column sample is compared with the FP64 oracle at
the fused kernels' bounds (5e-3 W/m2, 0.01 K/day)."""
import json
import re
import tempfile
import time

import numpy as np
import pytest

from rrtmgp_b200 import synthetic as S

from test_gpu_scale import _take

pytestmark = pytest.mark.gpu
HR_TOL = 0.01
FLUX_TOL = 5e-3


@pytest.fixture(scope="module")
def solvers():
    """(Fused_solver, tables, gases) by dense."""
    from rrtmgp_b200.solver import Fused_solver, Radiation_solver
    out = {}
    for dense in (False, True):
        t = {"lw": S.make_kdist("lw", dense=dense), "sw": S.make_kdist("sw", dense=dense),
             "cloud_lw": S.make_cloud_luts("lw"), "cloud_sw": S.make_cloud_luts("sw"), "aer": S.make_aerosol_luts()}
        gases = S.ATM_GASES_DENSE if dense else S.ATM_GASES
        base = Radiation_solver(t["lw"], t["sw"], t["cloud_lw"], t["cloud_sw"], gases, aerosol_sw=t["aer"],
                                delta_aerosol=True)
        out[dense] = Fused_solver(base), t, gases
    return out


def _grid(gpu, ncol, nlay, dense, aerosols, seed):
    import torch
    from rrtmgp_b200.solver import atm_to_device
    atm = S.make_atmosphere(ncol, nlay, seed=seed, clouds=True, trace_gases=dense)
    rng = np.random.default_rng(seed)
    atm["sfc_alb_dif"] = rng.uniform(0.02, 0.9, atm["sfc_alb_dif"].shape)
    d = atm_to_device(atm, torch.float32, gpu)
    if aerosols:
        atm["aerosols"], atm["rh"] = S.make_aerosols(atm["play"], seed=seed + 1)
        d["aerosols"] = {k: torch.as_tensor(v, dtype=torch.float32, device=gpu) for k, v in atm["aerosols"].items()}
        d["rh"] = torch.as_tensor(atm["rh"], dtype=torch.float32, device=gpu)
    return atm, d


def launches(call, count):
    """[(kernel, CTAs, threads per CTA)] of the `count` fused and per-stage kernels that call launches, as
    ("lw_forward_kernel<8, false, 256, 3>", 592, 256).  The profiler drops kernels that its clock places
    outside its window, so call is kept away from both ends of it, and repeated where one is
    missing all the same."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    for _ in range(5):
        with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
            torch.zeros(1, device="cuda")
            torch.cuda.synchronize()
            time.sleep(0.05)
            call()
            torch.cuda.synchronize()
            time.sleep(0.05)
            torch.zeros(1, device="cuda")
            torch.cuda.synchronize()
        with tempfile.TemporaryDirectory() as d:
            p.export_chrome_trace(d + "/trace.json")
            with open(d + "/trace.json") as f:
                events = json.load(f)["traceEvents"]
        found = [(re.search(r"([ls]w_(forward|adjoint|solver)\w*(<[^>]*>)?)", e["name"]), e) for e in events
                 if e.get("cat") == "kernel"]
        found = [(m.group(1), e["args"]["grid"][0], e["args"]["block"][0], e["ts"]) for m, e in found if m]
        if len(found) == count:
            break
    assert len(found) == count, found
    return [f[:3] for f in sorted(found, key=lambda f: f[3])]


def _check(got, ref, cols, what):
    for k in ref:
        if k in got:
            e = float(np.max(np.abs(got[k][:, cols].double().cpu().numpy() - ref[k])))
            assert e < (HR_TOL if k == "heating_rate" else FLUX_TOL), f"{what} {k}: {e:.3e}"


def test_split_leaves_no_second_wave_of_clusters(solvers, gpu):
    """147 x 40 in the shortwave: CTAs of five warps, three per SM, 444 places for 441 CTAs in clusters of three --
    but clusters do not cross GPCs, so some would wait for a second wave.  Clusters of two fit."""
    fused, _, _ = solvers[False]
    _, d = _grid(gpu, 147, 40, False, False, 5)
    fused.solve_sw(d)
    (name, ctas, threads), = launches(lambda: fused.solve_sw(d), 1)
    assert name.startswith("sw_forward_split_kernel<8, false") and (ctas, threads) == (2 * 147, 160)


@pytest.mark.parametrize("ncol,nlay,dense,aerosols,lw,sw", [
    # two or three capped CTAs share an SM
    (880, 60, False, False, "8, D, 256, 3", "8, D, 512, 1"),
    (880, 72, False, False, "8, D, 320, 2", "8, D, 320, 2"),
    (880, 96, False, True, "8, D, 384, 2", "8, D, 384, 2"),
    (880, 128, False, False, "16, D, 512, 1", "8, D, 512, 2"),
    (880, 64, True, True, "8, D, 256, 3", "8, D, 512, 1"),
    (880, 80, True, False, "8, D, 320, 2", "8, D, 320, 2"),
    (880, 96, True, True, "8, D, 384, 2", "8, D, 384, 2"),
    (880, 104, True, False, "16, D, 512, 1", "8, D, 512, 2"),
    # two shortwave CTAs do not fit, or leave the L1 too little: no cap
    (880, 104, False, True, "16, D, 512, 1", "8, D, 512, 1"),
    (880, 128, False, True, "16, D, 512, 1", "8, D, 512, 1"),
    (880, 128, True, False, "16, D, 512, 1", "8, D, 512, 1"),
    (880, 104, True, True, "16, D, 512, 1", "8, D, 512, 1"),
    # longwave chunk length by waves: two of 8 layers against one of 16, three against two
    (400, 72, False, False, "16, D, 512, 1", "8, D, 320, 2"),
    (520, 60, True, False, "16, D, 512, 1", "8, D, 512, 1"),
    (400, 112, False, False, "8, D, 512, 1", "8, D, 512, 2"),
    # one CTA per SM at most: no cap
    (140, 72, False, False, "8, D, 512, 1", "8, D, 512, 1"),
    (140, 96, True, True, "8, D, 512, 1", "8, D, 512, 1")])
def test_forward_instance_and_values(oracle_mod, solvers, gpu, ncol, nlay, dense, aerosols, lw, sw):
    fused, t, gases = solvers[dense]
    atm, d = _grid(gpu, ncol, nlay, dense, aerosols, 300 + nlay)
    out = {}

    def call():
        out["lw"] = fused.solve_lw(d)
        out["sw"] = fused.solve_sw(d, with_aerosols=aerosols)

    b = "true" if dense else "false"
    assert [n for n, _, _ in launches(call, 2)] == ["lw_forward_kernel<" + lw.replace("D", b) + ">",
                                                  "sw_forward_kernel<" + sw.replace("D", b) + ">"]
    cols = np.arange(0, ncol, max(1, ncol // 24))
    few = _take(atm, cols)
    extra = {}
    if aerosols:
        few["aerosols"] = {k: v[:, cols] for k, v in atm["aerosols"].items()}
        few["rh"] = atm["rh"][:, cols]
        extra = {"aerosol_tables": t["aer"], "delta_aerosol": True}
    _check(out["lw"], oracle_mod.forward_lw(oracle_mod.GasOptics(t["lw"], gases), oracle_mod.CloudOptics(t["cloud_lw"]),
                                            few), cols, "lw")
    _check(out["sw"], oracle_mod.forward_sw(oracle_mod.GasOptics(t["sw"], gases), oracle_mod.CloudOptics(t["cloud_sw"]),
                                            few, **extra), cols, "sw")


@pytest.mark.parametrize("nlay", [8, 47, 49, 56, 64, 65, 80, 81, 88, 96])
def test_fp64_longwave_solver_chunks(oracle_mod, solvers, gpu, nlay):
    """One angle in FP64: chunks of 8 layers where their blocks nearly fill the 20 warps of an SM (3 - 6, 9
    or 10 chunks), else of 16; each at the edges of its range against the oracle."""
    import torch
    from rrtmgp_b200 import api
    _, t, gases = solvers[False]
    atm = S.make_atmosphere(37, nlay, seed=40 + nlay, clouds=False)
    go = oracle_mod.GasOptics(t["lw"], gases).gas_optics_lw(atm["play"], atm["plev"], atm["tlay"], atm["tsfc"], atm["gases"],
                                                            atm["tlev"])
    emis = np.random.default_rng(5).uniform(0.8, 1.0, (37, 16))
    up, dn = oracle_mod.rte_lw(t["lw"]["bnd_limits_gpt"], go["tau"], True, go, emis)
    kd = api.Gas_optics_rrtmgp(t["lw"], gases)
    src = {k: torch.as_tensor(v, dtype=torch.float64, device=gpu).contiguous() for k, v in go.items()}
    e = torch.as_tensor(emis, device=gpu)
    out = {}
    (name, _, threads), = launches(lambda: out.update(f=api.Rte_lw.rte_lw(kd.bands, src["tau"], True, src, e)), 1)
    chunks = -(-nlay // 8)
    cl = 8 if chunks <= 6 or chunks in (9, 10) else 16
    assert name.startswith(f"lw_solver_chunked<double, {cl}, ") and threads == 32 * -(-nlay // cl)
    for got, ref in zip(out["f"], (up, dn)):
        np.testing.assert_allclose(got.cpu().numpy(), ref, rtol=1e-10, atol=1e-10 * np.abs(ref).max())
