"""Which compiled instance of the kernels a call runs, in which launch, and its values.

Grids too small to fill the chip share each column's g-points between CTAs (the split kernels); the
tests with a few dozen columns run those.  Kernel, grid and block are read from the profiler."""
import json
import re
import tempfile

import numpy as np
import pytest

from rrtmgp_b200 import synthetic as S

pytestmark = pytest.mark.gpu


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


def launches(call):
    """[(kernel, CTAs, threads per CTA)] of the fused and the per-stage kernels that call launches, as
    ("lw_forward_kernel<8, false, 256, 3>", 592, 256)."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    with tempfile.TemporaryDirectory() as d:
        p.export_chrome_trace(d + "/trace.json")
        with open(d + "/trace.json") as f:
            events = json.load(f)["traceEvents"]
    found = [(re.search(r"([ls]w_(forward|adjoint|solver)\w*(<[^>]*>)?)", e["name"]), e) for e in events
             if e.get("cat") == "kernel"]
    return [(m.group(1), e["args"]["grid"][0], e["args"]["block"][0]) for m, e in found if m]


def test_split_leaves_no_second_wave_of_clusters(solvers, gpu):
    """147 x 40 in the shortwave: CTAs of five warps, three per SM, 444 places for 441 CTAs in clusters of three --
    but clusters do not cross GPCs, so some would wait for a second wave.  Clusters of two fit."""
    fused, _, _ = solvers[False]
    _, d = _grid(gpu, 147, 40, False, False, 5)
    fused.solve_sw(d)
    (name, ctas, threads), = launches(lambda: fused.solve_sw(d))
    assert name.startswith("sw_forward_split_kernel<8, false") and (ctas, threads) == (2 * 147, 160)
