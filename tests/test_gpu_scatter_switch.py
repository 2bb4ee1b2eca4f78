"""HFGPU_SCATTER and HFGPU_WARP_SCATTER choose the staged scatter: the kernels
that run are the ones asked for.

`single` is one thread per quartet, `grouped` the lanes of a warp per quartet,
for FP64 lists and for FP32 ones (a cutoff above every bound).  That the two
forms give the same F is tests/test_gpu_parity.py's
test_grouped_and_single_thread_scatter_agree."""
import numpy as np
import pytest

from helpers import perturbed_density, system


def scatter_kernels(sh, p0, p, cutoff):
    from torch.profiler import ProfilerActivity, profile
    from hfcode_b200.fock import FockBuilder
    n = sh.nb
    fb = FockBuilder(sh)
    fb.fock_build_initial_diag(np.zeros((n, n)), p0, 1e-10)
    with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as prof:
        fb.fock_build_non_diag_mixed(np.zeros((n, n)), p, 1e-10, cutoff)
    fb.close()
    names = {e.key for e in prof.key_averages()}
    return {f for f in ("k_scatter_staged", "k_scatter_warp") if any(f in k for k in names)}, names


@pytest.mark.gpu
@pytest.mark.parametrize("cutoff,real", [(0.0, "double"), (1e3, "float")])
@pytest.mark.parametrize("env,want", [
    ({"HFGPU_SCATTER": "single"}, "k_scatter_staged"),
    ({"HFGPU_SCATTER": "grouped"}, "k_scatter_warp"),
    ({"HFGPU_WARP_SCATTER": "0"}, "k_scatter_staged"),
    ({"HFGPU_WARP_SCATTER": "100000000"}, "k_scatter_warp"),
    ({"HFGPU_SCATTER": "grouped", "HFGPU_WARP_SCATTER": "0"}, "k_scatter_staged"),
])
def test_switch_chooses_the_scatter(monkeypatch, env, want, cutoff, real):
    for k in ("HFGPU_SCATTER", "HFGPU_WARP_SCATTER"):
        monkeypatch.delenv(k, raising=False)
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    _, _, sh, p0 = system("alkane2_mix")
    forms, names = scatter_kernels(sh, p0, perturbed_density(p0, 10), cutoff)
    assert forms == {want}, env
    assert all(real + ">" in k for k in names if want in k)
