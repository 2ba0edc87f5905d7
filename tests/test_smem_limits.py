"""A kernel's limit of dynamic shared memory belongs to the process, not to an
engine: an engine with a smaller neighbour list must not take it away from an
engine with a larger one."""
import numpy as np
import pytest

from host_engine import host, host_library  # noqa: F401


def _engine(form, cap):
    from komd_gb300 import gpu, lattice
    s = lattice.argon_fcc(6, rho=0.8442, t_star=0.722, seed=3, jitter=0.05)
    cell = float(s.high[0]) / 3.0
    full = dict(atm_sign=gpu.ATM_SIGN_PHYSICAL, atm_enum=gpu.ATM_ENUM_FULL, virial_mode=gpu.VIRIAL_CORRECT)
    kw = {"fp64": dict(precision=gpu.FP64), "fp32_compat": {}, "fp32_full": full,
          "verlet": dict(skin=0.3, **full)}[form]   # caps past the half-list pass: k_lj_atm
    g = gpu.GpuSystem(s, gpu.make_config(s.low, s.high, cell, cutoff=2.5, cutoff_3b=2.0, nu=0.073, atm_list_cap=cap,
                                         terms=gpu.TERM_LJ | gpu.TERM_ATM, **kw))
    g.update_container()
    g.forces()
    return g


# staging per neighbour: 8 warps x 64 bytes in FP64, 8 x 32 in FP32; the larger one is
# above 48 KB, with 92 only together with the kernel's static arrays
CAPS = [("fp64", 112, 88), ("fp64", 92, 64), ("fp32_compat", 320, 224), ("fp32_full", 320, 224), ("verlet", 320, 240)]


def _larger_still_works(form, large, small):
    from komd_gb300 import gpu
    a = _engine(form, large)
    b = _engine(form, small)
    a.forces()
    a.measure(gpu.MEASURE_ENERGY)
    a.step(1)
    b.step(1)
    fa, fb = a.download()[2], b.download()[2]
    a.close()
    b.close()
    return fa, fb


@pytest.mark.parametrize("form,large,small", CAPS)
def test_a_smaller_engine_leaves_the_limit(host, form, large, small):  # noqa: F811
    _larger_still_works(form, large, small)


@pytest.mark.gpu
@pytest.mark.parametrize("form,large,small", CAPS)
def test_a_smaller_engine_leaves_the_limit_gpu(form, large, small):
    fa, fb = _larger_still_works(form, large, small)
    # FP64 and the fixed-point triplet sums are independent of the capacity; the
    # others sum the same FP32 terms in the same list order
    assert np.isfinite(fa).all() and np.array_equal(fa, fb)
