"""The tuner never ends slower than the library's own choice: that form is a candidate."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def closed_mesh_batch(n):
    """Queries inside a closed mesh: one of them visits thousands of nodes, so one search per
    warp (the library's choice for a batch this small) is several times faster than a lane
    each, and than packets."""
    import snch_lbvh_gb300 as snch
    import torch
    from snch_lbvh_gb300 import meshes
    s = snch.Scene(*meshes.noisy_icosphere(5, 1.0, 0.01, seed=0))
    s.compute_silhouettes()
    s.build_bvh()
    g = torch.Generator(device="cuda").manual_seed(2)
    return s, torch.rand(n, 3, generator=g, device="cuda") - 0.5


@pytest.mark.parametrize("n", [3000, 20_011])
def test_own_choice_is_a_candidate(n):
    import snch_lbvh_gb300 as snch
    s, p = closed_mesh_batch(n)
    s.set_option(snch.OPT_PACKET, 0)  # the tuner does not depend on what the scene had
    ms = s.autotune(p, p)
    for kind in ("nearest", "silhouette"):
        assert (2, 128, 2, 0) in ms[kind]
        assert s.search_config(kind) == min(ms[kind], key=ms[kind].get)
        assert s.search_config(kind) == (2, 128, 2, 0), ms[kind]


def test_c_entry_writes_its_seven_times():
    """The entry point of the first seven configurations writes no more than their times."""
    import snch_lbvh_gb300 as snch
    s, p = closed_mesh_batch(3000)
    out = np.full(20, -7.0, np.float32)
    ptr = C.c_void_p(p.data_ptr())
    snch.check(snch.lib().snch_autotune(s._h, None, ptr, len(p), None, ptr, None, len(p),
                                        out.ctypes.data_as(C.c_void_p), None))
    assert (out[:14] > 0).all() and (out[14:] == -7.0).all()
    assert s.search_config("silhouette") == (2, 128, 2, 0)
