"""Simulations whose steps never stream tiles (the k-nearest cap, the particle
packing) hold neither candidate lists nor recorded tiles."""
import math

import pytest

from uph_b200 import deck as D

pytestmark = pytest.mark.gpu


def _bytes(params):
    torch = pytest.importorskip("torch")
    from uph_b200.sim import Simulation
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    with Simulation(params):
        used = free - torch.cuda.mem_get_info()[0]
    return used


def test_no_stream_arrays_where_nothing_streams():
    d = D.dam_break(tank=(2.0, 3.0), column=(1.0, 2.0), dx=(2.0 / 200000) ** 0.5, layers=2,
                    eta=math.sqrt(91 / (4.0 * math.pi)))
    _bytes(d.uph_params())  # the context and the library's own
    streaming, capped = _bytes(d.uph_params()), _bytes(d.uph_params(knn_cap=40))
    d.params["flag_init_simul"] = 0
    packing = _bytes(d.uph_params())
    # 1.3 pi (2 h 1.07 / dx)^2 = 136 to 144 candidates of two bytes, less the cut's 12 bytes
    assert streaming - capped > 200 * d.n_fluid
    assert streaming - packing > 200 * d.n_fluid
