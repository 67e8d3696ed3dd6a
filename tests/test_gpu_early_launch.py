"""The stage kernels read their stage input ahead of their own wait for the
kernel before them; the input is handed over by the stage's published number
(publish_input and input_ready in csrc/dycore_kernels.cuh), the same word for
every stage of a handle.  A run of many stages, and a captured graph whose
stages carry the same numbers at every replay, give the bits of stages launched
the ordinary way (an explicit z chunk: the z march).  Grids with rows that
share 32-byte sectors between blocks, several waves of blocks, and an immersed
domain, whose stage takes two launches of each kernel."""
import numpy as np
import pytest

from porturb_b200 import Dycore, cases
from helpers import gpu_run

pytestmark = pytest.mark.gpu

CASES = {
    "immersed_ragged": lambda: cases.small_mixed(nx=101, ny=67, nz=75),
    "three_tracers": lambda: cases.small_mixed(nx=90, ny=40, nz=64, ntr=3, immersed=False),
    "one_wave": lambda: cases.small_mixed(nx=30, ny=24, nz=24),
    "thin": lambda: cases.small_mixed(nx=120, ny=4, nz=96, immersed=False),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_many_stages_give_the_bits_of_ordinary_launches(name, gpu_lib):
    case = CASES[name]()
    _, _, g = gpu_run(case, "f32", 0, 0.0)
    dt = 0.9 * g.compute_time_step()
    a = gpu_run(case, "f32", 20, dt)
    b = gpu_run(case, "f32", 20, dt, z_chunk=16)
    assert np.isfinite(a[0]).all()
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_replayed_graph_gives_the_bits_of_direct_calls(name, precision, gpu_lib):
    import torch
    case = CASES[name]()
    stream = torch.cuda.Stream()

    def handle():
        return gpu_run(case, precision, 0, 0.0, stream=stream.cuda_stream)[2]

    g = handle()
    dt = 0.9 * g.compute_time_step()
    for _ in range(4):
        g.advance(dt, 1)
    g.synchronize()
    want = g.get_conserved()
    g.close()
    g = handle()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        g.advance(dt, 1)
    with torch.cuda.stream(stream):
        for _ in range(3):
            graph.replay()
    g.advance(dt, 1)
    g.synchronize()
    got = g.get_conserved()
    del graph
    g.close()
    for x, y in zip(want, got):
        assert np.array_equal(x, y)
