"""A large system takes its memory from what a closed one left: none is mapped
for the second of two alike."""
import pytest

from soil_b200 import system, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("consumer", [0.0, 1e3])
def test_a_second_large_system_maps_no_memory(consumer):
    import torch
    torch.zeros(1, device="cuda")
    w = W.mono("reuse-large", 330, 1048576, 0.30, 1e-3, 0, harmonic_k=consumer)
    c = system.Context(0)
    free = []
    for _ in range(3):
        s = system.from_workload(c, w)
        s.step(30)
        s.sync()
        free.append(torch.cuda.mem_get_info()[0])
        s.close()
    assert free[1] >= free[0] and free[2] >= free[0], free
    c.close()
