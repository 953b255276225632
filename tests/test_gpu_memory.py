"""Device memory that the cooperative substeps add to a context, over that of the schedules that
launch a kernel per stage (a step of one substep takes those), whose lists their records share."""
import pytest

pytestmark = pytest.mark.gpu


def _bytes(form, n_sub, N, nc):
    import torch

    import brownian_gb300 as bg

    def make():
        return bg.Simulation(32, N, nc, mass_colloid=335.1, sig_colloid=4.0, sigma=4.0, Dr=0.001, n_sub=n_sub,
                             precision=bg.FP64 if form == "fp64" else bg.FP32C)

    make().close()  # (what the process itself takes)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    sim = make()
    used = free - torch.cuda.mem_get_info()[0]
    sim.close()
    return used


@pytest.mark.parametrize("form", ["fp64", "fp32c"])
def test_memory_of_the_cooperative_substeps(form):
    # 8 bytes a particle for the list of the active ones, 48 a sphere and substep, and in the FP64 form 64 for
    # each event record over the 192 of the lists in whose place they lie; allocations are rounded up
    N, nc = 327680, 60
    more = 8 * N + 48 * nc * 10 + (64 * (N // 16 + 65536) if form == "fp64" else 0)
    assert _bytes(form, 10, N, nc) <= _bytes(form, 1, N, nc) + more + (6 << 20)
