"""The phase stamps of the last edit that the persistent kernel ran: one for the start, the begin, every
level down, the leaves, every level up and the end. An edit that runs as a chain of launches takes no
stamps, so it leaves the count and the stamps as they were."""
import pytest

pytestmark = pytest.mark.gpu

LEVELS = 9


def sphere(svdag_lib, radius):
    return svdag_lib.MyGpuSphereEditor((200.0, 210.0, 190.0), radius, 3, is_adding=True).to_edit()


@pytest.mark.parametrize("phase_kernels", [False, True])
def test_a_chain_takes_no_stamps(svdag_lib, phase_kernels):
    g = svdag_lib.MyGPUHashDAG(LEVELS, pool_bytes=1 << 28, phase_kernels=phase_kernels)
    for radius in (3.0, 60.0):
        g.edit(sphere(svdag_lib, radius))
        assert len(g.last_edit_phase_times()) == 0
    g.free()


def test_a_chain_leaves_the_persistent_edits_stamps(svdag_lib):
    g = svdag_lib.MyGPUHashDAG(LEVELS, pool_bytes=1 << 28, persistent=True)
    g.edit(sphere(svdag_lib, 3.0))
    stamps = list(g.last_edit_phase_times())
    leaf = LEVELS - 2
    assert len(stamps) == 2 + leaf + 1 + (leaf + 1) + 1
    assert stamps == sorted(stamps) and stamps[0] > 0
    g.edit(sphere(svdag_lib, 60.0))  # estimated at far more than 400 leaves: a chain
    g.edit(svdag_lib.MyGpuSphereErosionEditor((200.0, 210.0, 190.0), 40.0, 13).to_edit())
    assert list(g.last_edit_phase_times()) == stamps
    g.free()
