"""What the launch rules choose: kernels, grids and shared memory as launched."""
import pytest

from conftest import kernel_launches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("setting", [1, 2, 3, 5, 7])
def test_pair_setting_is_the_resident_warps(torch_cuda, setting):
    """The force kernel's one-warp blocks ask for the shared memory that leaves
    four times the setting of them on an SM (setting 7 is what the registers
    of the force-only kernel allow)."""
    from spgnb import systems as S
    from spgnb.batch import Batch
    props = torch_cuda.cuda.get_device_properties(0)
    b = Batch(S.batch_systems(2, seed=15, n_min=1500, n_max=4000), use_graphs=0)
    b.set_tuning(b.tuning()["prune_buffer"], setting, 5, 10)
    found = [k for k in kernel_launches(torch_cuda, lambda: (b.run(1), b.progress())) if "k_pair8" in k["name"]]
    b.close()
    assert found
    for k in found:
        assert k["block"] == [32, 1, 1]
        reserved = 1024  # by the runtime, for each block
        assert props.shared_memory_per_multiprocessor // (k["shared"] + reserved) == 4 * setting
