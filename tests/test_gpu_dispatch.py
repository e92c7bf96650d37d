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


@pytest.mark.parametrize("waters,cutoff,one_sided,two_sided", [
    (2000, 8.0, "k_search<4>", "k_search<4>"),
    # past sixteen clusters an SM two-sided tables, twice as long, take a warp
    # each: two warps' shares would not fit what they can stage
    (5000, 8.0, "k_search<2>", "k_search<1>"),
    (7000, 12.0, "k_search<2>", "k_search<1>"),
    (9300, 8.0, "k_search<1>", "k_search<1>"),
])
def test_search_teams(torch_cuda, waters, cutoff, one_sided, two_sided):
    """The search of a build and the two-sided one that dH/dlambda asks for."""
    from spgnb import systems as S
    from spgnb.engine import SoftCorePath
    n_solute = 80
    L = ((waters + n_solute) / 0.0334) ** (1.0 / 3.0)
    s = S.water_system(waters, L, 61, n_solute=n_solute, cutoff=cutoff, skin=2.0)
    p = SoftCorePath(S.fep_system(s, n_perturbed=8))

    def searches(fn):
        return [k["name"] for k in kernel_launches(torch_cuda, fn) if "k_search" in k["name"]]

    built = searches(lambda: p.update(0, forced=True))
    again = searches(lambda: p.dhdl())
    assert len(built) == 1 and one_sided in built[0]
    assert len(again) == 1 and two_sided in again[0]
