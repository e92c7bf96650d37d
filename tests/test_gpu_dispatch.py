"""What the launch rules choose: kernels, grids and shared memory as launched."""
import pytest

from conftest import in_fresh_process, kernel_launches

pytestmark = pytest.mark.gpu

SETTINGS = (1, 2, 3, 5, 7)
# waters, cutoff, the search of a build, the two-sided one that dH/dlambda asks for
SEARCHES = (
    (2000, 8.0, "k_search<4>", "k_search<4>"),
    # past sixteen clusters an SM two-sided tables, twice as long, take a warp
    # each: two warps' shares would not fit what they can stage
    (5000, 8.0, "k_search<2>", "k_search<1>"),
    (7000, 12.0, "k_search<2>", "k_search<1>"),
    (9300, 8.0, "k_search<1>", "k_search<1>"),
)


def traced():
    """The force kernel's launches under each setting, and each search's."""
    import torch
    from spgnb import systems as S
    from spgnb.batch import Batch
    from spgnb.engine import SoftCorePath
    pairs, searches = {}, []
    for setting in SETTINGS:
        b = Batch(S.batch_systems(2, seed=15, n_min=1500, n_max=4000), use_graphs=0)
        b.set_tuning(b.tuning()["prune_buffer"], setting, 5, 10)
        pairs[setting] = [k for k in kernel_launches(torch, lambda: (b.run(1), b.progress()))
                          if "k_pair8" in k["name"]]
        b.close()
    for waters, cutoff, *_ in SEARCHES:
        L = ((waters + 80) / 0.0334) ** (1.0 / 3.0)
        s = S.water_system(waters, L, 61, n_solute=80, cutoff=cutoff, skin=2.0)
        p = SoftCorePath(S.fep_system(s, n_perturbed=8))
        searches.append([[k["name"] for k in kernel_launches(torch, fn) if "k_search" in k["name"]]
                         for fn in (lambda: p.update(0, forced=True), lambda: p.dhdl())])
    return {"pairs": pairs, "searches": searches}


@pytest.fixture(scope="module")
def launched(torch_cuda):
    return in_fresh_process("test_gpu_dispatch", "traced")


@pytest.mark.parametrize("setting", SETTINGS)
def test_pair_setting_is_the_resident_warps(torch_cuda, launched, setting):
    """The force kernel's one-warp blocks ask for the shared memory that leaves
    four times the setting of them on an SM (setting 7 is what the registers
    of the force-only kernel allow)."""
    per_sm = torch_cuda.cuda.get_device_properties(0).shared_memory_per_multiprocessor
    found = launched["pairs"][str(setting)]
    assert found
    for k in found:
        assert k["block"] == [32, 1, 1]
        reserved = 1024  # by the runtime, for each block
        assert per_sm // (k["shared"] + reserved) == 4 * setting


@pytest.mark.parametrize("case", range(len(SEARCHES)))
def test_search_teams(launched, case):
    for names, want in zip(launched["searches"][case], SEARCHES[case][2:]):
        assert len(names) == 1 and want in names[0]
