"""The front end of the native host path where threads share an engine."""
import pytest
import torch

import helpers


@pytest.mark.parametrize("mods", [False, True])
def test_scan_backward_kernels_are_complete_when_they_are_found(mods):
    """A thread takes the plan as complete once it finds the reverse kernel in it, so that one is set last."""
    class Plan:
        bwd = bwd_mods = 0

        def __init__(self):
            self.__dict__["order"] = []

        def __setattr__(self, name, value):
            assert value
            self.order.append(name)

    eng = helpers.mamba2_engine(1, 2, 128, 128, 64, torch.bfloat16, d_skip=True)
    eng._plan = Plan()
    assert eng._native_bwd(1, 2, False, mods, 0) == 1
    assert sorted(eng._plan.order) == sorted(["head_sum", "bwd_mods" if mods else "bwd"])
    assert eng._plan.order[-1] == ("bwd_mods" if mods else "bwd")


def test_split_counts_survive_a_cleared_table():
    class Cleared(dict):
        def __contains__(self, key):  # another thread clears the table behind this look
            found = super().__contains__(key)
            self.clear()
            return found

    dec = helpers.decode_engine(2, 8, 2, 1, 1000, 64, torch.float16)._decode
    want = dec.pick_splits(2, 1000)
    dec._splits = Cleared(dec._splits)
    assert dec.pick_splits(2, 1000) == want


def test_extension_for_another_torch_is_rebuilt(tmp_path):
    import __graft_entry__ as entry
    out, dep = tmp_path / "x.so", tmp_path / "x.cpp"
    dep.write_text("")
    assert entry.host_is_stale(str(out), [str(dep)], "built for A")
    out.write_bytes(b"\0..built for A\0")
    assert not entry.host_is_stale(str(out), [str(dep)], "built for A")
    assert entry.host_is_stale(str(out), [str(dep)], "built for B")
