"""What an engine launches is built with the engine, not in a call that serves it; two threads build a kernel once."""
import threading

import torch

from attentionengine_b200 import CustomIO, LinearAttentionEngine, examples as helpers, meta_tensor
from attentionengine_b200 import runtime as rt


def _no_builds(monkeypatch):
    def build(*_):
        raise AssertionError("a build after the engine was made")
    monkeypatch.setattr(rt, "compile_module", build)


def test_decode_engine_has_its_kernels(monkeypatch):
    dec = helpers.decode_engine(2, 32, 8, 1, 1000, 128, torch.float16)._decode
    _no_builds(monkeypatch)
    assert dec._pick(2, 1000) == (4, True) and dec.cut_kernel is not None


def test_group_of_more_rows_than_a_tile_is_never_cut():
    dec = helpers.decode_engine(2, 150, 1, 1, 8192, 128, torch.float16)._decode
    assert dec.cut_kernel is None and dec._pick(2, 1000)[1] is False
    assert dec.schedule(torch.tensor([8192, 5000, 1, 8000]), device="cpu")["intervals"] == 0


def test_scan_of_few_walks_has_its_kernels(monkeypatch):
    metas = tuple(meta_tensor(1, 4, 4096, n, dtype=torch.bfloat16) for n in (128, 128, 128))
    plain = LinearAttentionEngine(metas, custom_io=CustomIO({}))
    block = helpers.mamba2_engine(1, 8, 8192, 128, 64, torch.bfloat16, d_skip=True)
    full = helpers.mamba2_engine(8, 80, 8192, 128, 64, torch.bfloat16, d_skip=True)
    _no_builds(monkeypatch)
    plain._segment_kernels(128, False)
    block._segment_kernels(64, True)
    assert not full._cut_kernels


def test_threads_build_the_segment_kernels_once(monkeypatch):
    metas = tuple(meta_tensor(8, 80, 1024, n, dtype=torch.bfloat16) for n in (128, 128, 64))
    eng = LinearAttentionEngine(metas, custom_io=CustomIO({}))
    compile_module, built, got = rt.compile_module, [], []

    def build(src, name, *rest):
        built.append(name)
        threading.Event().wait(0.1)  # the others run into it
        return compile_module(src, name, *rest)

    monkeypatch.setattr(rt, "compile_module", build)
    threads = [threading.Thread(target=lambda: got.append(eng._segment_kernels(64, False))) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert sorted(built) == ["ae_linear_fwd", "ae_linear_segments"] and len(set(map(id, (x for pair in got for x in pair)))) == 2
