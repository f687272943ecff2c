"""A wait that ran out inside a kernel reaches whoever collects results: the flags are set here as a kernel would set them."""
import asyncio
import ctypes as C
from types import SimpleNamespace

import pytest
import torch

from vox_serve_b200 import _lib
from vox_serve_b200._lib import VoxB200Error


@pytest.fixture
def flags(monkeypatch):
    word = C.c_uint64(0)
    monkeypatch.setattr(_lib, "_wait_flags", word)
    return word


def test_check_waits_names_the_kernel_and_clears(flags):
    _lib.check_waits()
    for i, name in enumerate(_lib.WAIT_KINDS):
        flags.value = 1 << (8 * i)
        with pytest.raises(VoxB200Error, match=name):
            _lib.check_waits()
        assert flags.value == 0
        _lib.check_waits()


def test_next_call_raises_before_it_launches(flags, monkeypatch):
    calls = []
    monkeypatch.setattr(_lib, "_lib", SimpleNamespace(vb_fake=lambda *a: calls.append(a) or 0))
    _lib.call("vb_fake", 1)
    flags.value = 1
    with pytest.raises(VoxB200Error, match="ran out"):
        _lib.call("vb_fake", 2)
    _lib.call("vb_fake", 3)
    assert calls == [(1,), (3,)]


def _request():
    return SimpleNamespace(lm_output_tokens=[], lm_output_audio_tokens=[], done_lm_generation=False, finish_reason=None, next_position_id=1,
                           pending_tokens=None, sampling_config=None, input_tokens=None)


def _steps():
    from vox_serve_b200.model.bobavik import BobavikModel
    from vox_serve_b200.model.orpheus import OrpheusModel
    from vox_serve_b200.worker.depth import DepthModelWorker

    lm = SimpleNamespace(stop_token_id=99, max_tokens=50, max_positions=50)
    ids, done = torch.tensor([[7, 1]]), SimpleNamespace(synchronize=lambda: None)
    yield lambda r: OrpheusModel.sampling_host(lm, ids[:, :1], [r], ids_host=ids[:, :1], ready=done)
    yield lambda r: BobavikModel.sampling_host(lm, ids[:, :1], [r], ids_host=ids[:, :1], ready=done)
    depth = SimpleNamespace(model=lm, decode_mask=torch.ones(2, dtype=torch.bool), feats=None)
    yield lambda r: DepthModelWorker._update_req_states(depth, [r], ids, done)


@pytest.mark.parametrize("kind", range(3))
def test_a_step_with_an_expired_wait_gives_no_token(flags, kind):
    step = list(_steps())[kind]
    good, bad = _request(), _request()
    asyncio.run(step(good))
    assert len(good.lm_output_tokens) == 1
    flags.value = 1 << 16
    with pytest.raises(VoxB200Error, match="prompt attention"):
        asyncio.run(step(bad))
    assert bad.lm_output_tokens == [] and not bad.done_lm_generation
