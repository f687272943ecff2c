"""Which decoders run channels-last, and what the kernels' C entries refuse: nothing is launched here."""
import pytest

from vox_serve_b200 import _lib
from vox_serve_b200.tokenizer.mimi import MimiConfig, fits_channels_last
from vox_serve_b200.tokenizer.snac import SNAC


@pytest.mark.parametrize("kw,fits", [({}, True), (dict(decoder_dim=1024, decoder_rates=(8,)), False), (dict(decoder_dim=1024, decoder_rates=(8, 8)), True),
                                     (dict(decoder_dim=512), False), (dict(latent_dim=96), False)])
def test_snac_rule(kw, fits):
    assert SNAC(device="cpu", **kw)._fits_channels_last() == fits


@pytest.mark.parametrize("kw,fits", [({}, True), (dict(last_kernel_size=16), True), (dict(last_kernel_size=17), False), (dict(num_heads=4), True),
                                     (dict(num_heads=2), False), (dict(n_filters=48), False), (dict(n_q=65), False)])
def test_mimi_rule(kw, fits):
    assert fits_channels_last(MimiConfig(**kw)) == fits


A = 1 << 20                                              # an address on a 16-byte boundary that nothing reads


def _conv(**off):
    p = {k: A + off.get(k, 0) for k in ("y", "y2", "x", "w", "bias", "resid", "scale", "noise", "alpha")}
    return (p["y"], p["y2"], p["x"], 32 * 8, 8, p["w"], p["bias"], p["resid"], 32 * 8, p["scale"], p["noise"], 8, p["alpha"], 2, 1, 0, 32, 32, 32, 1, 1,
            0, 8, 32 * 8, None)


@pytest.mark.parametrize("name,make,operands", [
    ("vb_cl_conv", _conv, ("y", "y2", "x", "w", "bias", "resid", "scale", "alpha")),
    ("vb_cl_dwconv7", lambda **o: (A + o.get("y", 0), A + o.get("x", 0), 64, A + o.get("w", 0), A + o.get("bias", 0), A + o.get("a", 0), A + o.get("b", 0),
                                   0, 64, 8, 1, 0, 8, None), ("y", "x", "w", "bias", "a", "b")),
    ("vb_cl_last_conv", lambda **o: (A, A + o.get("x", 0), 64, A, A, 0, 64, 8, 7, 3, 0, 8, 0, None), ("x",)),
    ("vb_cl_layernorm", lambda **o: (A + o.get("y", 0), A + o.get("x", 0), A + o.get("w", 0), A + o.get("b", 0), 0, 64, 1e-5, None), ("y", "x", "w", "b")),
    ("vb_cl_chunk_attention", lambda **o: (A, A + o.get("x", 0), 0, 64, 1, 8, 1e4, None), ("x",))])
def test_entries_refuse_pointers_off_their_boundary(name, make, operands):
    """(with no batch entries: an accepted call returns without a launch)"""
    fn = getattr(_lib.load(), name)
    assert fn(*make()) == 0
    for op in operands:
        assert fn(*make(**{op: 4})) != 0 and b"boundar" in _lib.load().vb_last_error(), op
