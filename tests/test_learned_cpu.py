"""Warm-start network host logic without a GPU: parameter layout and the weights file."""
from __future__ import annotations

import pytest


def test_parameter_layout():
    from iane_gb300.learned import LAYERS, WarmStartNet

    net = WarmStartNet("cpu", seed=0)
    n = 0
    for name, ci, co, _ in LAYERS:
        assert net.offsets[name] == (n, n + co * ci * 27)
        n += co * ci * 27 + co
    assert net.size == n == net.master.numel()
    assert 300_000 < n < 600_000


def test_weights_file_round_trip(tmp_path):
    import torch

    from iane_gb300.learned import WarmStartNet

    net = WarmStartNet("cpu", seed=4)
    path = tmp_path / "w.bin"
    net.save(path)
    other = WarmStartNet("cpu", seed=5)
    assert not torch.equal(other.master, net.master)
    other.load(path)
    assert torch.equal(other.master, net.master)
    assert torch.equal(other.p16, net.master.to(torch.bfloat16))
    raw = bytearray(path.read_bytes())
    raw[0] ^= 0xFF
    path.write_bytes(bytes(raw))
    with pytest.raises(ValueError):
        other.load(path)
    path.write_bytes(bytes(path.read_bytes()[:100]))
    with pytest.raises(ValueError):
        other.load(path)


def test_conv3_refuses_too_deep_a_volume_for_every_kernel():
    # 4 planes to a brick, 65535 bricks: refused before any CUDA call, for channels in whole octets (the
    # tensor cores') as for others; the pointers are never read
    from iane_gb300 import _lib

    lib = _lib.lib()
    for conv3 in (lib.iane_gb_cnn_conv3, lib.iane_gb_cnn_conv3_simt):
        for c0, co in ((16, 16), (3, 5)):
            status = conv3(16, c0, None, 0, 4 * 65535 + 1, 1, 1, 16, None, co, 16, None, None, 0, None, None)
            assert status == -2 and "too deep" in _lib.last_error()
