"""Growth of a scratch buffer: the outgrown one stays alive, the new one has at least twice its size, slots are separate."""
import weakref

import torch


def test_scratch_keeps_what_it_outgrows(monkeypatch):
    from noeira_b200.ops import streams
    monkeypatch.setattr(streams, "ws_key", lambda device: (str(device), streams.slot()))
    pool, dev = streams.Scratch(16), torch.device("cpu")
    first = weakref.ref(pool.get(dev, 4))
    assert first().numel() == 16 and pool.get(dev, 16) is first()
    second = weakref.ref(pool.get(dev, 17))
    assert second().numel() == 32 and first() is not None
    assert pool.get(dev, 100).numel() == 100 and first() is not None and second() is not None
    monkeypatch.setattr(streams, "slot", lambda: 1)
    assert pool.get(dev, 4).numel() == 16


def test_column_sums_and_norms_draw_from_growing_scratch():
    from noeira_b200.nn import conv, layers, transformer
    from noeira_b200.ops.streams import Scratch
    for get in (conv._scratch, transformer._scratch, layers._colsum_workspace):
        assert isinstance(get.__self__, Scratch)


def test_world_model_workspace_holds_the_norm_partials():
    import ctypes

    from noeira_b200._native import cuda_lib
    from noeira_b200.models.world_model import workspace_floats
    lib = cuda_lib()
    for rows in (1, 64, 1000, 16448, 1 << 20):
        for dim in (64, 2048, 14336, 16384, 32768):
            assert 2 * lib.nb_norm_split(ctypes.c_int(rows)) * dim <= workspace_floats(lib, rows, dim)
