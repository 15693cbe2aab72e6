"""The scratch of an n-token call outlives its replacement where a captured graph holds its address."""
import weakref

import torch


def test_captured_scratch_is_kept_and_bounded(monkeypatch):
    from gemq_b200.inference.moe_block import _QuantFusedMoEBase
    capturing = [False]
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: capturing[0])
    blk, dev = _QuantFusedMoEBase(), torch.device("cpu")
    first = weakref.ref(blk._prefill_buffer(100, dev))
    assert blk._prefill_buffer(60, dev) is first()
    blk._prefill_buffer(200, dev)
    assert first() is None                       # eager only: given back
    capturing[0] = True
    kept = weakref.ref(blk._prefill_buffer(150, dev))
    capturing[0] = False
    larger = blk._prefill_buffer(250, dev)
    assert kept() is not None and larger is not kept() and larger.numel() >= 400
    capturing[0] = True
    for n in range(100, 5000, 7):                # graphs of growing batches
        assert blk._prefill_buffer(n, dev).numel() >= n
    sizes = [b.numel() for b in blk._graph_scratch]
    assert len(sizes) <= 8 and sum(sizes) <= 2 * sizes[-1]
