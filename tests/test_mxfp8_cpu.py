"""The cache of quantised expert weights (host side; the quantisers are stood in for)."""
import torch


def test_quantised_weight_is_not_taken_for_another_tensor_at_the_same_address(monkeypatch):
    from kolmogorov_moe_architecture_b200.ops import mxfp8
    monkeypatch.setattr(mxfp8, "_WCACHE", {})
    monkeypatch.setattr(mxfp8, "quant_rows", lambda w: (w.clone(), None))
    memory = bytearray(4 * 8)
    first = torch.frombuffer(memory, dtype=torch.float32)
    first.fill_(1.0)
    a = mxfp8._weight_quant(first, "rows")
    assert mxfp8._weight_quant(first, "rows") is a                         # unchanged: kept
    first.mul_(2.0)
    assert mxfp8._weight_quant(first, "rows")[0][0] == 2.0                 # changed in place: made anew
    version = first._version
    del first
    second = torch.frombuffer(memory, dtype=torch.float32)                 # what an allocator does with freed memory
    for _ in range(version - second._version):
        second.fill_(5.0)
    assert second._version == version
    assert mxfp8._weight_quant(second, "rows")[0][0] == 5.0
    assert len(mxfp8._WCACHE) == 1
    third = torch.ones(8)
    del second
    mxfp8._weight_quant(third, "rows")
    assert len(mxfp8._WCACHE) == 1                                         # copies of freed weights are dropped
