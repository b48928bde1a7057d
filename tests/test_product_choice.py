"""Which form of the gate/up product a prompt portion takes: by its sizes alone."""
import pytest

from tiny_transformer_inference_engine_b200.ops import CudaOps


@pytest.mark.parametrize("rows,hidden,K,fused", [
    (2048, 11008, 4096, True), (1024, 11008, 4096, True), (4096, 18176, 4544, True), (2048, 16384, 2048, True), (2048, 8192, 2048, True),
    (2000, 11008, 4096, False), (2047, 16384, 2048, False), (1300, 18176, 4544, False), (5000, 18176, 4544, True),      # ragged last tiles
    (768, 16384, 2048, False), (1023, 16384, 2048, False),                                                            # fewer than 1,024 rows
    (1280, 4096, 4096, False), (1024, 8192, 2048, False), (2048, 8192, 1024, False), (8192, 4096, 1024, False),      # few waves, small K
])
def test_gate_up_form_by_sizes(rows, hidden, K, fused):
    assert CudaOps._fused_swiglu_wins(148, rows, hidden, K) is fused
