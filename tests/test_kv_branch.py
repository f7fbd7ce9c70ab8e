"""SMs that the salient rows' K/V product keeps to beside the query projection."""
import pytest

from dyllm_b200 import model


@pytest.mark.parametrize("rows,columns,want", [
    (4096, 4096, 40), (8192, 4096, 80), (6144, 4096, 60), (8191, 4096, 80),      # 256, 512, 384 tiles of 148 SMs' waves
    (2560, 4096, 0), (4608, 4096, 0), (16384, 4096, 0),                          # 136, 8, 12 SMs idle
    (1, 4096, 0), (2048, 4096, 0), (2560, 2048, 0),                              # one wave
])
def test_sms_beside_the_query_projection(monkeypatch, rows, columns, want):
    monkeypatch.setitem(model._sm_counts, "gpu", 148)
    assert model._kv_ctas(rows, columns, "gpu") == want
