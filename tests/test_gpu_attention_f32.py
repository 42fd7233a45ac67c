"""The f32 attention kernel over more than a wave of blocks: ragged rows and keys, one to ten tiles, masked positions."""
import numpy as np
import pytest

from oxionnx_b200 import models
from oxionnx_b200.session import Session

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,seq", [(80, 33), (75, 64), (40, 65), (40, 127), (26, 129), (25, 190), (15, 257), (13, 383), (8, 630)])
def test_many_blocks_are_the_separate_nodes_bit_for_bit(batch, seq):
    graph, weights, feeds, _ = models.build_bert_dynamic_int8(batch=batch, seq=seq, hidden=128, heads=2, ffn=128, layers=1, vocab=100)
    f = feeds()
    f["attention_mask"][:, (seq + 1) // 2:] = 0
    f["attention_mask"][0] = 1
    out = {}
    for kept in (False, True):
        session = Session.builder().with_keep_intermediates(kept).build_from_graph(graph, weights)
        out[kept] = session.run(f)["hidden"]
        assert kept or [s["kernel"] for s in session.steps()].count("attention_f32") == 1
        session.close()
    assert np.array_equal(out[False], out[True])
