"""Device memory around prompts and weights: what is allocated when, and what happens when the card is nearly full."""
import pytest

import helpers as H
from velox_b200 import lib as L
from velox_b200.modelspec import LLAMA3_8B_INT4

pytestmark = pytest.mark.gpu


def spec_of(fmt, **kw):
    base = dict(name="ws", d_model=512, n_layers=2, n_q_heads=8, n_kv_heads=2, head_dim=64, ffn_dim=1408, vocab=1024, weight_fmt=fmt, head_fmt=fmt)
    return LLAMA3_8B_INT4.scaled(**{**base, **kw})


def test_long_prompt_keeps_the_captured_step():
    """The step captured before the first long prompt is still replayed after it: another context turns an option of the whole
    process that changes how many kernels a step of five int8 rows launches, and the step's count stays that of the capture."""
    spec = spec_of(L.FMT_I8PC)
    eng, other = H.build_engine(spec, 72, 640, max_batch=5), H.build_engine(spec, 72, 32)
    for slot in range(5):
        eng.reserve(slot, 640)
        eng.prefill(H.prompt_tokens(spec, 72 + slot, 40), slot)
    eng.build_graph()

    def launches_of_a_step():
        before = eng.launch_count()
        eng.decode(1)
        eng.sync()
        return eng.launch_count() - before
    captured = launches_of_a_step()
    eng.prefill(H.prompt_tokens(spec, 72, 600), 0)
    other.set_option("gemv_multirow", 0)
    try:
        assert launches_of_a_step() == captured
        eng.set_option("pdl", 1)  # drops the captured step
        assert launches_of_a_step() != captured
    finally:
        other.set_option("gemv_multirow", 1)
    eng.close(), other.close()
