"""Device memory around prompts and weights: what is allocated when, and what happens when the card is nearly full."""
import numpy as np
import pytest
import torch

import helpers as H
from velox_b200 import lib as L
from velox_b200.engine import Engine
from velox_b200.modelspec import LLAMA3_8B_INT4

pytestmark = pytest.mark.gpu


def spec_of(fmt, **kw):
    base = dict(name="ws", d_model=512, n_layers=2, n_q_heads=8, n_kv_heads=2, head_dim=64, ffn_dim=1408, vocab=1024, weight_fmt=fmt, head_fmt=fmt)
    return LLAMA3_8B_INT4.scaled(**{**base, **kw})


def free_bytes():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("fmt", [L.FMT_Q4G32, L.FMT_I8PC, L.FMT_F16])
def test_prompts_of_growing_length_allocate_twice_at_most(fmt):
    eng = H.build_engine(spec_of(fmt), 71, 2048)
    eng.reserve(0, 2048)
    seen = set()
    for n in (20, 60, 130, 300, 520, 700, 1100, 2000):
        eng.prefill(H.prompt_tokens(eng.spec, 71, n))
        seen.add(free_bytes())
    eng.close()
    assert len(seen) <= 2


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


def test_prompt_in_a_nearly_full_card():
    """A lean context whose chunk buffers do not fit takes shorter chunks: the logits of the roomy run up to the rounding of other
    row tiles (2^-11 of the fp16 cache)."""
    spec = spec_of(L.FMT_Q4G32, d_model=2048, n_q_heads=16, n_kv_heads=4, head_dim=128, ffn_dim=8192)
    prompt = H.prompt_tokens(spec, 73, 4000)
    got = []
    for left in (None, 300 << 20):  # the buffers of 4096 rows: 34 + 50 + 34 + 34 + 134 MB and 134 MB of parts
        eng = Engine(spec, max_seq_len=4096, lean_weights=True)
        eng.load_synthetic(73)
        eng.set_option("prefill_rows", 4096)
        eng.reserve(0, 4096)
        eng.prefill(prompt[:17])
        hog = torch.empty(free_bytes() - left, dtype=torch.uint8, device="cuda") if left else None
        try:
            eng.prefill(prompt)
        finally:
            del hog
            torch.cuda.empty_cache()
        got.append(eng.logits())
        eng.close()
    assert np.max(np.abs(got[0] - got[1])) <= 1e-2


def test_group64_weights_in_a_nearly_full_card():
    """The tile-major copies of group-64 weights are left out where only the weights themselves fit; gate and up have one copy, not two."""
    spec = spec_of(L.FMT_Q4G64REF, d_model=2048, n_layers=4, n_q_heads=16, n_kv_heads=4, head_dim=128, ffn_dim=8192, vocab=32000, embed_fmt=L.FMT_Q4G64REF)
    packed = sum(rows * cols for _, _, rows, cols, _, _ in spec.tensors() if rows > 1) * 9 // 16
    prompt, got, sizes = H.prompt_tokens(spec, 74, 12), [], []
    for left in (None, 400 << 20):
        hog = torch.empty(free_bytes() - left, dtype=torch.uint8, device="cuda") if left else None
        try:
            eng = Engine(spec, max_seq_len=64)
        finally:
            del hog
            torch.cuda.empty_cache()
        eng.load_synthetic(74)
        eng.reserve(0, 64)
        eng.prefill(prompt)
        eng.decode(3)
        got.append(eng.logits())
        n = L.C.c_uint64()
        L.check(L.load().vb_weight_bytes(eng.h, L.C.byref(n)))
        sizes.append(n.value)
        eng.close()
    assert packed <= sizes[1] < 1.01 * packed + (1 << 20) and sizes[0] <= 2 * sizes[1]
    assert np.max(np.abs(got[0] - got[1])) <= 1e-2  # (the rounding of the fp16 cache apart)


def test_int8_prompts_without_room_for_copies():
    """Prompts of 129 to 256 rows of an int8 model that may not, or cannot, hold fp16 copies of its weights read the packed ones: no copies
    and no room for converted weights (70 MB a matrix); longer ones take that way too where the card has no such room."""
    spec = spec_of(L.FMT_I8PC, n_layers=2, d_model=2048, n_q_heads=16, n_kv_heads=4, head_dim=128, ffn_dim=17408)
    ora, _ = H.build_oracle(spec, 75, 320)
    prompt = H.prompt_tokens(spec, 75, 300)
    want = {}
    for pos, t in enumerate(prompt):
        ora.forward_step(int(t), pos)
        want[pos + 1] = ora.logits.copy()
    for n in (130, 200, 257, 300):
        for resident_gb, left in ((40, None), (0, None), (40, 120 << 20)):
            eng = H.build_engine(spec, 75, 320)
            eng.set_option("tc_resident_gb", resident_gb)
            eng.reserve(0, 320)
            eng.prefill(prompt[:20])
            hog = torch.empty(free_bytes() - left, dtype=torch.uint8, device="cuda") if left else None
            before = free_bytes()
            try:
                eng.prefill(prompt[:n])
            finally:
                used = before - free_bytes()
                del hog
                torch.cuda.empty_cache()
            assert np.max(np.abs(eng.logits() - want[n])) <= 1e-2, (n, resident_gb, left)
            if n <= 257 and (resident_gb, left) != (40, None):
                assert used <= 110 << 20, (n, used)  # buffers of 320 rows: 3 + 4 + 3 + 3 + 22 MB and 22 MB of parts
            eng.close()
