"""ks_model_sample_step: the device lists the logits that can survive the min-p filter, the host draws.  Every token has to be
the one the CPU sampler (sample.rs:9-81) takes from the whole row, on the paths of one, two and several slots, with the
filter off, with more survivors than the list holds, and greedy."""
import numpy as np
import pytest

from ksearch_b200 import F16, F32, CudaContext, KsError, _lib, synth
from ksearch_b200 import model as ksm
from ksearch_b200.sample import sample_softcap_min_p

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("act", [F32, F16])
@pytest.mark.parametrize("n", [1, 2, 5])
def test_sample_step_takes_the_cpu_samplers_tokens(n, act):
    c = CudaContext(0, flags=1)
    cfg = ksm.tiny_config(max_seq=64, n_slots=n, act=act)
    cfg.vocab = 8193                      # not a multiple of anything the kernels use
    cfg.sigma_embd = 2e-5                 # flat logits: many survivors
    model = ksm.GemmaCudaModel.synthetic(c, cfg, seed=31)
    slots = [model.slot_alloc() for _ in range(n)]
    ids = [int(t) for t in synth.token_ids(31, "ids", n, cfg.vocab)]
    for step, (temp, min_p) in enumerate([(0.8, 0.05), (1.5, 0.3), (0.7, 1e-4), (4.0, 1e-3), (1.0, 0.0), (0.0, 0.05), (1.0, 1.0), (0.9, 2.0)]):
        seeds = [1000 * step + 7 * s for s in slots]
        got = model.sample_step(ids, 0, [temp] * n, [min_p] * n, seeds)
        want = [sample_softcap_min_p(model.read_debug(1, s), cfg.softcap, temp, min_p, seeds[s]) for s in slots]
        assert got == want, (temp, min_p)
        ids = got
    assert [model.seq_len(s) for s in slots] == [8] * n
    model.close()
    c.close()


def test_sample_step_rewinds_after_a_wait_that_gave_up():
    """The persistent kernel told to wait for something nobody writes: the blocking step reports KS_ERR_TIMEOUT and leaves the
    slot where it was, as decode_token does; the same step afterwards gives the token it gives without the stall."""
    c = CudaContext(0, flags=1)
    cfg = ksm.tiny_config(max_seq=48)
    model = ksm.GemmaCudaModel.synthetic(c, cfg, seed=32)
    ids = [int(t) for t in synth.token_ids(32, "ids", 6, cfg.vocab)]
    args = (0, [0.8], [0.05], [77])

    def run(stall):
        model.slot_reset(0)
        model.prefill(0, ids[:4])
        model.sample_step([ids[4]], *args)
        if stall:
            model.debug_set(model.POLL_LIMIT, 2000)
            model.debug_set(model.STALL, 1)
            with pytest.raises(KsError) as ei:
                model.sample_step([ids[5]], *args)
            assert ei.value.code == _lib.ERR_TIMEOUT and model.seq_len(0) == 5
            model.debug_set(model.STALL, 0)
            model.debug_set(model.POLL_LIMIT, 1 << 21)
        tok = model.sample_step([ids[5]], *args)
        assert model.seq_len(0) == 6
        return tok, model.read_debug(1, 0)

    model.slot_alloc()
    tok, logits = run(False)
    again, after = run(True)
    assert again == tok and np.array_equal(after, logits)
    model.close()
    c.close()


@pytest.mark.parametrize("min_p", [0.05, 0.9, 2.0, 0.0])
def test_sample_step_with_a_draw_that_rounds_to_one(ctx, min_p):
    """splitmix32 within 128 of 2^32 is 1.0 as a float: the CPU sampler then runs past every token and takes the row's last."""
    cfg = ksm.tiny_config(max_seq=32)
    model = ksm.GemmaCudaModel.synthetic(ctx, cfg, seed=35)
    model.slot_alloc()
    for seed in (1109269, 138204815, 280706243, 1109268):
        got = model.sample_step([7], 0, [0.8], [min_p], [seed])
        want = sample_softcap_min_p(model.read_debug(1, 0), cfg.softcap, 0.8, min_p, seed)
        assert got == [want] and (min_p == 2.0 or want == cfg.vocab - 1)
    model.close()
