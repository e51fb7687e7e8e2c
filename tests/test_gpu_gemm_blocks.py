"""A long step's token blocks in more than one launch of the tensor-core GEMM, which a matrix takes whose k is long and whose
tiles fill the SMs badly: that there are that many launches, and what the later ones (their first token, a shorter last group)
leave in the residual stream, its sums of squares, the K/V cache and the logits. Few SMs to count with make small matrices
such ones: 2 or 4 row tiles of k 10 240 are split over three blocks each apart, over one together."""
import numpy as np
import pytest

import oracle
from silicon_violetto_b200 import build, engine as E, synth, vlt
from tests.test_gpu_parity import TOL, same_state

pytestmark = pytest.mark.gpu
SHAPE = dict(n_layers=1, n_heads=4, n_kv=2, hd=64, vocab=256, eps=1e-5, theta=500000.0, page=16)
DOWN = dict(SHAPE, d=256, ffn=10240)  # the residual epilogue with its sums of squares
QKV = dict(SHAPE, d=10240, ffn=256)   # the qkv epilogue; norms from sums of squares of 80 row tiles


@pytest.fixture(scope="module", autouse=True)
def built():
    build.build()


@pytest.fixture(scope="module")
def weights(tmp_path_factory):
    made = {}

    def get(which, int8_group):
        key = (which["d"], int8_group)
        if key not in made:
            made[key] = tmp_path_factory.mktemp("w") / "w.vlt"
            synth.write_target(made[key], which, seed=0, int8_group=int8_group, std=0.02 * (256 / which["d"]) ** 0.5)  # (logits as large as the small models')
        return made[key]

    return get


def _engine(path, n, sms):
    kw = dict(max_seqs=1, max_step_tokens=n, max_chunk=n, max_seq_len=2 * n + 16, max_head_rows=n)
    return E.Engine(path, E.EngineConfig(global_kv_tokens=2 * n + 32, **kw), E.Tuning(sm_count=sms)), kw


def _launches(eng, kind, n):
    before = eng.launches()
    eng.bench_matmul(kind, n, variant=2, reps=1)
    return eng.launches() - before


# 300 and 512 tokens: two blocks, apart; 1 040: five blocks, as three and two.
@pytest.mark.parametrize("int8_group", [None, 0])
@pytest.mark.parametrize("sms,n,launches", [(0, 300, 1), (6, 300, 2), (6, 512, 2), (18, 1040, 2)])
def test_the_residual_of_token_blocks_apart_matches_the_oracle(weights, int8_group, sms, n, launches):
    path = weights(DOWN, int8_group)
    prod, kw = _engine(path, n, sms)
    assert _launches(prod, "down", n) == launches
    orc = oracle.Engine(path, kv_tokens=2 * n + 32, **kw)
    a = prod.new_seq()
    assert orc.new_seq() == a
    runs = [(a, np.random.default_rng(n).integers(0, 256, n).astype(np.uint32), E.Rows.ALL, False)]
    out = prod.debug_step(runs, E.StepOptions(read_logits=True))
    orc.step(runs)
    assert float(np.abs(out.logits - orc.array("logits").reshape(-1, 256)).max()) <= TOL[int8_group]
    same_state(prod, orc, 1, n)
    prod.close()


@pytest.mark.parametrize("int8_group", [None, 0])
@pytest.mark.parametrize("sms,n", [(12, 300), (12, 512), (36, 1040)])
def test_the_qkv_epilogue_of_token_blocks_apart_is_that_of_one_launch(weights, int8_group, sms, n):
    """The same sums in another order: K and V within one unit in the last place of bf16 (2^-7 of the value; 1e-4 for sums near 0,
    k 10 240 products of fp32 rounding)."""
    path, tokens, got = weights(QKV, int8_group), np.random.default_rng(n).integers(0, 256, n).astype(np.uint32), []
    for s, launches in ((0, 1), (sms, 2)):
        eng, _ = _engine(path, n, s)
        assert _launches(eng, "qkv", n) == launches
        a = eng.new_seq()
        out = eng.debug_step([(a, tokens, E.Rows.ALL, False)], E.StepOptions(read_logits=True))
        got.append((out.logits, [vlt.from_bf16(eng.debug_read(c).view(np.uint16)) for c in ("k_cache", "v_cache")]))
        eng.close()
    (logits0, caches0), (logits1, caches1) = got
    for c0, c1 in zip(caches0, caches1):
        assert np.abs(c0).max() > 0.5 and (np.abs(c0 - c1) <= 2.0 ** -7 * np.abs(c0) + 1e-4).all()
    assert float(np.abs(logits0 - logits1).max()) <= TOL[int8_group]
