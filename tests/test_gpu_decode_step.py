"""Steps of at most 8 tokens of a plain decoder as one launch, against the separate kernels (which a tuning knob still asks for):
logits, hidden rows and the K/V cache, over sizes where the launch divides its work differently -- weight rows of less than a
stage, of several, of a part that is not whole, groups of warps that share a row or stay idle, several row tiles and attention
units to a block, contexts around the edges of pages and splits -- and over activations that fp16 does not hold as they are.

Both multiply the same bf16 activations; sums are in another order, and through it a rounding to bf16 (2^-9) falls otherwise now
and then: over two layers the results may differ by a few such roundings' share, 1e-2 in the 2-norm; over 26 layers by 3e-2.
"""
import numpy as np
import pytest

from silicon_violetto_b200 import build, engine as E, synth, vlt

pytestmark = pytest.mark.gpu
BASE = dict(n_layers=2, hd=64, vocab=512, eps=1e-5, theta=500000.0, page=16)
SHAPES = {
    "narrow": dict(BASE, d=256, n_heads=4, n_kv=2, ffn=512),
    "uneven": dict(BASE, d=2304, n_heads=12, n_kv=3, ffn=6144),  # two groups a row and three, parts of 256 bytes
    "wide": dict(BASE, d=4096, n_heads=16, n_kv=8, ffn=8192, n_layers=1),                   # two row tiles a block, four groups a row
}
RUNS = {  # (context, new tokens) per sequence
    "one": [(17, 1)],
    "first": [(0, 8)],
    "drafts": [(700, 5)],
    "mixed": [(16, 1), (0, 2), (131, 4)],
    "eight": [(15, 1), (1, 1), (33, 1), (300, 1), (128, 1), (0, 1), (129, 1), (64, 1)],
}


@pytest.fixture(scope="module", autouse=True)
def built():
    build.build()


@pytest.fixture(scope="module")
def weights(tmp_path_factory):
    made = {}

    def get(shape, int8, std=0.02):
        key = (shape, int8, std)
        if key not in made:
            made[key] = tmp_path_factory.mktemp("w") / "w.vlt"
            synth.write_target(made[key], SHAPES[shape], seed=3, int8_group=0 if int8 else None, std=std)
        return made[key]

    return get


def _engines(path, sms=0):
    cfg = dict(max_seqs=8, max_step_tokens=256, max_chunk=256, global_kv_tokens=4096, max_seq_len=1024, max_head_rows=8)
    return [E.Engine(path, E.EngineConfig(**cfg), E.Tuning(sm_count=sms, attn_keys_per_cta=k)) for k in (0, 128)]


def _ids(n, seed, vocab=512):
    return np.random.default_rng(seed).integers(0, vocab, n).astype(np.uint32)


def _context(eng, n, seed):
    s = eng.new_seq()
    for a in range(0, n, 256):
        eng.step([E.Run(s, _ids(n, seed)[a:a + 256])], E.StepOptions(head=E.Rows.NONE))
    return s


def _near(got, want, bound=1e-2):
    got, want = np.asarray(got, np.float64), np.asarray(want, np.float64)
    assert np.isfinite(got).all()
    assert np.linalg.norm(got - want) <= bound * np.linalg.norm(want)


def _compare(engines, runs, launches=None, bound=1e-2, caches=("k_cache", "v_cache"), **opts):
    opts = E.StepOptions(head=E.Rows.ALL, hidden=E.Rows.ALL, read_logits=True, **opts)
    outs, kept = [], []
    for i, eng in enumerate(engines):
        seqs = [_context(eng, n, 10 + j) for j, (n, _) in enumerate(runs)]
        before = eng.launches()
        outs.append(eng.step([E.Run(s, _ids(k, 50 + j)) for j, (s, (_, k)) in enumerate(zip(seqs, runs))], opts))
        if launches is not None and i == 0:
            assert eng.launches() - before <= launches  # (embedding, the layers and the head, hidden rows, sampling, acceptance)
        kept.append([vlt.from_bf16(eng.debug_read(c).view(np.uint16)) for c in caches])
        for s in seqs:
            eng.free_seq(s)
    _near(outs[0].logits, outs[1].logits, bound)
    _near(outs[0].hidden, outs[1].hidden, bound)
    for a, b in zip(*kept):
        _near(a, b, bound)
    return outs


@pytest.mark.parametrize("runs", RUNS)
@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_the_one_launch_matches_the_separate_kernels(weights, shape, int8, runs):
    _compare(_engines(weights(shape, int8)), RUNS[runs], launches=6)


@pytest.mark.parametrize("sms", [11, 40])
@pytest.mark.parametrize("int8", [False, True])
def test_blocks_with_several_tiles_and_units(weights, int8, sms):
    _compare(_engines(weights("narrow", int8), sms), RUNS["eight"], launches=6)


# Activations below and above what the fp16 words may hold: embeddings of 2e-4; of 50 with feed-forwards of 1e5 (and one key a row: scores
# of 1e8 would pick another key for a rounding).
@pytest.mark.parametrize("std,runs", [(2e-4, RUNS["mixed"]), (50.0, [(0, 1)] * 3)])
def test_activations_that_fp16_does_not_hold(weights, std, runs):
    _compare(_engines(weights("narrow", True, std)), runs, launches=6)


# The two sets of words take turns: steps of all sizes one after the other, among them some of the separate kernels'.
def test_steps_of_changing_sizes(weights):
    engines = _engines(weights("narrow", True))
    streams = [[_context(eng, n, 70 + n) for n in (40, 3, 200)] for eng in engines]
    for i, counts in enumerate([(1, 1, 1), (8,), (3, 2, 3), (1,), (9, 1, 1), (5, 1), (1, 1, 1), (2,)]):
        outs = [eng.step([E.Run(s, _ids(k, 90 + 8 * i + j)) for j, (s, k) in enumerate(zip(seqs, counts))], E.StepOptions(head=E.Rows.LAST, read_logits=True)) for eng, seqs in zip(engines, streams)]
        _near(outs[0].logits, outs[1].logits)


# A tapped layer ends a launch.
def test_taps_between_launches(weights):
    engines = _engines(weights("uneven", True))
    for eng in engines:
        eng.set_taps([0, 1])
    a, b = _compare(engines, RUNS["mixed"], read_taps=True)
    _near(vlt.from_bf16(np.asarray(a.taps, np.uint16)), vlt.from_bf16(np.asarray(b.taps, np.uint16)))


# The reference's own architecture: o, gate_up, down and the next layer's qkv in one launch, up to a MUDD mix (in front of layers 24
# and 47) -- rows of 768 bytes (a stage half full), of a stage and a quarter, and feed-forwards of two parts and a bit.
@pytest.mark.parametrize("hidden,ffn", [(384, 640), (1280, 2112)])
@pytest.mark.parametrize("runs", ["one", "drafts", "mixed", "eight"])
def test_the_reference_architecture(tmp_path, hidden, ffn, runs):
    path = tmp_path / "w.vlt"
    synth.write_limite(path, n_layers=26, hidden=hidden, n_kv=1 if hidden == 384 else 2, ffn=ffn, vocab=512, seed=5)
    cfg = dict(max_seqs=8, max_step_tokens=256, max_chunk=256, global_kv_tokens=8 * 1024, max_seq_len=1024, max_head_rows=8)
    _compare([E.Engine(path, E.EngineConfig(**cfg), E.Tuning(gemm_min_rows=m)) for m in (0, 9)], RUNS[runs], launches=4 * 26 + 12, bound=3e-2, caches=())
