"""The stand-alone acceptance step (`spec_accept_static`) bit for bit against the oracle at the sizes where its kernels take
another path: rows of whole groups of 8 ids on 16-byte boundaries (asynchronous copies) and others, a last portion of every
length, fewer ids than a block's share, and rows too long for shared memory; drafts outside the vocabulary; on a graph."""
import numpy as np
import pytest

import oracle
from silicon_violetto_b200 import build, engine as E
from tests.test_zz_no_alloc import _case, _static

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    build.build()


@pytest.mark.parametrize("streams,k,vocab", [
    (1, 1, 8), (2, 3, 1), (3, 4, 130), (2, 2, 1024), (2, 2, 1032), (1, 4, 2047), (2, 5, 8192), (1, 15, 9001), (2, 4, 128256), (1, 2, 409600), (1, 2, 409608), (1, 1, 411003)])
def test_decisions_at_odd_sizes_are_the_oracles(streams, k, vocab):
    import torch
    pb, qb, drafts, seeds, pos0 = _case(streams, k, vocab, 17 + vocab, 0.7)
    got = _static(torch, pb, qb, drafts, 0.7, seeds, pos0)
    assert np.array_equal(got, np.stack(oracle.spec_accept(pb, qb, drafts, 0.7, seeds, pos0)))


def test_a_misaligned_row_and_rows_of_one_value_and_of_infinities():
    """p starts two bytes off a 16-byte boundary; a row all equal, and one with -inf (masked ids) and a single finite id."""
    import torch
    streams, k, vocab = 2, 3, 4096
    pb, qb, drafts, seeds, pos0 = _case(streams, k, vocab, 5, 1.0)
    pb[0, 0], qb[0, 0] = 0x3F80, 0x3F80
    pb[1, 1] = 0xFF80
    pb[1, 1, 77] = 0x4000
    qb[1, 1, 1000:] = 0xFF80
    drafts = oracle.draw_drafts(qb, 1.0, seeds, pos0)
    want = np.stack(oracle.spec_accept(pb, qb, drafts, 1.0, seeds, pos0))
    dev = lambda a, t: torch.from_numpy(np.ascontiguousarray(a).view(t)).cuda()  # noqa: E731
    p = torch.empty(pb.size + 1, dtype=torch.int16, device="cuda")
    p[1:] = dev(pb, np.int16).reshape(-1)
    q, d, s, o = dev(qb, np.int16), dev(drafts.astype(np.uint32), np.int32), dev(seeds, np.int64), dev(pos0, np.int32)
    out = torch.full((3, streams), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    E.spec_accept_static(p.data_ptr() + 2, q.data_ptr(), d.data_ptr(), streams, k, vocab, 1.0, s.data_ptr(), o.data_ptr(), out[0].data_ptr(), out[1].data_ptr(),
                         out[2].data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert np.array_equal(out.cpu().numpy().view(np.uint32), want)


def test_drafts_past_the_vocabulary_are_read_as_0_and_outputs_may_replace_the_drafts():
    import torch
    streams, k, vocab = 4, 1, 2000
    pb, qb, drafts, seeds, pos0 = _case(streams, k, vocab, 9, 1.0)
    drafts[1], drafts[3] = vocab, 0xFFFFFFFF
    want = np.stack(oracle.spec_accept(pb, qb, np.where(drafts < vocab, drafts, 0), 1.0, seeds, pos0))
    dev = lambda a, t: torch.from_numpy(np.ascontiguousarray(a).view(t)).cuda()  # noqa: E731
    p, q, d, s, o = dev(pb, np.int16), dev(qb, np.int16), dev(drafts.astype(np.uint32), np.int32), dev(seeds, np.int64), dev(pos0, np.int32)
    out = torch.full((2, streams), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    E.spec_accept_static(p.data_ptr(), q.data_ptr(), d.data_ptr(), streams, k, vocab, 1.0, s.data_ptr(), o.data_ptr(), out[0].data_ptr(), d.data_ptr(), out[1].data_ptr(),
                         torch.cuda.current_stream().cuda_stream)
    assert np.array_equal(np.stack([out[0].cpu().numpy(), d.reshape(-1).cpu().numpy(), out[1].cpu().numpy()]).view(np.uint32), want)


def test_the_step_is_captured_on_a_graph_and_replayed_on_new_inputs():
    import torch
    streams, k, vocab = 3, 4, 5000
    cases = [_case(streams, k, vocab, seed, 0.8) for seed in (1, 2)]
    dev = lambda a, t: torch.from_numpy(np.ascontiguousarray(a).view(t)).cuda()  # noqa: E731
    tensors = [[dev(a, t) for a, t in zip((c[0], c[1], c[2].astype(np.uint32), c[3], c[4]), (np.int16, np.int16, np.int32, np.int64, np.int32))] for c in cases]
    live = [t.clone() for t in tensors[0]]
    out = torch.full((3, streams), -1, dtype=torch.int32, device="cuda")
    call = lambda: E.spec_accept_static(*[t.data_ptr() for t in live[:3]], streams, k, vocab, 0.8, live[3].data_ptr(), live[4].data_ptr(), out[0].data_ptr(), out[1].data_ptr(),  # noqa: E731
                                        out[2].data_ptr(), torch.cuda.current_stream().cuda_stream)
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call()
    for c, ts in zip(cases[::-1], tensors[::-1]):
        for a, b in zip(live, ts):
            a.copy_(b)
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy().view(np.uint32), np.stack(oracle.spec_accept(c[0], c[1], c[2], 0.8, c[3], c[4])))
