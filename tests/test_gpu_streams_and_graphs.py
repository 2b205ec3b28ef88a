"""What a call shares with other calls: scratch on two streams, and the memory a captured graph writes into."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from test_gpu_parity import device_weight, make_case, to_dev  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def S():
    import skyrl_tx_rocm_b200 as S

    return S


def _block(S, seed, m, hidden, inter, rank=8, na=3):
    x, wgu, ga, gb, s, ids = make_case(seed, m, hidden, 2 * inter, rank, na, w_std=0.05)
    _, wd, da, db, _, _ = make_case(seed + 1, m, inter, hidden, rank, na, w_std=0.05)
    (_, pgu), (_, pd) = device_weight(S, wgu), device_weight(S, wd)
    lgu = S.pack_lora(to_dev(ga), to_dev(gb), to_dev(s), in_features=hidden, padded_out_features=2 * inter)
    ld = S.pack_lora(to_dev(da), to_dev(db), to_dev(s), in_features=inter, padded_out_features=hidden)
    return to_dev(x), to_dev(ids), (None, pgu, lgu, pd, ld)


def _block_call(S, seed):
    x, ids, parts = _block(S, seed, 1500, 512, 1536)
    return lambda: S.w8a8_mlp_block(x, *parts, ids, enabled=True)


def _linear_call(S, seed):
    x, ids, (_, pgu, lgu, _, _) = _block(S, seed, 1500, 512, 1536)
    return lambda: S.w8a8_lora_linear(x, pgu, lgu, adapter_ids=ids, enabled=True)


@pytest.mark.parametrize("make", [_block_call, _linear_call])
def test_calls_on_two_streams_do_not_share_scratch(S, make):
    calls = [make(S, 3), make(S, 30)]
    want = [c() for c in calls]
    streams = [torch.cuda.Stream() for _ in calls]
    got = [None, None]
    torch.cuda.synchronize()
    for _ in range(10):
        for i, c in enumerate(calls):
            with torch.cuda.stream(streams[i]):
                got[i] = c()
    torch.cuda.synchronize()
    assert all(torch.equal(g, w) for g, w in zip(got, want))
    S.check_status()


def test_a_chunked_stack_keeps_its_workspace_over_its_streams(S):
    from skyrl_tx_rocm_b200.stack import MLPStack

    x, ids, parts = _block(S, 5, 2304, 256, 512)
    want = MLPStack([parts] * 2, num_chunks=1)(x, ids).clone()
    stack = MLPStack([parts] * 2, num_chunks=2)
    stack(x, ids)
    with torch.cuda.stream(stack._side):     # the side stream now has a buffer of its own
        S.w8a8_mlp_block(x, *parts, ids, enabled=True)
    torch.cuda.synchronize()
    for _ in range(3):
        assert torch.equal(stack(x, ids), want)
    S.check_status()


@pytest.mark.parametrize("m", [64, 300])
def test_a_captured_step_owns_the_memory_it_writes(S, m):
    """A larger call after the capture makes the operators take larger buffers: the graph must not go on writing into
    what they gave back."""
    from skyrl_tx_rocm_b200.stack import MLPStack

    x, ids, parts = _block(S, 7, m, 256, 512)
    stack = MLPStack([parts] * 3, num_chunks=1)
    big_x, big_ids, big_parts = _block(S, 9, 4096, 256, 512)
    want = stack(x, ids).clone()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        stack(x, ids)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = stack(x, ids)
    for stream in (torch.cuda.current_stream(), side):
        with torch.cuda.stream(stream):
            S.w8a8_mlp_block(big_x, *big_parts, big_ids, enabled=True)
    torch.cuda.synchronize()
    fill = [torch.full((1 << 18,), 0x5a, dtype=torch.uint8, device="cuda") for _ in range(400)]   # reuses what was given back
    torch.cuda.synchronize()
    for _ in range(2):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    assert all(int((f != 0x5a).sum()) == 0 for f in fill)
    S.check_status()


def test_two_captures_do_not_share_a_workspace(S):
    x, ids, parts = _block(S, 11, 300, 256, 512)
    graphs, outs = [torch.cuda.CUDAGraph() for _ in range(2)], []
    want = S.w8a8_mlp_block(x, *parts, ids, enabled=True)
    for g in graphs:
        with torch.cuda.graph(g):
            first = S.w8a8_mlp_block(x, *parts, ids, enabled=True)
            second = S.w8a8_mlp_block(x, *parts, ids, enabled=True, reuse_routing=True)
        outs.append((first, second))
    del graphs[0], outs[0], g     # the first graph's memory goes with it
    torch.cuda.empty_cache()
    fill = torch.full((64 << 20,), 0x5a, dtype=torch.uint8, device="cuda")
    for _ in range(2):
        graphs[0].replay()
        torch.cuda.synchronize()
        assert all(torch.equal(o, want) for o in outs[0])
    assert int((fill != 0x5a).sum()) == 0
    S.check_status()


def test_a_captured_stack_owns_its_activations(S):
    """A forward of another shape replaces the stack's buffers; the graph must not go on writing into the old ones."""
    from skyrl_tx_rocm_b200.stack import MLPStack

    x, ids, parts = _block(S, 13, 64, 1024, 512)
    stack = MLPStack([parts] * 3, num_chunks=1)
    want = stack(x, ids).clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = stack(x, ids)
    stack(x[:16].contiguous(), ids[:16].contiguous())
    torch.cuda.synchronize()
    fill = [torch.full(x.shape, 3.0, dtype=torch.bfloat16, device="cuda") for _ in range(200)]
    for _ in range(2):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    assert all(bool((f == 3.0).all()) for f in fill)
    S.check_status()
