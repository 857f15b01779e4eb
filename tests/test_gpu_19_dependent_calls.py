"""Calls behind one another on a stream with nothing synchronised in between, eager and in a graph.

The kernels are programmatic dependents (csrc/pdl.cuh): each may start before the one in front of it has ended.  So every
call here changes what the one in front of it still reads (cache cells, partials in the workspace, queries) or
reads what that one still writes, with other values each time, and has to give the bytes that it gives when the device
is idle before each call.
"""
import numpy as np
import pytest
import torch

from pth_flash_attn_b200 import capi, host, ops, planner

pytestmark = pytest.mark.gpu

INPUTS = 5
# D, Hq, Hkv, query lengths, keys in front of them, kind of reservation: every kernel, with and without pieces
SHAPES = {
    "decode": (128, 8, 2, [1] * 6, [2999, 40, 700, 5000, 0, 130], "decode"),
    "decode_d64": (64, 16, 2, [1] * 4, [4000, 63, 900, 128], "decode"),
    "decode_d256": (256, 12, 2, [1] * 3, [3000, 500, 64], "decode"),
    "verify": (128, 32, 8, [4, 4, 3], [2000, 100, 0], "decode"),
    "drafter": (128, 16, 4, [16, 16, 12], [3000, 500, 0], "decode"),
    "pair_pieces": (128, 32, 8, [1, 1, 90, 1, 200], [6000, 50, 400, 10, 0], "mixed"),
    "pair_whole": (128, 32, 8, [1, 1, 90, 1, 200], [6000, 50, 400, 10, 0], "prefill"),
    "pair_d64": (64, 8, 2, [1, 70, 1], [3000, 300, 100], "mixed"),
    "pair_d256": (256, 12, 2, [1, 50, 2], [2000, 0, 300], "mixed"),
    "cluster": (128, 8, 1, [30], [4000], "prefill"),
}


class Layer:
    """A cache, a plan, and INPUTS sets of queries, keys and values for it."""

    def __init__(self, D, Hq, Hkv, qlens, priors, kind):
        gen = torch.Generator(device="cuda").manual_seed(D + Hq + len(qlens))
        lens = [q + p for q, p in zip(qlens, priors)]
        pages = [-(-n // 16) for n in lens]
        storage = torch.zeros((sum(pages), 16, Hkv, 2 * D + 8), dtype=torch.uint8, device="cuda")
        cells, words = storage.view(torch.int8), storage.view(torch.float32)
        streams = (cells[..., :D], cells[..., D + 4:2 * D + 4], words[..., D // 4], words[..., D // 2 + 1])
        self.views = host.CacheViews.from_tensors(*streams)
        table = torch.zeros((len(lens), max(pages)), dtype=torch.int32)
        slots, first = [], 0
        for r, n in enumerate(pages):
            table[r, :n] = torch.arange(first, first + n)
            slots.append(torch.arange(first * 16, first * 16 + lens[r]))
            first += n
        self.slots = torch.cat(slots).cuda()
        T, N = sum(qlens), sum(lens)
        ws = {"decode": planner.workspace_token_splits(max_num_seqs=len(lens), q_dec_max=max(qlens), Hkv=Hkv, D=D, num_sms=148),
              "mixed": 8 * T, "prefill": 0}[kind]
        plan = planner.plan_launch(num_tokens=T, num_reqs=len(lens), max_query_len=max(qlens), G=Hq // Hkv, Hkv=Hkv, D=D,
                                   num_sms=148, is_prefill=kind != "decode", ws_token_splits=ws)
        self.q = [torch.randn((T, Hq, D), generator=gen, device="cuda").to(torch.bfloat16) for _ in range(INPUTS)]
        self.kv = [torch.randn((2, N, Hkv, D), generator=gen, device="cuda").to(torch.bfloat16) for _ in range(INPUTS)]
        self.q_now = self.q[0].clone()
        starts = torch.tensor(np.concatenate([[0], np.cumsum(qlens)]), dtype=torch.int32, device="cuda")
        self.rest = (*streams, table.cuda(), torch.tensor(lens, dtype=torch.int32, device="cuda"), starts, max(qlens), plan.wm,
                     plan.num_splits, D ** -0.5, torch.full(plan.ws_o_shape, float("nan"), device="cuda"),
                     torch.full(plan.ws_lse_shape, float("nan"), device="cuda"))
        self.storage = storage

    def write(self, i):
        host.write_kv(self.kv[i][0], self.kv[i][1], self.views, self.slots)

    def attend(self, q, out):
        ops.pth_flash_attn_fwd(out, q, *self.rest)

    def result(self):
        return torch.full_like(self.q[0], float("nan"))


def _alone(layer, step, count=INPUTS):
    want = []
    for i in range(count):
        torch.cuda.synchronize()
        out = layer.result()
        step(i, out)
        torch.cuda.synchronize()
        want.append(out)
    assert all(not torch.equal(a, b) and a.isfinite().all() for a, b in zip(want, want[1:]))
    return want


def _check(layer, step, order, captured, repeats):
    """step(i, out) for every i of the order behind one another: the bytes of step(i, out) on an idle device."""
    want = _alone(layer, step)
    outs = [layer.result() for _ in order]

    def chain():
        for i, out in zip(order, outs):
            step(i, out)
    if captured:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            chain()
    differing = torch.zeros((), dtype=torch.int32, device="cuda")
    for _ in range(repeats):
        for out in outs:
            out.fill_(float("nan"))
        graph.replay() if captured else chain()
        for i, out in zip(order, outs):
            differing += (out.view(torch.int16) != want[i].view(torch.int16)).any().to(torch.int32)
    assert int(differing) == 0, f"{int(differing)} of {repeats * len(order)} calls differ"
    assert capi.load_library().device_status() == 0


ORDER = [0, 3, 1, 4, 2, 1, 0, 2, 4, 3, 0, 1, 2, 3, 4] * 2


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_the_writer_and_the_op_on_the_same_cells(shape, captured):
    layer = Layer(*SHAPES[shape])

    def step(i, out):
        layer.write(i)
        layer.attend(layer.q[i], out)
    _check(layer, step, ORDER, captured, repeats=20)


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_calls_over_one_workspace(shape, captured):
    layer = Layer(*SHAPES[shape])
    layer.write(0)
    _check(layer, lambda i, out: layer.attend(layer.q[i], out), ORDER, captured, repeats=20)


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("shape", ["decode", "pair_pieces", "pair_whole", "cluster"])
def test_queries_and_results_of_other_streams(shape, captured):
    """The queries come from a second stream and the result is taken by it, joined by events on both sides."""
    layer = Layer(*SHAPES[shape])
    second = torch.cuda.Stream()
    taken = layer.result()

    def step(i, out):
        main = torch.cuda.current_stream()
        layer.write(i)
        second.wait_stream(main)
        with torch.cuda.stream(second):
            layer.q_now.copy_(layer.q[i])
        main.wait_stream(second)
        layer.attend(layer.q_now, taken)
        second.wait_stream(main)
        with torch.cuda.stream(second):
            out.copy_(taken)
        main.wait_stream(second)
    _check(layer, step, ORDER, captured, repeats=20)
