"""Passes that run as CUDA graphs with rewritten parameters against the same passes launched kernel by kernel."""

import pytest
import torch

from substation_b200 import Encoder, layouts as L, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('mask_mode', ['philox', 'explicit'])
@pytest.mark.parametrize('B,S', [(2, 128), (3, 40)])
def test_rewritten_graphs_match_plain_launches(mask_mode, B, S):
    """New inputs and buffers every pass, inference passes in between, and a switch of the handle that changes which
    kernels a pass launches: same bits as plain launches, every time."""
    dev, lay, E = torch.device('cuda:0'), L.uniform_layouts(), 128
    table = L.validate(lay)
    gen = torch.Generator(device=dev).manual_seed(3)
    encs = [Encoder('', B, S, 2, E, lay, torch.float16, 0.1, 0.1, 0.1, 0.1, mask_mode=mask_mode, seed=7).to(dev)
            for _ in range(2)]
    encs[1].load_state_dict(encs[0].state_dict())
    encs[1].set_graphs(False)
    if mask_mode == 'explicit':
        masks = {n: (torch.rand(L.shape_of(table[n], encs[0].sizes), device=dev, generator=gen) >= 0.1).to(torch.uint8)
                 for n in L.MASKS}
        for e in encs:
            e.set_masks(masks)
    keep = []
    for step in range(9):
        x = torch.randn(B, S, E, device=dev, generator=gen).half()
        dy = torch.randn(B, S, E, device=dev, generator=gen).half()
        if step == 6:
            for e in encs:                              # one kernel per reference operator from here on
                e._check(ops._lib.load().sb_encoder_set_fusion(e._handle, 0))
        got = []
        for e in encs:
            e.zero_grad(set_to_none=True)
            xi = x.clone().requires_grad_(True)
            y = e(xi)
            y.backward(dy)
            got.append([y.detach(), xi.grad] + [p.grad for p in e.params])
            if step % 3 == 2:
                with torch.no_grad():
                    got[-1].append(e(x))
        keep.append(got)                                # nothing is freed: no buffer comes back
        assert all(torch.equal(a, b) for a, b in zip(*got)), step
    captures, runs = encs[0].graph_stats()
    # passes without and with score tensors (before and after the switch) have graphs of their own, two per direction:
    # forward 8 + 4 passes, backward 6 + 3, the first of each kind launched plainly
    assert captures == 2 + 2 + 2 + 1 and runs == 12 + 9 - 4 - captures
    assert encs[1].graph_stats() == (0, 0)
    assert ops.device_error() == 0


def _pair(**kw):
    encs = [Encoder('', 2, 128, 2, 128, L.uniform_layouts(), torch.float16, 0.1, 0.1, 0.1, 0.1, seed=7, **kw).to('cuda:0')
            for _ in range(2)]
    encs[1].load_state_dict(encs[0].state_dict())
    encs[1].set_graphs(False)
    return encs


def test_alternating_mask_modes_keep_their_graphs():
    """A program that uses generated and explicit masks in turn: each mode's passes find their graphs again."""
    encs, dev = _pair(), torch.device('cuda:0')
    table = L.validate(L.uniform_layouts())
    gen = torch.Generator(device=dev).manual_seed(3)
    masks = {n: (torch.rand(L.shape_of(table[n], encs[0].sizes), device=dev, generator=gen) >= 0.1).to(torch.uint8)
             for n in L.MASKS}
    for step in range(24):
        x, dy = (torch.randn(2, 128, 128, device=dev, generator=gen).half() for _ in range(2))
        got = []
        for e in encs:
            e.set_masks(masks)
            e.mask_mode = 'explicit' if step % 3 == 2 else 'philox'
            e.zero_grad(set_to_none=True)
            xi = x.clone().requires_grad_(True)
            y = e(xi)
            y.backward(dy)
            got.append([y.detach(), xi.grad] + [p.grad for p in e.params])
        assert all(torch.equal(a, b) for a, b in zip(*got)), step
    captures, replays = encs[0].graph_stats()
    assert captures == 8 and replays == 2 * 24 - 4 - 8        # two per direction and mode; the first of each runs plainly


def test_passes_that_keep_changing_their_kernels_are_not_captured_each_time():
    encs, dev = _pair(keep_all_intermediates=True), torch.device('cuda:0')
    gen = torch.Generator(device=dev).manual_seed(5)
    steps = 60
    for step in range(steps):
        x = torch.randn(2, 128, 128, device=dev, generator=gen).half()
        got = []
        for e in encs:
            if e._handle is not None:
                e._check(ops._lib.load().sb_encoder_set_fusion(e._handle, int(step * step % 7 < 3)))
            with torch.no_grad():
                got.append(e(x))
        assert torch.equal(*got), step
    captures, replays = encs[0].graph_stats()
    assert replays > 0 and captures <= 5 + steps // 8


def test_one_module_used_by_two_threads():
    """Host calls on one handle take turns: inference from two threads, a stream each, gives what it gives one by one.
    (128 tokens: no operator of these passes uses the handle's workspaces.)"""
    import threading
    dev = torch.device('cuda:0')
    enc = Encoder('', 1, 128, 2, 128, L.uniform_layouts(), torch.float16, 0., 0., 0., 0.).to(dev)
    gen = torch.Generator(device=dev).manual_seed(9)
    xs = [[torch.randn(1, 128, 128, device=dev, generator=gen).half() for _ in range(100)] for _ in range(2)]
    with torch.no_grad():
        want = [[enc(x) for x in part] for part in xs]
    torch.cuda.synchronize()
    got = [[], []]

    def work(i):
        with torch.no_grad(), torch.cuda.stream(torch.cuda.Stream(dev)):
            got[i] += [enc(x) for x in xs[i]]
            torch.cuda.current_stream().synchronize()
    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for part, ref in zip(got, want):
        assert len(part) == len(ref) and all(torch.equal(a, b) for a, b in zip(part, ref))
    assert ops.device_error() == 0
