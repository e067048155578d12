"""Passes whose intermediates nobody looks at (autograd's default path: attention without score tensors, activations in
their logical order, act' in a contraction's epilogue) against passes that keep every intermediate, same inputs and masks.

The two round differently, not more: the keeping pass rounds the scores, ALPHA and DATTN_DROP to 16 bits between its
operators, the other one the unnormalised exponentials and the row sum's GAMMA.  Each is a relative error of half a unit
(2^-11, bf16 2^-8) per tensor on the path, a handful of them in a row: 8 half-units is the bound used (GELU: no
derivative jumps)."""

import ctypes

import pytest
import torch

from substation_b200 import Encoder, layouts as L, _lib
from tests.layer_harness import run_private_case, uniform_or_feature_major

pytestmark = pytest.mark.gpu
HALF = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}


def _passes(B, S, H, dtype, p, mode, lay, seed, activation='gelu'):
    dev, E = torch.device('cuda:0'), 64 * H
    table = L.validate(lay)
    gen = torch.Generator(device=dev).manual_seed(seed)
    sizes = L.sizes_map(B, S, H, E)
    x0 = torch.randn(L.shape_of(table['X'], sizes), device=dev, generator=gen).to(dtype)
    dy = torch.randn(x0.shape, device=dev, generator=gen).to(dtype)
    masks = {n: (torch.rand(L.shape_of(table[n], sizes), device=dev, generator=gen) >= p).to(torch.uint8) for n in L.MASKS}
    state, out = None, []
    for keep in (True, False):
        enc = Encoder('', B, S, H, E, lay, dtype, p, p, p, p, activation=activation, mask_mode=mode, seed=5,
                      keep_all_intermediates=keep).to(dev)
        with torch.no_grad():
            if state is None:
                # unit-variance projections: the keeping pass rounds the scores to 16 bits, an error in ALPHA of half a unit
                # times the score, which the bound above counts once only because scores stay of order one
                for q in enc.params:
                    q.copy_((torch.randn(q.shape, device=dev, generator=gen) * (1.1 / E ** 0.5)).to(dtype))
                enc.S1.fill_(1)
                enc.S2.fill_(1)
                state = enc.state_dict()
            else:
                enc.load_state_dict(state)
        if mode == 'explicit':
            enc.set_masks(masks)
        assert (enc.private_arena_bytes(dev) is None) == keep
        x = x0.clone().requires_grad_(True)
        y = enc(x)
        y.backward(dy)
        got = {'Y': y.detach(), 'DX': x.grad, **{n: q.grad for n, q in zip(enc._param_names, enc.params)}}
        enc.philox_offset = 0
        with torch.no_grad():                                # nothing is kept for a backward pass here
            got['Y of inference'] = enc(x0)
        out.append(got)
        err = ctypes.c_int(0)
        lib = _lib.load(_lib.dtype_key(dtype))
        _lib.check(lib.sb_device_error(None, ctypes.byref(err)), lib)
        assert err.value == 0
    return out


@pytest.mark.parametrize('B,S,H,dtype,p,mode,layouts', [
    (1, 128, 2, torch.float16, 0.0, 'philox', 'uniform'),            # one tile, nothing dropped
    (2, 16, 8, torch.float16, 0.1, 'philox', 'uniform'),             # rows shorter than a copy box
    (3, 77, 4, torch.float16, 0.1, 'philox', 'uniform'),             # rows off the 16-byte grid: padded copies
    (3, 77, 4, torch.float16, 0.1, 'explicit', 'uniform'),
    (2, 130, 4, torch.float16, 0.1, 'explicit', 'uniform'),          # two columns in the second tile
    (2, 136, 4, torch.bfloat16, 0.1, 'philox', 'uniform'),
    (2, 512, 4, torch.float16, 0.1, 'explicit', 'uniform'),
    (1, 1000, 2, torch.float16, 0.6, 'philox', 'uniform'),           # threshold with its top bit set, eight tiles
    (40, 256, 4, torch.float16, 0.1, 'philox', 'uniform'),           # more items than a round of the machine
    (160, 72, 2, torch.bfloat16, 0.1, 'philox', 'uniform'),
    (5, 512, 8, torch.float16, 0.1, 'philox', 'feature_major'),      # activations change order on the way in and out
    (3, 77, 4, torch.float16, 0.1, 'philox', 'feature_major'),
    (2, 256, 4, torch.float16, 0.1, 'explicit', 'feature_major'),    # the caller's masks keep their order
])
def test_private_passes_match_passes_that_keep_everything(B, S, H, dtype, p, mode, layouts):
    kept, private = _passes(B, S, H, dtype, p, mode, uniform_or_feature_major(layouts), seed=B * 1000 + S)
    for name, want in kept.items():
        got = private[name]
        assert torch.isfinite(got).all(), name
        err = ((got.double() - want.double()).norm() / want.double().norm()).item()
        assert err <= 8 * HALF[dtype], (name, err)


@pytest.mark.parametrize('B,S,H,mode', [(1, 2048, 4, 'philox'), (3, 1920, 4, 'philox'), (1, 2000, 8, 'explicit')])
def test_long_streams_of_key_tiles(B, S, H, mode):
    """dQ items over 15 and 16 key tiles: element warps and product warp hand the two 16-bit tiles over in turn, with nothing
    but the barriers to keep one from running ahead of the other (a stall would end in the wait limit and be reported)."""
    kept, private = _passes(B, S, H, torch.float16, 0.1, mode, L.uniform_layouts(), seed=S)
    for name, want in kept.items():
        err = ((private[name].double() - want.double()).norm() / want.double().norm()).item()
        assert err <= 8 * HALF[torch.float16], (name, err)


@pytest.mark.parametrize('B,S,H,dtype,activation,mode,layouts', [
    (2, 128, 4, torch.float16, 'relu', 'philox', 'uniform'),         # split-K clusters with bias, activation, dropout
    (1, 77, 8, torch.float16, 'gelu', 'explicit', 'uniform'),
    (2, 64, 4, torch.bfloat16, 'relu', 'explicit', 'uniform'),
    (16, 77, 8, torch.float16, 'relu', 'philox', 'uniform'),         # the activation's backward in dXlin2's epilogue over
    (16, 77, 8, torch.bfloat16, 'relu', 'philox', 'uniform'),        # 1232 tokens: a last tile with 208 of 256 rows, the
    (16, 77, 8, torch.float16, 'gelu', 'explicit', 'uniform'),       # last block of 32 with 16
    (12, 200, 12, torch.bfloat16, 'gelu', 'philox', 'uniform'),
    (5, 100, 16, torch.float16, 'relu', 'philox', 'feature_major'),  # other orders and padded rows
    (4, 512, 16, torch.float16, 'relu', 'explicit', 'uniform'),
    (8, 128, 4, torch.float16, 'relu', 'philox', 'uniform'),         # the last token count with two sweeps over the keys,
    (8, 128, 4, torch.float16, 'gelu', 'philox', 'uniform'),
    (1, 1025, 4, torch.float16, 'relu', 'philox', 'uniform'),        # and the first with one
])
def test_default_path_against_the_oracle(B, S, H, dtype, activation, mode, layouts):
    enc, dlin1 = run_private_case(B, S, H, layouts=layouts, activation=activation, mask_mode=mode, seed=S, dtype=dtype,
                                  tol=1e-2 if dtype == torch.float16 else 5e-2)
    # LINB1's gradient is the column sums of DLIN1 as stored: fp32 sums, one rounding to 16 bits
    got, want = enc.LINB1.grad.double().cpu(), torch.from_numpy(dlin1).sum((0, 1))
    assert ((got - want).norm() / want.norm()).item() <= HALF[dtype] + 1e-5
    lib = _lib.load(_lib.dtype_key(dtype))
    _lib.check(lib.sb_encoder_set_timing(enc._handle, 1), lib)
    x = torch.zeros(L.shape_of(enc._table['X'], enc.sizes), device='cuda:0', dtype=dtype, requires_grad=True)
    enc(x).sum().backward()
    names = [n for n, _ in enc.op_times()]
    assert ('dXlin2+bdrlb' in names) == (B * S >= 1232), names


def test_private_passes_with_projections_stored_unit_by_unit():
    """KKQQVV as QHBPJ (the order shipped for B=96, L=128 with the original module)."""
    lay = L.uniform_layouts()
    lay['forward_interm'] = [(n, 'QHBPJ' if n == 'KKQQVV' else d) for n, d in lay['forward_interm']]
    kept, private = _passes(2, 256, 4, torch.float16, 0.1, 'philox', lay, seed=3)
    for name, want in kept.items():
        err = ((private[name].double() - want.double()).norm() / want.double().norm()).item()
        assert err <= 8 * HALF[torch.float16], (name, err)


@pytest.mark.parametrize('B,activation', [(1, 'relu'), (1, 'gelu'), (4, 'gelu')])
def test_row_maxima_that_rise_by_more_than_the_lag(B, activation):
    """Scores that grow along the keys by far more than 2^8 per tile: every tile raises the reference maximum and
    rescales what has been summed so far (keys scaled up with their position).  ReLU layers sweep the keys of 512 tokens
    twice, the others once (with ReLU only outputs are compared: rounding decides about whole elements behind its step)."""
    dev, S, H = torch.device('cuda:0'), 512, 2
    E = 64 * H
    enc = Encoder('', B, S, H, E, L.uniform_layouts(), torch.float16, 0., 0., 0., 0., activation=activation).to(dev)
    ref = Encoder('', B, S, H, E, L.uniform_layouts(), torch.float16, 0., 0., 0., 0., activation=activation,
                  keep_all_intermediates=True).to(dev)
    gen = torch.Generator(device=dev).manual_seed(1)
    with torch.no_grad():
        for n, q in zip(enc._param_names, enc.params):
            q.copy_((torch.randn(q.shape, device=dev, generator=gen) * (0.25 if n == 'WKQV' else 0.05)).half())
        enc.S1.fill_(1)
        enc.S2.fill_(1)
    ref.load_state_dict(enc.state_dict())
    x = torch.randn(B, S, E, device=dev, generator=gen) * torch.linspace(0.2, 3, S, device=dev)[None, :, None]
    outs = []
    for e in (ref, enc):
        xi = x.half().requires_grad_(True)
        y = e(xi)
        y.backward(torch.ones_like(y) * torch.linspace(-1, 1, E, device=dev).half())
        outs.append([y.detach(), xi.grad] + [q.grad for q in e.params])
    for a, b in list(zip(*outs))[:1 if activation == 'relu' else None]:
        assert torch.isfinite(b).all()
        # the keeping pass rounds scores of up to ~100 to 16 bits before exponentiating: errors of 2^-5 in ALPHA
        assert ((a.double() - b.double()).norm() / a.double().norm()).item() <= 2.0 ** -5


@pytest.mark.parametrize('B,S,H,dtype,mode', [
    (1, 19, 2, torch.float16, 'philox'),                             # all token counts off the 8 grid: rows of the
    (1, 77, 8, torch.float16, 'explicit'),                           # head-first tensors are padded to it
    (1, 130, 8, torch.bfloat16, 'philox'),
    (5, 100, 16, torch.float16, 'philox'),
    (3, 333, 8, torch.float16, 'philox'),
])
def test_token_counts_off_the_vector_grid(B, S, H, dtype, mode):
    for layouts in ('uniform', 'feature_major'):
        kept, private = _passes(B, S, H, dtype, 0.1, mode, uniform_or_feature_major(layouts), seed=S)
        for name, want in kept.items():
            err = ((private[name].double() - want.double()).norm() / want.double().norm()).item()
            assert torch.isfinite(private[name]).all() and err <= 8 * HALF[dtype], (layouts, name, err)


@pytest.mark.parametrize('M,N,K', [(128, 64, 256), (1, 1024, 512), (77, 1024, 1000), (256, 3072, 1024), (130, 520, 320),
                                   (200, 72, 4096), (1024, 77, 1024)])
def test_split_k_clusters(M, N, K):
    """Contractions with a side of at most 256 against float64: edges of the 128 x 64 tile, K that does not divide among
    the CTAs, both majors of both operands.  Bound: half a unit of the 16-bit result plus fp32 sums of K products."""
    from substation_b200 import ops
    dev = torch.device('cuda:0')
    gen = torch.Generator(device=dev).manual_seed(M + N + K)
    for am in (False, True):
        for bm in (False, True):
            a = torch.randn((K, M) if am else (M, K), device=dev, generator=gen).half()
            b = torch.randn((K, N) if bm else (N, K), device=dev, generator=gen).half()
            c = torch.zeros(M, N, device=dev, dtype=torch.float16)
            ops.einsum(('km' if am else 'mk') + ',' + ('kn' if bm else 'nk') + '->mn', a, b, c)
            want = (a.T if am else a).double() @ (b if bm else b.T).double()
            err = ((c.double() - want).norm() / want.norm()).item()
            assert err <= 2.0 ** -11 + K ** 0.5 * 2.0 ** -23, (am, bm, err)


@pytest.mark.parametrize('B,S,layouts', [(2, 128, 'uniform'), (3, 77, 'uniform'), (2, 128, 'feature_major')])
def test_private_passes_are_timed_operator_by_operator(B, S, layouts):
    """``sb_encoder_set_timing`` covers private passes, also those that run in other orders or with padded rows."""
    dev, H = torch.device('cuda:0'), 8                       # wide enough for the fused contractions of few tokens
    lay = uniform_or_feature_major(layouts)
    enc = Encoder('', B, S, H, 64 * H, lay, torch.float16, 0.1, 0.1, 0.1, 0.1).to(dev)
    nf, nb = enc.private_arena_bytes(dev)
    lib = _lib.load()
    _lib.check(lib.sb_encoder_set_timing(enc._handle, 1), lib)
    arena, barena, garena = (torch.empty(n, dtype=torch.uint8, device=dev) for n in (nf, nb, enc.arena_bytes('grads')))
    x = torch.randn(L.shape_of(L.validate(lay)['X'], enc.sizes), device=dev).half()
    y, dx, weights = torch.empty_like(x), torch.empty_like(x), [p.detach() for p in enc.params]
    changes = ['relayout'] if layouts == 'feature_major' else []
    for _ in range(2):
        enc.forward_private(x, weights, arena, y)
        assert enc.launch_count() == 7
        enc.backward_private(y, enc.views('grads', garena), barena, weights, arena, x, dx)
        names, ms = zip(*enc.op_times())
        assert all(t > 0 for t in ms)
        for part in (['QKV-fused+aib', 'attention', 'out', 'bdrln1', 'lin1+bad', 'lin2', 'bdrln2'],
                     ['bsb+blnrd1', 'attention-backward', 'dWQKV-fused']):
            assert [n for n in names if n in part] == part, names
        assert list(names[:1] + names[-1:]) == changes * 2 or not changes and 'relayout' not in names
        assert names.count('relayout') == 4 * len(changes)


def test_attention_forward_stays_within_the_sm_budget(tmp_path):
    """Two CTAs per SM of the whole device, one per SM of a budget: never on more SMs than the library may use."""
    import json
    from substation_b200 import ops
    dev, B, S, H = torch.device('cuda:0'), 8, 512, 16
    sms = torch.cuda.get_device_properties(dev).multi_processor_count
    enc = Encoder('', B, S, H, 64 * H, L.uniform_layouts(), torch.float16, 0.1, 0.1, 0.1, 0.1).to(dev)
    enc.set_graphs(False)
    x = torch.randn(B, S, 64 * H, device=dev).half()
    grids = []
    try:
        for budget in (0, 100):
            ops.set_sm_budget(budget)
            with torch.no_grad(), torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
                enc(x)
                torch.cuda.synchronize()
            path = tmp_path / f'{budget}.json'
            prof.export_chrome_trace(str(path))
            grids += [e['args']['grid'][0] for e in json.load(open(path))['traceEvents'] if 'flash_fwd_kernel' in e.get('name', '')]
    finally:
        ops.set_sm_budget(0)
    assert grids == [2 * sms, 100]


@pytest.mark.parametrize('keep', [True, False])
def test_rows_beyond_2048_are_refused_with_and_without_score_tensors(keep):
    dev, S = torch.device('cuda:0'), 2056
    enc = Encoder('', 1, S, 1, 64, L.uniform_layouts(), torch.float16, 0., 0., 0., 0., keep_all_intermediates=keep).to(dev)
    assert enc.private_arena_bytes(dev) is None
    with pytest.raises(_lib.SubstationError, match='2048'):
        enc(torch.zeros(1, S, 64, device=dev).half())


def _stack(layers):
    from substation_b200.stack import EncoderStack
    st = EncoderStack(layers, 2, 128, 2, 128, L.uniform_layouts(), dropout_p=0.1, device='cuda:0', seed=5, activation='gelu',
                      weight_std=0.1)
    gen = torch.Generator(device='cuda:0').manual_seed(4)
    return st, *(torch.randn(2, 128, 128, device='cuda:0', generator=gen).half() for _ in range(2))


def test_stack_shows_the_intermediates_of_its_last_pass_when_asked():
    """``fwd`` and ``bwd`` of a stack hold every named intermediate, also those of a pass that had kept none: same bits as a
    raw pass over the same input, masks included; later passes keep them as they go."""
    st, x, dy = _stack(1)
    enc = st.layers[0]
    st.forward(x)
    st.backward(dy)
    st.wait_gradients()
    fwd = enc.views('forward', torch.zeros(enc.arena_bytes('forward'), dtype=torch.uint8, device=x.device))
    bwd = enc.views('backward', torch.zeros(enc.arena_bytes('backward'), dtype=torch.uint8, device=x.device))
    grads = enc.views('grads', torch.zeros(enc.arena_bytes('grads'), dtype=torch.uint8, device=x.device))
    dead = ('BETA', 'WKKWQQWVV', 'SB1_LINW1', 'LIN2', 'DATTN_DROP', 'DLN2', 'DLN1', 'DXATT')
    for step in range(2):
        enc.philox_offset = 4 * step
        enc.forward_raw(x, st.weights[0], fwd, torch.empty_like(x))
        enc.backward_raw(dy, grads, bwd, st.weights[0], fwd, x, torch.empty_like(x))
        for got, want in ((st.fwd[0], fwd), (st.bwd, bwd)):
            assert set(got) == set(want)
            assert all(torch.equal(got[n], want[n]) for n in want if n not in dead + ('__arena__',))
        assert enc.philox_offset == 4 * step + 4
        st.forward(x)
        st.backward(dy)
        enc.philox_offset = 4 * step + 4
    st, x, dy = _stack(2)
    st.forward(x)
    with torch.no_grad():
        st.layers[1].params[0].add_(1)
    with pytest.raises(RuntimeError, match='weights changed'):
        st.fwd


@pytest.mark.parametrize('when', ['before', 'between'])
def test_stack_runs_on_when_a_layer_is_switched_to_debug(when):
    st, x, dy = _stack(3)
    ref, _, _ = _stack(3)
    y, dx = ref.forward(x), ref.backward(dy)
    if when == 'before':
        st.layers[1].enable_debug = True
    got_y = st.forward(x)
    st.layers[1].enable_debug = True
    got_dx = st.backward(dy)
    st.wait_gradients()
    for a, b in ((got_y, y), (got_dx, dx), (st.grads[1]['LINB1'], ref.grads[1]['LINB1'])):
        assert ((a.double() - b.double()).norm() / b.double().norm()).item() <= 3 * 8 * HALF[torch.float16]
