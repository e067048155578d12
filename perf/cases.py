"""The encoder layer's performance cases: what is timed when somebody asks whether a change made the layer faster.

Every case goes through the package's public interface as a program that uses the layer does: ``Encoder`` under
autograd for a training step, ``Encoder`` under ``torch.no_grad`` for inference, ``EncoderStack`` for several layers
without autograd.  Dropout masks come from the kernels (``mask_mode='philox'``, the module's default), buffers from
torch's allocator (also the default).  Heads are 64 wide in every case (H = E/64, as in the BERT family); what varies
is the batch, the sequence length, the width, the storage type, the activation, the direction and the memory layouts.

A case is a dict of plain values:

mode     'train': forward and backward through autograd, input gradient and twelve parameter gradients returned;
         'infer': forward alone, no gradients, no dropout;
         'stack': ``layers`` layers forward and backward through ``EncoderStack``
batch, seq, embed    B, L and E; the feed-forward width is 4*E
dtype    'fp16' or 'bf16' storage (accumulation is fp32 either way)
activation           'relu' or 'gelu'
layouts  'uniform': every tensor token-major with its features innermost; 'feature_major': the dim orders of the
         configuration file shipped for B=8, L=512 with the original module, most activations feature-major
"""

import torch

from substation_b200 import Encoder, layouts as L
from substation_b200.stack import EncoderStack

HEAD = 64
DROPOUT = 0.1
WEIGHT_STD = 0.02
DTYPES = {'fp16': torch.float16, 'bf16': torch.bfloat16}
# dim orders of the configuration shipped for B=8, L=512, where they are not the logical ones
FEATURE_MAJOR = {
    'X': 'IBJ', 'SB2': 'IBJ',
    'DROP1MASK': 'IBJ', 'SB1_LINW1': 'UBJ', 'DROP2': 'UBJ', 'LIN1': 'UBJ', 'DROP2_LINW2': 'IBJ', 'LN2': 'IBJ',
    'LN2STD': 'JB', 'LN2DIFF': 'JBI', 'DROP2MASK': 'UBJ', 'DROP3MASK': 'JBI', 'LN1': 'IBJ', 'LN1DIFF': 'JBI',
    'DLN2': 'IBJ', 'DRESID2': 'IBJ', 'DLIN2': 'IBJ', 'DDROP2': 'UBJ', 'DLIN1': 'UBJ', 'DLIN1_LINW1': 'IBJ',
    'DLN1': 'IBJ', 'DATT': 'IBJ',
}


def _case(name, mode, batch, seq, embed, dtype, activation, layouts='uniform', layers=1):
    c = {'mode': mode, 'batch': batch, 'seq': seq, 'embed': embed, 'dtype': dtype, 'activation': activation,
         'layouts': layouts, 'layers': layers}
    if name:
        c['name'] = name
    return c


def listed():
    return [
        # the headline workload: one BERT-large layer, B=8, L=512
        _case('train_b8_l512', 'train', 8, 512, 1024, 'fp16', 'relu'),
        # the large-batch, short-sequence pre-training phase of the same layer
        _case('train_b96_l128', 'train', 96, 128, 1024, 'fp16', 'relu'),
        # the smallest configuration: a few short sequences (fine-tuning on one example at a time), latency counts
        _case('train_b2_l128', 'train', 2, 128, 1024, 'fp16', 'relu'),
        # bfloat16 and GELU, what most training recipes use now, at a question-answering length
        _case('train_b16_l384_bf16_gelu', 'train', 16, 384, 1024, 'bf16', 'gelu'),
        # a narrower layer with sequences padded to the longest of the batch: no tile size divides 200
        _case('train_b12_l200_e768', 'train', 12, 200, 768, 'bf16', 'gelu'),
        # an odd length (sentence pairs, image patches plus a class token): nothing is a multiple of the vector width
        _case('train_b16_l77_e512', 'train', 16, 77, 512, 'fp16', 'gelu'),
        # long documents
        _case('train_b2_l1024', 'train', 2, 1024, 1024, 'fp16', 'gelu'),
        # a program that still passes the original module's layout configuration
        _case('train_b8_l512_feature_major', 'train', 8, 512, 1024, 'fp16', 'relu', 'feature_major'),
        # serving one request
        _case('infer_b1_l128', 'infer', 1, 128, 1024, 'fp16', 'gelu'),
        # offline inference over batches
        _case('infer_b64_l256_bf16', 'infer', 64, 256, 1024, 'bf16', 'gelu'),
        # several layers of a model in a row, gradients of each layer in a bucket of its own
        _case('stack4_b8_l512', 'stack', 8, 512, 1024, 'fp16', 'gelu', layers=4),
    ]


def _cost(c):
    """Time of a pass in arbitrary units: contractions, then scores (which every pass reads and writes often)."""
    tokens = c['batch'] * c['seq']
    once = tokens * (24.0 * c['embed'] ** 2 + 600.0 * c['embed'] * c['seq'])
    return once * c['layers'] * (1 if c['mode'] == 'infer' else 3)


def draw(rng):
    """One more case: any mode, storage type, activation and width of the listed ones; lengths log-uniform over
    16..1024 with every third an arbitrary (often odd) number and the others multiples of 8 or 64; batches
    log-uniform up to what keeps the case no dearer than the largest listed one."""
    limit = max(_cost(c) for c in listed() if c['mode'] != 'stack')
    while True:
        mode = rng.choices(['train', 'infer', 'stack'], [6, 3, 1])[0]
        step = rng.choice([1, 8, 64])
        seq = max(16, int(round(2 ** rng.uniform(4, 10) / step)) * step)
        embed = rng.choice([512, 768, 1024])
        batch = int(round(2 ** rng.uniform(0, 6.6)))
        # the shipped layouts are for the training step of the full-width layer
        layouts = 'feature_major' if mode == 'train' and embed == 1024 and rng.random() < 0.15 else 'uniform'
        dtype = 'fp16' if mode == 'stack' else rng.choice(['fp16', 'bf16'])
        # ReLU's step at zero makes a bf16 training step's (or a stack's) gradients differ from a correct one's by more
        # than can be told from a mistake, so those are drawn with GELU
        activation = 'gelu' if mode == 'stack' or dtype == 'bf16' else rng.choice(['relu', 'gelu'])
        c = _case(None, mode, batch, seq, embed, dtype, activation, layouts, rng.randint(2, 4) if mode == 'stack' else 1)
        if _cost(c) <= limit:
            return c


def _layouts(case):
    lay = L.uniform_layouts()
    if case['layouts'] == 'feature_major':
        for key in ('params', 'forward_interm', 'backward_interm'):
            lay[key] = [(n, FEATURE_MAJOR.get(n, dims)) for n, dims in lay[key]]
        lay['input'], lay['output'] = ('X', FEATURE_MAJOR['X']), ('SB2', FEATURE_MAJOR['SB2'])
    return lay


def _fill(enc, lay, gen):
    """Weights as a model in training has them: matrices ~N(0, 0.02), scales near one, biases small."""
    with torch.no_grad():
        for (name, _), prm in zip(lay['params'], enc.params):
            r = torch.randn(prm.shape, device=prm.device, generator=gen) * WEIGHT_STD
            prm.copy_(r + 1 if name in ('S1', 'S2') else r)


def prepare(case, seed):
    dev = torch.device('cuda', torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(int(seed))
    lay, dtype = _layouts(case), DTYPES[case['dtype']]
    heads = case['embed'] // HEAD
    sizes = L.sizes_map(case['batch'], case['seq'], heads, case['embed'])
    shape = L.shape_of(lay['input'][1], sizes)
    state = {'mode': case['mode']}
    if case['mode'] == 'stack':
        stack = EncoderStack(case['layers'], case['batch'], case['seq'], heads, case['embed'], lay, dropout_p=DROPOUT,
                             device=dev, seed=int(seed) % 65521, activation=case['activation'], dtype=dtype)
        state['layer'] = stack
    else:
        p = DROPOUT if case['mode'] == 'train' else 0.0
        enc = Encoder('', case['batch'], case['seq'], heads, case['embed'], lay, dtype, p, p, p, p,
                      activation=case['activation'], seed=int(seed) % 65521).to(dev)
        _fill(enc, lay, gen)
        state['layer'] = enc
    state['x'] = torch.randn(shape, device=dev, generator=gen).to(dtype)
    if case['mode'] == 'train':
        state['x'].requires_grad_(True)
    if case['mode'] != 'infer':
        state['dy'] = torch.randn(shape, device=dev, generator=gen).to(dtype)
    return state


def run(state):
    layer, x = state['layer'], state['x']
    if state['mode'] == 'infer':
        with torch.no_grad():
            return {'y': layer(x)}
    if state['mode'] == 'train':
        x.grad = None
        layer.zero_grad(set_to_none=True)
        y = layer(x)
        y.backward(state['dy'])
        out = {'y': y.detach(), 'dx': x.grad}
        out.update((name, prm.grad) for name, prm in layer.named_parameters())
        return out
    y = layer.forward(x)
    dx = layer.backward(state['dy'])
    layer.wait_gradients()
    out = {'y': y, 'dx': dx}
    for i, grads in enumerate(layer.grads):
        out.update(('%d.%s' % (i, n), grads[n]) for n in layer.layers[i]._param_names)
    return out


def work(case):
    """Input and weights read once, outputs (with gradients) written once; the multiply-adds of the contractions."""
    tokens, e, layers = case['batch'] * case['seq'], case['embed'], case['layers']
    weights = 12 * e * e + 13 * e
    acts = tokens * e
    flops = layers * (2.0 * tokens * 12 * e * e + 4.0 * tokens * case['seq'] * e)
    if case['mode'] == 'infer':
        return {'bytes': 2 * (weights + 2 * acts), 'flops': flops}
    return {'bytes': 2 * (2 * layers * weights + 4 * acts), 'flops': 3 * flops}


def tolerance(case):
    """Four times what the layer differs from itself by when the attention operators run one by one (scores rounded to
    16 bits between them, sums in another order) instead of fused, worst of forty drawn cases and the listed ones.
    Largest values seen (2-norm; largest element): inference 2.5e-4; 2.8e-3 in fp16 and 1.8e-3; 2.3e-2 in bf16, a
    training step with GELU 7.8e-4; 8.7e-3 in fp16 and 6.2e-3; 7.4e-2 in bf16, a stack of four layers 1.3e-3; 1.5e-2.
    ReLU's derivative jumps at zero: a pre-activation that rounding moves across it changes its gradient by all of
    its value, 6.9e-3; 0.59 in fp16."""
    if case['mode'] == 'infer':
        return {'rel': 1e-3, 'max': 1.2e-2} if case['dtype'] == 'fp16' else {'rel': 8e-3, 'max': 0.1}
    if case['mode'] == 'stack':
        return {'rel': 5e-3, 'max': 6e-2}
    if case['activation'] == 'relu':
        return {'rel': 2.8e-2, 'max': 0.99}
    return {'rel': 3e-3, 'max': 4e-2} if case['dtype'] == 'fp16' else {'rel': 2.5e-2, 'max': 0.3}
