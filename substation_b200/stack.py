"""A stack of encoder layers run through the raw (non-autograd) passes, with
data-parallel gradient reduction overlapped with the rest of backward.

The reference times one layer (pytorch_module/run_encoder.py:345-383); a BERT-large
encoder is 24 of them with independent weights.  Forward keeps what each layer's
backward needs alive (one arena per layer, allocated once and reused every step; every
named intermediate, as views in ``fwd`` and ``bwd``, with ``keep_all_intermediates`` or
once somebody asks for one of the two);
backward walks the layers in reverse with ONE shared arena for backward
intermediates, writes layer l's 12 parameter gradients into bucket l and starts
its sum-allreduce at once, so the reduction of layer l runs beside the backward of
layer l-1 (parameter gradients become final in the order
DS2,DB2 -> DLINW2 -> ... -> DWKQV -> DBKQV, i.e. at the end of the layer's backward).
"""

import torch

from . import layouts as L
from .data_parallel import GradientBucketReducer
from .encoder import Encoder


class EncoderStack:
    def __init__(self, num_layers, batch_size, max_seq_len, num_heads, embedding_size, layouts,
                 dropout_p=0.1, device='cuda', mask_mode='philox', seed=0, activation='relu',
                 weight_std=0.02, group=None, dtype=torch.float16, keep_all_intermediates=None):
        self.device = torch.device(device)
        self.layers = []
        gen = torch.Generator(device=self.device).manual_seed(seed)
        for l in range(num_layers):
            enc = Encoder('', batch_size, max_seq_len, num_heads, embedding_size, layouts, dtype,
                          dropout_p, dropout_p, dropout_p, dropout_p, mask_mode=mask_mode, seed=seed + l,
                          activation=activation, keep_all_intermediates=keep_all_intermediates).to(self.device)
            with torch.no_grad():
                for (name, _), prm in zip(layouts['params'], enc.params):
                    if name in ('WKQV', 'WO', 'LINW1', 'LINW2'):
                        prm.copy_((torch.randn(prm.shape, device=self.device, generator=gen) * weight_std).to(dtype))
                    elif name in ('S1', 'S2'):
                        prm.fill_(1.0)
                    else:
                        prm.zero_()
            self.layers.append(enc)
        e0 = self.layers[0]
        self.table = L.validate(layouts)
        shape_x = L.shape_of(self.table['X'], e0.sizes)
        self.weights = [[p.detach() for p in enc.params] for enc in self.layers]
        # private passes (no score tensors in memory) unless somebody wants to look at the intermediates
        sizes = e0.private_arena_bytes(self.device)
        self.private = sizes is not None
        self._named = None                               # (fwd, bwd): views of every intermediate, once they are wanted
        self._kept = ['nothing'] * num_layers            # how each layer's last forward pass kept what its backward needs
        self._redo = [None] * num_layers                 # (Philox offset, weight versions) of that pass
        self._dy0 = None                                 # what layer 0's last backward pass was given
        if self.private:
            self._arenas = [torch.empty(sizes[0], dtype=torch.uint8, device=self.device) for _ in self.layers]
            self._barena = torch.empty(sizes[1], dtype=torch.uint8, device=self.device)
        else:
            self._name_intermediates()
        # activations between layers: acts[l] is the input of layer l, acts[-1] the output
        self.acts = [torch.empty(shape_x, dtype=dtype, device=self.device) for _ in range(num_layers + 1)]
        self.dacts = [torch.empty(shape_x, dtype=dtype, device=self.device) for _ in range(2)]
        self.reducer = GradientBucketReducer(e0.arena_bytes('grads'), self.device, group=group, buffers=num_layers, dtype=dtype)
        self.grads = [enc.views('grads', self.reducer.arenas[l]) for l, enc in enumerate(self.layers)]
        if mask_mode == 'explicit':
            raise NotImplementedError('the stack draws its masks in the kernels (Philox); explicit masks are a '
                                      'single-layer testing facility')

    def _name_intermediates(self):
        """Buffers for every named intermediate; passes fill them from now on, and what the last passes kept privately is
        computed again from the activations between the layers (same weights and masks)."""
        e0 = self.layers[0]
        if self._named is None:
            self._named = ([enc.views('forward', torch.empty(enc.arena_bytes('forward'), dtype=torch.uint8, device=self.device))
                            for enc in self.layers],
                           e0.views('backward', torch.empty(e0.arena_bytes('backward'), dtype=torch.uint8, device=self.device)))
        again = [l for l, kept in enumerate(self._kept) if kept == 'private']
        if not again:
            return
        fwd, bwd = self._named
        out = torch.empty_like(self.acts[0])
        for l in again:
            enc, (offset, versions) = self.layers[l], self._redo[l]
            if versions != [w._version for w in self.weights[l]]:
                raise RuntimeError('the weights changed after the pass whose intermediates are asked for; '
                                   'build the stack with keep_all_intermediates=True')
            now, enc.philox_offset = enc.philox_offset, offset
            enc.forward_raw(self.acts[l], self.weights[l], fwd[l], out)
            enc.philox_offset = now
            self._kept[l] = 'named'
        if self._dy0 is not None and 0 in again:
            grads = e0.views('grads', torch.empty(e0.arena_bytes('grads'), dtype=torch.uint8, device=self.device))
            e0.backward_raw(self._dy0, grads, bwd, self.weights[0], fwd[0], self.acts[0], out)

    @property
    def fwd(self):
        """Per layer, name -> forward intermediate of the last pass.  Asking makes this and later passes keep them all."""
        self._name_intermediates()
        return self._named[0]

    @property
    def bwd(self):
        """Name -> backward intermediate of the layer that ran last.  Asking makes this and later passes keep them all."""
        self._name_intermediates()
        return self._named[1]

    def memory_bytes(self):
        e0, n = self.layers[0], len(self.layers)
        total = n * e0.arena_bytes('grads')
        if self.private:
            total += n * self._arenas[0].numel() + self._barena.numel()
        if self._named is not None:
            total += n * e0.arena_bytes('forward') + e0.arena_bytes('backward')
        return total

    def forward(self, X):
        self.acts[0].copy_(X)
        self._dy0 = None
        self._kept = ['nothing'] * len(self.layers)
        for l, enc in enumerate(self.layers):
            # (a layer whose switches changed since, enable_debug for one, has no private passes any more)
            plans = enc._private_plans(self.acts[l].device) if self._named is None else None
            if plans is None:
                enc.forward_raw(self.acts[l], self.weights[l], self.fwd[l], self.acts[l + 1])
                self._kept[l] = 'named'
            else:
                self._redo[l] = (enc.philox_offset, [w._version for w in self.weights[l]])
                enc._forward_private(plans, self.acts[l], self.weights[l], self._arenas[l], self.acts[l + 1])
                self._kept[l] = 'private'
        return self.acts[-1]

    def backward(self, DY, trace=None):
        """Returns dX; gradients of layer l are in ``self.grads[l]`` once ``wait_gradients`` returns.

        ``trace``: an empty list to be filled with one (layer, event at the end of that layer's backward, event at
        the end of its bucket's allreduce or None) per layer, plus a leading ('start', event, None): what
        ``overlap_trace`` turns into times.  The allreduce events are recorded on a stream of their own that
        waits for each reduction in turn, so tracing does not change what the compute stream waits for."""
        cur = DY
        tracing = trace is not None and self.device.type == 'cuda'
        if tracing:
            if self.__dict__.get('_trace_stream') is None:
                self._trace_stream = torch.cuda.Stream(self.device)
            ev = torch.cuda.Event(enable_timing=True)
            ev.record()
            trace.append(('start', ev, None))
        for l in range(len(self.layers) - 1, -1, -1):
            self.reducer.wait(l)                         # bucket l free again (previous step's reduction done)
            out = self.dacts[l & 1]
            enc = self.layers[l]
            plans = enc._private_plans(cur.device) if self._kept[l] == 'private' else None
            if plans is not None:
                enc._backward_private(plans, cur, self.grads[l], self._barena, self.weights[l], self._arenas[l],
                                      self.acts[l], out)
            else:
                enc.backward_raw(cur, self.grads[l], self.bwd, self.weights[l], self.fwd[l], self.acts[l], out)
            if l == 0:
                self._dy0 = cur
            if tracing:
                done = torch.cuda.Event(enable_timing=True)
                done.record()
            self.reducer.reduce_async(l)
            if tracing:
                reduced = None
                works = self.reducer.pending[l % len(self.reducer.arenas)]
                if works:
                    with torch.cuda.stream(self._trace_stream):
                        for w in works:
                            w.wait()
                        reduced = torch.cuda.Event(enable_timing=True)
                        reduced.record()
                trace.append((l, done, reduced))
            cur = out
        return cur

    @staticmethod
    def overlap_trace(trace):
        """Times in ms since the start of the traced backward: [[layer, backward done, allreduce done or None], ...]
        in the order the layers ran (last layer first).  Call after the device has finished the step."""
        start = trace[0][1]
        return [[l, round(start.elapsed_time(done), 3), None if red is None else round(start.elapsed_time(red), 3)]
                for l, done, red in trace[1:]]

    def wait_gradients(self):
        self.reducer.drain()
