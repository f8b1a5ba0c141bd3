"""ZeRO-3 / FSDP training engine over the library's all-gather and reduce-scatter.

Every unit of the model (embedding, each decoder layer, output head) is one flat bf16 buffer cut
into equal shards, one per rank. A training step:

  forward    for unit u: all-gather(u+1) runs on the communication stream while unit u computes;
             only each unit's input is kept (activation checkpointing), and the activations of the last layers
             while they fit a part of the memory that is free (`_layers_kept`).
  backward   in reverse: all-gather(u-1) is prefetched, unit u is recomputed and differentiated,
             its flat gradient is reduce-scattered (sum, then scaled by 1/ranks inside AdamW) on the
             communication stream, and the fused AdamW kernel updates this rank's shard right
             behind it, all overlapped with the backward compute of unit u-1.

Shards, gather buffers and gradient buffers live in symmetric memory registered as windows, so
the collectives run zero-copy over NVLink. With a host-only communicator (no GPU) the same code
runs synchronously on CPU tensors, which is how the engine is tested against plain autograd.

Reference parity: the reference serves this pattern through ncclAllGather / ncclReduceScatter on
user-registered buffers (src/collectives.cc, src/register/register.cc: ncclCommWindowRegister).
"""
import ctypes

import torch

from .. import _lib
from ..core import mem_alloc, mem_free
from ..models import llama as M
from ..models import llama_fused


def _align(n, a):
    return (n + a - 1) // a * a


# elements of a unit from which one rank updates it in pieces, each a quarter of that at least: a piece's launch and event cost the host 15 us,
# the update of 2^22 elements takes 17 us of the GPU's time (28 bytes each at 6.7 TB/s)
kEarlyUpdate = 1 << 24


# bytes that a program may have allocated since the last decision on kept layers (losses that it collects) without another one
kDrift = 16 << 20


class _Unit:
    pass


class _Kept:
    """Activations that the units from `first` on keep for the backward of one step; they are what can be done without when memory runs out."""

    def __init__(self, first, units):
        self.first, self.units, self.acts, self.ran_out = first, units, {}, False

    def spare(self, fn):
        """fn(), and if memory runs out in it once more without kept activations. fn may have started, but not changed anything."""
        try:
            return fn()
        except torch.OutOfMemoryError:
            if self.first == self.units:
                raise
        # behind the handler, which holds on to what the failed call had
        self.ran_out, self.first = True, self.units
        self.acts.clear()
        return fn()


class FSDPEngine:
    def __init__(self, comm, cfg, device="cuda", seed=0, lr=1e-4, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1, symmetric=True, init_on_device=False,
                 keep_layers=None):
        """keep_layers: how many layers may keep their activations for the backward at most (0: all are computed again there); None: as many as
        memory allows. What they take stays with the framework's allocator between steps (torch.cuda.empty_cache() gives it back)."""
        self.comm, self.cfg, self.device = comm, cfg, torch.device(device)
        self.keep_layers = keep_layers
        self.cuda = self.device.type == "cuda"
        if self.cuda and self.device.index is None:
            self.device = torch.device("cuda", torch.cuda.current_device())
        self.n, self.rank = comm.nranks, comm.rank
        self.lr, self.betas, self.eps, self.wd = lr, betas, eps, weight_decay
        self.step_count = 0
        self.symmetric = symmetric and self.cuda
        self._allocs = []
        self._wins = []
        self.lib = comm.lib            # collectives and memory: the communicator's library
        self.own = _lib.load()         # the optimizer kernel always comes from this package's library
        if self.cuda:
            self.own.b200FusedAdamW.argtypes = [ctypes.c_void_p] * 5 + [ctypes.c_size_t] + [ctypes.c_float] * 6 + [ctypes.c_int, ctypes.c_void_p]
            self.fused = llama_fused.FusedUnits(cfg, self.own)
        specs = M.unit_specs(cfg)
        self.units = []
        gen = torch.Generator().manual_seed(seed)
        for name, shapes in specs:
            u = _Unit()
            u.name, u.shapes, u.numel = name, shapes, M.numel(shapes)
            u.padded = _align(u.numel, self.n * 128)
            u.shard = u.padded // self.n
            if init_on_device and self.cuda:
                # large models: draw the unit on the GPU (same seed on every rank), keep this rank's slice
                dgen = torch.Generator(device=self.device).manual_seed(seed * 1000003 + len(self.units))
                full = torch.zeros(u.padded, dtype=torch.bfloat16, device=self.device)
                off = 0
                for _, shape in shapes:
                    cnt = 1
                    for sdim in shape:
                        cnt *= sdim
                    if len(shape) == 1:
                        full[off:off + cnt] = 1.0
                    else:
                        full[off:off + cnt] = (torch.randn(cnt, generator=dgen, device=self.device) * 0.02).to(torch.bfloat16)
                    off += cnt
            else:
                full = torch.zeros(u.padded, dtype=torch.bfloat16)
                full[:u.numel] = M.init_flat(shapes, gen)      # every rank draws the same stream, keeps its slice
            mine = full[self.rank * u.shard:(self.rank + 1) * u.shard]
            u.param = self._buffer(u.shard, torch.bfloat16)
            u.param.copy_(mine)
            u.grad = self._buffer(u.shard, torch.bfloat16)
            u.master = mine.float().to(self.device)
            u.m = torch.zeros(u.shard, dtype=torch.float32, device=self.device)
            u.v = torch.zeros(u.shard, dtype=torch.float32, device=self.device)
            self.units.append(u)
        # One rank's shards are the whole units: they are gathered and reduced where they lie (nothing is copied).
        biggest = max(u.padded for u in self.units) if self.n > 1 else 0
        self.gbuf = [self._buffer(biggest, torch.bfloat16) for _ in range(2 if self.n > 1 else 0)]
        self.ggrad = [self._buffer(biggest, torch.bfloat16) for _ in range(2 if self.n > 1 else 0)]
        if self.cuda:
            self.comm_stream = torch.cuda.Stream(device=self.device)
            ev = lambda: torch.cuda.Event()   # noqa: E731
            self.ev_gathered = [ev() for _ in range(2)]
            self.ev_free = [ev() for _ in range(2)]
            self.ev_grad_ready = [ev() for _ in range(2)]
            self.ev_grad_free = [ev() for _ in range(2)]
            self.ev_ready = ev()
            for e in self.ev_free + self.ev_grad_free:
                e.record()
        self.collectives = 0      # all-gathers + reduce-scatters issued (for reporting)
        self.kernels = 0          # AdamW launches
        self.layers_kept = 0      # whose activations the last step kept for its backward (for reporting)
        self._kept_for = None     # (tokens, memory held and allowed), bytes in use, layers: the last decision of `_layers_kept`

    # ------------------------------------------------------------------ memory
    def _buffer(self, numel, dtype):
        if not self.symmetric:
            return torch.zeros(numel, dtype=dtype, device=self.device)
        from ..utils.perf import tensor_at
        es = torch.empty(0, dtype=dtype).element_size()
        nbytes = _align(numel * es, 4096)
        ptr = mem_alloc(nbytes, self.lib)
        raw = tensor_at(ptr, nbytes)
        raw.zero_()
        self._wins.append(self.comm.register_window(raw))
        self._allocs.append(ptr)
        return raw[:numel * es].view(dtype)

    def close(self):
        if self.cuda:
            torch.cuda.synchronize()
        for w in self._wins:
            self.comm.deregister_window(w)
        for p in self._allocs:
            mem_free(p, self.lib)
        self._wins, self._allocs = [], []

    # ------------------------------------------------------------------ communication
    def _whole(self, idx, slot):
        """Where all of the unit's parameters lie once they are gathered."""
        u = self.units[idx]
        return self.gbuf[slot][:u.padded] if self.n > 1 else u.param

    def _whole_grad(self, idx, gslot):
        u = self.units[idx]
        return self.ggrad[gslot][:u.padded] if self.n > 1 else u.grad

    def _gather(self, idx, slot):
        u = self.units[idx]
        dst = self._whole(idx, slot)
        if self.cuda:
            with torch.cuda.stream(self.comm_stream):
                self.comm_stream.wait_event(self.ev_free[slot])
                self.comm.all_gather(u.param, dst, stream=self.comm_stream)
                self.ev_gathered[slot].record(self.comm_stream)
        else:
            self.comm.all_gather(u.param, dst)
        self.collectives += 1

    def _wait_gathered(self, slot):
        if self.cuda:
            torch.cuda.current_stream().wait_event(self.ev_gathered[slot])

    def _release(self, slot):
        if self.cuda:
            self.ev_free[slot].record(torch.cuda.current_stream())

    def _update_early(self, idx, lo, hi):
        """One rank: AdamW on elements [lo, hi) of the unit, whose gradients are final and whose weights this step reads no more."""
        self.ev_ready.record(torch.cuda.current_stream())
        self.comm_stream.wait_event(self.ev_ready)
        self._adamw(self.units[idx], self.comm_stream, lo, hi)

    def _reduce_and_update(self, idx, gslot, hi=None):
        """Reduce-scatter of the unit's gradients into its gradient shard, then AdamW on the shard (its first `hi` elements, if the others are through)."""
        u = self.units[idx]
        src = self._whole_grad(idx, gslot)
        if self.cuda:
            self.ev_grad_ready[gslot].record(torch.cuda.current_stream())
            with torch.cuda.stream(self.comm_stream):
                self.comm_stream.wait_event(self.ev_grad_ready[gslot])
                self.comm.reduce_scatter(src, u.grad, stream=self.comm_stream)
                self.ev_grad_free[gslot].record(self.comm_stream)
                self._adamw(u, self.comm_stream, 0, hi)
        else:
            self.comm.reduce_scatter(src, u.grad)
            self._adamw(u, None)
        self.collectives += 1

    def _adamw(self, u, stream, lo=0, hi=None):
        b1, b2 = self.betas
        step = self.step_count
        if self.cuda:
            rc = self.own.b200FusedAdamW(u.master.data_ptr() + 4 * lo, u.m.data_ptr() + 4 * lo, u.v.data_ptr() + 4 * lo, u.grad.data_ptr() + 2 * lo,
                                         u.param.data_ptr() + 2 * lo, (u.shard if hi is None else hi) - lo, self.lr, b1, b2, self.eps, self.wd, 1.0 / self.n, step, stream.cuda_stream)
            _lib.check(rc, "b200FusedAdamW", self.own)
            self.kernels += 1
            return
        g = u.grad.float() / self.n
        u.m.mul_(b1).add_(g, alpha=1 - b1)
        u.v.mul_(b2).addcmul_(g, g, value=1 - b2)
        mhat = u.m / (1 - b1 ** step)
        denom = u.v.sqrt() / (1 - b2 ** step) ** 0.5 + self.eps
        u.master.mul_(1 - self.lr * self.wd).addcdiv_(mhat, denom, value=-self.lr)
        u.param.copy_(u.master.to(torch.bfloat16))

    def _grad_flat(self, idx, gslot):
        """The unit's flat gradient buffer, to be written behind `_take_grads`."""
        return self._whole_grad(idx, gslot)[:self.units[idx].numel]

    def _take_grads(self, idx, gslot):
        """What follows may write the unit's gradients: the reduce-scatter that read the buffer last is through, the padding is zero."""
        u = self.units[idx]
        if self.cuda and self.n > 1:
            torch.cuda.current_stream().wait_event(self.ev_grad_free[gslot])
        if u.padded > u.numel:
            self._whole_grad(idx, gslot)[u.numel:u.padded].zero_()

    def _write_grads(self, idx, gslot, grads):
        self._take_grads(idx, gslot)
        flat = self._grad_flat(idx, gslot)
        off = 0
        for g in grads:
            flat[off:off + g.numel()].copy_(g.reshape(-1))
            off += g.numel()

    # ------------------------------------------------------------------ one training step
    def step(self, tokens, targets):
        """tokens, targets: int64 [B, S] (host or device). Returns the loss of this rank as a 0-d tensor."""
        if not self.cuda:
            return self._step(tokens, targets)
        with torch.cuda.device(self.device):   # kernels and events go to the current device's streams, whichever the caller has current
            return self._step(tokens, targets)

    def _layers_kept(self, tokens):
        """How many layers, counted from the last, keep their activations for the backward instead of computing them again there: as many as leave
        half of the memory that the framework's allocator can still get (of what is free, and within the process's memory fraction) beyond what the
        step takes anyway (the logits, every layer's input, one layer's activations). Two layers of hidden 4096 and ffn 14336 with 2048 tokens: 420 MB. Under capture, and where the allocator does
        not tell, none. At most `keep_layers`, which a step that ran out of memory halves.

        The driver is asked (60 us, and many milliseconds while other processes keep it busy) only when the allocator holds or may hold other
        memory than at the last decision for as many tokens: while it does not, the step runs in the memory that it ran in before."""
        c, layers = self.cfg, len(self.units) - 2
        most = layers if self.keep_layers is None else min(layers, self.keep_layers)
        if most <= 0 or torch.cuda.is_current_stream_capturing():
            return 0
        try:
            stats = torch.cuda.memory_stats_as_nested_dict(self.device)
            reserved, used = stats["reserved_bytes"]["all"]["current"], stats["allocated_bytes"]["all"]["current"]
            fraction = torch.cuda.get_per_process_memory_fraction(self.device)
            decided, now = self._kept_for, (tokens, most, reserved, fraction)
            if decided and decided[0] == now and used <= decided[1] + kDrift:
                return decided[2]
            free, total = torch.cuda.mem_get_info(self.device)
            room = min(free, max(0, int(fraction * total) - reserved)) + reserved - used
        except (RuntimeError, KeyError):
            return 0
        each = self.fused.activation_bytes(tokens)
        needed = self._backward_bytes(tokens) + 2 * tokens * (c.vocab + layers * c.hidden)
        kept = max(0, min(most, (room // 2 - needed) // each))
        self._kept_for = (now, used, kept)
        return kept

    def _backward_bytes(self, tokens):
        """What the backward of a layer allocates, its activations among it."""
        c = self.cfg
        return self.fused.activation_bytes(tokens) + 2 * tokens * (8 * c.hidden + 2 * c.ffn)

    def _step(self, tokens, targets):
        cfg, U = self.cfg, len(self.units)
        self.step_count += 1
        tokens = tokens.to(self.device, non_blocking=True)
        targets = targets.to(self.device, non_blocking=True)
        rope = M.rope_tables(cfg, tokens.shape[1], self.device)
        saved = [None] * U

        def params(idx, slot, need_grad):
            u = self.units[idx]
            vs = M.views(self._whole(idx, slot)[:u.numel], u.shapes)
            if need_grad:
                vs = {k: t.detach().requires_grad_(True) for k, t in vs.items()}
            return vs

        def run(idx, vs, x):
            if idx == 0:
                return M.embed(tokens, vs)
            if idx == U - 1:
                return M.head_loss(x, vs, cfg, targets)
            return M.decoder_layer(x, vs, cfg, rope)

        # shapes and modes that the row kernels fit: the layers and the head have their backward written out
        fused = self.fused if self.cuda and llama_fused.applies(cfg, tokens, targets) else None
        shape = tuple(tokens.shape)

        def weights(idx, slot):
            return self._whole(idx, slot)[:self.units[idx].numel]

        layers_kept = self._layers_kept(tokens.numel()) if fused else 0
        kept = _Kept(U - 1 - layers_kept if layers_kept else U, U)

        # forward (the head is differentiated at once: its recompute would be wasted work)
        self._gather(0, 0)
        x = add = None   # a layer leaves its output as two terms
        for idx in range(U - 1):
            self._gather(idx + 1, (idx + 1) % 2)
            self._wait_gathered(idx % 2)
            with torch.no_grad():
                if fused and idx:
                    saved[idx], x, add, *acts = kept.spare(lambda: fused.layer(x, add, weights(idx, idx % 2), rope, shape, keep=idx >= kept.first))
                    if acts:
                        kept.acts[idx] = acts[0]
                    del acts
                else:
                    saved[idx] = x
                    x = run(idx, params(idx, idx % 2, False), x)
                    x = x.view(-1, cfg.hidden) if fused else x
            self._release(idx % 2)
        # head: forward + backward
        idx = U - 1
        slot = idx % 2
        self._wait_gathered(slot)
        if fused:
            loss, gx = kept.spare(lambda: fused.head(x, add, weights(idx, slot), self._grad_flat(idx, slot), targets.reshape(-1).contiguous(),
                                                     before=lambda: self._take_grads(idx, slot)))
            self._release(slot)
        else:
            vs = params(idx, slot, True)
            xin = x.detach().requires_grad_(True)
            loss = run(idx, vs, xin)
            names = [n for n, _ in self.units[idx].shapes]
            grads = torch.autograd.grad(loss, [xin] + [vs[n] for n in names])
            self._release(slot)
            self._write_grads(idx, slot, grads[1:])
            gx = grads[0]
            del grads, vs, xin
        self._reduce_and_update(idx, slot)
        del x, add
        if kept.acts:   # a layer's backward updates weights on its way and cannot be begun again: whether its memory is there shows before the first
            kept.spare(lambda: torch.empty(self._backward_bytes(tokens.numel()), dtype=torch.uint8, device=self.device) if kept.acts else None)
        if kept.ran_out:
            self.keep_layers = layers_kept // 2
        self.layers_kept = len(kept.acts)
        # backward through the layers and the embedding; the last layer's parameters are still gathered from the forward
        for idx in range(U - 2, -1, -1):
            slot = idx % 2
            u = self.units[idx]
            if idx - 1 >= 0:
                self._gather(idx - 1, (idx - 1) % 2)
            self._wait_gathered(slot)
            if fused and idx:
                # one rank's large units: the optimizer takes the weights as their gradients come (it is bound by memory, the rest of the
                # backward by the tensor cores), and little of it is left behind the last unit
                done = [u.shard]
                if self.n == 1 and u.numel >= kEarlyUpdate:
                    def ready(lo):
                        if done[0] - lo < kEarlyUpdate // 4:
                            return   # goes with the next piece, or with the rest
                        self._update_early(idx, lo, done[0])
                        done[0] = lo
                else:
                    ready = None
                acts = [kept.acts.pop(idx)] if idx in kept.acts else None   # no name of its own: the layer lets go of it bit by bit
                gx = fused.layer_backward(saved[idx], weights(idx, slot), self._grad_flat(idx, slot), rope, shape, gx, ready,
                                          before=lambda: self._take_grads(idx, slot), kept=acts)
                del acts
                self._release(slot)
                self._reduce_and_update(idx, slot, done[0])
                saved[idx] = None
                continue
            if fused and llama_fused.embedding_applies(tokens):
                self._take_grads(idx, slot)
                fused.embedding_backward(tokens, gx, self._grad_flat(idx, slot))
                self._release(slot)
                self._reduce_and_update(idx, slot)
                continue
            vs = params(idx, slot, True)
            names = [n for n, _ in self.units[idx].shapes]
            gx = gx.view(*shape, cfg.hidden) if fused else gx
            with torch.enable_grad():
                if idx == 0:
                    out = run(idx, vs, None)
                    grads = (None,) + torch.autograd.grad(out, [vs[n] for n in names], gx)
                else:
                    xin = saved[idx].detach().requires_grad_(True)
                    out = run(idx, vs, xin)
                    grads = torch.autograd.grad(out, [xin] + [vs[n] for n in names], gx)
            self._release(slot)
            self._write_grads(idx, idx % 2, grads[1:])
            self._reduce_and_update(idx, idx % 2)
            gx = grads[0]
            saved[idx] = None
            del grads, vs, out
        if self.cuda:
            torch.cuda.current_stream().wait_stream(self.comm_stream)
        return loss.detach()

    # ------------------------------------------------------------------ inspection
    def full_params(self):
        """List of whole flat fp32 parameter buffers (gathers every unit; for tests)."""
        out = []
        for idx, u in enumerate(self.units):
            self._gather(idx, 0)
            self._wait_gathered(0)
            if self.cuda:
                torch.cuda.synchronize()
            out.append(self._whole(idx, 0)[:u.numel].float().cpu().clone())
            self._release(0)
        return out
