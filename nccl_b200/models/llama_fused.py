"""Forward and backward of the decoder's units with this package's own row kernels, for the sharded engine on a GPU.

The functions do what `llama.decoder_layer` and `llama.head_loss` do under autograd with checkpointing, over the same flat
buffers, with the backward written out:

  * RMSNorm (with the residual addition before it), rotary embedding, SwiGLU and cross entropy are one kernel each way
    (src/contrib/train_ops.cu) in place of chains of framework operations;
  * wq | wk | wv and w_gate | w_up lie next to each other in the flat buffer and are one matrix each;
  * weight gradients are written where the reduce-scatter reads them, and the recomputation leaves out the last product,
    whose result no gradient needs; a layer whose activations were kept is not computed again.

Between kernels everything is bf16 as before; sums, exponentials and rotations are held in fp32. The forward rounds where the
operations of `llama` round, so that both give the same loss up to the order of sums; the backward rounds each result once.
"""
import ctypes

import torch
import torch.nn.functional as F
from torch.nn.attention import SDPBackend
from torch.overrides import _get_current_function_mode_stack
from torch.utils._device import DeviceContext
from torch.utils._python_dispatch import _get_current_dispatch_mode_stack

from .. import _lib
from . import llama as M

_P, _I = ctypes.c_void_p, ctypes.c_int
_ENTRIES = {
    "b200RmsNorm": [_P] * 6 + [_I, _I, ctypes.c_float, _P],
    "b200RmsNormBackward": [_P] * 8 + [_I, _I, _P],
    "b200RmsNormBackwardCtas": [_I],
    "b200Rope": [_P] * 3 + [_I] * 5 + [_P],
    "b200RopeBackward": [_P] * 7 + [_I] * 5 + [_P],
    "b200SwiGlu": [_P] * 2 + [_I, _I, _P],
    "b200SwiGluBackward": [_P] * 2 + [_I, _I, _P],
    "b200CrossEntropy": [_P] * 5 + [_I, _I, _P],
    "b200EmbeddingBackward": [_P] * 4 + [_I] * 3 + [_P],
    "b200EmbeddingBackwardWork": [_I, _I],
}


def _watched():
    """Whether something in the framework looks into, or changes, the single operations: the row kernels would pass it by. A default
    device is a function mode too, but changes none of them."""
    return (torch.is_autocast_enabled("cuda") or torch.is_anomaly_enabled() or torch.jit.is_tracing() or torch.compiler.is_compiling() or
            bool(_get_current_dispatch_mode_stack()) or any(not isinstance(m, DeviceContext) for m in _get_current_function_mode_stack()) or
            torch._C._autograd._top_saved_tensors_default_hooks(False) is not None or torch._C._functorch.peek_interpreter_stack() is not None)


def applies(cfg, tokens, targets):
    """Whether a step on a GPU takes this path: shapes that the kernels' 16-byte accesses fit, gradients wanted, and nothing that watches the
    operations (autocast, anomaly detection, dispatch and function modes, hooks for saved tensors, tracing, function transforms).
    Everything else goes through `llama` and autograd."""
    h, d = cfg.hidden, cfg.head_dim
    return (h % 8 == 0 and h <= 16384 and d > 0 and d % 16 == 0 and d * cfg.heads == h and cfg.heads % cfg.kv_heads == 0 and cfg.ffn % 8 == 0 and
            cfg.vocab % 8 == 0 and tokens.dim() == 2 and tokens.numel() > 0 and targets.dtype == torch.int64 and targets.numel() == tokens.numel() and
            torch.is_grad_enabled() and not _watched())


def embedding_applies(tokens):
    """64-bit ids, and no more of them than the kernel takes: each is compared with all others. 8192 uniform ids of 4096 channels 78 us against
    762 by autograd, all of them the same id 90 against 471."""
    return tokens.dtype == torch.int64 and tokens.numel() <= 8192


class FusedUnits:
    """The units of one configuration; `lib` is this package's library."""

    def __init__(self, cfg, lib):
        self.cfg, self.lib = cfg, lib
        self._call = {}
        for name, types in _ENTRIES.items():
            fn = getattr(lib, name)
            fn.argtypes = types
            fn.restype = ctypes.c_size_t if name.endswith("Work") else ctypes.c_int
            self._call[name] = fn

    def _run(self, name, *args):
        rc = self._call[name](*args, torch.cuda.current_stream().cuda_stream)
        if rc:
            _lib.check(rc, name, self.lib)

    # ------------------------------------------------------------------ kernels
    def norm(self, x, gain, add=None, need_rstd=False):
        """(x + add, its RMSNorm, 1 / rms per row or None)."""
        h = torch.empty_like(x)
        total = x if add is None else torch.empty_like(x)
        rstd = torch.empty(x.shape[0], dtype=torch.float32, device=x.device) if need_rstd else None
        self._run("b200RmsNorm", x.data_ptr(), None if add is None else add.data_ptr(), gain.data_ptr(), total.data_ptr(), h.data_ptr(),
                  rstd.data_ptr() if need_rstd else None, x.shape[0], x.shape[1], self.cfg.eps)
        return total, h, rstd

    def norm_backward(self, x, gain, rstd, dh, res, dgain):
        """Gradient of x (plus `res`); the gain's goes into dgain."""
        rows, hidden = x.shape
        dx = torch.empty_like(x)
        partial = torch.empty(self._call["b200RmsNormBackwardCtas"](rows), hidden, dtype=torch.float32, device=x.device)
        self._run("b200RmsNormBackward", x.data_ptr(), gain.data_ptr(), rstd.data_ptr(), dh.data_ptr(), None if res is None else res.data_ptr(),
                  dx.data_ptr(), dgain.data_ptr(), partial.data_ptr(), rows, hidden)
        return dx

    def rope(self, qkv, rope, seq):
        c = self.cfg
        self._run("b200Rope", qkv.data_ptr(), rope[0].data_ptr(), rope[1].data_ptr(), qkv.shape[0], seq, c.heads, c.kv_heads, c.head_dim)

    def rope_backward(self, dq, dk, dv, rope, tokens, seq):
        """[tokens, (heads + 2 kv_heads) * head_dim] from the gradients [B, heads, S, head_dim] of attention's inputs."""
        c = self.cfg
        out = torch.empty(tokens, (c.heads + 2 * c.kv_heads) * c.head_dim, dtype=dq.dtype, device=dq.device)
        parts = [t if t.stride(3) == 1 and not any(s % 8 for s in t.stride()[:3]) and t.data_ptr() % 16 == 0 else t.clone(memory_format=torch.contiguous_format)
                 for t in (dq, dk, dv)]
        strides = (ctypes.c_longlong * 9)(*[s for t in parts for s in t.stride()[:3]])
        self._run("b200RopeBackward", *[t.data_ptr() for t in parts], strides, out.data_ptr(), rope[0].data_ptr(), rope[1].data_ptr(),
                  tokens, seq, c.heads, c.kv_heads, c.head_dim)
        return out

    def swiglu(self, gu):
        act = torch.empty(gu.shape[0], gu.shape[1] // 2, dtype=gu.dtype, device=gu.device)
        self._run("b200SwiGlu", gu.data_ptr(), act.data_ptr(), act.shape[0], act.shape[1])
        return act

    def swiglu_backward(self, gu, dact):
        """In place: gu becomes the gradients of gate and up, dact becomes silu(gate) * up."""
        self._run("b200SwiGluBackward", gu.data_ptr(), dact.data_ptr(), dact.shape[0], dact.shape[1])

    def cross_entropy(self, logits, targets):
        """Mean loss; logits become their gradient."""
        rows, vocab = logits.shape
        loss = torch.empty((), dtype=torch.float32, device=logits.device)
        work = torch.empty(rows + 1, dtype=torch.float32, device=logits.device)
        ok = torch.empty((), dtype=torch.bool, device=logits.device)
        self._run("b200CrossEntropy", logits.data_ptr(), targets.data_ptr(), loss.data_ptr(), work.data_ptr(), ok.data_ptr(), rows, vocab)
        torch._assert_async(ok, "a target is no class of the vocabulary")
        return loss

    # ------------------------------------------------------------------ units
    def _layer_views(self, flat):
        c = self.cfg
        h, qkv, f = c.hidden, (c.heads + 2 * c.kv_heads) * c.head_dim, c.ffn
        return M.views(flat, [("norm1", (h,)), ("wqkv", (qkv, h)), ("wo", (h, h)), ("norm2", (h,)), ("w_gu", (2 * f, h)), ("w_down", (h, f))])

    def _up_to_attention(self, x, add, p, rope, shape, keep, backward):
        """(x + add, norm1's output and 1 / rms, q, k, v as attention takes them, its output [B, heads, S, head_dim]). The output carries what
        its backward takes if `backward`; with `keep`, which is for a later one, only if that is no more than `activation_bytes` counts."""
        c, (B, S) = self.cfg, shape
        x, h, rstd = self.norm(x, p["norm1"], add=add, need_rstd=backward)
        qkv = torch.mm(h, p["wqkv"].t())
        self.rope(qkv, rope, S)
        q, k, v = (t.transpose(1, 2) for t in qkv.view(B, S, c.heads + 2 * c.kv_heads, c.head_dim).split((c.heads, c.kv_heads, c.kv_heads), dim=2))
        with torch.set_grad_enabled(backward):
            if backward:
                q, k, v = (t.detach().requires_grad_(True) for t in (q, k, v))
                if keep and torch._fused_sdp_choice(q, k, v, is_causal=True, enable_gqa=True) == SDPBackend.MATH.value:
                    q, k, v = (t.detach() for t in (q, k, v))   # single operations: S x S probabilities per head, and k and v for every head
            return x, h, rstd, (q, k, v), F.scaled_dot_product_attention(q, k, v, is_causal=True, enable_gqa=True)

    def activation_bytes(self, tokens):
        """What `layer` hands over to its backward for so many tokens, beside its input."""
        c = self.cfg
        return tokens * (2 * (4 * c.hidden + (c.heads + 2 * c.kv_heads) * c.head_dim + 2 * c.ffn) + 4 * c.heads + 8)

    def _to_product(self, x, add, p, rope, shape, keep, backward):
        """(x + add, (norm1's output and 1 / rms, q, k, v, attention's output, norm2's sum, output and 1 / rms, gate and up))."""
        x, h1, rstd1, qkv, a = self._up_to_attention(x, add, p, rope, shape, keep, backward)
        o = a.detach().transpose(1, 2).reshape(x.shape)
        x2, h2, rstd2 = self.norm(x, p["norm2"], add=torch.mm(o, p["wo"].t()), need_rstd=backward)
        return x, (h1, rstd1, qkv, a, x2, h2, rstd2, torch.mm(h2, p["w_gu"].t()))

    def layer(self, x, add, flat, rope, shape, keep=False):
        """The layer of input x + add (add may be None), [B * S, hidden] with shape = (B, S): its input, its output as two terms that the next
        unit's norm adds up, and with `keep` what `layer_backward` would compute again (unless attention would save much more than that)."""
        p = self._layer_views(flat)
        x, acts = self._to_product(x, add, p, rope, shape, keep, keep)
        out = x, acts[4], torch.mm(self.swiglu(acts[7]), p["w_down"].t())
        return out + (acts,) if keep and acts[3].requires_grad else out

    def layer_backward(self, x, flat, gflat, rope, shape, gy, ready=None, before=None, kept=None):
        """Gradient of the layer's input; the weights' gradients go into gflat (laid out like flat). before() is called ahead of the first
        write into gflat, ready(lo) is told that from element lo on the gradients are written and the weights are read no more. `kept` holds
        what came from `layer` as the one element of a list, which is emptied: with no reference elsewhere it goes as it is used."""
        p, g = self._layer_views(flat), self._layer_views(gflat)
        begin = flat.data_ptr()

        def done(name):
            if ready:
                ready((p[name].data_ptr() - begin) // flat.element_size())

        h1, rstd1, qkv, a, x2, h2, rstd2, gu = kept.pop() if kept else self._to_product(x, None, p, rope, shape, False, True)[1]
        o = a.detach().transpose(1, 2).reshape(x.shape)
        act = torch.mm(gy, p["w_down"])
        self.swiglu_backward(gu, act)
        if before:
            before()   # the recomputation does not wait for whoever still reads gflat
        torch.mm(gy.t(), act, out=g["w_down"])
        done("w_down")
        del act
        dh = torch.mm(gu, p["w_gu"])
        torch.mm(gu.t(), h2, out=g["w_gu"])
        done("w_gu")
        del gu, h2
        g2 = self.norm_backward(x2, p["norm2"], rstd2, dh, gy, g["norm2"])
        torch.mm(g2.t(), o, out=g["wo"])
        do = torch.mm(g2, p["wo"]).view(shape[0], shape[1], self.cfg.heads, self.cfg.head_dim).transpose(1, 2)
        done("wo")
        dqkv = self.rope_backward(*torch.autograd.grad(a, qkv, do), rope, x.shape[0], shape[1])
        del a, qkv, o, do
        dh = torch.mm(dqkv, p["wqkv"])
        torch.mm(dqkv.t(), h1, out=g["wqkv"])
        return self.norm_backward(x, p["norm1"], rstd1, dh, g2, g["norm1"])

    def embedding_backward(self, tokens, gx, gflat):
        """The gradient of the table, into gflat."""
        c, ids = self.cfg, tokens.reshape(-1).contiguous()
        work = torch.empty(self._call["b200EmbeddingBackwardWork"](ids.numel(), c.hidden), dtype=torch.float32, device=ids.device)
        self._run("b200EmbeddingBackward", ids.data_ptr(), gx.data_ptr(), gflat.data_ptr(), work.data_ptr(), ids.numel(), c.vocab, c.hidden)

    def head(self, x, add, flat, gflat, targets, before=None):
        """(mean loss, gradient of the hidden states x + add); the weights' gradients go into gflat, before() ahead of them."""
        shapes = M.head_shapes(self.cfg)
        p, g = M.views(flat, shapes), M.views(gflat, shapes)
        x, h, rstd = self.norm(x, p["norm"], add=add, need_rstd=True)
        logits = torch.mm(h, p["out"].t())
        loss = self.cross_entropy(logits, targets)
        dh = torch.mm(logits, p["out"])
        if before:
            before()
        torch.mm(logits.t(), h, out=g["out"])
        return loss, self.norm_backward(x, p["norm"], rstd, dh, None, g["norm"])
