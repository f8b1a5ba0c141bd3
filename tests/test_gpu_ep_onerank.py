"""Expert-parallel groups of one rank: the local dispatch / combine kernels against PyTorch and against the general kernels
(which a split-phase call of the same group takes)."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def comm():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from nccl_b200 import Communicator, get_unique_id
    torch.cuda.set_device(0)
    c = Communicator(1, 0, get_unique_id())
    yield c
    c.destroy()


def _batch(T, E, K, H, seed, drop):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(T, H, device="cuda", generator=g).bfloat16()
    idx = torch.rand(T, E, device="cuda", generator=g).topk(K, dim=1).indices
    if drop:
        idx = torch.where(torch.rand(T, K, device="cuda", generator=g) < drop, torch.full_like(idx, -1), idx)
    return x, idx.contiguous(), torch.rand(T, K, device="cuda", generator=g)


# max_sms 1 makes one CTA serve several batches of 64 tokens; 256 experts and top-16 are the limits
@pytest.mark.parametrize("T,cap,E,K,H,max_sms,drop", [(1, 1, 1, 1, 128, 0, 0.0), (5, 9, 256, 8, 640, 0, 0.2), (64, 64, 32, 16, 1024, 0, 0.0),
                                                      (131, 140, 8, 3, 384, 1, 0.1), (700, 700, 16, 9, 7168, 0, 0.0), (2000, 2048, 8, 2, 128, 3, 0.3)])
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("layout", ["expert_major", "rank_major"])
def test_local_kernels_match_the_general_ones(comm, T, cap, E, K, H, max_sms, drop, fp8, layout):
    from nccl_b200.ops.ep import ExpertParallel
    ep = ExpertParallel(comm, E, cap, H, max_sms=max_sms, layout=layout)
    got = {}
    for split in (False, True, False):   # the general kernels in between: the handle's records serve both
        x, idx, w = _batch(T, E, K, H, 7, drop)
        lead = (E, cap) if layout == "expert_major" else (1, cap)
        toks = torch.zeros(*lead, H, dtype=torch.uint8 if fp8 else torch.bfloat16, device="cuda")
        scales = torch.zeros(*lead, H // 128, device="cuda") if fp8 else None
        toks, scales, counts = ep.dispatch(x, idx, w, fp8=fp8, toks=toks, scales=scales, send_only=split)
        if split:
            ep.complete()
        y = toks
        if fp8:
            y = (toks.view(torch.float8_e4m3fn).float().view(*lead, H // 128, 128) * scales.unsqueeze(-1)).view(*lead, H).bfloat16()
        out = ep.combine(y, send_only=split)
        if split:
            ep.complete()
        mixed = ep.combine(y)   # a whole combine after a split dispatch as well
        torch.cuda.synchronize()
        assert torch.equal(out, mixed)
        rows = [out, counts] + ([toks, ep.recv_topk_idx, ep.recv_topk_weights] + ([scales] if fp8 else []) if layout == "rank_major" else [])
        if got:
            assert all(torch.equal(a, b) for a, b in zip(rows, got["rows"]))   # bit for bit: same arithmetic in the same order
        got["rows"] = rows
        valid = (idx >= 0)
        assert torch.equal(counts.long(), torch.bincount(idx[valid], minlength=E))
        if layout == "expert_major":
            ref = x.float() * (w * valid).sum(1, keepdim=True)
        else:
            ref = x.float() * valid.any(1, keepdim=True)
        # e4m3 keeps 3 mantissa bits (2^-4 of the value), or 2^-9 of the block's scale among the subnormals; bf16 rounds twice
        tol = (2 ** -4 if fp8 else 2 ** -7) * ref.abs() + (2 ** -8 * x.float().abs().amax() * (1 + w.sum(1).max()) if fp8 else 1e-6)
        assert ((out.float() - ref).abs() <= tol).all()
    assert comm.async_error() == 0
    ep.destroy()


def test_expert_named_twice_and_tokens_at_eight_bytes(comm):
    from nccl_b200.ops.ep import ExpertParallel
    ep = ExpertParallel(comm, 4, 16, 256)
    x, idx, w = _batch(16, 4, 2, 256, 3, 0.0)
    raw = torch.zeros(16 * 256 + 4, dtype=torch.bfloat16, device="cuda")
    shifted = raw[4:].view(16, 256).copy_(x)   # 8-byte aligned: stays with the general kernel
    a = ep.dispatch(x, idx, w, fp8=True)[2].clone()
    b = ep.dispatch(shifted, idx, w, fp8=True)[2].clone()
    assert torch.equal(a, b)
    idx[:] = 1   # 32 claims for 16 rows: what does not fit is left out, nothing is written outside
    toks, _, counts = ep.dispatch(x, idx, w, fp8=False)
    torch.cuda.synchronize()
    assert counts.tolist() == [0, 16, 0, 0]
    idx.copy_(_batch(16, 4, 2, 256, 3, 0.0)[1])
    toks, _, counts = ep.dispatch(x, idx, w, fp8=False)
    out = ep.combine(toks)
    torch.cuda.synchronize()
    torch.testing.assert_close(out.float(), x.float() * w.sum(1, keepdim=True), rtol=2 ** -7, atol=1e-6)
    ep.destroy()


@pytest.mark.parametrize("layout", ["expert_major", "rank_major"])
def test_outputs_over_inputs(comm, layout):
    """A result may lie in the memory of what it is made from: the rows are read before any result is stored."""
    from nccl_b200.ops.ep import ExpertParallel
    T, E, K, H = 600, 4, 2, 1024
    ep = ExpertParallel(comm, E, T, H, layout=layout)
    x, idx, w = _batch(T, E, K, H, 11, 0.1)
    valid = idx >= 0
    y = ep.dispatch(x, idx, w, fp8=False)[0].clone()
    want = ep.combine(y).clone()
    scale = (w * valid).sum(1, keepdim=True) if layout == "expert_major" else valid.any(1, keepdim=True)
    torch.testing.assert_close(want.float(), x.float() * scale, rtol=2 ** -7, atol=1e-6)
    for shift in (0, 1, 5):   # rows of the input that the first row of the result lies behind its start
        z = torch.empty(y.numel() + shift * H, dtype=y.dtype, device="cuda")
        z[:y.numel()] = y.view(-1)
        out = z[shift * H:(shift + T) * H].view(T, H)
        assert torch.equal(ep.combine(z[:y.numel()].view(y.shape), out=out), want)
    for shift in (0, 3):      # the tokens lie in the tensor that they are dispatched to
        toks = torch.zeros_like(y)
        inside = toks.view(-1, H)[shift:shift + T] if shift + T <= toks.numel() // H else toks.view(-1, H)[:T]
        inside.copy_(x)
        got, _, counts = ep.dispatch(inside, idx, w, fp8=False, toks=toks)
        assert torch.equal(counts.long(), torch.bincount(idx[valid], minlength=E))
        assert torch.equal(ep.combine(got), want)
    torch.cuda.synchronize()
    assert comm.async_error() == 0
    ep.destroy()


@pytest.mark.parametrize("layout", ["expert_major", "rank_major"])
def test_counts_outside_the_gpu(comm, layout):
    """Expert counts may be asked for in pinned host memory; memory that the GPU cannot reach is refused with an error."""
    from nccl_b200.ops.ep import ExpertParallel
    ep = ExpertParallel(comm, 8, 32, 256, layout=layout)
    x, idx, w = _batch(32, 8, 2, 256, 5, 0.2)
    want = torch.bincount(idx[idx >= 0], minlength=8).cpu()
    pinned = torch.zeros(8, dtype=torch.int32).pin_memory()
    ep.dispatch(x, idx, w, fp8=False, counts=pinned)
    torch.cuda.synchronize()
    assert torch.equal(pinned.long(), want)
    with pytest.raises(Exception):
        ep.dispatch(x, idx, w, fp8=False, counts=torch.zeros(8, dtype=torch.int32))
    torch.cuda.synchronize()
    assert torch.equal(ep.dispatch(x, idx, w, fp8=False)[2].long().cpu(), want)
    torch.cuda.synchronize()
    assert comm.async_error() == 0
    ep.destroy()


@pytest.mark.parametrize("layout", ["expert_major", "rank_major"])
def test_calls_in_a_row_leave_no_counts_behind(comm, layout):
    """Tickets are taken before the payload is through: calls behind each other without waiting, of changing sizes, none among them."""
    from nccl_b200.ops.ep import ExpertParallel
    E, K, H, cap = 64, 6, 2048, 900
    ep = ExpertParallel(comm, E, cap, H, layout=layout)
    got, want = [], []
    for T in (900, 1, 513, 64, 899, 3):
        x, idx, w = _batch(T, E, K, H, T, 0.2)
        counts = torch.full((E,), 7, dtype=torch.int32, device="cuda")
        toks = ep.dispatch(x, idx, w, fp8=False, counts=counts)[0].clone()
        valid = idx >= 0
        scale = (w * valid).sum(1, keepdim=True) if layout == "expert_major" else valid.any(1, keepdim=True)
        got.append((counts, ep.combine(toks)[:T].clone()))
        want.append((torch.bincount(idx[valid], minlength=E), x.float() * scale))
    torch.cuda.synchronize()
    for (c, out), (cr, ref) in zip(got, want):
        assert torch.equal(c.long(), cr)
        torch.testing.assert_close(out.float(), ref, rtol=2 ** -7, atol=1e-6)
    assert comm.async_error() == 0
    ep.destroy()


@pytest.mark.parametrize("T,H,max_sms", [(1, 128, 0), (33, 384, 0), (200, 640, 1)])
@pytest.mark.parametrize("fp8", [False, True])
def test_tokens_at_sixteen_bytes(comm, T, H, max_sms, fp8):
    """Tokens that start on 16 bytes, but not on 32, give the bytes that aligned ones give, and nothing beside the rows is written."""
    from nccl_b200.ops.ep import ExpertParallel
    ep = ExpertParallel(comm, 8, T, H, max_sms=max_sms, layout="rank_major")
    x, idx, w = _batch(T, 8, 2, H, 11, 0.1)
    dt, off = (torch.uint8, 16) if fp8 else (torch.bfloat16, 8)
    got = []
    for at_in, at_out in ((0, 0), (8, 0), (0, off), (8, off)):
        xs = torch.empty(T * H + 16, dtype=torch.bfloat16, device="cuda")[at_in:at_in + T * H].view(T, H).copy_(x)
        buf = torch.full((T * H + 64,), 7, dtype=dt, device="cuda")
        toks = buf[at_out:at_out + T * H].view(1, T, H)
        assert xs.data_ptr() % 32 == 2 * at_in and toks.data_ptr() % 32 == (16 if at_out else 0)
        scales = torch.zeros(1, T, H // 128, device="cuda") if fp8 else None
        ep.dispatch(xs, idx, w, fp8=fp8, toks=toks, scales=scales)
        torch.cuda.synchronize()
        assert (buf[:at_out] == 7).all() and (buf[at_out + T * H:] == 7).all()
        used = (idx >= 0).any(1)
        got.append((toks[0][used].clone(), scales[0][used].clone() if fp8 else None))
    for toks, scales in got[1:]:
        assert torch.equal(toks, got[0][0]) and (not fp8 or torch.equal(scales, got[0][1]))
    if not fp8:
        assert torch.equal(got[0][0], x[(idx >= 0).any(1)])
    ep.destroy()


@pytest.mark.parametrize("layout", ["expert_major", "rank_major"])
@pytest.mark.parametrize("T,K,H", [(1, 1, 128), (37, 3, 384), (65, 4, 640), (6000, 4, 4096), (2700, 8, 4096)])
def test_results_at_sixteen_bytes(comm, T, K, H, layout):
    """Combine with rows and results that start on 16 bytes, but not on 32, gives the bytes that aligned ones give: on each side of the lines
    between accesses of 16 and 32 bytes."""
    from nccl_b200.ops.ep import ExpertParallel
    E = 16
    ep = ExpertParallel(comm, E, T, H, layout=layout)
    x, idx, w = _batch(T, E, K, H, 13, 0.1)
    toks, _, _ = ep.dispatch(x, idx, w, fp8=False)
    y = toks if layout == "expert_major" else torch.randn(1, T, H, device="cuda").bfloat16()
    want = None
    for at_in, at_out in ((0, 0), (8, 0), (0, 8), (8, 8)):
        ys = torch.empty(y.numel() + 16, dtype=torch.bfloat16, device="cuda")[at_in:at_in + y.numel()].view(y.shape).copy_(y)
        buf = torch.full((T * H + 32,), 7.0, dtype=torch.bfloat16, device="cuda")
        out = ep.combine(ys, out=buf[at_out:at_out + T * H].view(T, H))
        torch.cuda.synchronize()
        assert (buf[:at_out] == 7).all() and (buf[at_out + T * H:] == 7).all()
        want = out.clone() if want is None else want
        assert torch.equal(out, want)
    used = (idx >= 0).any(1)
    if layout == "rank_major":
        assert torch.equal(want, y[0] * used[:, None])
    else:   # one bf16 rounding of an fp32 sum of at most eight products
        ref = x.double() * (w.double() * (idx >= 0)).sum(1, keepdim=True)
        assert ((want.double() - ref).abs() <= 2 ** -8 * ref.abs() + 2 ** -20 * x.double().abs() * w.double().sum(1, keepdim=True)).all()
    ep.destroy()
