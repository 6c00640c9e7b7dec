"""Edge sizes of the kernels whose dispatch depends on the shape, against plain PyTorch in fp32 or fp64 (needs a B200).

Tolerances: a bf16 result differs from the exact one by up to 2^-9 relative per element from its own rounding; attention rounds
the probabilities and dS to bf16 as well, which the products average over many keys.  So 1e-2 in the 2-norm for one product and
2e-2 / 3e-2 for attention forward / backward, as in the kernels' main tests; copies and single-rounding sums are exact.
"""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _dev():
    return torch.device("cuda", 0)


def _status_ok():
    from fairscale_b200 import _native

    torch.cuda.synchronize()
    assert _native.read_status(_dev()) == 0


def _rel_err(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-12)).item()


def _attention_ref(x, H):
    B, S, W = x.shape
    D = W // (3 * H)
    q, k, v = x.view(B, S, 3, H, D).permute(2, 0, 3, 1, 4)
    s = (q @ k.transpose(-1, -2)) / math.sqrt(D)
    s = s.masked_fill(torch.ones(S, S, dtype=torch.bool, device=x.device).triu(1), float("-inf"))
    return (torch.softmax(s, -1) @ v).transpose(1, 2).reshape(B, S, H * D)


# one row, less than a tile, one row more or less than a tile of 128 and a pair of tiles, an odd number of tiles whose last
# pair has one tile (with more items than SMs too, so that the persistent kernels meet both kinds of item), a long ragged one
@pytest.mark.parametrize("B,S,H,D", [(1, 1, 1, 64), (2, 5, 2, 128), (2, 77, 3, 64), (1, 127, 2, 128), (2, 129, 2, 128), (1, 255, 2, 64),
                                     (3, 257, 2, 128), (1, 385, 2, 64), (2, 384, 3, 64), (40, 300, 8, 64), (24, 650, 16, 128), (2, 1543, 4, 128)])
def test_attention_any_length(B, S, H, D):
    from fairscale_b200.ops import attention

    torch.manual_seed(S)
    x = (torch.randn(B, S, 3 * H * D, device=_dev()) * 0.7).bfloat16().requires_grad_()
    o = attention.causal_attention(x, H)
    assert attention.BACKEND == "tcgen05"
    go = torch.randn_like(o)
    o.backward(go)
    _status_ok()
    ref = x.detach().float().requires_grad_()
    oref = _attention_ref(ref, H)
    oref.backward(go.float())
    assert _rel_err(o, oref) < 2e-2
    g, gr = x.grad.view(B, S, 3, H, D), ref.grad.view(B, S, 3, H, D)
    for i in range(3):
        # with one or five keys dQ and dK are (almost) zero: measure them against the whole gradient there
        scale = gr[:, :, i].norm() if S > 64 else gr.norm()
        assert ((g[:, :, i].float() - gr[:, :, i]).norm() / scale).item() < 3e-2, i


def test_attention_ragged_rows_do_not_mix():
    """A sequence's last tile must not see the next sequence of the batch, and rows past the end are not written."""
    from fairscale_b200.ops.attention import causal_attention

    torch.manual_seed(0)
    B, S, H, D = 3, 200, 2, 64
    x = torch.randn(B, S, 3 * H * D, device=_dev()).bfloat16()
    go = torch.randn(B, S, H * D, device=_dev()).bfloat16()
    whole = x.clone().requires_grad_()
    o = causal_attention(whole, H)
    o.backward(go)
    for b in range(B):
        one = x[b : b + 1].clone().requires_grad_()
        ob = causal_attention(one, H)
        ob.backward(go[b : b + 1])
        assert torch.equal(ob[0], o[b]) and torch.equal(one.grad[0], whole.grad[b])
    # a view that starts off a 16-byte boundary, and a gradient that is not contiguous
    flat = torch.empty(B * S * 3 * H * D + 1, device=_dev(), dtype=torch.bfloat16)
    odd = flat[1:].view(B, S, -1)
    odd.copy_(x)
    odd.requires_grad_()
    od = causal_attention(odd, H)
    od.backward(go.transpose(0, 1).contiguous().transpose(0, 1))
    assert torch.equal(od, o) and torch.equal(odd.grad, whole.grad)
    _status_ok()


def test_attention_ragged_infinities_stay_where_they_are():
    from fairscale_b200.ops.attention import causal_attention

    torch.manual_seed(0)
    S, D = 150, 64
    x = torch.randn(1, S, 3 * D, device=_dev()).bfloat16()
    x[0, 140, D : 2 * D] = float("inf")  # one key: no query before it may notice
    a = causal_attention(x, 1)
    y = x.clone()
    y[0, 140, D : 2 * D] = 0
    assert torch.equal(a[0, :140], causal_attention(y, 1)[0, :140])


@pytest.mark.parametrize("S,D", [(300, 64), (300, 128), (512, 64), (512, 128)])
def test_attention_rows_whose_first_keys_score_minus_infinity(S, D):
    """A whole first key tile at -inf leaves the later keys as they are."""
    from fairscale_b200.ops.attention import causal_attention

    torch.manual_seed(S + D)
    H = 2
    x = torch.randn(2, S, 3, H, D, device=_dev()).bfloat16()
    x[:, :, 0, :, 0] = 1.0
    x[:, :128, 1, :, 0] = float("-inf")
    x = x.view(2, S, 3 * H * D)
    o, ref = causal_attention(x, H), _attention_ref(x.float(), H)
    _status_ok()
    assert torch.isfinite(ref[:, 128:]).all() and torch.isfinite(o[:, 128:]).all()
    assert _rel_err(o[:, 128:], ref[:, 128:]) < 2e-2


def test_attention_of_ragged_lengths_under_autocast():
    """Autocast to another 16-bit type casts what torch's operator takes; bf16 autocast leaves the kernels in place."""
    from fairscale_b200.ops import attention

    torch.manual_seed(0)
    x = torch.randn(1, 77, 3 * 2 * 64, device=_dev()).bfloat16()
    for dtype, backend in ((torch.float16, "torch-sdpa"), (torch.bfloat16, "tcgen05")):
        with torch.autocast("cuda", dtype):
            o = attention.causal_attention(x, 2)
        assert o.dtype == dtype and attention.BACKEND == backend
        assert _rel_err(o, _attention_ref(x.float(), 2)) < 2e-2


# (B, S, H): short, few heads and long, many heads and long, beyond the longest
@pytest.mark.parametrize("B,S,H,trains,infers", [(1, 77, 2, True, True), (1, 2500, 2, False, False), (2, 2500, 4, True, False), (1, 5601, 8, False, False),
                                                 (70, 100, 10, True, False)])
def test_attention_of_ragged_lengths_runs_where_it_is_faster(B, S, H, trains, infers):
    from fairscale_b200.ops import attention

    torch.manual_seed(0)
    x = torch.randn(B, S, 3 * H * 64, device=_dev()).bfloat16()
    with torch.no_grad():
        o = attention.causal_attention(x, H)
    assert (attention.BACKEND == "tcgen05") == trains  # the same kernels with and without gradients
    y = x.clone().requires_grad_()
    assert torch.equal(attention.causal_attention(y, H), o) and (attention.BACKEND == "tcgen05") == trains
    with torch.inference_mode():
        i = attention.causal_attention(x, H)
    assert (attention.BACKEND == "tcgen05") == infers
    assert _rel_err(i.clone(), o) < 2e-2
    _status_ok()


@pytest.mark.parametrize("D", [64, 128])
def test_attention_scales_of_either_sign(D):
    """A scale that is zero or negative is taken at multiples of 128, as it always was."""
    from fairscale_b200.ops.attention import causal_attention

    torch.manual_seed(D)
    H = 2
    x = torch.randn(1, 384, 3, H, D, device=_dev()).bfloat16()
    for scale in (-1.0, 0.0, 1.0):
        y = x.clone()
        y[:, :, 0] *= scale
        want = _attention_ref(y.view(1, 384, -1).float(), H)
        assert _rel_err(causal_attention(x.view(1, 384, -1), H, scale / math.sqrt(D)), want) < 2e-2
    _status_ok()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("S,E,M", [(64, 4, 1024), (820, 4, 512), (48, 16, 33), (8, 2, 8)])
def test_moe_rows_match_index_ops(S, E, M, dtype):
    """Dispatch and combine of one rank on the row kernels against the index formulation that the CPU runs."""
    import torch.distributed as dist

    from fairscale_b200.nn.moe import top2gate
    from fairscale_b200.nn.moe.moe_layer import _Combine, _Dispatch

    if not dist.is_initialized():
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1)
    group = dist.group.WORLD
    torch.manual_seed(S + M)
    logits = torch.randn(S, E, device=_dev()) + torch.linspace(2, 0, E, device=_dev())  # crowded first experts: some choices overflow
    noise = top2gate.gumbel_rsample(logits.shape, logits.device)
    x = torch.randn(S, M, device=_dev()).to(dtype)
    dy = torch.randn(S, M, device=_dev()).to(dtype)
    got = {}
    for where, cast in (("gpu", lambda t: t), ("cpu", lambda t: t.cpu())):
        lg, xx = (cast(t).detach().clone().requires_grad_() for t in (logits, x))
        route = top2gate.top2_route(lg, cast(noise))
        rows = _Dispatch.apply(xx, route, group, E)
        weight = cast(torch.arange(1, E + 1, device=_dev())).to(dtype).view(E, 1, 1)  # experts that differ, or the gates' gradient is zero
        out = _Combine.apply(rows * weight, route.gate, route, group, E)
        out.backward(cast(dy))
        got[where] = [t.detach().cpu() for t in (rows, out, xx.grad, lg.grad)]
    _status_ok()
    assert torch.equal(got["gpu"][0], got["cpu"][0])
    eps = {torch.float32: 1e-5, torch.float16: 2e-3, torch.bfloat16: 1.6e-2}[dtype]  # gates differ by fp32 rounding, so results by a last bit
    for a, b in zip(got["gpu"][1:], got["cpu"][1:]):
        torch.testing.assert_close(a.float(), b.float(), rtol=eps, atol=eps * b.float().abs().max().item())


# a gate that changes what the routing kernels made: choices dropped out of place and in place, a smaller capacity
@pytest.mark.parametrize("change", ["replace", "in_place", "capacity"])
def test_moe_rows_follow_a_route_that_was_changed(change):
    import torch.distributed as dist

    from fairscale_b200.nn.moe import GroupedExperts, MOELayer, Top2Gate

    if not dist.is_initialized():
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1)

    class PickyGate(Top2Gate):
        def route(self, x):
            r = super().route(x)
            if change == "capacity":
                small = r.capacity // 2
                return r._replace(capacity=small, keep=r.keep & (r.slot < small), slot=r.slot * (r.slot < small))
            allowed = (torch.arange(r.keep.shape[0], device=r.keep.device) % 3 > 0).unsqueeze(1)
            if change == "in_place":
                r.keep.logical_and_(allowed)
                return r
            return r._replace(keep=r.keep & allowed)

    torch.manual_seed(1)
    S, E, M = 96, 4, 64
    layer = MOELayer(PickyGate(M, E), GroupedExperts(E, M, 2 * M)).to(_dev()).to(torch.bfloat16)
    seen = {}
    layer.experts[0].register_forward_hook(lambda m, i, o: seen.update(rows=i[0].detach(), out=o))
    x = torch.randn(1, S, M, device=_dev()).bfloat16().requires_grad_()
    torch.full((64 << 20,), float("nan"), device=_dev())  # memory that the layer's buffers may be taken from
    route = {}
    inner = layer.gate.route
    layer.gate.route = lambda t: route.setdefault("r", inner(t))
    layer(x.view(E, S // E, M)).float().sum().backward()
    r = route["r"]
    want = torch.zeros(E * r.capacity, M, device=_dev(), dtype=torch.bfloat16)
    for k in range(2):
        kept = r.keep[:, k]
        want[(r.expert * r.capacity + r.slot)[kept, k]] = x.detach().view(S, M)[kept]
    assert torch.equal(seen["rows"].reshape(-1, M), want)
    assert torch.isfinite(x.grad).all() and all(torch.isfinite(p.grad).all() for p in layer.parameters())
    assert not r.keep.all()
    _status_ok()


def test_moe_row_gradients_can_be_differentiated():
    """create_graph: what the CPU formulation offers (a gradient that is differentiable in the incoming one) holds on the GPU."""
    import torch.distributed as dist

    from fairscale_b200.nn.moe import top2gate
    from fairscale_b200.nn.moe.moe_layer import _Combine, _Dispatch

    if not dist.is_initialized():
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1)
    torch.manual_seed(3)
    S, E, M = 64, 4, 40
    logits = torch.randn(S, E, device=_dev()) + torch.linspace(2, 0, E, device=_dev())
    noise = top2gate.gumbel_rsample(logits.shape, logits.device)
    x, dy = torch.randn(S, M, device=_dev()), torch.randn(S, M, device=_dev())
    got = {}
    for where, cast in (("gpu", lambda v: v.detach().clone()), ("cpu", lambda v: v.detach().cpu())):
        xx, gg, dd = (cast(v).requires_grad_() for v in (x, logits, dy))
        route = top2gate.top2_route(gg, cast(noise))
        scale = cast(torch.arange(1.0, E + 1, device=_dev())).view(E, 1, 1)
        out = _Combine.apply(_Dispatch.apply(xx, route, dist.group.WORLD, E) * scale, route.gate, route, dist.group.WORLD, E)
        first = torch.autograd.grad(out, (xx, route.gate), dd, create_graph=True)
        (second,) = torch.autograd.grad(sum(f.pow(2).sum() for f in first), dd)
        got[where] = [v.detach().cpu() for v in (*first, second)]
    _status_ok()
    for a, b in zip(got["gpu"], got["cpu"]):
        torch.testing.assert_close(a, b, rtol=1e-4, atol=1e-4 * b.abs().max().item())


def test_moe_experts_may_reuse_their_output_buffer():
    """The layer keeps no hold on the experts' output: a second forward may overwrite it before the first one's backward."""
    import torch.distributed as dist

    from fairscale_b200.nn.moe import MOELayer, Top2Gate

    if not dist.is_initialized():
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1)
    S, E, M = 64, 4, 32

    class Scale(torch.autograd.Function):
        @staticmethod
        def forward(ctx, x, scale, buf):
            ctx.scale = scale
            out = torch.empty_like(x) if buf is None else buf
            return torch.mul(x, scale, out=out.view(x.shape)).view(x.shape)

        @staticmethod
        def backward(ctx, g):
            return g * ctx.scale, None, None

    class Experts(torch.nn.Module):
        grouped = True

        def __init__(self, buf):
            super().__init__()
            self.buf, self.scale = buf, torch.arange(1.0, E + 1, device=_dev()).view(E, 1, 1)

        def __len__(self):
            return E

        def forward(self, x):
            return Scale.apply(x, self.scale, self.buf)

    torch.manual_seed(5)
    x1, x2 = (torch.randn(E, S // E, M, device=_dev()) for _ in range(2))
    gate = Top2Gate(M, E).to(_dev())
    grads = []
    for buf in (None, torch.empty(E, 2 * S // E, M, device=_dev())):
        layer = MOELayer(gate, Experts(buf))
        x = x1.clone().requires_grad_()
        gate.zero_grad()
        torch.manual_seed(6)  # the gate's noise
        y = layer(x)
        layer(x2)
        y.pow(2).sum().backward()
        grads.append((x.grad, gate.wg.weight.grad.clone()))
    _status_ok()
    for a, b in zip(*grads):
        torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-5)


# (M, N, K): below, at and above the 128 x 64 / 128 x 128 tiles, K of one block, K no multiple of a block, K with fewer
# blocks than a cluster could split
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("M,N,K", [(8, 8, 64), (77, 1000, 1024), (128, 64, 512), (136, 72, 520), (256, 200, 136), (264, 128, 4096)])
@pytest.mark.parametrize("block_n,splits", [(64, 1), (64, 8), (128, 1), (128, 2), (128, 4)])
def test_cluster_split_k_gemm(M, N, K, a_mn, b_mn, block_n, splits):
    from ctypes import c_int, c_void_p

    from fairscale_b200.ops import _bind

    _bind._SIGNATURES.setdefault("fsb_gemm_bf16_cluster_k", [c_void_p] * 6 + [c_int] * 14 + [c_void_p, c_void_p])
    torch.manual_seed(M + N + K)
    a = torch.randn((K, -(-M // 8) * 8), device=_dev()).bfloat16()[:, :M] if a_mn else torch.randn((M, K), device=_dev()).bfloat16()
    b = torch.randn((K, N) if b_mn else (N, K), device=_dev()).bfloat16()
    bias = torch.randn(N, device=_dev()).bfloat16()
    aux = torch.randn(M, N, device=_dev()).bfloat16()
    ref = (a.t() if a_mn else a).double() @ (b if b_mn else b.t()).double()

    def run(epi, dtype=torch.bfloat16, use_bias=False, use_aux=False, pre=None, into=None, accumulate=0):
        c = into if into is not None else torch.full((M, N), float("nan"), device=_dev(), dtype=dtype)
        code = _bind.fn("fsb_gemm_bf16_cluster_k")(
            a.data_ptr(), b.data_ptr(), c.data_ptr(), bias.data_ptr() if use_bias else None, aux.data_ptr() if use_aux else None,
            _bind.ptr(pre), M, N, K, a.stride(0), b.stride(0), N, N, int(a_mn), int(b_mn), epi, int(dtype == torch.float32), accumulate,
            block_n, splits, _bind.status_ptr(_dev()), _bind.stream_ptr(_dev()))
        assert code == (-1 if splits > -(-K // 64) else 0)
        return c

    if splits > -(-K // 64):
        run(0)  # refused: a CTA of the cluster would have no K block
        return
    assert _rel_err(run(0), ref) < 1e-2
    f32 = run(0, torch.float32)
    assert _rel_err(f32, ref) < 1e-5
    assert _rel_err(run(0, torch.float32, into=f32.clone(), accumulate=1), 2 * ref) < 1e-5
    with_bias = ref + bias.double()
    pre = torch.empty(M, N, device=_dev(), dtype=torch.bfloat16)
    assert _rel_err(run(2, use_bias=True, pre=pre), torch.nn.functional.gelu(with_bias)) < 1e-2
    assert _rel_err(pre, with_bias) < 1e-2
    assert _rel_err(run(3, use_bias=True, use_aux=True), with_bias + aux.double()) < 1e-2
    z = aux.double().requires_grad_()
    torch.nn.functional.gelu(z).sum().backward()
    assert _rel_err(run(4, use_aux=True), ref * z.grad) < 1e-2
    assert torch.equal(run(0, torch.float32), f32)  # the cluster sums in a fixed order
    _status_ok()


# The persistent GEMM kernels by name, whatever the dispatch makes of the size: 1 one CTA per tile, 2 CTA pairs (256 x 256 tiles).
# Whole tiles, remainders in M, N and K, fewer tiles than one wave of either kernel, more than one wave of both.
@pytest.mark.parametrize("plan", [1, 2])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (264, 328, 136), (520, 264, 1000), (1000, 264, 8192), (2600, 2056, 520), (8200, 1800, 264)])
def test_persistent_gemm_kernels(M, N, K, a_mn, b_mn, plan):
    from ctypes import c_int, c_void_p

    from fairscale_b200.ops import _bind

    _bind._SIGNATURES.setdefault("fsb_gemm_bf16_plan", [c_void_p] * 6 + [c_int] * 13 + [c_void_p] * 2)
    torch.manual_seed(M + N + K)
    a, b, aux = (torch.randn(*s, device=_dev()).bfloat16() for s in ((M, K), (N, K), (M, N)))
    bias = torch.randn(N, device=_dev()).bfloat16()
    sa, sb = (t.t().contiguous() if mn else t for t, mn in ((a, a_mn), (b, b_mn)))
    ref = a.double() @ b.double().t()

    def run(epi, dtype=torch.bfloat16, use_aux=False, pre=None, accumulate=0, into=None):
        c = torch.full((M, N), float("nan"), device=_dev(), dtype=dtype) if into is None else into
        _bind.call("fsb_gemm_bf16_plan", sa.data_ptr(), sb.data_ptr(), c.data_ptr(), bias.data_ptr() if epi in (1, 2, 3) else None,
                   aux.data_ptr() if use_aux else None, _bind.ptr(pre), M, N, K, sa.stride(0), sb.stride(0), N, N, int(a_mn), int(b_mn),
                   epi, int(dtype == torch.float32), accumulate, plan, _bind.status_ptr(_dev()), _bind.stream_ptr(_dev()))
        return c

    assert _rel_err(run(0), ref) < 1e-2
    f32 = run(0, torch.float32)
    assert _rel_err(f32, ref) < 1e-5
    assert _rel_err(run(0, torch.float32, into=f32.clone(), accumulate=1), 2 * ref) < 1e-5
    with_bias = ref + bias.double()
    assert _rel_err(run(1), with_bias) < 1e-2
    pre = torch.empty(M, N, device=_dev(), dtype=torch.bfloat16)
    assert _rel_err(run(2, pre=pre), torch.nn.functional.gelu(with_bias)) < 1e-2
    assert _rel_err(pre, with_bias) < 1e-2
    assert _rel_err(run(3, use_aux=True), with_bias + aux.double()) < 1e-2
    z = aux.double().requires_grad_()
    torch.nn.functional.gelu(z).sum().backward()
    assert _rel_err(run(4, use_aux=True), ref * z.grad) < 1e-2
    assert _rel_err(run(5, use_aux=True), ref + aux.double()) < 1e-2
    assert torch.equal(run(0, torch.float32), f32)
    _status_ok()


# The CTA-pair kernel with tiles of 512 x 256 (plan 3): one tile, remainders in M, N and K, more tiles than pairs, stacked problems, a
# bias that starts off a 16-byte boundary.  It sums K in the order of the 256 x 256 tiles: every result is the same to the bit.
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("E,M,N,K", [(1, 512, 256, 64), (1, 520, 264, 8), (1, 776, 1000, 264), (1, 5128, 4360, 520), (3, 1032, 264, 200), (5, 2056, 2056, 136)])
def test_wide_pair_gemm(E, M, N, K, a_mn, b_mn):
    from ctypes import c_int, c_longlong, c_void_p

    from fairscale_b200.ops import _bind

    _bind._SIGNATURES.setdefault("fsb_gemm_bf16_plan", [c_void_p] * 6 + [c_int] * 13 + [c_void_p] * 2)
    _bind._SIGNATURES.setdefault("fsb_gemm_bf16_batched_plan", [c_void_p] * 6 + [c_int] * 8 + [c_longlong] * 5 + [c_int] * 6 + [c_void_p, c_void_p])
    torch.manual_seed(M + N + K)
    a, b = (torch.randn(*s, device=_dev()).bfloat16() for s in ((E, M, K), (E, N, K)))
    bias = torch.randn(E * N + 1, device=_dev()).bfloat16()[1:].view(E, N)
    sa, sb = (t.transpose(1, 2).contiguous() if mn else t for t, mn in ((a, a_mn), (b, b_mn)))
    ref = a.double() @ b.double().transpose(1, 2)

    def run(epi, plan):
        c = torch.full((E, M, N), float("nan"), device=_dev(), dtype=torch.bfloat16)
        ptrs = (sa.data_ptr(), sb.data_ptr(), c.data_ptr(), bias.data_ptr() if epi else None, None, None)
        tail = (int(a_mn), int(b_mn), epi, 0, 0, plan, _bind.status_ptr(_dev()), _bind.stream_ptr(_dev()))
        if E == 1:
            _bind.call("fsb_gemm_bf16_plan", *ptrs, M, N, K, sa.stride(1), sb.stride(1), N, 0, *tail)
        else:
            _bind.call("fsb_gemm_bf16_batched_plan", *ptrs, E, M, N, K, sa.stride(1), sb.stride(1), N, 0, sa.stride(0), sb.stride(0), M * N, 0, N, *tail)
        return c

    for epi, want in ((0, ref), (1, ref + bias.double().unsqueeze(1))):
        got = run(epi, 3)
        assert _rel_err(got, want) < 1e-2
        assert torch.equal(got, run(epi, 2))
    _status_ok()


@pytest.mark.parametrize("plan", [0, 1, 2])
@pytest.mark.parametrize("E,C,K,N", [(2, 256, 256, 256), (3, 257, 72, 264), (3, 257, 264, 264), (4, 410, 512, 2048), (1, 300, 64, 256), (17, 300, 264, 520)])
def test_batched_gemm_edges(E, C, K, N, plan):
    """Stacked problems on either kernel (0: the dispatch's choice); remainders must not leak into the next problem."""
    from ctypes import c_int, c_longlong, c_void_p

    from fairscale_b200.ops import _bind, gemm

    _bind._SIGNATURES.setdefault("fsb_gemm_bf16_batched_plan", [c_void_p] * 6 + [c_int] * 8 + [c_longlong] * 5 + [c_int] * 6 + [c_void_p, c_void_p])
    torch.manual_seed(C)
    x = torch.randn(E, C, K, device=_dev()).bfloat16()
    w = torch.randn(E, N, K, device=_dev()).bfloat16()
    dy = torch.randn(E, C, N, device=_dev()).bfloat16()
    b = torch.randn(E, N, device=_dev()).bfloat16()
    call = _bind.call

    def planned(name, *args, **kw):
        if plan == 1 or (plan == 2 and min(args[7:9]) >= 256):  # the pairs take M and N from 256 on
            name, args = name + "_plan", args[:-2] + (plan,) + args[-2:]
        call(name, *args, **kw)

    _bind.call = planned
    try:
        y, _ = gemm.batched_linear_forward(x, w, b)
        act, pre = gemm.batched_linear_forward(x, w, b, gelu=True, save_pre_activation=True)
        dx, dw = gemm.batched_linear_dgrad(dy, w), gemm.batched_linear_wgrad(dy, x)
        dx_act = gemm.batched_linear_dgrad(dy, w, dgelu_pre=x)
    finally:
        _bind.call = call
    _status_ok()
    want = torch.baddbmm(b.double().unsqueeze(1), x.double(), w.double().transpose(1, 2))
    z = x.double().requires_grad_()
    torch.nn.functional.gelu(z).sum().backward()
    for e in range(E):
        assert _rel_err(y[e], want[e]) < 1e-2 and _rel_err(pre[e], want[e]) < 1e-2
        assert _rel_err(act[e], torch.nn.functional.gelu(want[e])) < 1e-2
        d = dy[e].double() @ w[e].double()
        assert _rel_err(dx[e], d) < 1e-2 and _rel_err(dx_act[e], d * z.grad[e]) < 1e-2
        assert _rel_err(dw[e], dy[e].double().t() @ x[e].double()) < 1e-2


def test_products_beyond_the_pair_threshold():
    """The dispatch's own way onto CTA pairs; M, N and K no multiples of the tiles."""
    from ctypes import c_int, c_longlong

    from fairscale_b200.ops import _bind
    from fairscale_b200.ops.gemm import batched_linear_forward, linear_dgrad, linear_forward, linear_wgrad

    _bind._SIGNATURES.setdefault("fsb_gemm_plan_of", [c_longlong] + [c_int] * 6)
    plan_of, sms = _bind.fn("fsb_gemm_plan_of"), torch.cuda.get_device_properties(0).multi_processor_count
    torch.manual_seed(8)
    M, N, K = 8200, 4360, 4360
    assert plan_of(1, M, N, K, K, K, sms) == plan_of(1, M, K, N, N, K, sms) == plan_of(1, N, K, M, N, K, sms) == plan_of(4, 2048, N, K, K, K, sms) == 0
    x, w, dy = (torch.randn(*s, device=_dev()).bfloat16() for s in ((M, K), (N, K), (M, N)))
    b, res = torch.randn(N, device=_dev()).bfloat16(), torch.randn(M, N, device=_dev()).bfloat16()
    # fp32 oracle: its own sums differ by 1e-6, far below one rounding to bf16
    assert _rel_err(linear_forward(x, w, b, residual=res)[0], x.float() @ w.float().t() + b.float() + res.float()) < 1e-2
    assert _rel_err(linear_dgrad(dy, w), dy.float() @ w.float()) < 1e-2
    assert _rel_err(linear_wgrad(dy, x), dy.float().t() @ x.float()) < 1e-2
    xe, we, be = x[:8192].view(4, 2048, K), torch.randn(4, N, K, device=_dev()).bfloat16(), torch.randn(4, N, device=_dev()).bfloat16()
    y, _ = batched_linear_forward(xe, we, be)
    for e in range(4):
        assert _rel_err(y[e], xe[e].float() @ we[e].float().t() + be[e].float()) < 1e-2
    _status_ok()


@pytest.mark.parametrize("E,rows,H", [(1, 1, 8), (3, 63, 256), (4, 410, 2048), (2, 5000, 264)])
def test_batched_column_sum(E, rows, H):
    from fairscale_b200.ops.reduce import batched_column_sum

    torch.manual_seed(rows)
    x = torch.randn(E, rows, H, device=_dev()).bfloat16()
    want = x.double().sum(1)
    # fp32 sums of `rows` terms and one rounding to bf16
    torch.testing.assert_close(batched_column_sum(x).double(), want, rtol=2**-8, atol=1e-5 * rows)
    assert torch.equal(batched_column_sum(x)[-1], batched_column_sum(x[-1:])[0])


# one column group per thread up to 4096 columns (part of a warp, one, two to eight warps with one to four rows side by side, nine
# to sixteen), one CTA per row beyond; row counts that are no multiple of the rows a CTA takes at a time, and more rows than the
# persistent grid takes in one round
@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("rows,H", [(1, 8), (3, 264), (5, 2048), (7, 2056), (2, 4096), (3, 4104), (1801, 768),
                                    (9, 24), (37, 64), (40001, 128), (10007, 256), (5003, 264), (5003, 520), (601, 1032), (903, 2304)])
def test_norm_backward_edges(rows, H, rms):
    from fairscale_b200.ops import norm

    torch.manual_seed(rows + H)
    x, dy = (torch.randn(rows, H, device=_dev()).bfloat16() for _ in range(2))
    w = torch.randn(H, device=_dev()).bfloat16()
    b = None if rms else torch.randn(H, device=_dev()).bfloat16()
    y, mean, rstd = norm.norm_forward(x, w, b, 1e-5, rms)
    dx, dw, db = norm.norm_backward(dy, x, w, mean, rstd, rms, b is not None)
    _status_ok()
    xd, wd = x.double(), w.double()
    mu = 0 if rms else xd.mean(-1, keepdim=True)
    rs = torch.rsqrt((xd - mu).pow(2).mean(-1, keepdim=True) + 1e-5)
    xh, g = (xd - mu) * rs, dy.double() * wd
    assert _rel_err(y, xh * wd + (0 if b is None else b.double())) < 4e-3  # one rounding to bf16
    assert _rel_err(dx, rs * (g - (0 if rms else g.mean(-1, keepdim=True)) - xh * (g * xh).mean(-1, keepdim=True))) < 4e-3
    assert _rel_err(dw, (dy.double() * xh).sum(0)) < 4e-3
    if not rms:
        assert _rel_err(db, dy.double().sum(0)) < 4e-3
    # the residual branch's gradient goes into dx before it is rounded
    res = torch.randn(rows, H, device=_dev()).bfloat16()
    both, dw2, _ = norm.norm_backward(dy, x, w, mean, rstd, rms, b is not None, residual=res)
    want = rs * (g - (0 if rms else g.mean(-1, keepdim=True)) - xh * (g * xh).mean(-1, keepdim=True)) + res.double()
    assert _rel_err(both, want) < 4e-3 and torch.equal(dw, dw2)


def test_small_gradients_land_in_their_flat_window():
    """Bias and norm gradients are written where the flat gradient wants them; a second use goes through autograd's sum."""
    from fairscale_b200.nn.misc.flatten_params_wrapper import GradArena
    from fairscale_b200.ops import norm
    from fairscale_b200.ops.gemm import linear

    torch.manual_seed(0)
    d = 64
    arena = GradArena(d * d + 3 * d)
    w, b, g, be = ((torch.randn(s, device=_dev()) * 0.1).bfloat16().requires_grad_() for s in ((d, d), (d,), (d,), (d,)))
    x = torch.randn(100, d, device=_dev()).bfloat16()

    def grads():
        y = linear(norm.layer_norm(x, g, be), w, b)
        return torch.autograd.grad(linear(y, w, b).float().sum(), (w, b, g, be))

    want = grads()
    off = 0
    for p in (w, b, g, be):
        p._fsb_grad_slot = (arena, off, p.shape)
        off += p.numel()
    got = grads()
    _status_ok()
    for a, r in zip(got, want):
        assert torch.equal(a, r)
    base = arena.buffer.data_ptr()
    assert got[2].data_ptr() == base + 2 * (d * d + d) and got[3].data_ptr() == base + 2 * (d * d + 2 * d)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_multi_tensor_norm_and_scale_edges(dtype):
    """Less than a vector, whole and ragged chunks, tensors that start off a 16-byte boundary, infinities."""
    from fairscale_b200.ops import _bind, multi_tensor

    torch.manual_seed(0)
    chunk = _bind.fn("fsb_adam_chunk_size")()
    flat = torch.randn(4 * chunk + 64, device=_dev()).to(dtype)
    ts = [torch.randn(n, device=_dev()).to(dtype) for n in (1, 7, 8, 9, 2049, chunk, chunk + 3, 3 * chunk + 17)] + [flat[3 : chunk + 40], flat[2 * chunk + 1 :]]
    want = math.sqrt(sum(t.double().pow(2).sum().item() for t in ts))
    assert abs(multi_tensor.l2_norm(ts).item() / want - 1) < 1e-5  # fp32 sums, split over threads and chunks
    flag = torch.zeros(1, dtype=torch.int32, device=_dev())
    copies = [t.clone() for t in ts[:-2]] + [flat.clone()[3 : chunk + 40]]
    wants = [(c.float() * 0.3).to(dtype) for c in copies]
    multi_tensor.scale_(copies, torch.tensor([0.3], device=_dev()), flag)
    for c, r in zip(copies, wants):
        assert torch.equal(c, r)
    assert int(flag) == 0
    copies[-1][-1] = float("inf")
    multi_tensor.scale_(copies, torch.tensor([1.0], device=_dev()), flag)
    assert int(flag) == 1


# head sizes whose rows do and do not divide 256 threads, fewer rows than a step of four takes, more tokens than the grid
@pytest.mark.parametrize("B,S,H,D", [(1, 1, 1, 8), (2, 5, 3, 80), (1, 7, 1, 2048), (1, 3, 1, 2056), (3, 700, 2, 64), (2, 33, 32, 128)])
def test_rope_edges(B, S, H, D):
    from fairscale_b200.ops.rope import _rope_apply, rope_reference

    torch.manual_seed(D)
    qkv = torch.randn(B, S, 3, H, D, device=_dev()).bfloat16()
    for backward in (False, True):
        got = _rope_apply(qkv, 10000.0, backward, 3)
        want = rope_reference(qkv.double(), 10000.0, backward, 3)
        assert _rel_err(got, want) < 4e-3  # one rounding to bf16, angles in fp32
        assert torch.equal(got[:, :, 2], qkv[:, :, 2])
    _status_ok()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,V", [(1, 8), (3, 512), (5, 32000), (7, 2056)])
def test_vocab_cross_entropy_pieces(rows, V, dtype):
    """Loss, statistics and gradient of one vocabulary shard; masked (-inf, lowest finite) logits, targets of other shards."""
    from fairscale_b200.ops.loss import ce_backward, ce_forward

    torch.manual_seed(V)
    x = (torch.randn(rows, V, device=_dev()) * 4).to(dtype)
    x[:, : V // 4] = float("-inf")  # a thread's first logits among them
    if V > 8:
        x[:, V // 4 : V // 2] = torch.finfo(dtype).min
    v0 = 1000
    t = torch.randint(V // 2, V, (rows,), device=_dev()) + v0
    if rows > 1:
        t[0] = 3  # another rank's token
    loss, lse, stats = ce_forward(x, t, ignore_index=-(2**62), vocab_start=v0, want_stats=True)
    xd = x.double()
    want = torch.logsumexp(xd, -1)
    tl = torch.where(t >= v0, xd.gather(1, (t - v0).clamp(min=0).unsqueeze(1)).squeeze(1), torch.zeros((), device=_dev(), dtype=torch.float64))
    tol = 2e-6 if dtype == torch.float32 else 1e-4  # fp32 logits: expf and fp32 sums; bf16: the fast exponential
    torch.testing.assert_close(lse.double(), want, rtol=tol, atol=tol)
    torch.testing.assert_close(loss.double(), want - tl, rtol=tol, atol=10 * tol)
    torch.testing.assert_close((stats[:, 0] + stats[:, 1].log()).double(), want, rtol=tol, atol=tol)
    g = torch.rand(rows, device=_dev())
    before = x.clone()
    dx = ce_backward(x, t, lse, g, 1.0, ignore_index=-(2**62), vocab_start=v0, inplace=True)
    p = torch.softmax(before.double(), -1)
    onehot = torch.zeros_like(p)
    for r in range(rows):
        if t[r] >= v0:
            onehot[r, t[r] - v0] = 1
    torch.testing.assert_close(dx.double(), (p - onehot) * g.double().unsqueeze(1), rtol=2e-5 if dtype == torch.float32 else 1e-2, atol=1e-6 if dtype == torch.float32 else 1e-4)
    if dtype == torch.float32:
        assert torch.equal(x, before)  # fp32 logits may be the caller's own
    _status_ok()


# one vector of NaN (with few columns all that its thread sees), a whole row of it, infinities on their own and beside NaN
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("V", [8, 512, 2056, 32000])
def test_cross_entropy_keeps_nan_and_infinity(V, dtype):
    from fairscale_b200.ops.loss import ce_forward

    torch.manual_seed(V)
    inf, nan = float("inf"), float("nan")
    x = torch.randn(7, V, device=_dev()).to(dtype)
    x[0, :8] = nan
    x[1] = nan
    x[2, 3] = inf
    x[3, 3], x[3, 5] = inf, inf
    x[4, 3], x[4, V - 1] = inf, nan
    x[5] = -inf
    t = torch.full((7,), V // 2, device=_dev())
    t[2:4] = 0
    loss, lse, stats = ce_forward(x, t, want_stats=True)
    want = torch.logsumexp(x.double(), -1)
    assert torch.isnan(want[[0, 1, 4]]).all() and (want[2:4] == inf).all() and want[5] == -inf
    torch.testing.assert_close(lse.double(), want, rtol=1e-4, atol=1e-4, equal_nan=True)
    torch.testing.assert_close(loss.double(), want - x.double().gather(1, t.unsqueeze(1)).squeeze(1), rtol=1e-4, atol=1e-3, equal_nan=True)
    # what another rank's shard makes of the pieces: NaN comes through, also from a shard that holds nothing else
    other = torch.tensor([0.5, 2.0, 0.25], device=_dev()).expand(7, 3)
    both = torch.stack([stats, other])
    top = both[..., 0].max(0).values
    merged = top + (both[..., 1] * torch.exp(both[..., 0] - top)).sum(0).log()
    assert torch.isnan(merged[[0, 1, 4]]).all() and torch.isfinite(merged[5:]).all()
    _status_ok()


# one CTA per tile and CTA pairs, both with more tiles than one wave
@pytest.mark.parametrize("M,N,K", [(4104, 2568, 512), (8200, 8200, 4096)])
def test_products_on_two_streams_and_in_a_graph_keep_their_tiles(M, N, K):
    """The run-time tile hand-out belongs to a stream: a product that waits on one stream while many are enqueued on another,
    and one replayed from a graph, share no counter with them."""
    from ctypes import c_void_p

    from fairscale_b200.fair_dev.testing.testing import gpu_delay
    from fairscale_b200.ops import _bind
    from fairscale_b200.ops.gemm import _launch

    _bind._SIGNATURES.setdefault("fsb_gemm_sched_slot", [c_void_p])
    slot = _bind.fn("fsb_gemm_sched_slot")
    torch.manual_seed(0)
    a, b = torch.randn(M, K, device=_dev()).bfloat16(), torch.randn(N, K, device=_dev()).bfloat16()
    want = torch.empty(M, N, device=_dev(), dtype=torch.bfloat16)

    def product(out):
        _launch(a, b, out, M, N, K, False, False)

    product(want)
    assert _rel_err(want, a.float() @ b.float().t()) < 1e-2
    outs = [torch.full_like(want, float("nan")) for _ in range(6)]
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    slots = [slot(_bind.stream_ptr(_dev())), slot(s1.cuda_stream), slot(s2.cuda_stream)]
    assert min(slots) > 0 and len(set(slots)) == 3 and slot(s1.cuda_stream) == slots[1]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        assert slot(_bind.stream_ptr(_dev())) == 0
        product(outs[0])
    torch.cuda.synchronize()
    with torch.cuda.stream(s1):
        gpu_delay(3.0)  # so that all of the other stream's products are enqueued before these start
        for i in (1, 2):
            product(outs[i])
    with torch.cuda.stream(s2):
        for _ in range(80):
            product(outs[3])
        product(outs[4])
    with torch.cuda.stream(s1):
        graph.replay()
        product(outs[5])
    torch.cuda.synchronize()
    for o in outs:
        assert torch.equal(o, want)
    _status_ok()


def test_fp32_cross_entropy_gradient_can_be_differentiated():
    """create_graph: fp32 logits, whose gradient is differentiable in the incoming one on the CPU, offer that on the GPU too."""
    from fairscale_b200.ops.loss import ce_backward

    torch.manual_seed(4)
    x, t = torch.randn(64, 32, device=_dev()), torch.randint(0, 32, (64,), device=_dev())
    lse, g = torch.logsumexp(x, -1), torch.rand(64, device=_dev())
    got = {}
    for where, cast in (("gpu", lambda v: v.detach().clone()), ("cpu", lambda v: v.detach().cpu())):
        gg = cast(g).requires_grad_()
        dx = ce_backward(cast(x), cast(t), cast(lse), gg, 1.0)
        got[where] = [v.detach().cpu() for v in (dx, *torch.autograd.grad(dx.pow(2).sum(), gg))]
    for a, b in zip(got["gpu"], got["cpu"]):
        torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("rms", [False, True])
def test_norm_gradients_of_no_rows_are_zero(rms):
    """Also where they are windows of a flat gradient, which is used as it stands."""
    from fairscale_b200.nn.misc.flatten_params_wrapper import GradArena
    from fairscale_b200.ops import norm

    H = 64
    x = torch.empty(0, H, device=_dev(), dtype=torch.bfloat16)
    w = torch.ones(H, device=_dev(), dtype=torch.bfloat16)
    b = None if rms else torch.zeros_like(w)
    y, mean, rstd = norm.norm_forward(x, w, b, 1e-5, rms)
    assert y.shape == x.shape
    arena = GradArena(2 * H)
    arena.buffer = torch.full((2 * H,), float("nan"), device=_dev(), dtype=torch.bfloat16)
    windows = ((arena, 0, w.shape), (arena, H, w.shape))
    for slots in ((None, None), windows):
        torch.full((1 << 20,), float("nan"), device=_dev())  # memory that the results may be taken from
        dx, dw, db = norm.norm_backward(x, x, w, mean, rstd, rms, not rms, slots)
        assert dx.shape == x.shape and not dw.any() and (rms or not db.any())
    assert not arena.buffer[: H if rms else 2 * H].any()
    _status_ok()


def _off(t):
    """The same values in a contiguous view that starts two bytes (fp32: four) after a 16-byte boundary."""
    flat = torch.empty(t.numel() + 8, dtype=t.dtype, device=t.device)
    view = flat[1 : 1 + t.numel()].view(t.shape)
    view.copy_(t)
    assert view.data_ptr() % 16 != 0 and view.is_contiguous()
    return view


def test_views_that_start_off_a_16_byte_boundary():
    """The wrappers hand kernels with 16-byte accesses a copy; results are those of aligned tensors."""
    import torch.distributed as dist

    from fairscale_b200.ops import norm
    from fairscale_b200.ops.attention import causal_attention
    from fairscale_b200.ops.loss import ce_backward, ce_forward
    from fairscale_b200.ops.reduce import batched_column_sum, column_sum
    from fairscale_b200.ops.rope import rope_qkv
    from fairscale_b200.parallel.fused_tp import _LinearReduceScatter

    if not dist.is_initialized():
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1)
    torch.manual_seed(7)

    def randn(*shape):
        return torch.randn(*shape, device=_dev()).bfloat16()

    def both(f, *args):
        want, got = f(*args), f(*(_off(a) for a in args))
        for w, g in zip(want, got):
            assert torch.equal(w, g)

    def norms(x, dy, w, b, res):
        out = []
        for rms, bias in ((False, b), (True, None)):
            y, mean, rstd = norm.norm_forward(x, w, bias, 1e-5, rms)
            out += [y, *(t for t in norm.norm_backward(dy, x, w, mean, rstd, rms, not rms, residual=res) if t is not None)]
        return out

    for H in (256, 4104):
        both(norms, randn(5, H), randn(5, H), randn(H), randn(H), randn(5, H))
    both(lambda x: [column_sum(x)], randn(70, 264))
    both(lambda x: [batched_column_sum(x)], randn(3, 70, 264))
    both(lambda x: [rope_qkv(x)], randn(2, 5, 3, 2, 64))
    both(lambda x: [causal_attention(x, 2)], randn(1, 128, 3 * 2 * 64))
    x, w, g = randn(64, 128), randn(256, 128), randn(64, 256)

    def row_parallel(gg):
        xx, ww = x.clone().requires_grad_(), w.clone().requires_grad_()
        return torch.autograd.grad(_LinearReduceScatter.apply(xx, ww, None, dist.group.WORLD), (xx, ww), gg)

    both(row_parallel, g)
    t = torch.randint(0, 512, (9,), device=_dev())
    for dtype in (torch.bfloat16, torch.float32):
        logits = torch.randn(9, 512, device=_dev()).to(dtype)
        lse = ce_forward(logits, t)[1]
        torch.testing.assert_close(ce_forward(_off(logits), t)[1], lse, rtol=1e-4, atol=1e-4)
        up = torch.rand(9, device=_dev())
        torch.testing.assert_close(ce_backward(_off(logits), t, lse, up, 1.0), ce_backward(logits.clone(), t, lse, up, 1.0), rtol=1e-2, atol=1e-4)
    _status_ok()


# few tiles (split over K), one CTA per tile; CTA pairs share the code of the latter
@pytest.mark.parametrize("M,N,K", [(136, 264, 512), (2600, 2056, 128)])
def test_gemm_outputs_and_epilogue_operands_at_any_element(M, N, K):
    from fairscale_b200.ops.gemm import EPI_BIAS_GELU, EPI_BIAS_RESIDUAL, EPI_DGELU, EPI_RESIDUAL, _launch

    torch.manual_seed(M)
    a, b, aux = (torch.randn(*s, device=_dev()).bfloat16() for s in ((M, K), (N, K), (M, N)))
    bias = torch.randn(N, device=_dev()).bfloat16()

    def run(place, epi=0, dtype=torch.bfloat16, use_aux=False, pre=False, accumulate=False):
        c = place(torch.ones(M, N, device=_dev(), dtype=dtype))
        out = place(torch.zeros(M, N, device=_dev(), dtype=torch.bfloat16)) if pre else None
        _launch(a, b, c, M, N, K, False, False, epi, bias=place(bias), aux=place(aux) if use_aux else None, aux_out=out, accumulate=accumulate)
        return [t for t in (c, out) if t is not None]

    for kw in (dict(), dict(dtype=torch.float32), dict(dtype=torch.float32, accumulate=True), dict(epi=EPI_BIAS_GELU, pre=True),
               dict(epi=EPI_BIAS_RESIDUAL, use_aux=True), dict(epi=EPI_DGELU, use_aux=True), dict(epi=EPI_RESIDUAL, use_aux=True)):
        for want, got in zip(run(lambda t: t, **kw), run(_off, **kw)):
            assert torch.equal(want, got), kw
    _status_ok()


def test_frozen_parameters_claim_no_window_of_a_flat_gradient():
    """Their gradients go nowhere: a window would keep a whole flat gradient alive that no backward takes."""
    from fairscale_b200.nn.misc.flatten_params_wrapper import GradArena
    from fairscale_b200.ops import norm
    from fairscale_b200.ops.gemm import linear
    from fairscale_b200.ops.mlp import mlp

    torch.manual_seed(9)
    d = 64
    arena = GradArena(5 * d * d)
    shapes = dict(g=(d,), b=(d,), w=(d, d), wb=(d,), w1=(2 * d, d), b1=(2 * d,), w2=(d, 2 * d), b2=(d,))
    p, off = {}, 0
    for name, shape in shapes.items():
        p[name] = torch.randn(shape, device=_dev()).bfloat16() * 0.1
        p[name]._fsb_grad_slot = (arena, off, p[name].shape)
        off += p[name].numel()
    x = torch.randn(40, d, device=_dev()).bfloat16().requires_grad_()
    y = linear(norm.layer_norm(x, p["g"], p["b"]), p["w"], p["wb"], residual=x)
    mlp(y, p["w1"], p["b1"], p["w2"], p["b2"], residual=y).float().sum().backward()
    assert torch.isfinite(x.grad).all()
    assert arena.buffer is None and not arena.claimed
    _status_ok()


def _row_sums(p, four_by_four):
    """fp32 sums over the keys of a row, ``p [rows, keys]``, steps of 128 keys: in the order of the keys (per 32 keys four partial
    sums of pairs, the four sums of a step one after the other), or with a running sum for each half of a step."""
    import numpy as np

    p = np.pad(p, ((0, 0), (0, -p.shape[1] % 128))).astype(np.float32)
    run = np.zeros((2, p.shape[0]), np.float32)
    for j in range(0, p.shape[1], 128):
        step = p[:, j:j + 128]
        if four_by_four:
            rs = np.zeros(p.shape[0], np.float32)
            for c in range(0, 128, 32):
                acc = [np.zeros(p.shape[0], np.float32) for _ in range(4)]
                for i in range(0, 32, 2):
                    acc[(i >> 1) & 3] = acc[(i >> 1) & 3] + (step[:, c + i] + step[:, c + i + 1])
                rs = rs + ((acc[0] + acc[1]) + (acc[2] + acc[3]))
            run[0] = run[0] + rs
        else:
            for h in (0, 1):
                acc = [np.zeros(p.shape[0], np.float32) for _ in range(4)]
                for i in range(0, 64, 2):
                    for k in (0, 1):
                        acc[2 * ((i >> 1) & 1) + k] = acc[2 * ((i >> 1) & 1) + k] + step[:, 64 * h + i + k]
                run[h] = run[h] + ((acc[0] + acc[2]) + (acc[1] + acc[3]))
    return run[0] + run[1]


@pytest.mark.parametrize("S,D", [(128, 64), (128, 128), (715, 64), (715, 128), (1543, 128)])
def test_attention_adds_a_row_up_in_the_order_of_its_keys(S, D):
    """The normaliser of a row to the last bit.  Every score is a small integer and the scale makes the exponentials powers of two,
    so all that is rounded is the sum.  Bound: a last bit of the sum (1 to 1.02) is 1.2e-7 of its logarithm; the logarithm, below
    0.02, is itself good to 2 ulp of its value, 4e-9."""
    import numpy as np

    from fairscale_b200.ops import _bind, attention_native

    attention_native._bind_sigs()
    scale = float(np.float32(1) / np.float32(1.4426950408889634))  # times log2(e) in fp32: 1
    rng = np.random.default_rng(S + D)
    scores = rng.integers(-26, -13, S).astype(np.float32)
    scores[0] = 0.0  # the maximum of every row, met at its first key
    qkv = torch.zeros(1, S, 3, 1, D, dtype=torch.bfloat16, device=_dev())
    qkv[0, :, 0, 0, 0] = 1.0
    qkv[0, :, 1, 0, 0] = torch.from_numpy(scores).to(_dev())
    o = torch.empty(1, S, D, dtype=torch.bfloat16, device=_dev())
    lse = torch.empty(1, 1, S, dtype=torch.float32, device=_dev())
    _bind.call("fsb_attn_fwd", qkv.data_ptr(), o.data_ptr(), lse.data_ptr(), 1, S, 1, D, scale, _bind.status_ptr(_dev()), _bind.stream_ptr(_dev()))
    _status_ok()
    p = np.where(np.tril(np.ones((S, S), bool)), np.exp2(scores)[None], 0.0).astype(np.float32)
    want, divided = _row_sums(p, True).astype(np.float64), _row_sums(p, False).astype(np.float64)
    assert want.max() < 1.02 and (want != divided).mean() > 0.1  # the two orders can be told apart
    assert np.abs(lse.cpu().numpy()[0, 0].astype(np.float64) - np.log(want)).max() < 1e-8


@pytest.mark.parametrize("plan", [1, 2])
@pytest.mark.parametrize("M,N,K", [(256, 264, 72), (300, 264, 72), (520, 1032, 200)])
def test_packed_gelu_is_the_scalar_one_to_the_bit(M, N, K, plan):
    """GELU and GELU' of whole 16-byte pieces are computed two values per instruction, those of a matrix whose width is no multiple of
    eight one at a time: one column less must not change a bit of the others.  Inputs reach the constant ends of the polynomial."""
    from ctypes import c_int, c_void_p

    from fairscale_b200.ops import _bind

    _bind._SIGNATURES.setdefault("fsb_gemm_bf16_plan", [c_void_p] * 6 + [c_int] * 13 + [c_void_p] * 2)
    torch.manual_seed(M + N)
    a, b, z = (torch.randn(*s, device=_dev()).bfloat16() for s in ((M, K), (N, K), (M, N)))
    b, z, bias = b * (2.0 / K**0.5), z * 2, torch.randn(N, device=_dev()).bfloat16()

    def run(epi, n):
        c = torch.full((M, N), float("nan"), device=_dev(), dtype=torch.bfloat16)
        pre = torch.empty_like(c)
        _bind.call("fsb_gemm_bf16_plan", a.data_ptr(), b.data_ptr(), c.data_ptr(), bias.data_ptr() if epi == 2 else None, z.data_ptr() if epi == 4 else None,
                   pre.data_ptr() if epi == 2 else None, M, n, K, K, K, N, N, 0, 0, epi, 0, 0, plan, _bind.status_ptr(_dev()), _bind.stream_ptr(_dev()))
        return c, pre

    for epi in (2, 4):
        (packed, pre), (scalar, pre_scalar) = run(epi, N), run(epi, N - 1)
        _status_ok()
        assert scalar[:, N - 1].isnan().all() and not packed.isnan().any()
        assert torch.equal(packed[:, : N - 1], scalar[:, : N - 1])
        if epi == 2:
            assert torch.equal(pre[:, : N - 1], pre_scalar[:, : N - 1])
            assert (pre.float().abs() > 5).any()


@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("H", [8, 264, 1024, 2048, 2056, 3000, 4096])
def test_a_row_is_normalised_alike_however_many_there_are(H, rms):
    """Rows of more than 2048 columns are kept as fp32 or as bf16 by their number (300 and 2048 lie on either side): to the bit the same."""
    from fairscale_b200.ops import norm

    torch.manual_seed(H)
    x = (torch.randn(2048, H, device=_dev()) * 3 + 1).bfloat16()
    w, b = torch.randn(H, device=_dev()).bfloat16(), None if rms else torch.randn(H, device=_dev()).bfloat16()
    many, few, one = (norm.norm_forward(x[:n], w, b, 1e-5, rms) for n in (2048, 300, 1))
    _status_ok()
    for m, f, o in zip(many, few, one):
        assert (m is None) == (f is None) == (o is None)
        if m is not None:
            assert torch.equal(m[:300], f) and torch.equal(m[:1], o)
    xd = x.double()
    want = xd if rms else xd - xd.mean(1, keepdim=True)
    want = want * torch.rsqrt((want * want).mean(1, keepdim=True) + 1e-5) * w.double() + (0 if rms else b.double())
    assert _rel_err(many[0], want) < 1e-2
