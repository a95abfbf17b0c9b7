"""The norm after a gated sum where a row waits in registers: runs that fill a warp's loads and do not, groups of one to eight warps'
parts and parts that are empty, one step over the widest row, with and without a result, a gate and its bias, chosen rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def want(x, w, groups, eps, alpha, delta, gate, bias):
    v = alpha * x.double()
    if delta is not None:
        d = delta.double()
        if gate is not None:
            d = d * torch.sigmoid(gate.double() + (bias.double() if bias is not None else 0.0))
        v = v + d
    v = v.reshape(v.shape[0], groups, -1)
    return (v / torch.sqrt((v * v).mean(-1, keepdim=True) + eps)).flatten(1) * w.double()


@pytest.mark.parametrize("W, groups", [(4, 1), (24, 3), (128, 8), (512, 1), (1000, 2), (1020, 5), (2048, 4), (4096, 1), (4096, 8), (4100, 1)])
@pytest.mark.parametrize("form", ["gate", "two slices", "no gate", "no result"])
def test_rows_in_registers(W, groups, form):
    from allpaca_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(W + groups)
    T, eps, alpha = 5, 1e-6, 1.7
    x, delta, gate = (torch.randn(T, W, generator=g, device="cuda") for _ in range(3))
    wide = torch.zeros(T, W + 8, device="cuda")
    wide[:, :W] = gate
    w, bias = 1.0 + 0.2 * torch.randn(W, generator=g, device="cuda"), torch.randn(W, generator=g, device="cuda")
    kw = {"alpha": alpha}
    if form != "no result":
        kw["delta"] = delta.unsqueeze(0)
    if form == "two slices":
        other = torch.randn(T, W, generator=g, device="cuda")
        kw["delta"] = torch.stack([delta, other])
        delta = delta + other
    if form in ("gate", "two slices"):
        kw.update(gate=wide[:, :W], gate_bias=bias)
    ref = want(x, w, groups, eps, alpha, delta if form != "no result" else None, gate if form in ("gate", "two slices") else None, bias)
    got, out = x.clone(), torch.empty(T, W, dtype=torch.bfloat16, device="cuda")
    ops.gated_postnorm(got, w, groups, eps, copy=out, **kw)
    assert float((got.double() - ref).abs().max()) <= 4e-6 * float(ref.abs().max())          # some 20 roundings of 2^-24
    assert torch.equal(out, got.bfloat16())
    if form == "no result":
        picked, rows = torch.empty(2, W, device="cuda"), torch.tensor([3, 1], dtype=torch.int32, device="cuda")
        before = x.clone()
        ops.gated_postnorm(x, w, groups, eps, alpha=alpha, rows=rows, out=picked)
        assert torch.equal(x, before) and torch.equal(picked, got[[3, 1]])


@pytest.mark.parametrize("W, groups", [(4, 1), (1020, 5), (2048, 4), (4096, 8)])
@pytest.mark.parametrize("slices", [1, 2])
@pytest.mark.parametrize("gated", ["bias", "gate", None])
def test_bits_of_the_general_kernel(W, groups, slices, gated):
    """Slices of zeros behind the same sums change nothing but the kernel: more than two of them take the general one."""
    from allpaca_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(W + slices)
    T = 9
    x, gate = (torch.randn(T, W, generator=g, device="cuda") for _ in range(2))
    delta = torch.zeros(4, T, W, device="cuda")
    delta[:slices] = torch.randn(slices, T, W, generator=g, device="cuda")
    w, bias = 1.0 + 0.2 * torch.randn(W, generator=g, device="cuda"), torch.randn(W, generator=g, device="cuda")
    results = []
    for n in (slices, 4):
        got = x.clone()
        ops.gated_postnorm(got, w, groups, 1e-6, alpha=1.7, delta=delta[:n], gate=gate if gated else None,
                           gate_bias=bias if gated == "bias" else None)
        results.append(got)
    assert torch.equal(*results)


def test_weight_and_bias_of_the_kernel_before():
    """A weight and a gate's bias that the kernel right ahead writes, one that lets the next kernel start early, are read as that one
    leaves them, unless the caller says that nothing in flight writes them."""
    from allpaca_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(3)
    T, W, rows = 4, 2048, 2048                               # a long kernel before: many rows, the vectors among its last
    x, delta, gate = (torch.randn(T, W, generator=g, device="cuda") for _ in range(3))
    source, ones = torch.randn(rows, W, generator=g, device="cuda"), torch.ones(W, device="cuda")
    for _ in range(20):
        made = torch.full((rows, W), float("nan"), device="cuda")
        got, want = x.clone(), x.clone()
        torch.cuda.synchronize()
        ops.gated_postnorm(source, ones, 4, 1e-6, out=made)
        ops.gated_postnorm(got, made[-1], 4, 1e-6, delta=delta, gate=gate, gate_bias=made[-2])
        torch.cuda.synchronize()
        ops.gated_postnorm(want, made[-1], 4, 1e-6, delta=delta, gate=gate, gate_bias=made[-2], settled=True)
        assert torch.equal(got, want)


def test_slices_of_no_sums():
    """At the C entry: no sums to add, and a count of slices all the same."""
    from allpaca_b200 import ops
    x, w = torch.randn(3, 512, device="cuda"), torch.ones(512, device="cuda")
    want = x.clone()
    ops.gated_postnorm(want, w, 4, 1e-6, alpha=1.7)
    ops.call(ops.core(), "ap_gated_postnorm", x.data_ptr(), 0, 3, 0, 2, x.numel(), 0, 0, 0, 1.7, w.data_ptr(),
             ops.dtype_code(w.dtype), 4, 1e-6, 1, 0, ops.AP_F32, 512, 0, ops.stream_handle())
    assert torch.equal(x, want)


@pytest.mark.parametrize("W, groups, slices", [(512, 1, 1), (2048, 4, 2), (4096, 8, 2)])
@pytest.mark.parametrize("T", [296, 297, 1023, 1024])
def test_rows_around_the_change_of_kernels(W, groups, slices, T):
    """As many rows as run at once and one more, and as many as take two slices of wide rows back: each row has the bits it has alone."""
    from allpaca_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(T + W)
    x, gate = (torch.randn(T, W, generator=g, device="cuda") for _ in range(2))
    delta = torch.randn(slices, T, W, generator=g, device="cuda")
    w, bias = 1.0 + 0.2 * torch.randn(W, generator=g, device="cuda"), torch.randn(W, generator=g, device="cuda")
    got = x.clone()
    ops.gated_postnorm(got, w, groups, 1e-6, alpha=1.7, delta=delta, gate=gate, gate_bias=bias)
    for r in (0, T // 2, T - 1):
        one = x[r:r + 1].clone()
        ops.gated_postnorm(one, w, groups, 1e-6, alpha=1.7, delta=delta[:, r:r + 1].contiguous(), gate=gate[r:r + 1], gate_bias=bias)
        assert torch.equal(one, got[r:r + 1])
