"""Each kernel alone against a plain float32/float64 torch computation, at sizes other than the
tiny models': widths and vocabularies that are no power of two, odd head counts, head sizes in
steps of 16 (and one that is not), long and short rows."""
import math

import numpy as np
import pytest
import torch

import plain_falcon as plain

pytestmark = pytest.mark.gpu

DTYPES = [torch.float32, torch.bfloat16]


def tol(dtype):
    return dict(atol=2e-5, rtol=1e-5) if dtype == torch.float32 else dict(atol=2e-2, rtol=2e-2)


@pytest.fixture(scope="module")
def K():
    from pytorch_transformers_b200 import kernels
    kernels.lib()
    return kernels


def rnd(*shape, dtype=torch.float32, scale=1.0, seed=0):
    g = torch.Generator().manual_seed(seed + sum(shape))
    return (torch.randn(*shape, generator=g) * scale).to(dtype).cuda()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("width", [7, 96, 1000, 4544])
def test_gather_rows(K, dtype, width):
    table = rnd(333, width, dtype=dtype)
    ids = torch.tensor([0, 332, 5, 5, 17], dtype=torch.int32).cuda()
    status = torch.zeros(1, dtype=torch.int32).cuda()
    out = K.gather_rows(ids, table, status)
    assert torch.equal(out, table[ids.long()])
    assert status.item() == 0
    bad = torch.tensor([1, 400], dtype=torch.int32).cuda()
    K.gather_rows(bad, table, status)
    assert status.item() == 1


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("width,scale", [(7, 1.0), (96, 3.0), (1000, 0.37), (4544, 1.7), (4546, 2.0)])
def test_embed_rows(K, dtype, width, scale):
    """Rows of a table widened to float32 and scaled there: what a gather, a widening and a product in float32 give."""
    table = rnd(333, width, dtype=dtype)
    ids = torch.tensor([0, 332, 5, 5, 17], dtype=torch.int32).cuda()
    status = torch.zeros(1, dtype=torch.int32).cuda()
    out = K.embed_rows(ids, table, scale, status)
    assert out.dtype == torch.float32 and torch.equal(out, table[ids.long()].float() * scale)
    assert status.item() == 0
    K.embed_rows(torch.tensor([1, -1], dtype=torch.int32).cuda(), table, scale, status)
    assert status.item() == 1


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("rows,width,eps", [(1, 64, 1e-5), (5, 96, 1e-6), (3, 4544, 1e-5), (2, 8192, 1e-5),
                                            (4, 1001, 1e-3), (2, 20000, 1e-5), (300, 4544, 1e-5), (2, 16384, 1e-5),
                                            (2, 16392, 1e-5), (7, 2056, 1e-5)])
def test_layernorm_and_pair(K, dtype, rows, width, eps):
    x = rnd(rows, width, dtype=dtype, scale=3.0) + 0.5
    g1, b1 = rnd(width, seed=1) + 1, rnd(width, seed=2)
    g2, b2 = rnd(width, seed=3) + 1, rnd(width, seed=4)
    ref1 = plain.layer_norm(x.double().cpu(), g1.double().cpu(), b1.double().cpu(), eps)
    ref2 = plain.layer_norm(x.double().cpu(), g2.double().cpu(), b2.double().cpu(), eps)
    y = K.norm(x, g1, b1, eps)
    torch.testing.assert_close(y.double().cpu(), ref1, **tol(dtype))
    y1, y2 = K.norm(x, g1, b1, eps, gain2=g2, bias2=b2)
    assert torch.equal(y1, y)
    torch.testing.assert_close(y2.double().cpu(), ref2, **tol(dtype))


@pytest.mark.parametrize("dtype", DTYPES)
def test_rmsnorm(K, dtype):
    x = rnd(6, 200, dtype=dtype, scale=2.0)
    g = rnd(200, seed=1) + 1
    xd = x.double().cpu()
    ref = xd / torch.sqrt((xd ** 2).mean(-1, keepdim=True) + 1e-6) * g.double().cpu()
    torch.testing.assert_close(K.norm(x, g, None, 1e-6, "rmsnorm").double().cpu(), ref, **tol(dtype))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("act", ["none", "gelu", "gelu_new", "relu"])
def test_bias_act(K, dtype, act):
    y = rnd(9, 333, dtype=dtype, scale=2.0)
    b = rnd(333, seed=5)
    ref = y.double().cpu() + b.double().cpu()
    ref = ref if act == "none" else plain.activation(ref, act)
    out = K.bias_act_(y.clone(), b, act)
    torch.testing.assert_close(out.double().cpu(), ref, **tol(dtype))
    out2 = K.bias_act_(y.clone(), None, act)
    ref2 = y.double().cpu() if act == "none" else plain.activation(y.double().cpu(), act)
    torch.testing.assert_close(out2.double().cpu(), ref2, **tol(dtype))


@pytest.mark.parametrize("dtype", DTYPES)
def test_residual(K, dtype):
    x, a, b = (rnd(11, 97, dtype=dtype, seed=s) for s in (1, 2, 3))
    ref = x.double() + (a.double() + b.double())
    torch.testing.assert_close(K.residual(x, a, b).double(), ref, **tol(dtype))
    torch.testing.assert_close(K.residual(x, a).double(), x.double() + a.double(), **tol(dtype))
    if dtype == torch.bfloat16:
        # one rounding of the float32 sum, not a rounding per addition
        exact = (x.float() + (a.float() + b.float())).bfloat16()
        assert torch.equal(K.residual(x, a, b), exact)


@pytest.mark.parametrize("m,n,k", [(1, 64, 64), (37, 101, 53), (64, 64, 16), (130, 4672 // 8, 71), (5, 1000, 96),
                                   (2, 65, 4544)])
@pytest.mark.parametrize("act,bias", [("none", False), ("gelu", True), ("none", True)])
def test_linear_f32(K, m, n, k, act, bias):
    x, w = rnd(m, k, seed=1), rnd(n, k, seed=2, scale=0.1)
    b = rnd(n, seed=3) if bias else None
    ref = x.double().cpu() @ w.double().cpu().T
    if bias:
        ref = ref + b.double().cpu()
    if act != "none":
        ref = plain.activation(ref, act)
    out = K.linear_f32(x, w, b, act)
    torch.testing.assert_close(out.double().cpu(), ref, atol=1e-5, rtol=1e-5)


def test_linear_f32_rows_do_not_depend_on_the_batch(K):
    x, w = rnd(70, 300, seed=1), rnd(129, 300, seed=2)
    full = K.linear_f32(x, w)
    for rows in ([0], [3, 4], list(range(65, 70))):
        part = K.linear_f32(x[rows].contiguous(), w)
        assert torch.equal(part, full[rows])


@pytest.mark.parametrize("m", [1, 16, 17, 32, 33, 64, 65, 131])
@pytest.mark.parametrize("n,k", [(64, 1024), (65, 1056), (2048, 1024), (7, 2048), (130, 2081), (64, 4100)])
def test_linear_f32_tiles_and_stretches(K, m, n, k):
    """Tiles of 16 to 128 rows with remainders, in either form (matrices of 64 outputs and K of 1,024 on in whole 16-byte words go to the
    tensor cores), K in several stretches, rows at odd words, rows that lie apart.
    An element's error: its chains are 16 products long, then about k / 32 sums, each a rounding of 2^-24 of the partial sum."""
    wide, w = rnd(m, k + 3, seed=1), rnd(n, k, seed=2, scale=0.1)
    b = rnd(n, seed=3)
    for x in (wide[:, :k], wide[:, :k].contiguous()):
        out = K.linear_f32(x, w, b)
        ref = x.double() @ w.double().T + b.double()
        bound = (16 + k / 32 + 6) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T + b.double().abs())
        assert ((out.double() - ref).abs() <= bound).all()
    assert torch.equal(K.linear_f32(wide[-1:, :k], w, b), K.linear_f32(wide[:, :k], w, b)[-1:])


@pytest.mark.parametrize("n,k", [(64, 1024), (65, 1028), (512, 256), (1000, 1028), (129, 2052), (4096, 2048), (4300, 1024), (9000, 300), (96, 33000)])
def test_linear_f32_on_tensor_cores(K, n, k):
    """Matrices that the tensor-core form takes, around its tiles of 128 outputs and 16 to 128 rows, with K in one to four stretches and
    an end inside a stage of 64; rows at odd words and apart; rows alone and in every size of tile the same bits. A product of
    three-term operands is off by 2^-24 of itself at most, 32 of them are summed cut off (12 sums of 16, 2^-23 each), and k / 32
    such sums are rounded additions. (This holds every element, loosely; the test of the 2-norm below holds the 24 bits.)"""
    wide, w = rnd(300, k + 3, seed=1), rnd(n, k, seed=2, scale=0.1)
    b = rnd(n, seed=3)
    ref = wide[:, :k].double() @ w.double().T
    size = wide[:, :k].double().abs() @ w.double().abs().T
    for m in (1, 15, 16, 17, 33, 64, 65, 128, 129, 300):
        for x in (wide[:m, :k], wide[:m, :k].contiguous()):
            out = K.linear_f32(x, w)
            assert ((out.double() - ref[:m]).abs() <= (k / 32 + 26) * 2.0 ** -24 * size[:m]).all()
            full = out if m == 1 else full
            assert torch.equal(out[:1], full[:1]) and torch.equal(K.linear_f32(x[-1:], w), out[-1:])
    out = K.linear_f32(wide[:40, :k], w, b, "gelu")
    torch.testing.assert_close(out.double().cpu(), plain.activation((ref[:40] + b.double()).cpu(), "gelu"), atol=1e-5, rtol=1e-5)


def multiply_adds(x, w, outputs):
    """x @ w.T in float32 multiply-adds as linear_f32.cu orders them: two chains of 16 products a step of 32 k, joined, and the steps' running
    total, K of 2,048 on in four stretches, of 1,024 on beside fewer than 2,048 outputs in two. (A product of two float32 values is exact in 64 bits.)"""
    steps = (x.shape[1] + 31) // 32
    pad = lambda t: torch.nn.functional.pad(t, (0, steps * 32 - t.shape[1])).double().reshape(t.shape[0], steps, 16, 2).permute(1, 3, 2, 0)
    a, b = pad(x), pad(w)      # [step][chain][16][rows]
    sums = torch.zeros(steps, 2, x.shape[0], w.shape[0], device=x.device)
    for i in range(16):
        sums = (sums.double() + a[:, :, i, :, None] * b[:, :, i, None, :]).float()
    sums = sums[:, 0] + sums[:, 1]
    ranks = 4 if x.shape[1] >= 2048 else 2 if x.shape[1] >= 1024 and outputs < 2048 else 1
    out = torch.zeros_like(sums[0])
    for part in sums.split((steps + ranks - 1) // ranks):
        total = torch.zeros_like(out)
        for step in part:
            total = total + step
        out = out + total
    return out


def norm_error(got, ref):
    return ((got.double() - ref).norm() / ref.norm()).item()


@pytest.mark.parametrize("kind", ["normal", "one sign", "cubed"])
@pytest.mark.parametrize("n,k", [(64, 1024), (512, 256), (1024, 1024), (1024, 4096), (1536, 6144), (6144, 1536), (4300, 2048), (5700, 2048),
                                 (6144, 4096), (9216, 1024), (9216, 4096), (18176, 4544), (4544, 18176)])
def test_linear_f32_on_tensor_cores_errs_no_more_than_multiply_adds(K, n, k, kind):
    """2-norm against 64 bits, whatever the number of outputs, of values whose sums cancel and of values of one sign (whose sums show
    what the tensor core cuts off). Operands of two terms are off by 4e-6, thirty times the bound and more."""
    make = {"normal": rnd, "one sign": lambda *s, seed: rnd(*s, seed=seed).abs(), "cubed": lambda *s, seed: rnd(*s, seed=seed) ** 3}[kind]
    x, w = make(40, k, seed=1), make(n, k, seed=2)
    some = w[torch.arange(0, n, max(1, n // 200), device="cuda")]
    ref = x.double() @ some.double().T
    got = K.linear_f32(x, w)[:, ::max(1, n // 200)]
    assert norm_error(got, ref) <= norm_error(multiply_adds(x, some, n), ref)


def test_linear_f32_products_of_terms(K):
    """One product an output, of values with 24 bits: off by what is left out (2^-24 at most), cut (2^-23) and put back for sums that are
    (2^-24). Without any one of the six products of terms it would be 2^-18 and more."""
    g = torch.Generator(device="cuda").manual_seed(3)
    x, w = torch.zeros(64, 1024, device="cuda"), 1 + torch.rand(512, 1024, generator=g, device="cuda")
    at = torch.randint(0, 1024, (64,), generator=g, device="cuda")
    x[torch.arange(64), at] = 1 + torch.rand(64, generator=g, device="cuda")
    ref = x.double() @ w.double().T
    assert ((K.linear_f32(x, w).double() - ref).abs() <= 2.0 ** -22 * ref).all()


@pytest.mark.parametrize("m", [1, 16, 17, 33, 131])
@pytest.mark.parametrize("n,k", [(40, 1024), (63, 1500), (130, 1027), (300, 2047), (33, 4100), (2100, 1026), (12, 2048)])
def test_linear_f32_multiply_adds_in_stretches(K, m, n, k):
    """What stays with the multiply-adds (fewer than 64 outputs, or rows that are no whole 16-byte words), K in one, two and four stretches
    among a cluster, copies of 4 and of 16 bytes. Bound: test_linear_f32_tiles_and_stretches."""
    wide, w = rnd(m, k + 4, seed=1), rnd(n, k, seed=2, scale=0.1)
    for x in (wide[:, :k], wide[:, :k].contiguous()):
        ref, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
        assert ((K.linear_f32(x, w).double() - ref).abs() <= (16 + k / 32 + 6) * 2.0 ** -24 * size).all()
    assert torch.equal(K.linear_f32(wide[-1:, :k], w), K.linear_f32(wide[:, :k], w)[-1:])


@pytest.mark.parametrize("scale", [1e-30, 1e-33, 1e-36, 1e-38, 1e34])
@pytest.mark.parametrize("n,k", [(1024, 1024), (640, 4096)])
def test_linear_f32_of_small_and_large_numbers(K, n, k, scale):
    """Down to numbers without a leading one (1e-38) and up to where the scale of the terms leaves float32: no further off than
    multiply-adds. A third term without that scale would lie under bfloat16's smallest number from 1e-33 down."""
    for x, w in ((rnd(40, k, seed=1) * scale, rnd(n, k, seed=2)), (rnd(40, k, seed=1), rnd(n, k, seed=2) * scale)):
        ref = x.double() @ w.double().T
        assert norm_error(K.linear_f32(x, w), ref) <= norm_error(multiply_adds(x, w, n), ref)


def test_linear_f32_of_values_without_three_terms(K):
    """Infinities, NaN, values that round to an infinity in bfloat16 and products beyond float32: what float32 multiply-adds give. Small
    numbers: the test above."""
    x, w = rnd(20, 1024, seed=1), rnd(70, 1024, seed=2)
    x[3, 7], x[5, 9], x[6, 1], x[7, 2] = math.inf, math.nan, 3.4e38, -3.4e38
    w[11, 7], w[12, 1], w[13, 30] = 0.0, 0.5, -math.inf
    # a product beyond float32 beside an infinity of the other sign has no number in float32 and one in 64 bits: zero times infinity instead
    x[6:8, 30] = 0.0
    x[8], w[20] = 1e30, 1e30
    out, ref = K.linear_f32(x, w), x.double() @ w.double().T
    inside = ref.abs() < 3.4028e38
    assert torch.equal(out.isnan(), ref.isnan()) and torch.equal(out[~inside & ~ref.isnan()], ref[~inside & ~ref.isnan()].clamp(-math.inf, math.inf).sign() * math.inf)
    size = x.double().abs() @ w.double().abs().T
    assert ((out.double() - ref).abs()[inside] <= 80 * 2.0 ** -24 * size[inside]).all()
    tiny = rnd(20, 1024, seed=4) * 1e-30
    torch.testing.assert_close(K.linear_f32(tiny, w[:64].nan_to_num(0, 1, -1).clamp(-4, 4)).double() * 1e30,
                               (tiny.double() @ w[:64].nan_to_num(0, 1, -1).clamp(-4, 4).double().T) * 1e30, atol=1e-5, rtol=1e-5)


def test_to_float(K):
    x = rnd(3, 1000, dtype=torch.bfloat16)
    assert torch.equal(K.to_float(x), x.float())


@pytest.mark.parametrize("m", [1, 5, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("n,k", [(100, 64), (4672, 4544), (71, 96), (1000, 18176 // 4)])
@pytest.mark.parametrize("act,bias,add,f32", [("none", False, False, False), ("gelu", True, False, False),
                                               ("none", True, True, False), ("none", False, False, True),
                                               ("relu", False, True, True)])
def test_skinny_linear(K, m, n, k, act, bias, add, f32):
    bf = torch.bfloat16
    x, w = rnd(m, k, dtype=bf, seed=1), rnd(n, k, dtype=bf, seed=2, scale=0.05)
    b = rnd(n, seed=3) if bias else None
    a = rnd(m, n, dtype=bf, seed=4) if add else None
    assert K.skinny_linear_takes(m, k)
    ref = x.double().cpu() @ w.double().cpu().T
    if bias:
        ref = ref + b.double().cpu()
    if act != "none":
        ref = plain.activation(ref, act)
    if add:
        ref = ref + a.double().cpu()
    out = K.skinny_linear(x, w, b, act, a, out_dtype=torch.float32 if f32 else bf)
    assert out.dtype == (torch.float32 if f32 else bf)
    if f32:
        torch.testing.assert_close(out.double().cpu(), ref, atol=1e-3, rtol=1e-4)
    else:
        torch.testing.assert_close(out.double().cpu(), ref, **tol(bf))


@pytest.mark.parametrize("m", [1, 7, 16, 17, 33, 64, 100, 128])
@pytest.mark.parametrize("n,k", [(100, 64), (4672, 4544), (71, 96), (18176 // 2, 4544), (333, 18176 // 4),
                                 (4544, 1160), (129, 1024), (128, 8)])
@pytest.mark.parametrize("act,bias,add,f32", [("none", False, False, False), ("gelu", True, False, False),
                                               ("none", True, True, False), ("relu", False, True, True)])
def test_tc_linear(K, m, n, k, act, bias, add, f32):
    """The tcgen05 linear layer: every number of rows up to 128, widths that are no multiple of the
    128-row tile or of the 64-wide k chunk, with and without the division of K over a cluster."""
    bf = torch.bfloat16
    x, w = rnd(m, k, dtype=bf, seed=1), rnd(n, k, dtype=bf, seed=2, scale=0.05)
    b = rnd(n, seed=3) if bias else None
    a = rnd(m, n, dtype=bf, seed=4) if add else None
    assert K.tc_linear_takes(m, k)
    ref = x.double().cpu() @ w.double().cpu().T
    if bias:
        ref = ref + b.double().cpu()
    if act != "none":
        ref = plain.activation(ref, act)
    if add:
        ref = ref + a.double().cpu()
    out = K.tc_linear(x, w, b, act, a, out_dtype=torch.float32 if f32 else bf)
    K.check_device_errors(x.device)
    assert out.dtype == (torch.float32 if f32 else bf)
    if f32:
        torch.testing.assert_close(out.double().cpu(), ref, atol=1e-3, rtol=1e-4)
    else:
        torch.testing.assert_close(out.double().cpu(), ref, **tol(bf))


def test_tc_linear_one_key_stands_out(K):
    """A single large product far along K, in a block's last chunk, must arrive in the sum: one weight
    row and one token get a matching spike at the last k."""
    bf = torch.bfloat16
    m, n, k = 48, 4544, 4544
    x, w = rnd(m, k, dtype=bf, seed=1, scale=0.01), rnd(n, k, dtype=bf, seed=2, scale=0.01)
    x[37, k - 1] = 8.0
    w[4001, k - 1] = 4.0
    out = K.tc_linear(x, w).float().cpu()
    K.check_device_errors(x.device)
    ref = (x.double().cpu() @ w.double().cpu().T).float()
    assert abs(out[37, 4001] - 32.0) < 0.5
    torch.testing.assert_close(out, ref, **tol(bf))


def test_tc_linear_refuses_what_it_does_not_take(K):
    from pytorch_transformers_b200.kernels import KernelError
    assert K.lib().ptb_tc_linear_max_rows() == K.TC_LINEAR_MAX_ROWS
    assert K.lib().ptb_tc_linear_k_multiple() == K.TC_LINEAR_K_MULTIPLE
    assert not K.tc_linear_takes(129, 64) and not K.tc_linear_takes(4, 36)
    bf = torch.bfloat16
    with pytest.raises(KernelError):
        K.tc_linear(rnd(129, 64, dtype=bf), rnd(16, 64, dtype=bf))
    with pytest.raises(KernelError):
        K.tc_linear(rnd(4, 36, dtype=bf), rnd(16, 36, dtype=bf))
    with pytest.raises(KernelError):
        K.tc_linear(rnd(4, 64), rnd(16, 64))


@pytest.mark.parametrize("m", [1, 8, 16])
@pytest.mark.parametrize("n,k,shares", [(8192, 32768, 2), (4096, 65568, 4)])
def test_skinny_linear_k_divided_among_blocks(K, m, n, k, shares):
    """512 and 256 tiles of 16 rows do not divide evenly over 148 SMs and K is long enough: 2 and 4 blocks
    per tile, partial sums through scratch memory, the last block by ticket runs the epilogue. Twice in a
    row: the tickets must be back at zero. The second K leaves a ragged last round."""
    bf = torch.bfloat16
    assert K._skinny_scratch_floats(m, n, k) == (n // 16) * shares * 16 * (8 if m <= 8 else 16)
    assert K._skinny_scratch_floats(m, 4544, 18176) == 0
    x, w = rnd(m, k, dtype=bf, seed=1, scale=0.3), rnd(n, k, dtype=bf, seed=2, scale=0.05)
    b, a = rnd(n, seed=3), rnd(m, n, dtype=bf, seed=4)
    ref = plain.activation(x.double().cpu() @ w.double().cpu().T + b.double().cpu(), "gelu") + a.double().cpu()
    for _ in range(2):
        out = K.skinny_linear(x, w, b, "gelu", a)
        torch.testing.assert_close(out.double().cpu(), ref, **tol(bf))
    assert int(K._ticket_arenas[x.device][0].abs().sum()) == 0


def test_two_divided_launches_at_the_same_time_do_not_share_their_tickets(K):
    """Two launches that divide K among blocks run side by side on two streams (as the two branches of a
    block do inside a step): each counts its blocks' arrivals in words of its own, so both give what
    they give alone. Tickets never wait for anybody, so a fault here shows as a wrong sum, not a hang."""
    bf = torch.bfloat16
    m, n, k = 8, 8192, 32768
    assert K._skinny_scratch_floats(m, n, k) > 0
    xs = [rnd(m, k, dtype=bf, seed=s, scale=0.3) for s in (1, 2)]
    ws = [rnd(n, k, dtype=bf, seed=s, scale=0.05) for s in (3, 4)]
    alone = [K.skinny_linear(x, w) for x, w in zip(xs, ws)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(10):
        outs = []
        for st, x, w in zip(streams, xs, ws):
            st.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(st):
                outs.append([K.skinny_linear(x, w) for _ in range(3)])
        for st in streams:
            torch.cuda.current_stream().wait_stream(st)
        torch.cuda.synchronize()
        for got, want in zip(outs, alone):
            for g in got:
                assert torch.equal(g, want)
    assert int(K._ticket_arenas[xs[0].device][0].abs().sum()) == 0
    # a launch's words are its own: consecutive launches get consecutive stretches of the arena
    a, b = K._tickets(100, xs[0].device), K._tickets(100, xs[0].device)
    assert a.data_ptr() != b.data_ptr() and a.numel() == 128


def test_skinny_linear_refuses_what_it_does_not_take(K):
    from pytorch_transformers_b200.kernels import KernelError
    assert K.lib().ptb_skinny_linear_max_rows() == K.SKINNY_MAX_ROWS
    assert K.lib().ptb_skinny_linear_k_multiple() == K.SKINNY_K_MULTIPLE
    assert not K.skinny_linear_takes(33, 64) and not K.skinny_linear_takes(4, 48)
    with pytest.raises(KernelError):
        K.skinny_linear(rnd(33, 64, dtype=torch.bfloat16), rnd(16, 64, dtype=torch.bfloat16))
    with pytest.raises(KernelError):
        K.skinny_linear(rnd(4, 48, dtype=torch.bfloat16), rnd(16, 48, dtype=torch.bfloat16))
    with pytest.raises(KernelError):
        K.skinny_linear(rnd(4, 64), rnd(16, 64))




def test_a_bounded_wait_that_runs_out_raises_on_the_host_and_leaves_the_device_usable(K):
    """Every wait on an mbarrier in the tcgen05 kernels gives up after a number of tries, raises a flag
    in device memory and lets the kernel return. Here a kernel waits 1,000 tries on a barrier at which
    nobody arrives (no fault, no hang: the wait simply runs out); the host's check then raises once,
    the flag is clean again afterwards, and a tcgen05 kernel still runs."""
    from pytorch_transformers_b200.kernels import KernelError
    dev = torch.device("cuda", torch.cuda.current_device())
    K.check_device_errors(dev)                           # clean before
    gave_up = K.selftest_bounded_wait(dev, tries=1000)
    with pytest.raises(KernelError, match="gave up waiting .*code 99"):
        K.check_device_errors(dev)
    assert int(gave_up.item()) == 1
    K.check_device_errors(dev)                           # raised once, clean again
    bf = torch.bfloat16
    x, w = rnd(40, 256, dtype=bf, seed=1), rnd(300, 256, dtype=bf, seed=2, scale=0.05)
    out = K.tc_linear(x, w)
    K.check_device_errors(dev)
    torch.testing.assert_close(out.double().cpu(), x.double().cpu() @ w.double().cpu().T, **tol(bf))
    with pytest.raises(KernelError):
        K.selftest_bounded_wait(dev, tries=0)


@pytest.mark.parametrize("kind", ["gated", "clamped", "plain", "plain on input"])
@pytest.mark.parametrize("width,inner", [(72, 136), (200, 1000), (1024, 8)])
@pytest.mark.parametrize("tile_rows", [0, 16, 32, 64, 128, 256])
def test_expert_tiles(K, kind, width, inner, tile_rows):
    """Experts with no rows, one, a tile's rows and one more, remainders of 16, several tiles; K and outputs that end within a
    stage or a block. The inner values are rounded to bfloat16 on both sides, so they may differ by one unit (2^-8 of
    themselves) where float32 sums fall on either side of a tie: that bounds a result's error through |W_down|."""
    counts = [0, 1, 15, 16, 17, 255, 256, 257, 0, 300]
    n_experts, tokens = len(counts), sum(counts)
    h = rnd(tokens, width, dtype=torch.bfloat16, seed=1)
    g = torch.Generator().manual_seed(5)
    ids = torch.repeat_interleave(torch.arange(n_experts), torch.tensor(counts))[torch.randperm(tokens, generator=g)]
    plain_kind = kind.startswith("plain")
    up = rnd(n_experts, inner if plain_kind else 2 * inner, width, dtype=torch.bfloat16, scale=width ** -0.5, seed=2)
    down = rnd(n_experts, width, inner, dtype=torch.bfloat16, scale=inner ** -0.5, seed=3)
    weights = rnd(tokens, 1, seed=4).abs()
    on_input = kind == "plain on input"
    y, rows = K.expert_rows(h, ids.int().reshape(-1, 1).cuda(), up, down, mma_tile_rows=tile_rows, plain_act="gelu" if plain_kind else None,
                            input_weights=weights if on_input else None, clamp=(1.0, 1.702) if kind == "clamped" else None)
    got = y[rows.long()]
    for e in range(n_experts):
        at = (ids == e).nonzero()[:, 0].cuda()
        z = h[at].double() @ up[e].double().T
        if plain_kind:
            a = plain.activation((z * weights[at].double() if on_input else z).cpu(), "gelu").cuda()
        elif kind == "clamped":
            gate, u = z[:, :inner].clamp(max=1.0), z[:, inner:].clamp(-1.0, 1.0)
            a = gate * torch.sigmoid(1.702 * gate) * (u + 1)
        else:
            a = z[:, :inner] * torch.sigmoid(z[:, :inner]) * z[:, inner:]
        a = a.bfloat16().double()
        bound = (2.0 ** -8 * a.abs() + 1e-5) @ down[e].double().abs().T + 1e-5
        assert ((got[at].double() - a @ down[e].double().T).abs() <= bound).all(), (kind, e)
    K.check_device_errors("cuda:0")


@pytest.mark.parametrize("kind", ["gated", "plain"])
@pytest.mark.parametrize("tile_rows", [16, 32, 64, 128, 256])
@pytest.mark.parametrize("n_experts", [40, 16, 6])
def test_expert_tiles_beyond_the_blocks(K, kind, tile_rows, n_experts):
    """More tiles than blocks stay on the device, so that a block walks several: its rings carry on from tile to tile at any
    stage (9 and 21 stages of k, each with a remainder), and tiles of different rows take turns in tensor memory; with fewer experts a
    little more than one round of tiles, and less than half of one, which choose other forms. The bound is that of test_expert_tiles."""
    width, inner = 520, 1304
    counts = [(1, 16, 17, 64, 65, 130, 0, 200)[e % 8] for e in range(n_experts)]
    h = rnd(sum(counts), width, dtype=torch.bfloat16, seed=1)
    ids = torch.repeat_interleave(torch.arange(n_experts), torch.tensor(counts))[torch.randperm(sum(counts), generator=torch.Generator().manual_seed(5))]
    up = rnd(n_experts, inner if kind == "plain" else 2 * inner, width, dtype=torch.bfloat16, scale=width ** -0.5, seed=2)
    down = rnd(n_experts, width, inner, dtype=torch.bfloat16, scale=inner ** -0.5, seed=3)
    y, rows = K.expert_rows(h, ids.int().reshape(-1, 1).cuda(), up, down, mma_tile_rows=tile_rows, plain_act="relu" if kind == "plain" else None)
    got = y[rows.long()]
    for e in range(n_experts):
        at = (ids == e).nonzero()[:, 0].cuda()
        z = h[at].double() @ up[e].double().T
        a = (z.relu() if kind == "plain" else z[:, :inner] * torch.sigmoid(z[:, :inner]) * z[:, inner:]).bfloat16().double()
        bound = (2.0 ** -8 * a.abs() + 1e-5) @ down[e].double().abs().T + 1e-5
        assert ((got[at].double() - a @ down[e].double().T).abs() <= bound).all(), (kind, e)
    K.check_device_errors("cuda:0")


@pytest.mark.parametrize("m", [1, 8, 9, 32])
@pytest.mark.parametrize("n,n_bf16,k", [(40, 8, 64), (8224, 8192, 2048), (50, 49, 4096), (10000, 9000, 256)])
def test_skinny_linear_split(K, m, n, n_bf16, k):
    """One pass over two matrices' rows: the first rounded, the others as float32 sums; borders inside a tile, K divided or not.
    The same kernel's whole results in either type have the same sums, so the same bits."""
    x, w = rnd(m, k, dtype=torch.bfloat16, seed=1), rnd(n, k, dtype=torch.bfloat16, scale=0.1, seed=2)
    a, b = K.skinny_linear_split(x, w, n_bf16)
    wide, rounded = K.skinny_linear(x, w, out_dtype=torch.float32), K.skinny_linear(x, w)
    assert torch.equal(a, rounded[:, :n_bf16]) and torch.equal(b, wide[:, n_bf16:])


@pytest.mark.parametrize("tokens,heads,kv,v_dim", [(1, 16, 4, 128), (5, 6, 3, 20), (700, 16, 4, 128), (2, 4, 1, 7)])
def test_talk_mix(K, tokens, heads, kv, v_dim):
    """Both forms (a thread an output, or four columns of a K/V group's heads) against float64."""
    wide, talk = rnd(tokens, heads, kv, v_dim, seed=1), rnd(heads, heads, seed=2)
    out = K.talk_mix(wide, talk, torch.float32).view(tokens, heads, v_dim)
    own = torch.arange(heads, device="cuda") // (heads // kv)
    per = wide.double()[:, :, own]                      # [tokens, g, h, v]: head g's weights on head h's values
    ref = torch.einsum("hg,tghv->thv", talk.double(), per)
    bound = heads * 2.0 ** -24 * torch.einsum("hg,tghv->thv", talk.double().abs(), per.abs()) + 1e-30
    assert ((out.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("width", [8, 1000, 4544])
def test_chain_of_launches_keeps_the_streams_order(K, width):
    """Kernels that may be placed while their predecessor still runs, one after the other on two buffers, each reading
    what the last one wrote and writing what it read, with a copy and an ordinary launch between: the same bits as with a
    synchronisation after each, as on the default stream, and as a replayed graph. Rows enough for several waves."""
    n, rounds = 3000, 6
    x0, gain, other = rnd(n, width, seed=1), 1 + rnd(width, scale=0.1, seed=2), rnd(n, width, seed=3)

    def chain(x, wait):
        for i in range(rounds):
            y = K.norm(x, gain, None, 1e-6, "rmsnorm")
            wait()
            K.scale_(x, 0.5)                # x after its reader
            wait()
            x.copy_(K.residual(x, y, other))
            wait()
            z = K.bias_act_(y, gain, "gelu")    # y after its readers
            wait()
            x.add_(z)                       # an ordinary launch
            wait()
        return K.to_float(x)

    want = chain(x0.clone(), torch.cuda.synchronize)
    assert torch.equal(chain(x0.clone(), lambda: None), want)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        assert torch.equal(chain(x0.clone(), lambda: None), want)
    torch.cuda.current_stream().wait_stream(side)
    x, graph = x0.clone(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = chain(x, lambda: None)
    for _ in range(2):
        x.copy_(x0)
        graph.replay()
        assert torch.equal(got, want)


@pytest.mark.parametrize("clamp", [None, (7.0, 1.702)])
def test_expert_units_at_large_gates(K, clamp):
    """Gates of either sign beyond where the exponential leaves float32 (results stay finite: an infinite one would meet the
    zeros of the second matrix), among them those whose 1 + exp(-gate) lies
    between 2^126 and 2^128: the unit is the float32 formula with a true division, rounded once to bfloat16 (2^-8 of
    itself beside the exponential's few units of 2^-24)."""
    g = torch.tensor([0.0, 1e-3, 0.5, 1.0, 3.0, 20.0, 50.0, 80.0, 86.0, 87.0, 87.5, 88.0, 88.5, 100.0, 1e4, 1e6])
    g = torch.cat([g, -g]).repeat_interleave(3).bfloat16()
    u = torch.tensor([1.0, 1e30, -3e4]).repeat(g.numel() // 3).bfloat16()
    h = torch.zeros(g.numel(), 8, dtype=torch.bfloat16)
    h[:, 0], h[:, 1] = g, u
    w = torch.zeros(1, 16, 8, dtype=torch.bfloat16)
    w[0, :8, 0], w[0, 8:, 1] = 1.0, 1.0
    down = torch.eye(8, dtype=torch.bfloat16)[None].contiguous()
    y, rows = K.expert_rows(h.cuda(), torch.zeros(g.numel(), 1, dtype=torch.int32, device="cuda"), w.cuda(), down.cuda(), clamp=clamp)
    got = y[rows.long()].cpu()
    g, u = g.float(), u.float()
    if clamp is not None:
        g, u, alpha = g.clamp(max=clamp[0]), u.clamp(-clamp[0], clamp[0]) + 1.0, clamp[1]
    else:
        alpha = 1.0
    ref = g / (1.0 + torch.exp(-alpha * g)) * u
    # what is smaller than float32's normal numbers may be flushed to zero
    for f in range(8):
        torch.testing.assert_close(got[:, f], ref.bfloat16().float(), rtol=2.0 ** -8, atol=2.0 ** -126, equal_nan=True)
