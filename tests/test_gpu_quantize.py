"""Parity of the quantisers, SwiGLU rows and combine kernels through the C ABI: E4M3 bytes
and fp32 scales bit-exact against the oracle and the reference's fixtures."""

import pytest
import torch

import inputs
from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
U8 = torch.uint8


def _ops():
    from mlops_b200 import ops

    return ops


def test_weight_blocks_match_reference_fixture(golden):
    ops = _ops()
    fixture = golden("quantize.pt")
    w = inputs.block_weight()
    for name, value in (("w_fp32", w), ("w_bf16", w.bfloat16())):
        data, scale = ops.quantize_blocks(value.to(DEV))
        assert torch.equal(data.cpu().view(U8), fixture[name + "_data"])
        assert torch.equal(scale.cpu(), fixture[name + "_scale"])


@pytest.mark.parametrize("shape", [(1, 128, 128), (2, 8, 8), (3, 200, 328), (1, 129, 4), (2, 64, 1000)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("special", [False, True])
def test_weight_blocks_of_aligned_and_unaligned_sources(shape, dtype, special):
    """The one-pass quantiser (16-byte loads) writes the bytes and scales of the value-by-value one,
    which serves a source one element off alignment; both equal the oracle where it is defined by
    finite values. Infinities and NaN: the maximum skips a NaN, an infinity makes the scale
    infinite, and a NaN quotient stays a NaN."""
    ops = _ops()
    g = torch.Generator().manual_seed(sum(shape))
    n = shape[0] * shape[1] * shape[2]
    w = (torch.randn(n, generator=g) * torch.rand(n, generator=g).mul(40).sub(20).exp2()).to(dtype).view(shape)
    if special:
        w.view(-1)[3] = float("nan")
        w[-1, -1, -1] = float("-inf")
    else:
        w[0, 0, :4] = 0
    store = torch.empty(n + 1, dtype=dtype, device=DEV)
    store[1:] = w.to(DEV).view(-1)
    q, s = ops.quantize_blocks(w.to(DEV))
    q_general, s_general = ops.quantize_blocks(store[1:].view(shape))
    assert torch.equal(q.view(U8), q_general.view(U8))
    assert torch.equal(s, s_general)
    if not special:
        q_ref, s_ref = O.quantize_blocks(w)
        assert torch.equal(q.cpu().view(U8), q_ref.view(U8)) and torch.equal(s.cpu(), s_ref)


def test_publication_writes_the_container_in_place():
    """`container.copy_(master)` fills the container's own buffers, a master that shares their
    memory or broadcasts included, and tells autograd that they changed."""
    from mlops_b200.weights import BlockFP8Weight

    ops = _ops()
    g = torch.Generator().manual_seed(5)
    master = torch.randn(3, 256, 128, generator=g).to(DEV)
    ref, ref_scale = ops.quantize_blocks(master)
    container = BlockFP8Weight(torch.zeros_like(ref), torch.zeros_like(ref_scale))
    data, scale, versions = container._data, container._scale, (container._data._version, container._scale._version)
    container.copy_(master)
    assert container._data is data and container._scale is scale
    assert torch.equal(data.view(U8), ref.view(U8)) and torch.equal(scale, ref_scale)
    assert data._version > versions[0] and scale._version > versions[1]
    container.copy_(master[:1])  # broadcast over the experts
    assert torch.equal(data.view(U8), ref[:1].expand_as(ref).view(U8))
    store = torch.empty(master.numel(), device=DEV)  # the master's memory holds the container's bytes
    shared = BlockFP8Weight(store.view(torch.float8_e4m3fn)[:master.numel()].view(3, 256, 128), torch.zeros_like(scale))
    store.view(3, 256, 128).copy_(master)
    shared.copy_(store.view(3, 256, 128))
    assert torch.equal(shared._data.view(U8), ref.view(U8))


def test_row_quantiser_matches_reference_fixture(golden):
    ops = _ops()
    fixture = golden("quantize.pt")
    x, gather = inputs.activation_rows()
    data, scale = ops.quantize_rows(x.to(DEV), gather=gather.to(DEV), gather_div=1, mode="row")
    assert torch.equal(data.cpu().view(U8), fixture["rows_data"])
    assert torch.equal(scale.cpu()[:, 0], fixture["rows_scale"])


@pytest.mark.parametrize("rows,width", [(300, 256), (64, 192), (1000, 7168), (33, 2048), (7, 8)])
@pytest.mark.parametrize("mode", ["1x128", "row"])
def test_quantize_rows_bit_exact(rows, width, mode):
    ops = _ops()
    g = torch.Generator().manual_seed(rows + width)
    x = torch.randn(rows, width, generator=g).bfloat16()
    x[0] = 0                     # all-zero row keeps the 1e-12 floor
    x[rows // 2] *= 30000        # values that saturate nothing after scaling
    gather = torch.randint(0, rows, (2 * rows,), generator=g).to(torch.int32)
    q_ref, s_ref = O.quantize_rows(x, gather=torch.div(gather, 2, rounding_mode="floor"), mode=mode)
    q, s = ops.quantize_rows(x.to(DEV), gather=gather.to(DEV), gather_div=2, mode=mode)
    assert torch.equal(q.cpu().view(U8), q_ref.view(U8))
    assert torch.equal(s.cpu(), s_ref)
    q2, s2 = ops.quantize_rows(x.to(DEV), mode=mode)  # no gather
    q2_ref, s2_ref = O.quantize_rows(x, mode=mode)
    assert torch.equal(q2.cpu().view(U8), q2_ref.view(U8)) and torch.equal(s2.cpu(), s2_ref)


def test_quantize_rows_writes_the_gathered_rows_into_a_given_slice():
    """`copy_out`: the quantiser also writes the bf16 rows it gathered, into a caller's slice
    (a pitched view of a larger buffer), bit for bit; the E4M3 result does not change."""
    ops = _ops()
    g = torch.Generator().manual_seed(21)
    x = torch.randn(90, 384, generator=g).bfloat16().to(DEV)
    gather = torch.randint(0, 90 * 3, (200,), generator=g).to(torch.int32).to(DEV)
    q_ref, s_ref = ops.quantize_rows(x, gather=gather, gather_div=3)
    big = torch.full((260, 384), float("nan"), dtype=torch.bfloat16, device=DEV)
    q, s, copy = ops.quantize_rows(x, gather=gather, gather_div=3, copy_out=big[30:230])
    assert copy.data_ptr() == big[30:230].data_ptr()
    assert torch.equal(big[30:230], x[torch.div(gather, 3, rounding_mode="floor").long()])
    assert big[:30].isnan().all() and big[230:].isnan().all()
    assert torch.equal(q.view(U8), q_ref.view(U8)) and torch.equal(s, s_ref)


def test_quantize_rows_empty():
    ops = _ops()
    q, s = ops.quantize_rows(torch.zeros(0, 256, dtype=torch.bfloat16, device=DEV))
    assert q.shape == (0, 256) and s.shape == (0, 2)


@pytest.mark.parametrize("rows,width", [(100, 512), (77, 640), (50, 80)])
@pytest.mark.parametrize("limit", [None, 1.5])
def test_swiglu_quantize(rows, width, limit):
    """fp32 SwiGLU differs from the CPU's by an ulp of expf at most, which can move a value
    across an E4M3 rounding boundary: bytes must agree on all but a 1e-3 fraction, and the
    bf16 activation within bf16 rounding."""
    ops = _ops()
    g = torch.Generator().manual_seed(rows)
    h = (torch.randn(rows, 2 * width, generator=g) * 2).bfloat16()
    act = O.swiglu(h, limit)
    q_ref, s_ref = O.quantize_rows(act, mode="1x128")
    q, s, a16 = ops.swiglu_quantize(h.to(DEV), limit=limit, quantized=True, rounded=True)
    same = (q.cpu().view(U8) == q_ref.view(U8)).float().mean().item()
    assert same > 0.999
    torch.testing.assert_close(s.cpu(), s_ref, rtol=1e-6, atol=0)
    mx, mean = O.rel_errors(a16.float().cpu(), act)
    assert mx <= 2e-2 and mean <= 2e-3


@pytest.mark.parametrize("limit", [None, 1.5])
def test_dswiglu_routed(limit):
    ops = _ops()
    g = torch.Generator().manual_seed(11)
    rows, width = 90, 256
    h = (torch.randn(rows, 2 * width, generator=g) * 2).bfloat16()
    r = torch.randn(rows, width, generator=g).bfloat16()
    route_weights = torch.rand(rows, generator=g)
    order = torch.randperm(rows, generator=g).to(torch.int32)
    ds_ref, gh_ref, as_ref = O.dswiglu_routed(h, r, route_weights[order.long()], limit)
    ds, gq, gs, gb, a_s = ops.dswiglu_routed(
        h.to(DEV), r.to(DEV), route_weights.to(DEV), order.to(DEV), limit=limit, quantized=True,
        rounded=True, scaled_activation=True,
    )
    torch.testing.assert_close(ds.cpu(), ds_ref, rtol=1e-5, atol=1e-5)
    for actual, expected in ((gb, gh_ref), (a_s, as_ref)):
        mx, mean = O.rel_errors(actual.float().cpu(), expected)
        assert mx <= 2e-2 and mean <= 2e-3
    q_ref, s_ref = O.quantize_rows(gh_ref, mode="1x128")
    torch.testing.assert_close(gs.cpu(), s_ref, rtol=1e-5, atol=0)
    assert (gq.cpu().view(U8) == q_ref.view(U8)).float().mean().item() > 0.995


def test_combine_matches_reference_fixture_and_oracle(golden):
    ops = _ops()
    fixture = golden("combine.pt")
    out = ops.combine(*(fixture[k].to(DEV) for k in ("source", "slots", "weights", "residual")))
    assert torch.equal(out.cpu(), O.combine(fixture["source"], fixture["slots"], fixture["weights"], fixture["residual"]))
    torch.testing.assert_close(out.cpu().float(), fixture["output"].float(), rtol=2 ** -7, atol=1e-6)
    g = torch.Generator().manual_seed(3)
    tokens, top_k, width = 200, 4, 384
    src = torch.randn(tokens * top_k, width, generator=g).bfloat16()
    slots = torch.randperm(tokens * top_k, generator=g).view(tokens, top_k).to(torch.int32)
    again = ops.dispatch_backward(src.to(DEV), slots.to(DEV))
    assert torch.equal(again.cpu(), O.combine(src, slots, None, None))
    assert torch.equal(again, ops.dispatch_backward(src.to(DEV), slots.to(DEV)))  # repeatable
    order = torch.randperm(tokens * top_k, generator=g).to(torch.int32)
    x = torch.randn(tokens, width, generator=g).bfloat16()
    rows = ops.dispatch(x.to(DEV), order.to(DEV), top_k)
    assert torch.equal(rows.cpu(), x[order.long() // top_k])


def test_scatter_quantiser_equals_the_gathered_quantiser_bit_for_bit():
    """Quantising every token once and writing its row to its K expert-ordered rows gives the
    bytes, the scales and the bf16 copies of the per-output-row gather (which is pinned above
    against the reference's `quantize_rows_fp8_reference`), including a width that is not a
    multiple of 128 and a slot outside the output, which is reported and skipped."""
    from mlops_b200 import ops
    from mlops_b200._lib import NativeError

    g = torch.Generator().manual_seed(31)
    tokens, top_k, experts = 700, 8, 64
    for width in (7168, 1000):
        x = torch.randn(tokens, width, generator=g).bfloat16().to(DEV)
        ids = torch.stack([torch.randperm(experts, generator=g)[:top_k] for _ in range(tokens)]).to(torch.int32).to(DEV)
        order, _offsets, slots, _counts = ops.sort_assignments(ids, experts)
        q_ref, s_ref, c_ref = ops.quantize_rows(x, gather=order, gather_div=top_k, with_copy=True)
        q, s, c = ops.quantize_rows_scatter(x, slots, with_copy=True)
        assert torch.equal(q.view(torch.uint8), q_ref.view(torch.uint8))
        assert torch.equal(s, s_ref) and torch.equal(c, c_ref)
    ops.check_status(DEV)
    bad = slots.clone()
    bad[3, 2] = tokens * top_k + 5
    ops.quantize_rows_scatter(x, bad)
    with pytest.raises(NativeError):
        ops.check_status(DEV)


@pytest.mark.parametrize("rows", [3, 5000])  # a warp per 256 columns / per row
@pytest.mark.parametrize("width", [8, 264, 768])
@pytest.mark.parametrize("limit", [None, 1.3])
def test_swiglu_over_the_whole_range_of_gates(rows, width, limit):
    """Gates from 2^-20 to 2^100, infinities and NaN: fp32 SwiGLU rounded once to bf16 is the float64
    value to one bf16 rounding (2^-8 relative, and 2^-20 of slack for the fp32 steps), values of the
    two forms of the reciprocal (changing at g = -80) alike; a NaN stays one."""
    ops = _ops()
    g = torch.Generator().manual_seed(rows + width)
    gate = torch.randn(rows, width, generator=g) * torch.rand(rows, width, generator=g).mul(12).sub(6).exp2()
    gate[0, :8] = torch.tensor([float("inf"), float("-inf"), float("nan"), 12.0, -12.0, 2.0 ** 100, -88.0, 0.0])
    up = torch.randn(rows, width, generator=g)
    h = torch.cat([gate, up], dim=1).bfloat16()
    _q, _s, act = ops.swiglu_quantize(h.to(DEV), limit=limit, quantized=False, rounded=True)
    gd, ud = h[:, :width].double(), h[:, width:].double()
    if limit is not None:
        cap = torch.tensor(limit, dtype=torch.float32).double()
        gd, ud = torch.where(gd > cap, cap, gd), ud.clamp(-cap, cap)
    expected = gd * torch.sigmoid(gd) * ud
    actual = act.cpu().double()
    odd = ~expected.isfinite() | gd.isnan() | gd.isinf() | (gd < -80)  # fp32 underflows or overflows there
    error = (actual - expected).abs()[~odd]
    assert (error <= expected.abs()[~odd] * (2.0 ** -8 + 2.0 ** -20) + 1e-37).all()
    if limit is None:
        assert actual[0, 2].isnan() and actual[0, 0].isinf() and actual[0, 1].isnan()


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("boundary", [True, False])
def test_a_nan_survives_every_quantiser_whatever_its_neighbours(value, boundary):
    """A NaN, or an infinity divided by its infinite scale, among eight values of which one lies on a
    rounding boundary of E4M3 (17 between 16 and 18 at scale 1: these eight are divided exactly) or none
    does: the NaN byte, and the other values as torch's division, clamp and cast give them at the
    kernel's scale."""
    ops = _ops()
    x = torch.randn(128, 128, generator=torch.Generator().manual_seed(3)).bfloat16()
    x[:, 0], x[:, 1], x[:, 2] = 448.0, 17.0 if boundary else 16.0, value  # scale 1 unless infinite
    wide = x.to(DEV)
    slots = torch.arange(128, dtype=torch.int32, device=DEV).view(128, 1)
    whole = torch.tensor([0, 128], dtype=torch.int32, device=DEV)
    store = torch.empty(128 * 128 + 1, dtype=torch.bfloat16, device=DEV)
    store[1:] = wide.view(-1)
    produced = {
        "1x128": ops.quantize_rows(wide), "row": ops.quantize_rows(wide, mode="row"),
        "scatter": ops.quantize_rows_scatter(wide, slots), "columns": ops.quantize_columns(wide, whole, 1),
        "blocks": [t[0] for t in ops.quantize_blocks(wide[None])],
        "blocks fp32": [t[0] for t in ops.quantize_blocks(wide.float()[None])],
        "blocks, unaligned": [t[0] for t in ops.quantize_blocks(store[1:].view(1, 128, 128))],
    }
    for name, (q, scale) in produced.items():
        got = q.cpu().float()
        expected = torch.clamp(x.float() / scale.cpu().float(), -448.0, 448.0).to(torch.float8_e4m3fn).float()
        assert expected[:, 2].isnan().all() and torch.equal(got.isnan(), expected.isnan()), name
        assert torch.equal(got.nan_to_num(0.0), expected.nan_to_num(0.0)), name


@pytest.mark.parametrize("limit", [None, 1.3])
def test_swiglu_holds_the_library_functions_in_fp32(limit):
    """silu of every finite bf16 gate in fp32, seen through the route-weight gradient (a one-hot r and up
    = 1 make it silu itself): the bits of `g * reciprocal(1 + exp(-g))`, and within 7 x 2^-24 of the float64
    value (exponential two ulp of 2^-23, sum, reciprocal and product half an ulp each)."""
    ops = _ops()
    gates = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    gates = gates[gates.isfinite()].view(-1, 8)  # eight consecutive patterns a row: neighbours in one thread
    rows = gates.shape[0]
    h13 = torch.cat([gates, torch.ones_like(gates)], dim=1).to(DEV)
    order, ones = torch.arange(rows, dtype=torch.int32, device=DEV), torch.ones(rows, device=DEV)
    g = gates.to(DEV).float()
    if limit is not None:
        g = g.clamp(max=limit)
    same = g * torch.reciprocal(1.0 + torch.exp(-g))
    exact = g.double() * torch.sigmoid(g.double())
    for column in range(8):
        r = torch.zeros(rows, 8, dtype=torch.bfloat16, device=DEV)
        r[:, column] = 1.0
        dscore = ops.dswiglu_routed(h13, r, ones, order, limit=limit, quantized=False, rounded=True)[0]
        assert torch.equal(dscore, same[:, column])
        normal = exact[:, column].abs() > 2.0 ** -120
        error = (dscore.double() - exact[:, column]).abs()[normal]
        assert (error <= 7 * 2.0 ** -24 * exact[:, column].abs()[normal]).all()


@pytest.mark.parametrize("tokens,width,top_k", [(1, 8, 1), (3, 1032, 2), (70, 2048, 3), (5, 7168, 8), (9, 264, 11)])
def test_row_kernels_at_the_edges_of_their_pieces(tokens, width, top_k):
    """Pieces of 512 (scatter quantiser) and 1024 columns (combine, gather), batches of 2, 4 and 8
    slots: widths that end inside a piece, more slots than a batch, and negative slots, which add
    nothing. Bit-equal to the oracle (one fp32 sum in slot order, one rounding)."""
    ops = _ops()
    g = torch.Generator().manual_seed(tokens * width + top_k)
    x = torch.randn(tokens, width, generator=g).bfloat16()
    order = torch.randperm(tokens * top_k, generator=g).to(torch.int32)
    slots = torch.empty(tokens * top_k, dtype=torch.int32)
    slots[order.long()] = torch.arange(tokens * top_k, dtype=torch.int32)
    slots = slots.view(tokens, top_k)
    rows = x[torch.div(order, top_k, rounding_mode="floor").long()]
    q_ref, s_ref = O.quantize_rows(rows, mode="1x128")
    q, s, copy = ops.quantize_rows_scatter(x.to(DEV), slots.to(DEV), with_copy=True)
    assert torch.equal(q.cpu().view(U8), q_ref.view(U8)) and torch.equal(s.cpu(), s_ref)
    assert torch.equal(copy.cpu(), rows) and torch.equal(ops.dispatch(x.to(DEV), order.to(DEV), top_k).cpu(), rows)
    if top_k <= 32:
        assert torch.equal(ops.scatter_rows(x.to(DEV), slots.to(DEV)).cpu(), rows)
    weights = torch.randint(-3, 2, (tokens, top_k), generator=g).float().exp2()  # products are exact, fused or not
    residual = torch.randn(tokens, width, generator=g).bfloat16()
    got = ops.combine(rows.to(DEV), slots.to(DEV), weights.to(DEV), residual.to(DEV))
    assert torch.equal(got.cpu(), O.combine(rows, slots, weights, residual))
    if top_k > 1:
        holes = slots.clone()
        holes[:, 1] = -1
        zeroed = weights.clone()
        zeroed[:, 1] = 0
        got = ops.combine(rows.to(DEV), holes.to(DEV), weights.to(DEV), residual.to(DEV))
        assert torch.equal(got.cpu(), O.combine(rows, slots, zeroed, residual))
    ops.check_status(DEV)
