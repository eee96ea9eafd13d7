"""The quantizers' fused forms against the passes they stand for, bit for bit: the two-level macro scaling inside
the quantizers, and stochastic rounding from a slot-ordered table."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from alto_b200 import _lib as L
from alto_b200 import _linear as E
from alto_b200.hadamard import HadamardFactory
from alto_b200.macro_block_scaling import macro_block_scaling

MX = L.FMT_MXFP4


def _transform():
    HadamardFactory.configure(block_size=16, randomized=True, dtype=torch.float32, seed=11)
    return HadamardFactory.create_transform(device="cuda")


def _matrix(rows, cols, kind, seed=0):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(rows, cols, generator=g) * torch.exp2(torch.randint(-12, 12, (rows, 1), generator=g).float())
    if kind == "special":
        r = torch.rand(rows, cols, generator=g)
        x = torch.where(r < 0.2, torch.zeros(()), x)
        x = torch.where((r >= 0.2) & (r < 0.3), -torch.zeros(()), x)
        x[: rows // 3] = 0.0
        x[rows // 2, cols // 2] = float("inf")
        x[rows - 1, 0] = float("-inf")
        x[0, cols - 1] = float("nan")
    return x.bfloat16().cuda()


def _sr(rounding, rows, cols, rht=None, slots=False):
    if rounding == "rtn":
        return E.RTN
    if slots:
        return dict(rounding=L.ROUND_SR_SLOTS, rand_bits=L.philox_slots(7, 1 << 31, rht, torch.device("cuda")),
                    rand_tile=L.SLOTS_TILE)
    tile = L.sr_tile_dims(rows, cols)
    return dict(rounding=L.ROUND_SR_BITS, rand_bits=L.philox_tile(7, 1 << 31, *tile, torch.device("cuda")), rand_tile=tile)


def _same(a, b):
    assert torch.equal(a.codes, b.codes) and torch.equal(a.scales, b.scales)


def test_macro_field_needs_its_flag():
    """A caller built against the struct without the field passes whatever lies behind it: not read."""
    x = _matrix(64, 128, "normal")
    guard = torch.full((64,), 77, dtype=torch.uint8, device="cuda")
    out = [torch.empty(64, 64, dtype=torch.uint8, device="cuda") for _ in range(2)]
    scales = [torch.empty(64, 4, dtype=torch.uint8, device="cuda") for _ in range(2)]
    L.quantize_rowwise(x, MX, out[0], scales[0], None)
    p = L._params(MX, x, L.ROUND_RTN, None, None, None, L.SCALE_PLAIN)
    p.macro_codes = guard.data_ptr()
    rc = L.lib().altob200_quantize_rowwise(x.data_ptr(), 64, 128, 128, L.C.byref(p), out[1].data_ptr(),
                                           scales[1].data_ptr(), None, L._stream())
    assert rc == 0 and (guard == 77).all()
    assert torch.equal(out[0], out[1]) and torch.equal(scales[0], scales[1])


# one tile, ragged last tiles in either direction, several tiles
SHAPES = [(64, 64), (128, 128), (96, 160), (160, 416), (416, 1056)]


@pytest.mark.parametrize("kind", ["normal", "special"])
@pytest.mark.parametrize("rounding", ["rtn", "sr"])
@pytest.mark.parametrize("shape", SHAPES + [(130, 96)])
def test_rowwise_macro_scaling(shape, rounding, kind):
    x = _matrix(*shape, kind)
    codes = torch.empty(shape[0], -(-shape[1] // 128), dtype=torch.uint8, device="cuda")
    got = E.quant_rows(x, MX, None, _sr(rounding, *shape), macro_codes=codes)
    scaled, factors = macro_block_scaling(x, axis=-1)
    _same(got, E.quant_rows(scaled, MX, None, _sr(rounding, *shape)))
    assert torch.equal(codes, factors)


@pytest.mark.parametrize("kind", ["normal", "special"])
@pytest.mark.parametrize("clip_mode", ["none", "static", "dynamic"])
@pytest.mark.parametrize("rotate", [False, True])
@pytest.mark.parametrize("rounding", ["rtn", "sr"])
@pytest.mark.parametrize("shape", SHAPES)
def test_colwise_macro_scaling(shape, rounding, rotate, clip_mode, kind):
    x = _matrix(*shape, kind)
    had = _transform() if rotate else None
    rht = had.device_params() if rotate else None
    codes = torch.empty(shape[1], -(-shape[0] // 128), dtype=torch.uint8, device="cuda")
    got = E.quant_cols(x, MX, None, rht, _sr(rounding, shape[1], shape[0], rht, slots=True), clip_mode=clip_mode,
                       macro_codes=codes)
    scaled, factors = macro_block_scaling(had(x, left_mul=True) if rotate else x, axis=0)
    _same(got, E.quant_cols(scaled, MX, None, None, _sr(rounding, shape[1], shape[0]), clip_mode=clip_mode))
    assert torch.equal(codes, factors)


@pytest.mark.parametrize("kind", ["normal", "special"])
@pytest.mark.parametrize("rounding", ["rtn", "sr"])
@pytest.mark.parametrize("batch", [1, 3])
@pytest.mark.parametrize("shape", SHAPES)
def test_2d_macro_scaling(shape, batch, rounding, kind):
    rows, cols = shape
    x = torch.stack([_matrix(rows, cols, kind, seed=i) for i in range(batch)])
    sr = _sr(rounding, batch * rows, cols)

    def quantised(t, **macro):
        out = [torch.empty(batch, rows, cols // 2, dtype=torch.uint8, device="cuda"),
               torch.empty(batch, cols, rows // 2, dtype=torch.uint8, device="cuda"),
               torch.empty(batch * L.packed_scale_bytes(rows, cols // 32), dtype=torch.uint8, device="cuda"),
               torch.empty(batch * L.packed_scale_bytes(cols, rows // 32), dtype=torch.uint8, device="cuda")]
        L.quantize_2d_batched(t, MX, out[0], out[1], None, out[2], out[3], **macro, **sr)
        return out

    codes = torch.empty(batch, -(-rows // 128), -(-cols // 128), dtype=torch.uint8, device="cuda")
    got = quantised(x, macro_codes=codes)
    scaled, factors = macro_block_scaling(x, axis=-1, use_2d_block=True)
    assert all(torch.equal(g, e) for g, e in zip(got, quantised(scaled)))
    assert torch.equal(codes, factors)


@pytest.mark.parametrize("kind", ["normal", "special"])
@pytest.mark.parametrize("rotate", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("fmt", [L.FMT_NVFP4, L.FMT_MXFP4])
@pytest.mark.parametrize("shape", SHAPES)
def test_stochastic_rounding_from_the_slot_ordered_table(shape, fmt, dtype, rotate, kind):
    x = _matrix(*shape, kind).to(dtype)
    rht = _transform().device_params() if rotate else None
    rows, cols = shape[1], shape[0]
    tile = _sr("sr", rows, cols)
    # the plain table spelled out as one word per element
    planes = tile["rand_bits"].repeat(1, -(-rows // 64), -(-cols // 64))[:, :rows, :cols // 2].contiguous()
    got = E.quant_cols(x, fmt, None, rht, _sr("sr", rows, cols, rht, slots=True))
    _same(got, E.quant_cols(x, fmt, None, rht, tile))
    _same(got, E.quant_cols(x, fmt, None, rht, dict(rounding=L.ROUND_SR_BITS, rand_bits=planes)))


def test_macro_scaling_is_refused_where_it_is_not_built():
    x = _matrix(64, 64, "normal")
    codes = torch.empty(64, 1, dtype=torch.uint8, device="cuda")
    with pytest.raises(L.Altob200Error):
        E.quant_rows(x.float(), MX, None, E.RTN, macro_codes=codes)
    with pytest.raises(L.Altob200Error):
        E.quant_cols(x, MX, None, None, _sr("sr", 64, 64), macro_codes=codes)
    with pytest.raises(L.Altob200Error):
        E.quant_2d(x, L.FMT_NVFP4, None, True, macro_codes=codes)


@pytest.mark.parametrize("block", [1, 32])
@pytest.mark.parametrize("transposed", [False, True])
@pytest.mark.parametrize("rows,ncols", [(32, 1), (128, 4), (160, 7), (4096, 45)])
def test_packed_scales(rows, ncols, transposed, block):
    shape = (rows // block, ncols)
    s = torch.randint(0, 256, shape[::-1] if transposed else shape, generator=torch.Generator().manual_seed(1), dtype=torch.uint8)
    s = s.t() if transposed else s
    full = torch.zeros(-(-rows // 128) * 128, -(-ncols // 4) * 4, dtype=torch.uint8)
    full[:rows, :ncols] = s.repeat_interleave(block, 0)
    # tiles of 128 rows x 4 columns; in a tile 32 x 16 bytes: row % 32, then row / 32, then the column
    packed = full.view(-1, 4, 32, full.shape[1] // 4, 4).permute(0, 3, 2, 1, 4).reshape(-1)
    assert torch.equal(E.pack_plain_scales(s.cuda() if not transposed else s.t().cuda().t(), rows, block > 1, block).cpu(), packed)


@pytest.mark.parametrize("counts", [[128], [0, 256, 0, 0, 128, 0], [128] * 300, [0, 0]])
def test_expert_of_every_row_group(counts):
    from alto_b200.grouped import group_experts_from_offsets
    offs = torch.tensor(counts, dtype=torch.int64).cumsum(0).to(torch.int32)
    rows = int(offs[-1]) + 200
    expect = [next((e for e, end in enumerate(offs.tolist()) if end > start), -1) for start in range(0, rows, 128)]
    assert group_experts_from_offsets(offs.cuda(), rows).tolist() == expect


@pytest.mark.parametrize("needs", [(True, False), (False, True), (False, False)])
@pytest.mark.parametrize("weight_2d", [False, True])
@pytest.mark.parametrize("recipe", ["nvfp4", "mxfp4", "mxfp8"])
def test_operands_of_gradients_that_are_not_asked_for(recipe, weight_2d, needs):
    from alto_b200 import mxfp4, mxfp8, nvfp4
    calls = {"nvfp4": lambda x, w: nvfp4._to_nvfp4_then_scaled_mm(x, w, False, weight_2d, True, use_outer_scale=True,
                                                                 use_hadamard=True),
             "mxfp4": lambda x, w: mxfp4._to_mxfp4_then_scaled_mm(x, w, False, weight_2d, True, True, "none", True),
             "mxfp8": lambda x, w: mxfp8._to_mxfp8_then_scaled_mm(x, w, "e4m3", False, False, weight_2d)}
    x0, w0, dy = _matrix(128, 192, "normal"), _matrix(160, 192, "normal", 1), _matrix(128, 160, "normal", 2)

    def step(need_x, need_w):
        _transform()
        torch.manual_seed(5)
        x, w = x0.clone().requires_grad_(need_x), w0.clone().requires_grad_(need_w)
        y = calls[recipe](x, w)
        if need_x or need_w:
            y.backward(dy)
        return y.detach(), x.grad, w.grad

    full, got = step(True, True), step(*needs)
    assert torch.equal(got[0], full[0])
    for need, g, f in zip(needs, got[1:], full[1:]):
        assert torch.equal(g, f) if need else g is None


@pytest.mark.parametrize("form", ["expanded", "overlapping", "column slice", "odd offset"])
def test_two_level_operands_of_views(form):
    """Rows the fused quantizers cannot read as they are give what a contiguous copy gives."""
    from alto_b200 import _two_level as T
    base = _matrix(160, 512, "normal")
    t = {"expanded": lambda: base[:1, :256].expand(96, 256),
         "overlapping": lambda: base.flatten().as_strided((96, 256), (64, 1)),
         "column slice": lambda: base[:96, 64:320],
         "odd offset": lambda: base[:96, 3:259]}[form]()
    makers = [lambda v: T.rows_operand(v, False), lambda v: T.cols_operand(v, False),
              lambda v: T.tiles_operands(v, False)[0]]
    if form == "column slice":   # the transform itself takes no overlapping or misaligned rows
        rht = _transform()
        makers.append(lambda v: T.cols_operand(v, False, "none", None, rht))
    for make in makers:
        got, want = make(t), make(t.contiguous())
        _same(got, want)
        assert torch.equal(got.macro.codes, want.macro.codes)


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("tile", [None, (64, 32), (5, 8), (3, 12), (64, 6)])
@pytest.mark.parametrize("rotate", [False, True])
@pytest.mark.parametrize("fmt", [L.FMT_NVFP4, L.FMT_MXFP4])
@pytest.mark.parametrize("shape", [(32, 8), (96, 160), (160, 416)])
def test_column_blocks_with_explicit_words(shape, fmt, rotate, tile, offset):
    """Words in vectors (16-byte aligned, whole groups of 16 rows) or one by one: the codes that the row-wise
    quantizer makes of the transposed matrix with the same words."""
    x = _matrix(*shape, "normal")
    rows, cols = shape[1], shape[0]                      # of the axis-last view
    n_rows, n_pairs = tile or (rows, cols // 2)
    g = torch.Generator().manual_seed(3)
    flat = torch.randint(-2 ** 31, 2 ** 31 - 1, (2 * n_rows * n_pairs + offset,), generator=g, dtype=torch.int32).cuda()
    table = flat[offset:].view(2, n_rows, n_pairs)
    planes = table[:, torch.arange(rows, device="cuda") % n_rows][:, :, torch.arange(cols // 2, device="cuda") % n_pairs]
    had = _transform() if rotate else None
    got = E.quant_cols(x, fmt, None, had.device_params() if rotate else None,
                       dict(rounding=L.ROUND_SR_BITS, rand_bits=table, rand_tile=tile or (0, 0)))
    view = (had(x, left_mul=True) if rotate else x).t().contiguous()
    _same(got, E.quant_rows(view, fmt, None, dict(rounding=L.ROUND_SR_BITS, rand_bits=planes.contiguous())))


def test_dynamic_clip_behind_a_rotation_sums_in_row_order():
    """Rotated columns of +-M whose running sum overflows in some orders of the rows and not in others: the block
    statistics, hence the codes, are those of the separate passes."""
    from alto_b200 import _two_level as T
    had = _transform()
    x = torch.zeros(128, 16, dtype=torch.bfloat16, device="cuda")
    x[torch.arange(16), torch.arange(16)] = 3.3e38
    got = T.cols_operand(x, False, "dynamic", None, had)
    scaled, factors = macro_block_scaling(had(x, left_mul=True), axis=0)
    _same(got, E.quant_cols(scaled, MX, None, None, E.RTN, clip_mode="dynamic"))
    assert torch.equal(got.macro.codes, factors)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("clip_mode", ["none", "dynamic"])
def test_two_level_gradients_draw_the_same_words_on_every_route(dtype, clip_mode, monkeypatch):
    """Rounding words of a gradient that is rotated inside the quantizer, before it, or in fp32: those of the
    plain table."""
    from types import SimpleNamespace
    from alto_b200 import _two_level as T
    had = _transform()
    g = (_matrix(160, 192, "normal") * 1e-3).to(dtype)
    ctx = SimpleNamespace(use_2dblock_x=False, use_uos=False, use_sr_grad=True, hadamard_transform=had,
                          clip_mode=clip_mode)
    torch.manual_seed(9)
    got = T._grad_operands(ctx, g, 160, 192)
    monkeypatch.setattr(L, "SLOTS_TILE", None)           # no view takes the slot-ordered table
    torch.manual_seed(9)
    want = T._grad_operands(ctx, g, 160, 192)
    for a, b in zip(got, want):
        _same(a, b)
        assert torch.equal(a.macro.codes, b.macro.codes)


@pytest.mark.parametrize("shape", [(64, 64), (160, 416)])
def test_macro_scaling_with_a_word_for_every_element(shape):
    """The fused row-wise and 2-D forms with full planes of words instead of a periodic table."""
    x = _matrix(*shape, "normal")
    g = torch.Generator().manual_seed(4)
    words = torch.randint(-2 ** 31, 2 ** 31 - 1, (2, shape[0], shape[1] // 2), generator=g, dtype=torch.int32).cuda()
    sr = dict(rounding=L.ROUND_SR_BITS, rand_bits=words)
    for two_d in (False, True):
        chunks = (-(-shape[0] // 128) if two_d else shape[0], -(-shape[1] // 128))
        codes = torch.empty(chunks, dtype=torch.uint8, device="cuda")
        scaled, factors = macro_block_scaling(x, axis=-1, use_2d_block=two_d)
        if two_d:
            got, want = E.quant_2d(x, MX, None, True, False, sr, codes), E.quant_2d(scaled, MX, None, True, False, sr)
        else:
            got, want = [E.quant_rows(x, MX, None, sr, macro_codes=codes)], [E.quant_rows(scaled, MX, None, sr)]
        for a, b in zip(got, want):
            _same(a, b)
        assert torch.equal(codes, factors)
