"""The kernels and call paths that the dispatch picks by size, at the edges of their tiles, against a dense product of
whole numbers (exact in every order of summation)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _operand(M, K, V, m, strategy, seed):
    import torch
    from venom_b200 import capi
    from venom_b200.synth import random_vnm_dense
    dense, cols, _ = random_vnm_dense(M, K, V, m, seed=seed, integer_values=True)
    d = torch.from_numpy(dense).cuda()
    c = torch.from_numpy(cols.view(np.int32)).cuda()
    values, meta, bad = capi.compress(d, c, V, m)
    assert bad == 0
    return d.float(), values, meta, c, capi.Prepared(values, meta, c, M, K, V, m, strategy=strategy)


def _ints(shape, seed):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randint(-4, 5, shape, generator=g, device="cuda").half()


# Few columns: every N up to 64 and beyond at the edges of tiles; k-tiles that split evenly, raggedly and not at all; ragged rows.
@pytest.mark.parametrize("N", [8, 16, 24, 32, 40, 64, 72, 136])
@pytest.mark.parametrize("cfg", [(128, 1024, 128, 16), (96, 520, 32, 8), (192, 2048, 64, 8), (704, 4480, 64, 32), (128, 512, 128, 4)])
@pytest.mark.parametrize("form", ["gather", "dense_b"])
def test_few_columns(N, cfg, form):
    import torch
    from venom_b200 import capi
    M, K, V, m = cfg
    d, _, _, _, prep = _operand(M, K, V, m, capi.STRATEGY_GATHER if form == "gather" else capi.STRATEGY_DENSE_B, seed=M + K)
    B = _ints((K, N), N)
    bias = _ints((M,), 3)
    want = d @ B.float()
    assert torch.equal(prep.spmm(B), want.half())
    assert torch.equal(prep.spmm(B, bias=bias, layout=capi.VNM_LAYOUT_NM), (want.half() + bias[:, None]).T)
    if form == "dense_b":
        assert torch.equal(prep.spmm_nk(B.T.contiguous()), want.half().T)
    assert prep.device_status() == 0


# Few columns: widths of 32 and 64 as well as 16, unsplit and split by 2 to 8, of 1, 2 and 4 vector blocks a tile: (form, V, row tiles, k-tiles, N, width, split).  The
# last k-tile is ragged.  Among them the sizes at which a split was taken that is slower than none (V = 128, 96 row tiles and 16 k-tiles; 23 and 8).
@pytest.mark.parametrize("cfg", [("dense_b", 64, 12, 20, 64, 32, 4), ("dense_b", 64, 23, 20, 40, 16, 2), ("dense_b", 64, 8, 7, 40, 16, 4), ("dense_b", 64, 1, 6, 8, 16, 6),
                                 ("dense_b", 64, 1, 7, 8, 16, 7), ("dense_b", 64, 75, 8, 40, 64, 1), ("dense_b", 64, 48, 8, 64, 32, 1), ("gather", 128, 32, 24, 40, 32, 2),
                                 ("gather", 128, 75, 32, 24, 32, 3), ("gather", 128, 23, 24, 64, 32, 5), ("gather", 128, 5, 32, 64, 32, 8), ("gather", 128, 32, 32, 40, 64, 4),
                                 ("gather", 128, 75, 8, 40, 64, 1), ("gather", 128, 96, 16, 32, 32, 1), ("gather", 128, 96, 16, 16, 16, 1), ("gather", 128, 23, 8, 64, 16, 1),
                                 ("gather", 64, 48, 32, 40, 64, 5), ("gather", 64, 12, 13, 24, 32, 8), ("gather", 64, 12, 8, 64, 32, 4), ("gather", 32, 8, 24, 40, 32, 6),
                                 ("gather", 32, 12, 24, 64, 64, 8), ("gather", 32, 23, 16, 64, 64, 4), ("gather", 32, 23, 8, 64, 64, 1), ("gather", 32, 74, 8, 24, 32, 1),
                                 ("gather", 32, 48, 13, 24, 32, 5), ("gather", 32, 75, 20, 24, 32, 3), ("gather", 32, 48, 12, 24, 32, 2), ("gather", 32, 288, 4, 64, 64, 1)])
def test_widths_and_splits_of_few_columns(cfg):
    import torch
    from venom_b200 import capi
    from venom_b200.synth import random_vnm_dense_cuda
    form, V, mtiles, ktiles, N, width, split = cfg
    M, K, m = 128 * mtiles, (128 * ktiles - 56 if form == "dense_b" else 256 * ktiles - 40), 8
    dense, cols = random_vnm_dense_cuda(M, K, V, m, seed=M + K)
    dense = torch.sign(dense) * torch.ceil(dense.abs() * 3)
    values, meta, bad = capi.compress(dense, cols, V, m)
    assert bad == 0
    prep = capi.Prepared(values, meta, cols, M, K, V, m, strategy=capi.STRATEGY_GATHER if form == "gather" else capi.STRATEGY_DENSE_B)
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        got = prep.config(N)
        assert got["tile_n"] == width and got["grid"] == mtiles * -(-N // width) * split
    B, bias = _ints((K, N), N), _ints((M,), 3)
    want = (dense.float() @ B.float()).half()
    assert torch.equal(prep.spmm(B), want)
    assert torch.equal(prep.spmm(B, bias=bias, layout=capi.VNM_LAYOUT_NM), (want + bias[:, None]).T)
    if form == "dense_b":
        assert torch.equal(prep.spmm_nk(B.T.contiguous()), want.T)
    assert prep.device_status() == 0


# Few tiles: one CTA an SM with the deep ring (eight k-tiles a CTA and more), two, and several waves of them; rings that do and do not go round.
@pytest.mark.parametrize("V", [128, 64, 32])
@pytest.mark.parametrize("ktiles", [7, 8, 9, 21])
@pytest.mark.parametrize("N", [72, 104, 200, 264])
@pytest.mark.parametrize("form", ["gather", "dense_b"])
def test_few_tiles_with_the_deep_ring(form, N, ktiles, V):
    import torch
    from venom_b200 import capi
    M, m = 160 if V == 32 else 192 if V == 64 else 256, 8
    K = 128 * ktiles - 56 if form == "dense_b" else 256 * ktiles - 40       # the last k-tile is ragged
    d, _, _, _, prep = _operand(M, K, V, m, capi.STRATEGY_GATHER if form == "gather" else capi.STRATEGY_DENSE_B, seed=M + K)
    prep.set_pair_mode(0)
    cfg = prep.config(N)
    assert cfg["tile_m"] == 128 and (cfg["smem_bytes"] > 110 * 1024) == (ktiles >= 8 or cfg["tile_n"] * (128 // V if form == "gather" else 1) > 128)
    B, bias = _ints((K, N), N), _ints((M,), 3)
    want = (d @ B.float()).half()
    assert torch.equal(prep.spmm(B), want)
    assert torch.equal(prep.spmm(B, bias=bias, layout=capi.VNM_LAYOUT_NM), (want + bias[:, None]).T)
    if form == "dense_b":
        assert torch.equal(prep.spmm_nk(B.T.contiguous()), want.T)
    assert prep.device_status() == 0


# SM pairs, 256 rows a tile: every width, columns that end inside a tile; one tile a cluster, whose columns both epilogue groups share,
# and two or three, the last of which they share; ragged rows.
@pytest.mark.parametrize("tiles", [1, 2, 3])
@pytest.mark.parametrize("N", [176, 192, 216, 240, 248, 504])
def test_pair_tiles_shared_by_both_epilogue_groups(N, tiles):
    import torch
    from venom_b200 import capi
    from venom_b200.synth import random_vnm_dense_cuda
    pairs = torch.cuda.get_device_properties(0).multi_processor_count // 2
    M, K, V, m = (256 * 3 if tiles == 1 else 256 * (pairs * (tiles - 1) + 2)) - 96, 264, 32, 8
    dense, cols = random_vnm_dense_cuda(M, K, V, m, seed=M + N)
    dense = torch.sign(dense) * torch.ceil(dense.abs() * 3)
    values, meta, bad = capi.compress(dense, cols, V, m)
    assert bad == 0
    prep = capi.Prepared(values, meta, cols, M, K, V, m, strategy=capi.STRATEGY_DENSE_B)
    prep.set_pair_mode(3)   # 256 rows a tile, not the kernel for few tiles
    assert prep.config(N)["tile_m"] == 256
    if N in (248, 504):
        assert prep.config(N)["tile_n"] == 256
    B, bias = _ints((K, N), N), _ints((M,), 3)
    want = (dense.float() @ B.float()).half()
    assert torch.equal(prep.spmm(B), want)
    assert torch.equal(prep.spmm(B, bias=bias, layout=capi.VNM_LAYOUT_NM), (want + bias[:, None]).T)
    assert torch.equal(prep.spmm_nk(B.T.contiguous(), bias=bias), (want + bias[:, None]).T)
    assert torch.equal(prep.spmm_nk(B.T.contiguous(), layout=capi.VNM_LAYOUT_MN), want)
    assert prep.device_status() == 0


# SM pairs: fewer k-tiles than the rings hold (three with 512 rows a tile, four with 256), as many, and more; one tile a cluster and several. The
# slots of the last round of the rings are not reported free, all others are.
@pytest.mark.parametrize("ktiles", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("tiles", [1, 2])
@pytest.mark.parametrize("rows", [3, 4])
def test_pair_kernel_ends_in_any_round_of_its_rings(rows, tiles, ktiles):
    import torch
    from venom_b200 import capi
    from venom_b200.synth import random_vnm_dense_cuda
    pairs = torch.cuda.get_device_properties(0).multi_processor_count // 2
    tile_m = 256 if rows == 3 else 512
    M, K, V, m, N = tile_m * (3 if tiles == 1 else pairs + 2), 128 * ktiles - 64, 32, 8, 216
    dense, cols = random_vnm_dense_cuda(M, K, V, m, seed=M + K)
    dense = torch.sign(dense) * torch.ceil(dense.abs() * 3)
    values, meta, bad = capi.compress(dense, cols, V, m)
    assert bad == 0
    prep = capi.Prepared(values, meta, cols, M, K, V, m, strategy=capi.STRATEGY_DENSE_B)
    prep.set_pair_mode(rows)
    assert prep.config(N)["tile_m"] == tile_m
    B = _ints((K, N), N)
    want = (dense.float() @ B.float()).half()
    for _ in range(20):      # launches of one shape behind one another, each beside the end of the one ahead
        out = prep.spmm(B)
        out_nk = prep.spmm_nk(B.T.contiguous())
    assert torch.equal(out, want) and torch.equal(out_nk, want.T)
    assert prep.device_status() == 0


# Several destinations: the last tile is staged in the operand rings, in slots that its last k-tile (any of them) was read from.
@pytest.mark.parametrize("ktiles", [1, 2, 3, 4])
@pytest.mark.parametrize("tiles", [1, 2])
@pytest.mark.parametrize("rows", [3, 4])
def test_last_tile_staged_in_the_rings(rows, tiles, ktiles):
    import torch
    from venom_b200 import capi
    pairs = torch.cuda.get_device_properties(0).multi_processor_count // 2
    M, K, V, m = 1024, 128 * ktiles, 64, 8
    N = 240 * 2 if tiles == 1 else 240 * pairs
    d, _, _, _, prep = _operand(M, K, V, m, capi.STRATEGY_DENSE_B, seed=K)
    prep.set_pair_mode(rows)
    B, bias = _ints((K, N), N), _ints((M,), 3)
    want = (d @ B.float()).half()
    for _ in range(10):
        outs = [torch.zeros((M, N), dtype=torch.float16, device="cuda") for _ in range(2)]
        outs_nm = [torch.zeros((N, M), dtype=torch.float16, device="cuda") for _ in range(2)]
        prep.spmm_multi(B, outs)
        prep.spmm_multi(B, outs_nm, bias=bias, layout=capi.VNM_LAYOUT_NM)
        assert all(torch.equal(o, want) for o in outs) and all(torch.equal(o, (want + bias[:, None]).T) for o in outs_nm)
    assert prep.device_status() == 0


# Gather kernel: a last wave of at most half of the SMs has its tiles cut in two, a fuller one has not.  Column tiles that end inside
# the first and the second half; more tiles than one a SM, so that whole and half tiles follow one another on it; five k-tiles a tile or more, the
# last one ragged, so that the rings go round and half-filled stages take the slots of whole ones.
@pytest.mark.parametrize("N", [96, 200, 256 + 72])
@pytest.mark.parametrize("rest", ["few", "one", "half", "more"])
@pytest.mark.parametrize("cfg", [(128, 16), (64, 16), (32, 8)])
def test_last_tiles_cut_in_two(cfg, rest, N):
    import torch
    from venom_b200 import capi
    from venom_b200.synth import random_vnm_dense_cuda
    V, m = cfg
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    bn = {128: 256, 64: 128, 32: 64}[V]
    ntiles = -(-N // bn)
    want_tiles = {"few": 5, "one": sms + 1, "half": sms + sms // 2, "more": sms + sms // 2 + 3}[rest]
    M, K = 128 * -(-want_tiles // ntiles), 32 * m * 4 + 320
    dense, cols = random_vnm_dense_cuda(M, K, V, m, seed=M + N)
    dense = torch.sign(dense) * torch.ceil(dense.abs() * 3)
    values, meta, bad = capi.compress(dense, cols, V, m)
    assert bad == 0
    prep = capi.Prepared(values, meta, cols, M, K, V, m, strategy=capi.STRATEGY_GATHER)
    prep.set_pair_mode(3)   # not the kernel for few tiles
    tiles = M // 128 * ntiles
    cut = V != 32 and 0 < tiles % sms <= sms // 2
    assert cut == (V != 32 and rest != "more")
    assert prep.config(N)["grid"] == min(sms, tiles + (tiles % sms if cut else 0))
    B, bias = _ints((K, N), N), _ints((M,), 3)
    want = (dense.float() @ B.float()).half()
    outs = [torch.zeros((N, M), dtype=torch.float16, device="cuda") for _ in range(2)]
    prep.spmm_multi(B, outs, bias=bias, layout=capi.VNM_LAYOUT_NM)
    assert all(torch.equal(o, (want + bias[:, None]).T) for o in outs)
    for mode in (0, 2):     # stores from tensor memory, through shared memory
        prep.set_epilogue(mode)
        assert torch.equal(prep.spmm(B), want)
        assert torch.equal(prep.spmm(B, bias=bias, layout=capi.VNM_LAYOUT_NM), (want + bias[:, None]).T)
    assert prep.device_status() == 0


# m = 4 in gather form (every row of B): the kernel that was measured to be the faster one by more than a tenth; results where the two meet.
@pytest.mark.parametrize("cfg", [(4096, 4096, 128, 16384, "large"), (1024, 4096, 128, 4096, "large"), (4096, 512, 128, 2048, "large"), (2048, 12288, 128, 2048, "large"),
                                 (4096, 512, 64, 4096, "large"), (2048, 1024, 64, 8192, "large"), (1024, 1024, 32, 4096, "large"), (4096, 1024, 32, 520, "large"),
                                 (1024, 4096, 128, 2048, "few"), (4096, 4096, 128, 520, "few"), (512, 2048, 64, 2048, "few"), (1024, 4096, 32, 256, "few")])
def test_kernel_of_an_operand_of_every_row(cfg):
    import torch
    from venom_b200 import capi
    from venom_b200.synth import random_vnm_dense_cuda
    M, K, V, N, want = cfg
    dense, cols = random_vnm_dense_cuda(M, K, V, 4, seed=M + K)
    dense = torch.sign(dense) * torch.ceil(dense.abs() * 3)
    values, meta, bad = capi.compress(dense, cols, V, 4)
    assert bad == 0
    prep = capi.Prepared(values, meta, cols, M, K, V, 4, strategy=capi.STRATEGY_GATHER)
    assert (prep.config(N)["stages"] == 16) == (want == "large")
    B = _ints((K, N), N)
    assert torch.equal(prep.spmm(B), (dense.float() @ B.float()).half())
    assert prep.device_status() == 0


# SM pairs: row tiles that do not fill the last pair (or group of four), fewer columns than a box, ragged columns.
@pytest.mark.parametrize("rows", [3, 4])
@pytest.mark.parametrize("cfg", [(128, 512, 128, 8, 248), (384, 264, 64, 8, 480), (640, 1152, 32, 16, 1000), (896, 1024, 64, 8, 72)])
def test_odd_row_tiles_on_sm_pairs(cfg, rows):
    import torch
    from venom_b200 import capi
    M, K, V, m, N = cfg
    d, _, _, _, prep = _operand(M, K, V, m, capi.STRATEGY_DENSE_B, seed=M + N)
    prep.set_pair_mode(rows)
    B = _ints((K, N), N)
    want = (d @ B.float()).half()
    assert torch.equal(prep.spmm(B), want)
    assert torch.equal(prep.spmm(B, layout=capi.VNM_LAYOUT_NM), want.T)
    assert torch.equal(prep.spmm_nk(B.T.contiguous()), want.T)
    assert prep.device_status() == 0


# A layer reads its input as it lies ([tokens, features], any leading dimensions) in either form, and goes through the copying
# path for one that it cannot read in place; edits of the arrays are seen by the next call.
@pytest.mark.parametrize("cfg", [(256, 512, 128, 16, (3, 8)), (96, 520, 32, 8, (1368,)), (1024, 1024, 64, 8, (2, 4, 8)), (384, 640, 128, 16, (1000,)), (128, 120, 64, 10, (8,))])
def test_layer_reads_its_input_in_place(cfg):
    import torch
    from venom_b200.nmv import SrnmSpmm
    M, K, V, m, lead = cfg
    d, values, meta, c, _ = _operand(M, K, V, m, None, seed=M + K)
    layer = SrnmSpmm(torch.nn.Linear(K, M).half().cuda(), 2, m, V)
    layer.values.data.copy_(values.reshape(-1))
    layer.metadata, layer.columns = meta, c
    layer.bias.data.copy_(_ints((M,), 5))
    x = _ints(lead + (K,), 7)
    want = ((x.reshape(-1, K).float() @ d.T).half() + layer.bias).reshape(lead + (M,))
    assert torch.equal(layer(x), want)
    wide = torch.zeros(lead + (K + 8,), dtype=torch.float16, device="cuda")
    wide[..., 8:] = x
    assert torch.equal(layer(wide[..., 8:]), want)
    layer.values.data.mul_(2)
    layer.values.add_(0)                       # an in-place edit that autograd counts
    assert torch.equal(layer(x), (((want - layer.bias).float() * 2).half() + layer.bias))


def test_product_reports_errors_as_before():
    import torch
    from venom_b200 import capi
    _, _, _, _, prep = _operand(128, 256, 64, 8, None, seed=1)
    for bad in (_ints((256, 12), 1), _ints((128, 16), 1), _ints((256, 16), 1).float(), _ints((16, 256), 1).T, _ints((256, 16), 1).cpu()):
        with pytest.raises(capi.VenomError):
            prep.spmm(bad)
    with pytest.raises(capi.VenomError):
        prep.spmm(_ints((256, 16), 1), bias=_ints((128,), 1))            # a bias needs layout NM
    prep.close()
    with pytest.raises(capi.VenomError):
        prep.spmm(_ints((256, 16), 1))


# Decompressor: pieces of 8 and of 4 columns, a last piece block that ends inside a row, a ragged last group and last tile, rows
# aligned to 8 bytes only.
@pytest.mark.parametrize("cfg", [(64, 96, 32, 16), (32, 1000, 32, 8), (32, 1032, 32, 16), (64, 100, 32, 20), (32, 84, 32, 12), (32, 4104, 32, 24), (128, 2304, 64, 32), (64, 4100, 64, 4)])
def test_decompress_pieces(cfg):
    import torch
    from venom_b200 import capi
    from venom_b200.synth import random_vnm_dense
    M, K, V, m = cfg
    dense, cols, _ = random_vnm_dense(M, K, V, m, seed=K)
    d = torch.from_numpy(dense).cuda()
    c = torch.from_numpy(cols.view(np.int32)).cuda()
    values, meta, bad = capi.compress(d, c, V, m)
    assert bad == 0
    assert torch.equal(capi.decompress(values, meta, c, M, K, V, m), d)


# A [tokens, features] activation of more rows than 65535 blocks of 64, which the gather form transposes first.
def test_gather_form_takes_millions_of_tokens():
    import torch
    from venom_b200 import capi
    M, K, V, m = 32, 32, 32, 16
    N = 65535 * 64 + 8
    d, _, _, _, prep = _operand(M, K, V, m, capi.STRATEGY_GATHER, seed=9)
    x = _ints((N, K), 4)
    out = torch.empty((N, M), dtype=torch.float16, device="cuda")
    workspace = torch.empty((K, N), dtype=torch.float16, device="cuda")
    rc = capi.lib().vnm_spmm_f16_nk_ws(prep._h, x.data_ptr(), K, N, None, out.data_ptr(), M, capi.VNM_LAYOUT_NM, workspace.data_ptr(), capi._stream())
    assert rc == 0, capi.lib().vnm_last_error_string()
    assert torch.equal(out, (x.float() @ d.T).half())
    assert prep.device_status() == 0


def _two_forms(M, K, V, m):
    """Token counts for which a layer wants its weight in different forms."""
    import ctypes as C
    from venom_b200 import capi
    form, first = C.c_int(), {}
    for n in (4096, 2048, 1024, 512, 256, 128, 64, 32, 16, 8):
        assert capi.lib().vnm_choose_form(M, K, V, 2, m, n, 1, C.byref(form)) == 0
        first.setdefault(form.value, n)
    assert len(first) == 2, first
    return first[capi.STRATEGY_GATHER], first[capi.STRATEGY_DENSE_B]


# Token counts that are no multiple of 16: the form that was measured to be the faster one by more than a tenth, where a product is mostly its start
# (few tokens, gather form) and where the gathers of unaligned rows count (dense-B form); and a multiple of 16 beside each.
@pytest.mark.parametrize("cfg", [(8192, 2048, 128, 16, 8, "gather"), (8192, 2048, 128, 16, 24, "gather"), (8192, 2048, 128, 16, 56, "gather"), (1024, 4096, 128, 16, 72, "gather"),
                                 (1024, 4096, 128, 16, 136, "gather"), (36864, 12288, 128, 16, 8, "gather"), (36864, 12288, 128, 16, 40, "gather"), (12288, 4096, 128, 32, 104, "gather"),
                                 (4096, 4096, 64, 32, 1368, "gather"), (12288, 12288, 128, 16, 1000, "gather"), (12288, 4096, 128, 8, 8, "dense_b"), (12288, 4096, 128, 8, 56, "dense_b"),
                                 (8192, 12288, 32, 8, 8, "dense_b"), (8192, 12288, 32, 8, 24, "dense_b"), (12288, 12288, 64, 16, 520, "dense_b"), (6912, 3784, 128, 8, 8152, "dense_b"),
                                 (8192, 2048, 128, 16, 32, "gather"), (36864, 12288, 128, 16, 48, "gather"), (8192, 12288, 32, 8, 64, "dense_b")])
def test_form_of_a_layer_at_odd_token_counts(cfg):
    import ctypes as C
    from venom_b200 import capi
    M, K, V, m, N, want = cfg
    form = C.c_int()
    assert capi.lib().vnm_choose_form(M, K, V, 2, m, N, 1, C.byref(form)) == 0
    assert form.value == (capi.STRATEGY_GATHER if want == "gather" else capi.STRATEGY_DENSE_B)


def _layer_of(values, meta, c, M, K, V, m):
    import torch
    from venom_b200.nmv import SrnmSpmm
    layer = SrnmSpmm(torch.nn.Linear(K, M, bias=False).half().cuda(), 2, m, V)
    layer.values = torch.nn.Parameter(values.reshape(-1), requires_grad=False)
    layer.metadata, layer.columns = meta, c
    return layer


# A graph captured at a token count that wants a form the weight is not held in yet: it uses the other one, and calls outside
# of it, before and after its replays, are not disturbed.
@pytest.mark.parametrize("warm", [0, 1])
def test_layer_captured_before_its_form_exists(warm):
    import torch
    M, K, V, m = 1024, 4096, 128, 16
    ns = _two_forms(M, K, V, m)
    d, values, meta, c, _ = _operand(M, K, V, m, None, seed=21)
    layer = _layer_of(values, meta, c, M, K, V, m)
    xs = [_ints((n, K), n) for n in ns]
    want = [(x.float() @ d.T).half() for x in xs]
    assert torch.equal(layer(xs[warm]), want[warm])
    x = xs[1 - warm].clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = layer(x)
    assert torch.equal(layer(xs[1 - warm]), want[1 - warm])
    graph.replay()
    assert torch.equal(y, want[1 - warm])
    x.mul_(2)
    graph.replay()
    assert torch.equal(y, (xs[1 - warm].float() * 2 @ d.T).half())
    assert torch.equal(layer(xs[warm]), want[warm])


# vnm_prepare on a stream that is being captured: refused in the global mode, allowed in the relaxed one, where the copy is filled by
# every replay and outlives the graph.
def test_prepare_under_capture():
    import ctypes as C
    import torch
    from venom_b200 import capi
    M, K, V, m, N = 256, 512, 64, 8, 64
    d, values, meta, c, _ = _operand(M, K, V, m, None, seed=5)
    B = _ints((K, N), 2)
    want = (d @ B.float()).half()
    out = torch.zeros((M, N), dtype=torch.float16, device="cuda")
    torch.cuda.synchronize()
    rt, L = C.CDLL("libcudart.so.12"), capi.lib()
    s = C.c_void_p(torch.cuda.Stream().cuda_stream)
    graph, run, h = C.c_void_p(), C.c_void_p(), C.c_void_p()
    assert rt.cudaStreamBeginCapture(s, 0) == 0
    assert L.vnm_prepare(values.data_ptr(), meta.data_ptr(), c.data_ptr(), M, K, V, 2, m, C.byref(h), s) == 2
    assert rt.cudaStreamEndCapture(s, C.byref(graph)) != 0
    rt.cudaGetLastError()
    assert rt.cudaStreamBeginCapture(s, 2) == 0
    assert L.vnm_prepare(values.data_ptr(), meta.data_ptr(), c.data_ptr(), M, K, V, 2, m, C.byref(h), s) == 0
    assert L.vnm_spmm_f16(h, B.data_ptr(), N, N, None, out.data_ptr(), N, 0, s) == 0
    assert rt.cudaStreamEndCapture(s, C.byref(graph)) == 0
    assert rt.cudaGraphInstantiate(C.byref(run), graph, C.c_ulonglong(0)) == 0
    for _ in range(2):
        out.zero_()
        torch.cuda.synchronize()
        assert rt.cudaGraphLaunch(run, s) == 0 and rt.cudaStreamSynchronize(s) == 0
        assert torch.equal(out, want)
    assert rt.cudaGraphExecDestroy(run) == 0 and rt.cudaGraphDestroy(graph) == 0
    out.zero_()
    torch.cuda.synchronize()
    assert L.vnm_spmm_f16(h, B.data_ptr(), N, N, None, out.data_ptr(), N, 0, None) == 0
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    assert L.vnm_destroy(h) == 0


# An operand that is still being re-packed behind other work of one stream: a product on another stream, plain or captured, waits.
@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("form", ["gather", "dense_b"])
@pytest.mark.parametrize("lies", ["kn", "nk"])     # nk in gather form: a transpose, and a product that starts beside it
def test_product_waits_for_an_operand_packed_on_another_stream(form, captured, lies):
    import torch
    from venom_b200 import capi
    M, K, V, m, N = 256, 1024, 64, 8, 64
    d, values, meta, c, _ = _operand(M, K, V, m, None, seed=13)
    B = _ints((K, N), 6)
    Bt = B.T.contiguous()
    want = (d @ B.float()).half()
    workspace, out = torch.empty((K, N), dtype=torch.float16, device="cuda"), torch.zeros((M, N), dtype=torch.float16, device="cuda")
    busy, other = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()

    def product():
        if lies == "kn":
            return prep.spmm(B, out=out)
        assert capi.lib().vnm_spmm_f16_nk_ws(prep._h, Bt.data_ptr(), K, N, None, out.data_ptr(), N, capi.VNM_LAYOUT_MN, workspace.data_ptr(), capi._stream()) == 0
    with torch.cuda.stream(busy):
        torch.cuda._sleep(50_000_000)
        prep = capi.Prepared(values, meta, c, M, K, V, m, strategy=capi.STRATEGY_GATHER if form == "gather" else capi.STRATEGY_DENSE_B)
    with torch.cuda.stream(other):
        if captured:
            graph = torch.cuda.CUDAGraph()
            graph.capture_begin()            # not torch.cuda.graph, which waits for the device first
            product()
            graph.capture_end()
            graph.replay()
        else:
            product()
    other.synchronize()
    assert torch.equal(out, want)
    assert prep.device_status() == 0


def test_layer_called_on_two_streams():
    import torch
    M, K, V, m = 1024, 4096, 128, 16
    d, values, meta, c, _ = _operand(M, K, V, m, None, seed=17)
    layer = _layer_of(values, meta, c, M, K, V, m)
    xs = [_ints((n, K), n) for n in _two_forms(M, K, V, m)]
    want = [(x.float() @ d.T).half() for x in xs]
    busy = torch.cuda.Stream()
    torch.cuda.synchronize()
    for x, w in zip(xs, want):
        with torch.cuda.stream(busy):
            torch.cuda._sleep(50_000_000)
            a = layer(x)             # re-packs the weight into the form that this token count wants
        assert torch.equal(layer(x), w)
        busy.synchronize()
        assert torch.equal(a, w)


# A layer holds its weight in each form that a token count has wanted, or in the one that it was given.
@pytest.mark.parametrize("form", [0, 1, 2])
def test_layer_holds_the_form_it_is_given(form):
    import torch
    from venom_b200 import spatha_module
    ext = spatha_module()
    M, K, V, m = 1024, 4096, 128, 16
    d, values, meta, c, _ = _operand(M, K, V, m, None, seed=23)
    layer = _layer_of(values, meta, c, M, K, V, m)
    layer.form = form
    ext.clear_cache()
    for n in _two_forms(M, K, V, m):
        x = _ints((n, K), n)
        want = (x.float() @ d.T).half()
        assert torch.equal(layer(x), want)
        wide = torch.zeros((n, K + 8), dtype=torch.float16, device="cuda")
        wide[:, :K] = x
        assert torch.equal(layer(wide[:, :K]), want)                  # through spmm(), a transposed view
        b = x.T.contiguous()
        assert torch.equal(ext.spmm(meta, c, layer.values, b, None, M, K, n, V, 2, m, values.numel(), 0, 32, 4, form), want)
    assert ext.cache_size() == 1 and ext.cached_copies() == (2 if form == 0 else 1)
    with pytest.raises(RuntimeError, match="form"):
        ext.linear(x, meta, c, layer.values, None, M, K, V, 2, m, 3)


def test_layer_without_a_dense_b_form():
    import torch
    M, K, V, m = 128, 280, 64, 10
    d, values, meta, c, _ = _operand(M, K, V, m, None, seed=3)
    layer = _layer_of(values, meta, c, M, K, V, m)
    layer.form = 2
    x = _ints((16, K), 1)
    assert torch.equal(layer(x), (x.float() @ d.T).half())


# A form that does not fit the device (193 GB) is an error of its own call only.
def test_form_that_does_not_fit():
    import torch
    from venom_b200 import capi, spatha_module
    M, K, V, m, N = 262144, 655360, 128, 256, 8
    ksp, nv, nm, nc = capi.sizes(M, K, V, m)
    values = torch.zeros(nv, dtype=torch.float16, device="cuda")
    meta = torch.full((nm,), 0x44444444, dtype=torch.int32, device="cuda")
    cols = torch.tensor([0, 1, 2, 3], dtype=torch.int32, device="cuda").repeat(nc // 4)
    x = torch.ones((N, K), dtype=torch.float16, device="cuda")
    for form in (2, 1, 2):
        call = lambda: spatha_module().linear(x, meta, cols, values, None, M, K, V, 2, m, form)
        if form == 2:
            with pytest.raises(RuntimeError, match="out of memory"):
                call()
        else:
            assert not call().any()
    assert torch.ones(4, device="cuda").sum().item() == 4             # no error left behind
    spatha_module().clear_cache()
