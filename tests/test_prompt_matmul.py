"""The two-SM prompt matmul (csrc/gemm_pair.cu): edges of its tiles against float64 on the dequantised weights, plain, with the fused
MLP's activation, and over the experts of a mixture (csrc/experts.cu).

Bounds.  Weights are rounded once to the activation dtype, so a product's error is at most u * sum|x w| with u = 2^-11 (fp16) or
(1 + 2^-8)(1 + 2^-11) - 1 (bf16 has eight significant bits; its expansion goes through fp16).  The 32-bit sum: a step of the tensor cores aligns its 16 products
and the accumulator to the largest of them and drops what falls below 2^-23 of it, 17 terms a step, so ACC = 2^-18 * sum|x w| covers
two steps' worth at full size (the later ones' drops are relative to sums that rarely reach sum|x w|).  A 16-bit result adds u * |y|."""
import pytest
import torch

pytestmark = pytest.mark.gpu

U = {torch.float16: 2.0 ** -11, torch.bfloat16: (1 + 2.0 ** -8) * (1 + 2.0 ** -11) - 1}
ACC = 2.0 ** -18


@pytest.fixture(scope="module")
def lbl(native_lib, cuda_device):
    from ipex_llm_b200.transformers import low_bit_linear
    yield low_bit_linear
    assert not native_lib.lowbit_gemm_wait_expired()


def weights(lbl, dev, seed, n, k, qtype, count=1):
    g = torch.Generator(device=dev).manual_seed(seed)
    out = []
    for _ in range(count):
        w = torch.empty(n, k, device=dev).normal_(0.0, 0.02, generator=g)
        qt = lbl.ggml_tensor_qtype[qtype]
        tiled = lbl.FP4Params(w, qtype=qt).to(dev).data
        out.append((tiled, lbl.dequantize_device_layout(tiled, (n, k), qt).double()))
    return out, qt


def acts(dev, seed, m, k, dtype):
    return torch.empty(m, k, device=dev).normal_(generator=torch.Generator(device=dev).manual_seed(seed)).to(dtype)


def product(x, w, u):
    """x w^T in 64 bits and the bound of a 32-bit sum over weights rounded to u"""
    return x @ w.T, (u + ACC) * (x.abs() @ w.abs().T)


# one row over a 16- / 128- / 256-token tile, a lone feature pair and an odd one, one k-block, K splits and several rounds of tiles
@pytest.mark.parametrize("m,n,k", [(65, 128, 64), (96, 384, 128), (129, 256, 4096), (256, 640, 192), (257, 128, 2048), (513, 2176, 320),
                                   (100, 4096, 1024), (1037, 19072, 64)])
@pytest.mark.parametrize("qtype,dtype", [("sym_int4", torch.float16), ("asym_int4", torch.bfloat16), ("nf4", torch.float16), ("fp8_e4m3", torch.bfloat16),
                                         ("fp8_e5m2", torch.float16), ("fp6", torch.bfloat16)])
def test_prompt_matmul_edges(lbl, cuda_device, qtype, dtype, m, n, k):
    [(w, wd)], qt = weights(lbl, cuda_device, m + n, n, k, qtype)
    x = acts(cuda_device, k, m, k, dtype)
    want, bound = product(x.double(), wd, U[dtype])
    y32 = lbl.lowbit_matmul(x, w, (n, k), qt, out_dtype=torch.float32)
    assert bool(((y32.double() - want).abs() <= bound + 1e-30).all())
    y = lbl.lowbit_matmul(x, w, (n, k), qt)
    assert torch.equal(y, y32.to(dtype))
    # bias and accumulation are added in 32 bits; a result that starts off a 16-byte boundary is written all the same
    bias = acts(cuda_device, 5, 1, n, dtype)[0]
    out = torch.empty(m * n + 1, dtype=dtype, device=cuda_device)[1:].view(m, n)
    out.copy_(acts(cuda_device, 6, m, n, dtype))
    old = out.double()
    lbl.lowbit_matmul(x, w, (n, k), qt, out=out, bias=bias, accumulate=True)
    # two 32-bit additions (2^-24 of each partial result), then one rounding to 16 bits: half a unit in the last place, at least half
    # of the format's smallest step
    base, terms = y32.double() + bias.double() + old, y32.double().abs() + bias.double().abs() + old.abs()
    u16, tiny = (2.0 ** -11, 2.0 ** -25) if dtype == torch.float16 else (2.0 ** -8, 0.0)
    assert bool(((out.double() - base).abs() <= 2.0 ** -22 * terms + u16 * base.abs() + tiny).all())


def test_prompt_matmul_without_scratch_for_partial_sums(lbl, native_lib, cuda_device):
    """a workspace too small for the K split the shape would take: the same product from whole K ranges"""
    m, n, k = 100, 256, 4096
    [(w, wd)], qt = weights(lbl, cuda_device, 3, n, k, "sym_int4")
    x = acts(cuda_device, 4, m, k, torch.float16)
    assert native_lib.lowbit_matmul_workspace_size(n, k, m, native_lib.DT_F16) > 256
    y, ws = torch.empty(m, n, dtype=torch.float32, device=cuda_device), torch.empty(256, dtype=torch.uint8, device=cuda_device)
    native_lib.lowbit_matmul_cuda(w.data_ptr(), qt, n, k, x.data_ptr(), native_lib.DT_F16, m, y.data_ptr(), native_lib.DT_F32, None, False,
                                  ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
    want, bound = product(x.double(), wd, U[torch.float16])
    assert bool(((y.double() - want).abs() <= bound).all())


def gated(x, wg, wu, u, act):
    """act(x wg^T) * (x wu^T) and its bound: both activations' slopes are below 1.13"""
    f = torch.nn.functional.silu if act == 0 else torch.nn.functional.gelu
    g, bg = product(x, wg, u)
    p, bp = product(x, wu, u)
    a = f(g)
    return a * p, 1.13 * bg * (p.abs() + bp) + a.abs() * bp + 1e-6 * (a * p).abs() + 1e-6 * p.abs()


@pytest.mark.parametrize("m,n,k", [(65, 128, 128), (257, 384, 64), (600, 1408, 512)])
@pytest.mark.parametrize("qtype,dtype,act", [("sym_int4", torch.bfloat16, 0), ("asym_int4", torch.float16, 1), ("nf4", torch.bfloat16, 0), ("fp6", torch.float16, 0),
                                             ("fp8_e4m3", torch.float16, 1)])
def test_prompt_mlp_edges(lbl, cuda_device, qtype, dtype, act, m, n, k):
    ((wg, g), (wu, p)), qt = weights(lbl, cuda_device, m, n, k, qtype, 2)
    x = acts(cuda_device, n, m, k, dtype)
    want, bound = gated(x.double(), g, p, U[dtype], act)
    y32 = lbl.mlp_forward(x, wg, wu, m, k, n, act, qt, out=torch.empty(m, n, dtype=torch.float32, device=cuda_device))
    assert bool(((y32.double() - want).abs() <= bound).all())
    assert torch.equal(lbl.mlp_forward(x, wg, wu, m, k, n, act, qt), y32.to(dtype))
    odd = torch.empty(m * n + 1, dtype=dtype, device=cuda_device)[1:].view(m, n)                  # not on a 16-byte boundary
    assert torch.equal(lbl.mlp_forward(x, wg, wu, m, k, n, act, qt, out=odd), y32.to(dtype))


@pytest.mark.parametrize("rows,experts,top_k,skew", [(1, 4, 2, False), (2, 3, 1, False), (40, 16, 4, False), (300, 4, 2, True), (700, 40, 2, False), (600, 2, 2, False)])
@pytest.mark.parametrize("qtype,dtype", [("sym_int4", torch.bfloat16), ("fp8_e4m3", torch.float16)])
def test_experts_of_many_tokens(lbl, cuda_device, qtype, dtype, rows, experts, top_k, skew):
    """unused experts, experts of one row, of more rows than a tile, every token on one expert; ids outside the table add nothing"""
    H, I = 256, 384
    ws, qt = weights(lbl, cuda_device, rows, I, H, qtype, 2 * experts)
    downs, _ = weights(lbl, cuda_device, rows + 1, H, I, qtype, experts)
    table = lambda ts: torch.tensor([t.data_ptr() for t, _ in ts], dtype=torch.int64, device=cuda_device)         # noqa: E731
    gen = torch.Generator(device=cuda_device).manual_seed(rows)
    ids = torch.randint(0, experts, (rows, top_k), generator=gen, device=cuda_device)
    if skew:
        ids[:, 0] = experts - 1
        ids[5, 1] = experts + 7
        ids[6, 0] = -1
    wgt = torch.rand(rows, top_k, generator=gen, device=cuda_device)
    x = acts(cuda_device, 1, rows, H, dtype)
    got = lbl.moe_forward_tokens(x, ids if skew else ids.int(), wgt, table(ws[:experts]), table(ws[experts:]), table(downs), H, I, qt)
    want = torch.zeros(rows, H, dtype=torch.float64, device=cuda_device)
    bound, u = torch.zeros_like(want), U[dtype]
    for e in range(experts):
        r, s = torch.where(ids == e)
        if not len(r):
            continue
        h, bh = gated(x[r].double(), ws[e][1], ws[experts + e][1], u, 0)
        bh = bh + u * (h.abs() + bh)                                          # the hidden rows are rounded to the activation dtype
        y, by = product(h, downs[e][1], u)
        by = by + (1 + u) * bh @ downs[e][1].abs().T
        by = by + u * (y.abs() + by)
        want.index_add_(0, r, y * wgt[r, s, None].double())
        bound.index_add_(0, r, by * wgt[r, s, None].double())
    bound = bound + u * want.abs() + 1e-7                                     # fp16's smallest step
    assert bool(((got.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("qtype,dtype", [("asym_int4", torch.float16), ("sym_int4", torch.bfloat16), ("nf4", torch.float16), ("fp8_e4m3", torch.bfloat16)])
def test_prompt_matmul_rings_over_many_rounds(lbl, cuda_device, qtype, dtype):
    """several tiles per cluster and 32-bit results, whose slow epilogue stalls the MMAs until every ring is full: each slot is refilled
    only after its readers have used what they loaded"""
    m, n, k = 2048, 14336, 1024
    [(w, wd)], qt = weights(lbl, cuda_device, 8, n, k, qtype)
    x = acts(cuda_device, 9, m, k, dtype)
    want, bound = product(x.double(), wd, U[dtype])
    first = lbl.lowbit_matmul(x, w, (n, k), qt, out_dtype=torch.float32)
    assert bool(((first.double() - want).abs() <= bound).all())
    for _ in range(8):
        assert torch.equal(lbl.lowbit_matmul(x, w, (n, k), qt, out_dtype=torch.float32), first)


@pytest.mark.parametrize("m,n,k", [(33, 128, 64), (64, 384, 128), (65, 256, 4096), (127, 640, 192), (200, 4096, 1024), (300, 2176, 320), (513, 19072, 64)])
@pytest.mark.parametrize("qtype", ["sym_int4", "fp8_e4m3", "fp8_e5m2", "fp6", "asym_int4", "nf4"])
def test_prompt_matmul_fp32_keeps_its_contract(lbl, native_lib, cuda_device, qtype, m, n, k):
    """32-bit activations to 2^-24 of sum|x w| (the bound of the GEMV's tests: 2e-6; nf4's table is held to 2^-17), no further off than the
    GEMV's passes of 32 rows, which a workspace of their size still gets"""
    [(w, wd)], qt = weights(lbl, cuda_device, m + n, n, k, qtype)
    x = acts(cuda_device, k, m, k, torch.float32)
    mag = x.double().abs() @ wd.abs().T
    want, tol = x.double() @ wd.T, (2e-6 if qtype != "nf4" else 2.0 ** -17 + 2e-6)
    y = lbl.lowbit_matmul(x, w, (n, k), qt)
    assert y.dtype == torch.float32 and bool(((y.double() - want).abs() <= tol * mag).all())
    small = native_lib.lowbit_matmul_workspace_size(n, k, 32, native_lib.DT_F32)
    ws, passes = torch.empty(small, dtype=torch.uint8, device=cuda_device), torch.empty_like(y)
    native_lib.lowbit_matmul_cuda(w.data_ptr(), qt, n, k, x.data_ptr(), native_lib.DT_F32, m, passes.data_ptr(), native_lib.DT_F32, None, False,
                                  ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
    assert bool(((passes.double() - want).abs() <= tol * mag).all())
    assert float((y.double() - want).norm()) <= 1.05 * float((passes.double() - want).norm())
    bias, out = acts(cuda_device, 5, 1, n, torch.float32)[0], torch.empty(m * n + 1, device=cuda_device)[1:].view(m, n)
    out.copy_(acts(cuda_device, 6, m, n, torch.float32))
    base = y.double() + bias.double() + out.double()
    terms = y.abs() + bias.abs() + out.abs()
    lbl.lowbit_matmul(x, w, (n, k), qt, out=out, bias=bias, accumulate=True)
    assert bool(((out.double() - base).abs() <= 2.0 ** -22 * terms.double() + 2e-6 * mag).all())
    # a strided or misaligned view of the activations, and 16-bit results, which keep to the GEMV
    assert torch.equal(lbl.lowbit_matmul(torch.cat([x, x], 1)[:, :k], w, (n, k), qt), y)
    half = lbl.lowbit_matmul(x, w, (n, k), qt, out_dtype=torch.float16)
    assert bool(((half.double() - want).abs() <= tol * mag + 2.0 ** -11 * want.abs() + 2.0 ** -25).all())


@pytest.mark.parametrize("m,n,k", [(48, 19200, 384), (64, 9600, 832), (65, 128, 64), (128, 2176, 1088), (129, 9600, 256), (385, 4736, 448), (257, 9728, 832),
                                   (512, 9728, 640)])
@pytest.mark.parametrize("qtype", ["sym_int4", "fp8_e4m3", "fp8_e5m2", "fp6"])
def test_prompt_matmul_fp32_tiles(lbl, native_lib, cuda_device, qtype, m, n, k):
    """tiles of 64 and of 128 tokens: the line between them, several rounds of units of either through the rings, k-blocks no multiple of the rings"""
    test_prompt_matmul_fp32_keeps_its_contract(lbl, native_lib, cuda_device, qtype, m, n, k)


@pytest.mark.parametrize("m,n,k", [(33, 9600, 192), (48, 19200, 384), (65, 128, 64), (97, 4736, 1088), (129, 9600, 256), (385, 4736, 448), (512, 9728, 640)])
def test_prompt_matmul_fp32_with_minima(lbl, native_lib, cuda_device, m, n, k):
    """the activations' sums beside the codes: both tiles' remainders, more than one unit per cluster, K ranges of an odd number of blocks;
    activations away from zero, where the minima are most of the result, to the same bound; a workspace without room for the sums"""
    test_prompt_matmul_fp32_keeps_its_contract(lbl, native_lib, cuda_device, "asym_int4", m, n, k)
    [(w, wd)], qt = weights(lbl, cuda_device, m + n, n, k, "asym_int4")
    x = acts(cuda_device, k, m, k, torch.float32) + 3
    want, mag = x.double() @ wd.T, x.double().abs() @ wd.abs().T
    size = native_lib.lowbit_matmul_workspace_size(n, k, m, native_lib.DT_F32)
    outs = []
    for room in (size, 256 * ((3 * m * k * 2 + 255) // 256)):                  # the second holds the planes alone
        ws, y = torch.full((room,), 255, dtype=torch.uint8, device=cuda_device), torch.empty(m, n, device=cuda_device)
        native_lib.lowbit_matmul_cuda(w.data_ptr(), qt, n, k, x.data_ptr(), native_lib.DT_F32, m, y.data_ptr(), native_lib.DT_F32, None, False,
                                      ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
        outs.append((y.double() - want).abs())
        assert bool((outs[-1] <= 2e-6 * mag).all())
    assert float(outs[0].norm()) <= 1.05 * float(outs[1].norm())


@pytest.mark.parametrize("qtype", ["sym_int4", "asym_int4", "nf4", "fp8_e4m3", "fp8_e5m2", "fp6"])
@pytest.mark.parametrize("m,n,k", [(33, 256, 192), (100, 1024, 2048)])
def test_mlp_fp32_in_a_workspace_without_sums(lbl, native_lib, cuda_device, qtype, m, n, k):
    """only asym_int4's minima need the activations' sums, and without room for them it runs in passes; less than that is refused"""
    [(gate, gd), (up, ud)], qt = weights(lbl, cuda_device, m, n, k, qtype, 2)
    x = acts(cuda_device, m, m, k, torch.float32)
    full = native_lib.lowbit_mlp_workspace_size(n, k, m, native_lib.DT_F32)
    room = full - 256 * ((k // 64 * ((m + 15) // 16 * 16) * 4 + 255) // 256)
    stream = torch.cuda.current_stream().cuda_stream

    def call(size):
        ws, y = torch.full((full,), 255, dtype=torch.uint8, device=cuda_device), torch.empty(m, n, device=cuda_device)
        native_lib.lowbit_mlp_cuda(gate.data_ptr(), up.data_ptr(), qt, n, k, x.data_ptr(), native_lib.DT_F32, m, y.data_ptr(), native_lib.DT_F32, 0,
                                   ws.data_ptr(), size, stream)
        assert bool((ws[size:] == 255).all())
        return y
    want, got = call(full), call(room)
    assert qtype == "asym_int4" or torch.equal(want, got)
    a, b = x.double() @ gd.T, x.double() @ ud.T
    mag = (x.double().abs() @ gd.abs().T) * b.abs() + (x.double().abs() @ ud.abs().T) * a.abs()
    for y in (want, got):                         # each product to 2e-6 of its magnitude, silu's slope at most 1.1
        assert bool(((y.double() - torch.nn.functional.silu(a) * b).abs() <= 3e-6 * mag + 1e-7).all())
    with pytest.raises(native_lib.LowBitNativeError, match="workspace too small"):
        call(room - 256)


@pytest.mark.parametrize("m,n,k", [(33, 9600, 192), (48, 19200, 832), (64, 1024, 8192), (65, 128, 64), (129, 9600, 256), (385, 4736, 448), (512, 9728, 1088)])
def test_prompt_matmul_fp32_through_the_table(lbl, native_lib, cuda_device, m, n, k):
    """nf4's two tiles per k-block: both tiles' remainders, rings that go round with two and with three expansion groups, the same bits each time"""
    test_prompt_matmul_fp32_keeps_its_contract(lbl, native_lib, cuda_device, "nf4", m, n, k)
    [(w, _)], qt = weights(lbl, cuda_device, 3, n, k, "nf4")
    x = acts(cuda_device, 4, m, k, torch.float32)
    first = lbl.lowbit_matmul(x, w, (n, k), qt)
    for _ in range(8):
        assert torch.equal(lbl.lowbit_matmul(x, w, (n, k), qt), first)


@pytest.mark.parametrize("qtype,dtype,m,n,k", [("sym_int4", torch.float16, 200, 4096, 4096), ("sym_int4", torch.float16, 500, 4096, 11008),
                                               ("sym_int4", torch.float16, 512, 4096, 11008), ("fp8_e4m3", torch.float16, 256, 4096, 4096),
                                               ("sym_int4", torch.bfloat16, 1500, 1024, 4096), ("nf4", torch.bfloat16, 512, 4096, 4096)])
def test_prompts_whose_k_range_stays_whole(lbl, native_lib, cuda_device, qtype, dtype, m, n, k):
    """a split is another order of the sums, which decode steps behind a prompt show: the same bits with and without room for partial sums"""
    p = lbl.FP4Params(torch.randn(n, k, device=cuda_device, generator=torch.Generator(device=cuda_device).manual_seed(k)) * 0.02,
                      qtype=lbl.ggml_tensor_qtype[qtype]).to(cuda_device)
    x = torch.randn(m, k, device=cuda_device, generator=torch.Generator(device=cuda_device).manual_seed(m)).to(dtype)
    room, dt = torch.empty(8 * m * n * 4, dtype=torch.uint8, device=cuda_device), lbl._TORCH_TO_DT[dtype]
    y = [torch.empty(m, n, dtype=dtype, device=cuda_device) for _ in range(2)]
    for out, size in zip(y, (room.numel(), 0)):
        native_lib.lowbit_matmul_cuda(p.data.data_ptr(), p.qtype, n, k, x.data_ptr(), dt, m, out.data_ptr(), dt, None, 0, room.data_ptr(), size,
                                      torch.cuda.current_stream().cuda_stream)
    assert torch.equal(*y)


@pytest.mark.parametrize("qtype,dtype", [("sym_int4", torch.float16), ("nf4", torch.bfloat16), ("fp8_e4m3", torch.float16)])
@pytest.mark.parametrize("n,k", [(1280, 1024), (14336, 384)])
def test_the_token_tile_changes_no_bit(lbl, native_lib, cuda_device, qtype, dtype, n, k):
    """a prompt's rows computed with those of longer prompts, in other tiles, K whole (no room for partial sums)"""
    p = lbl.FP4Params(torch.randn(n, k, device=cuda_device, generator=torch.Generator(device=cuda_device).manual_seed(k)) * 0.02,
                      qtype=lbl.ggml_tensor_qtype[qtype]).to(cuda_device)
    x = torch.randn(4000, k, device=cuda_device, generator=torch.Generator(device=cuda_device).manual_seed(n)).to(dtype)
    dt, st = lbl._TORCH_TO_DT[dtype], torch.cuda.current_stream().cuda_stream
    def rows(m):
        y, none = torch.empty(m, n, dtype=dtype, device=cuda_device), torch.empty(16, dtype=torch.uint8, device=cuda_device)
        native_lib.lowbit_matmul_cuda(p.data.data_ptr(), p.qtype, n, k, x.data_ptr(), dt, m, y.data_ptr(), dt, None, 0, none.data_ptr(), 0, st)
        return y
    longest = rows(4000)
    for m in (65, 70, 200, 512, 1000, 3999):
        assert torch.equal(rows(m), longest[:m]), m


@pytest.mark.parametrize("offset", [4, 8])
def test_scratch_off_a_16_byte_boundary(lbl, native_lib, cuda_device, offset):
    """shapes that would split K run it whole, within the same bounds; 32-bit activations, whose planes lie there, are refused"""
    m, n, k = 100, 2048, 4096
    ((wg, g), (wu, p)), qt = weights(lbl, cuda_device, 3, n, k, "sym_int4", 2)
    x = acts(cuda_device, 4, m, k, torch.float16)
    stream = torch.cuda.current_stream().cuda_stream
    y = torch.empty(m, n, dtype=torch.float32, device=cuda_device)

    def scratch(size):
        return torch.empty(size + 16, dtype=torch.uint8, device=cuda_device)[offset:]
    ws = scratch(native_lib.lowbit_matmul_workspace_size(n, k, m, native_lib.DT_F16))
    assert ws.data_ptr() % 16 == offset and ws.numel() > m * n * 8
    native_lib.lowbit_matmul_cuda(wg.data_ptr(), qt, n, k, x.data_ptr(), native_lib.DT_F16, m, y.data_ptr(), native_lib.DT_F32, None, False,
                                  ws.data_ptr(), ws.numel(), stream)
    want, bound = product(x.double(), g, U[torch.float16])
    assert bool(((y.double() - want).abs() <= bound).all())
    ws = scratch(native_lib.lowbit_mlp_workspace_size(n, k, m, native_lib.DT_F16))
    native_lib.lowbit_mlp_cuda(wg.data_ptr(), wu.data_ptr(), qt, n, k, x.data_ptr(), native_lib.DT_F16, m, y.data_ptr(), native_lib.DT_F32, 0,
                               ws.data_ptr(), ws.numel(), stream)
    want, bound = gated(x.double(), g, p, U[torch.float16], 0)
    assert bool(((y.double() - want).abs() <= bound).all())
    x = acts(cuda_device, 4, m, k, torch.float32)
    ws = scratch(native_lib.lowbit_matmul_workspace_size(n, k, m, native_lib.DT_F32))
    for rows in (1, m):
        with pytest.raises(RuntimeError):
            native_lib.lowbit_matmul_cuda(wg.data_ptr(), qt, n, k, x.data_ptr(), native_lib.DT_F32, rows, y.data_ptr(), native_lib.DT_F32, None, False,
                                          ws.data_ptr(), ws.numel(), stream)


@pytest.mark.parametrize("qtype,dtype", [("sym_int4", torch.float16), ("asym_int4", torch.bfloat16), ("nf4", torch.float16), ("fp8_e5m2", torch.bfloat16)])
@pytest.mark.parametrize("act", [0, 1])
@pytest.mark.parametrize("m,n,k", [(100, 2048, 4096), (65, 384, 2048), (150, 1024, 8192)])
def test_prompt_mlp_with_a_split_k_range(lbl, native_lib, cuda_device, qtype, dtype, act, m, n, k):
    """few tiles, long rows: gate and up partial sums in scratch, the activation in the second launch"""
    ((wg, g), (wu, p)), qt = weights(lbl, cuda_device, m, n, k, qtype, 2)
    x = acts(cuda_device, n, m, k, dtype)
    # a size of at least two splits: 8 bytes of partial sums per split, token and feature
    assert native_lib.lowbit_mlp_workspace_size(n, k, m, native_lib.DT_F16) >= 2 * 8 * m * n
    want, bound = gated(x.double(), g, p, U[dtype], act)
    y32 = lbl.mlp_forward(x, wg, wu, m, k, n, act, qt, out=torch.empty(m, n, dtype=torch.float32, device=cuda_device))
    assert bool(((y32.double() - want).abs() <= bound).all())
    assert torch.equal(lbl.mlp_forward(x, wg, wu, m, k, n, act, qt), y32.to(dtype))
