"""The one-rank GEMM kernel (``csrc/kernels/gemm_local.cu``): its choice of tile and split on the CPU, and on a GPU every
form of it (operands swapped or not, single CTAs and pairs, tile widths, pieces of K) against a float64 product, at sizes
with remainders in every dimension.

Bounds: the operands are multiplied exactly and summed in fp32 (int8: in 32-bit integers), so a 16-bit result is off by
its rounding, half a unit in the last of 8 (bf16) or 11 (fp16) bits, at most 2^-8 or 2^-11 of the value, plus the fp32 sums' K * 2^-24 of the sum of magnitudes; a tf32
product cuts each operand to 11 bits, so every term is off by at most 2 * 2^-10 of its magnitude, and the sums of 256 terms
and more here, whose cuts average out, by at most 2 * 2^-11.  int8 is exact."""
import ctypes
import os
import random
import re

import pytest
import torch

from iris_b200 import _native

TYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32, "int8": torch.int8}
CODE = {"bf16": 0, "fp16": 1, "fp32": 2, "int8": 3}
SIZE = {"bf16": 2, "fp16": 2, "fp32": 4, "int8": 1}


def _choice(m, n, k, dtype, sms=148):
    lib = _native.kernels()
    lib.iris_gemm_local_choice.restype = ctypes.c_double
    v = [ctypes.c_int() for _ in range(4)]
    t = lib.iris_gemm_local_choice(m, n, k, CODE[dtype], sms, *[ctypes.byref(x) for x in v])
    return [x.value for x in v] + [t]


@pytest.mark.skipif(not _native.kernels_available(), reason="native kernels not built")
def test_choice_is_launchable_for_every_size():
    rng = random.Random(3)
    for _ in range(3000):
        dtype = rng.choice(list(TYPES))
        g = 16 // SIZE[dtype]
        m = rng.choice([1, 2, 64, 128, 129, 256, 257, rng.randint(1, 40000)])
        n, k = g * rng.randint(1, 4000 // g + 1), g * rng.choice([1, 2, 8, 9, rng.randint(1, 20000 // g + 1)])
        swap, cg, tn, split, t = _choice(m, n, k, dtype, rng.choice([148, 132, 16, 1]))
        kblocks = -(-k * SIZE[dtype] // 128)
        assert swap in (0, 1) and cg in (1, 2) and t > 0
        assert 16 <= tn <= 256 and tn % (32 if dtype == "int8" else 16) == 0
        assert 1 <= split <= kblocks and split * cg <= 8
        assert not (swap and m > 256)


@pytest.mark.skipif(not _native.kernels_available(), reason="native kernels not built")
def test_overlapping_output_rows_are_refused():
    """Before any device is looked at; a single row has no pitch."""
    from iris_b200.ops import gemm as G
    lib = G._lib()
    for m, glu, refused in ((2, 0, True), (2, 1, True), (1, 0, False)):
        h = lib.iris_gemm_local_create(4096, 64, 8192, 64, 12288, 248, m, 256, 64, 0, -1, 0, 0, -1, 0, 0, 0, glu)
        assert h is None
        assert (b"row pitch is smaller" in lib.iris_gemm_local_last_error()) == refused


def test_split_handover_publishes_the_stores_of_every_lane():
    """The order in which a warp hands its partial sums over, read out of the source and run through the memory model's
    happens-before relation: each of 32 lanes stores into another CTA's shared memory, and what a relaxed arrival
    publishes is what its own thread knew at its last fence.  A thread knows its own stores and, after a warp barrier,
    those of all lanes; the arrivals have to publish all 32."""
    source = open(os.path.join(os.path.dirname(_native.__file__), "csrc", "kernels", "gemm_local.cu")).read()
    part = source[source.index("st_cluster_v4(at"):source.index("cluster_arrive();   // nothing more is sent")]
    part = re.sub(r"//[^\n]*", "", part)
    order = re.findall(r"\b(st_cluster_v4|__syncwarp|fence_acq_rel_cluster|mbar_arrive_cluster_relaxed)\(", part)
    order = order[:order.index("mbar_arrive_cluster_relaxed") + 1]
    assert order[0] == "st_cluster_v4"
    knows = [set() for _ in range(32)]
    released = [set() for _ in range(32)]
    for what in order:
        if what == "st_cluster_v4":
            for lane in range(32):
                knows[lane].add(lane)
        elif what == "__syncwarp":
            everything = set().union(*knows)
            knows = [set(everything) for _ in range(32)]
        elif what == "fence_acq_rel_cluster":
            released = [set(k) for k in knows]
    assert all(r == set(range(32)) for r in released)


def _operand(shape, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    if dtype == "int8":
        return torch.randint(-128, 128, shape, generator=g, device="cuda", dtype=torch.int32).to(torch.int8)
    return torch.randn(shape, generator=g, device="cuda").to(TYPES[dtype])


def _check(got, a, bt):
    exact = a.double() @ bt.double().t()
    if got.dtype == torch.int8:
        assert torch.equal(got, exact.to(torch.int64).to(torch.int8))
        return
    size = a.double().abs() @ bt.double().abs().t()
    unit = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -24}[got.dtype]
    bound = unit * exact.abs() + a.shape[1] * 2.0 ** -24 * size + 1e-30
    if got.dtype == torch.float32:
        bound = bound + 2.0 * 2.0 ** -11 * size
    assert bool(((got.double() - exact).abs() <= 1.01 * bound).all())


def _run(a, bt, out, swap=-1, cg=0, tn=0, split=0):
    from iris_b200.ops import gemm as G
    lib = G._lib()
    status = torch.zeros(16, dtype=torch.int32, device="cuda")
    name = [t for t, d in TYPES.items() if d == a.dtype][0]
    rc = lib.iris_gemm_local(a.data_ptr(), a.stride(0), bt.data_ptr(), bt.stride(0), out.data_ptr(), out.stride(0),
                             a.shape[0], bt.shape[0], a.shape[1], CODE[name], 0, status.data_ptr(), 2000000000, swap, cg,
                             tn, split, torch.cuda.current_stream().cuda_stream)
    assert rc == 0, lib.iris_gemm_local_last_error().decode()
    torch.cuda.synchronize()
    assert int(status[0]) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", list(TYPES))
@pytest.mark.parametrize("cg,split", [(1, 1), (2, 1), (1, 2), (1, 3), (1, 8), (2, 2), (2, 3), (2, 4)])
@pytest.mark.parametrize("swap", [0, 1])
def test_every_form_against_float64(dtype, cg, split, swap):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    g = 16 // SIZE[dtype]
    for i, (m, n, k) in enumerate([(1, g, 64 * g), (17, 40 * g, 81 * g), (130, 31 * g, 64 * g), (300, 65 * g, 145 * g)]):
        for tn in (32, 96, 256) if dtype == "int8" else (16, 48, 112, 256):
            a, bt = _operand((m, k + g), dtype, i)[:, :k], _operand((n, k), dtype, i + 9)   # a: rows at a pitch of k + g
            frame = torch.full((m + 2, n + 4 * g), 3, dtype=TYPES[dtype], device="cuda")
            out = frame[1:m + 1, g:g + n]
            _run(a, bt, out, swap, cg, tn, split)
            _check(out, a, bt)
            frame[1:m + 1, g:g + n] = 3
            assert bool((frame == 3).all()), "wrote outside the output"


WIDTHS = {"bf16": (48, 112, 176, 256), "fp16": (16, 128, 192, 240), "fp32": (16, 48, 96, 256), "int8": (32, 96, 160, 256)}


@pytest.mark.gpu
@pytest.mark.parametrize("kblocks", [1, 19])    # a tile's loads: a fraction of the ring, or several times round it
@pytest.mark.parametrize("dtype", list(TYPES))
@pytest.mark.parametrize("cg", [1, 2])
@pytest.mark.parametrize("swap", [0, 1])
def test_many_tiles_per_cta(dtype, cg, swap, kblocks):
    """Every form with at least five tiles for every CTA (or pair): two accumulators are in flight, so from the third tile
    on the MMAs wait for an accumulator that the epilogue gives back.  Tile widths of one to eight 128-byte pieces."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from iris_b200.ops import gemm as G
    lib, es = G._lib(), SIZE[dtype]
    g = 16 // es
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    status = torch.zeros(16, dtype=torch.int32, device="cuda")
    k = kblocks * 128 // es - (g if kblocks > 1 else 0)
    for i, tn in enumerate(WIDTHS[dtype]):
        tiles_r = 13
        tiles_c = -(-11 * (sms // cg) // (2 * tiles_r)) + 1
        rows, cols = (tiles_r - 1) * 128 * cg + 96, (tiles_c - 1) * tn + 16     # the last tile of either side is not full
        m, n = (cols, rows) if swap else (rows, cols)
        a, bt = _operand((m, k), dtype, i), _operand((n, k), dtype, i + 9)
        if dtype == "fp32":   # 11 significant bits, which tf32 holds: with one K block the cut bits do not average out
            a, bt = ((x.view(torch.int32) & -8192).view(torch.float32) for x in (a, bt))
        frame = torch.full((m + 2, n + 2 * g), 3, dtype=TYPES[dtype], device="cuda")
        out = frame[1:m + 1, g:g + n]
        h = lib.iris_gemm_local_create(a.data_ptr(), k, bt.data_ptr(), k, out.data_ptr(), out.stride(0), m, n, k, CODE[dtype], 0,
                                       status.data_ptr(), 2000000000, swap, cg, tn, 1, 0)
        assert h, lib.iris_gemm_local_last_error().decode()
        info = (ctypes.c_int * 6)()
        lib.iris_gemm_local_info(h, info)
        assert list(info)[:4] == [swap, cg, tn, 1] and tiles_r * tiles_c >= 5 * (info[4] // cg)
        assert lib.iris_gemm_local_launch(h, torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        lib.iris_gemm_local_destroy(h)
        assert int(status[0]) == 0
        _check(out, a, bt)
        frame[1:m + 1, g:g + n] = 3
        assert bool((frame == 3).all()), "wrote outside the output"


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(1, 2048, 4096), (64, 1456, 1448), (129, 2504, 1736), (2500, 2048, 512)])
@pytest.mark.parametrize("dtype", ["bf16", "int8"])
def test_choice_matches_and_repeats(m, n, k, dtype):
    """What the rule picks is right, gives the same bits each time, and the same through ``gemm`` and a prepared op of any
    collective form (one rank: all of them are the product)."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    import iris_b200 as iris
    from iris_b200.ops import gemm as G
    n, k = n // 16 * 16, k // 16 * 16
    a, bt = _operand((m, k), dtype, 1), _operand((n, k), dtype, 2)
    outs = [torch.empty((m, n), dtype=TYPES[dtype], device="cuda") for _ in range(2)]
    for o in outs:
        _run(a, bt, o)
    _check(outs[0], a, bt)
    assert torch.equal(outs[0], outs[1])
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        c = G.gemm(a, bt)
    side.synchronize()
    assert torch.equal(c, outs[0])
    ctx = iris.iris(256 << 20)
    ops = [G.gemm_all_scatter(ctx, [a], [bt])]
    if dtype == "bf16":
        ops += [G.gemm_all_reduce(ctx, [a], [bt], variant=v) for v in ("auto", "atomic", "one_shot", "two_shot")]
    for op in ops:
        assert op.local
        graph = torch.cuda.CUDAGraph()
        op()
        op.check()
        assert torch.equal(op.out[0], outs[0])
        op.out[0].zero_()
        with torch.cuda.graph(graph):
            op()
        graph.replay()
        op.check()
        assert torch.equal(op.out[0], outs[0])
        graph.reset()
        op.close()
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["store", "reduce"])
@pytest.mark.parametrize("c_cols", [320, 328])
def test_narrower_output_cuts_the_product_off(mode, c_cols):
    """``c_cols`` below the rows of B: the columns from there on are not written, not to the next row and not past the
    buffer's end (a guard band of 3s all round)."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    import iris_b200 as iris
    from iris_b200.ops import gemm as G
    m, n, k = 256, 512, 192
    a, bt = _operand((m, k), "bf16", 1), _operand((n, k), "bf16", 2)
    ctx = iris.iris(64 << 20)
    frame = ctx.full((m + 2, 336), 3, dtype=torch.bfloat16)
    op = G.FusedGemm(ctx, [a], [bt], mode, store_all=mode == "reduce", out=[frame[1:m + 1, :c_cols]], c_cols=c_cols)
    got = op()[0]
    op.check()
    _check(got, a, bt[:c_cols])
    frame[1:m + 1, :c_cols] = 3
    assert bool((frame == 3).all()), "wrote outside the output"
    own = G.FusedGemm(ctx, [a], [bt], mode, store_all=mode == "reduce", c_cols=320)
    own()
    own.check()
    assert own.out[0].shape == (m, 320)
    _check(own.out[0], a, bt[:320])
    op.close(), own.close(), ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("m,inter,k,dtype", [(1, 8, 64, "bf16"), (128, 1376, 512, "bf16"), (129, 200, 264, "fp16"),
                                             (700, 2744, 1032, "bf16"), (2048, 1024, 512, "fp16"),
                                             (4096, 8200, 264, "bf16"), (4000, 8192, 1288, "fp16")])
def test_gate_and_linear_projection_in_one(m, inter, k, dtype):
    """``swiglu=True`` against silu(a gate^T) * (a linear^T) in float64.  Off by the output's rounding, by the fp32 sums'
    K * 2^-24 of their magnitudes (times what either factor scales them by; silu' <= 1.1), and by 2^-20 of the value for
    the fast exponential and division."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    import iris_b200 as iris
    from iris_b200.ops import gemm as G
    a = _operand((m, k), dtype, 1)
    bt = (_operand((2 * inter, k), dtype, 2).float() / k ** 0.5).to(TYPES[dtype])
    frame = torch.full((m, inter + 16), 3, dtype=TYPES[dtype], device="cuda")
    ctx = iris.iris(256 << 20)
    op = G.all_gather_gemm(ctx, (m + 127) // 128 * 128, [bt], swiglu=True)
    op.a_full[0][:m].copy_(a)
    got = op()[0][:m]
    op.check()
    own = G.FusedGemm(ctx, [a], [bt], "store", out=[frame[:, 8:8 + inter]], swiglu=True)
    own()
    own.check()
    if m >= 4000:   # several tiles for every CTA or pair, see test_many_tiles_per_cta
        tiles = -(-m // (128 * own.cta_group)) * -(-inter // (own.bn // 2))
        assert tiles > 2 * (own.ctas_per_rank // own.cta_group)
    assert got.shape == (m, inter) and torch.equal(frame[:, 8:8 + inter], got)
    assert bool((frame[:, :8] == 3).all()) and bool((frame[:, 8 + inter:] == 3).all())
    g, u = a.double() @ bt[:inter].double().t(), a.double() @ bt[inter:].double().t()
    sg, su = (a.double().abs() @ b.double().abs().t() for b in (bt[:inter], bt[inter:]))
    exact = g * torch.sigmoid(g) * u
    unit = 2.0 ** -8 if dtype == "bf16" else 2.0 ** -11
    bound = (unit + 2.0 ** -20) * exact.abs() + k * 2.0 ** -24 * (1.1 * sg * u.abs() + g.abs() * su) + 2.0 ** -24
    assert bool(((got.double() - exact).abs() <= 1.01 * bound).all())
    with pytest.raises(ValueError):
        G.FusedGemm(ctx, [a], [bt], "store", swiglu=True, bn=64)
    op.close(), own.close(), ctx.close()
