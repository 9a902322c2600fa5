"""The tcgen05 attention kernel against a plain PyTorch fp32 softmax(Q K^T / sqrt(d)) V of the same inputs."""
import pytest
import torch

from iris_b200.ops.attention import attention_fwd

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)


def _reference(qkv, batch, seq, heads, causal):
    d = 128
    hl = heads * d
    q = qkv[:, :hl].float().view(batch, seq, heads, d).transpose(1, 2)
    k = qkv[:, hl:2 * hl].float().view(batch, seq, heads, d).transpose(1, 2)
    v = qkv[:, 2 * hl:].float().view(batch, seq, heads, d).transpose(1, 2)
    s = q @ k.transpose(-1, -2) / d ** 0.5
    if causal:
        mask = torch.ones((seq, seq), dtype=torch.bool, device=qkv.device).tril()
        s = s.masked_fill(~mask, float("-inf"))
    o = torch.softmax(s, dim=-1) @ v
    return o.transpose(1, 2).reshape(batch * seq, hl)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("batch,seq,heads", [(1, 128, 1), (2, 256, 3), (1, 1024, 2), (3, 384, 4)])
def test_attention_matches_fp32_softmax(batch, seq, heads, causal, dtype):
    g = torch.Generator(device="cuda").manual_seed(batch * 1000 + seq + heads)
    wide = torch.randn((batch * seq, 3 * heads * 128 + 64), generator=g, device="cuda").to(dtype)
    qkv = wide[:, 32:32 + 3 * heads * 128]           # a strided view: row pitch larger than the row
    out_full = torch.full((batch * seq, heads * 128 + 8), float("nan"), dtype=dtype, device="cuda")
    out = out_full[:, :heads * 128]
    status = torch.zeros(16, dtype=torch.int32, device="cuda")
    attention_fwd(qkv, out, batch, seq, heads, causal=causal, status=status)
    torch.cuda.synchronize()
    assert int(status[0]) == 0, f"a wait of the kernel ran out: {status[:8].tolist()}"
    ref = _reference(qkv, batch, seq, heads, causal)
    # P is rounded to 16 bits before the second product and so is the output: a few 2^-8 of the largest |v| average
    tol = 3 * 2.0 ** -8 * ref.abs().max().item() + 1e-3
    err = (out.float() - ref).abs().max().item()
    assert err <= tol, f"max err {err} > {tol}"
    assert bool(torch.isnan(out_full[:, heads * 128:].float()).all()), "wrote past the row"


def test_attention_large_logits_and_rejects_bad_shapes():
    """Scores far from zero (the running maximum moves from tile to tile) and argument checks."""
    g = torch.Generator(device="cuda").manual_seed(7)
    batch, seq, heads = 1, 512, 2
    qkv = (torch.randn((batch * seq, 3 * heads * 128), generator=g, device="cuda") * 3.0).to(torch.bfloat16)
    out = torch.empty((batch * seq, heads * 128), dtype=torch.bfloat16, device="cuda")
    attention_fwd(qkv, out, batch, seq, heads)
    torch.cuda.synchronize()
    ref = _reference(qkv, batch, seq, heads, True)
    assert (out.float() - ref).abs().max().item() <= 4 * 2.0 ** -8 * ref.abs().max().item() + 1e-3
    with pytest.raises((RuntimeError, ValueError)):
        attention_fwd(qkv[:500], out[:500], 1, 500, heads)       # seq not a multiple of 128
    with pytest.raises(TypeError):
        attention_fwd(qkv.float(), out, batch, seq, heads)


@pytest.mark.parametrize("batch,seq,heads,causal,dtype", [
    (1, 128, 5, False, torch.float16),      # one key tile: the second side of the split form has nothing to merge
    (2, 640, 14, True, torch.bfloat16),     # 140 query tiles: split form, odd and even numbers of key tiles
    (1, 2048, 3, False, torch.bfloat16),    # split form, a long chain
    (3, 640, 10, True, torch.float16),      # 150 query tiles: pairs, the last tile of every head alone
    (2, 384, 80, False, torch.bfloat16),    # pairs, several items per CTA, an incomplete last round
    (5, 1024, 30, True, torch.bfloat16),    # pairs, several groups of heads
])
def test_attention_both_forms(batch, seq, heads, causal, dtype):
    """The form in which two query tiles share their keys, and the one in which the keys of a query tile are shared out
    and merged.  Queries grow along the keys' order, so that running maxima move from tile to tile."""
    g = torch.Generator(device="cuda").manual_seed(seq + heads)
    t, w = batch * seq, heads * 128
    qkv = torch.randn((t, 3 * w), generator=g, device="cuda")
    ramp = torch.linspace(0.1, 4.0, seq, device="cuda").repeat(batch)[:, None]
    qkv[:, w:2 * w] *= ramp                                   # later keys: larger scores
    qkv[: t // 2, :w] *= 3.0
    qkv = qkv.to(dtype)
    outs = [torch.full((t, w), float("nan"), dtype=dtype, device="cuda") for _ in range(2)]
    status = torch.zeros(16, dtype=torch.int32, device="cuda")
    for out in outs:
        attention_fwd(qkv, out, batch, seq, heads, causal=causal, status=status)
    torch.cuda.synchronize()
    assert int(status[0]) == 0, f"a wait of the kernel ran out: {status[:8].tolist()}"
    assert torch.equal(outs[0], outs[1])
    v_max = qkv[:, 2 * w:].float().abs().max().item()
    unit = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for b in range(batch):
        rows = slice(b * seq, (b + 1) * seq)
        ref = _reference(qkv[rows], 1, seq, heads, causal)
        # every weight is rounded once (half a unit of it; the weights add up to 1), the output once more, and ex2.approx
        # is off by 2 units in 24 bits
        err = (outs[0][rows].float() - ref).abs().max().item()
        assert err <= 1.05 * unit * 2 * v_max, f"batch {b}: {err}"


@pytest.mark.parametrize("batch,heads", [(1, 1), (2, 40)])   # keys of a query tile shared out; pairs of query tiles
@pytest.mark.parametrize("key", [0, 5, 6, 7, 130, 255])
def test_attention_keeps_nan_and_infinity_of_a_key(batch, heads, key):
    """A NaN in one key reaches every query that may see it, whichever unit makes its exponential, and no other; a key whose
    scores are minus infinity weighs nothing."""
    g = torch.Generator(device="cuda").manual_seed(key)
    seq, w = 256, heads * 128
    qkv = torch.randn((batch * seq, 3 * w), generator=g, device="cuda").to(torch.bfloat16)
    out = torch.empty((batch * seq, w), dtype=torch.bfloat16, device="cuda")
    bad = qkv.clone()
    bad[key, w:w + 128] = float("nan")                        # batch 0, head 0
    attention_fwd(bad, out, batch, seq, heads, causal=True)
    nan = torch.isnan(out.float())
    want = torch.zeros_like(nan)
    want[key:seq, :128] = True
    assert torch.equal(nan, want)
    if key > 0:
        bad = qkv.clone()
        bad[:, :128] = bad[:, :128].abs() + 0.1               # head 0: positive queries, a key of minus infinity
        bad[key, w:w + 128] = float("-inf")
        attention_fwd(bad, out, batch, seq, heads, causal=True)
        ref = _reference(bad[:seq], 1, seq, heads, True)[:, :128]
        # as in test_attention_both_forms
        assert (out[:seq, :128].float() - ref).abs().max().item() <= 1.05 * 2.0 ** -7 * bad[:, 2 * w:].float().abs().max().item()


@pytest.mark.parametrize("batch,heads", [(1, 1), (2, 40)])   # keys of a query tile shared out; pairs of query tiles
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("key", [260, 390])                  # either side of the split form, not its first tile
def test_attention_largest_weight_is_exact(batch, heads, key, dtype):
    """The largest weight of a row is 1 in the 16 bits of P wherever its key lies: one key that weighs 2^x times the others,
    x from 0.1 to 7, with the only non-zero value, 1.  The output is 1 / (row sum) then, and off by its own rounding alone
    (half a unit, and 2^-20 for the fp32 sum and the exponentials)."""
    seq, w = 512, heads * 128
    qkv = torch.zeros((batch * seq, 3 * w), device="cuda")
    head = slice(128 * (heads - 1), 128 * heads)              # the last head, the last batch
    rows = slice((batch - 1) * seq, batch * seq)
    q, k, v = qkv[rows, :w][:, head], qkv[rows, w:2 * w][:, head], qkv[rows, 2 * w:][:, head]
    q[:, 3] = torch.linspace(0.8, 55.0, seq, device="cuda")
    k[key, 3], v[key] = 1.0, 1.0
    qkv = qkv.to(dtype)
    out = torch.empty((batch * seq, w), dtype=dtype, device="cuda")
    attention_fwd(qkv, out, batch, seq, heads, causal=False)
    x = qkv[rows, :w][:, head][:, 3].double() / 128 ** 0.5    # score of the key, natural logarithm
    exact = 1.0 / (1.0 + (seq - 1) * torch.exp(-x))
    bits = 8 if dtype == torch.bfloat16 else 11
    half = 0.5 * 2.0 ** (torch.floor(torch.log2(exact)) - (bits - 1))
    err = (out[rows, head].double() - exact[:, None]).abs().amax(1)
    assert bool((err <= half + exact * 2.0 ** -20).all()), f"up to {(err / half).max().item()} half units"


@pytest.mark.parametrize("batch,heads", [(1, 1), (2, 40)])   # keys of a query tile shared out; pairs of query tiles
def test_attention_masked_keys_weigh_nothing(batch, heads):
    """The values of later keys reach no query, not even as the smallest normal number times the largest bf16 value: the
    rows before them have the same bits as with zeros there."""
    g = torch.Generator(device="cuda").manual_seed(11)
    seq, w = 256, heads * 128
    qkv = torch.randn((batch * seq, 3 * w), generator=g, device="cuda").to(torch.bfloat16)
    outs = []
    for value in (0.0, 3.3e38):
        late = qkv.clone().view(batch, seq, 3 * w)
        late[:, 160:, 2 * w:] = value
        out = torch.empty((batch * seq, w), dtype=torch.bfloat16, device="cuda")
        attention_fwd(late.view(batch * seq, 3 * w), out, batch, seq, heads, causal=True)
        outs.append(out.view(batch, seq, w)[:, :160])
    assert bool(torch.isfinite(outs[0].float()).all())
    assert torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("batch,heads", [(1, 1), (2, 60)])   # keys of a query tile shared out; pairs of query tiles
@pytest.mark.parametrize("tile", [0, 1, 2])
def test_attention_tile_of_minus_infinity(batch, heads, tile):
    """128 keys, a whole tile, whose scores are minus infinity: they weigh nothing, also where they are the first that a
    row (or its half of the keys) meets."""
    g = torch.Generator(device="cuda").manual_seed(tile)
    seq, w = 384, heads * 128
    qkv = torch.randn((batch * seq, 3 * w), generator=g, device="cuda").to(torch.bfloat16)
    qkv[:, :128] = qkv[:, :128].abs() + 0.1                   # head 0: positive queries
    qkv[tile * 128:tile * 128 + 128, w:w + 128] = float("-inf")
    out = torch.empty((batch * seq, w), dtype=torch.bfloat16, device="cuda")
    attention_fwd(qkv, out, batch, seq, heads, causal=False)
    ref = _reference(qkv[:seq], 1, seq, heads, False)
    # as in test_attention_both_forms
    bound = 1.05 * 2.0 ** -7 * qkv[:, 2 * w:].float().abs().max().item()
    assert (out[:seq].float() - ref).abs().max().item() <= bound
