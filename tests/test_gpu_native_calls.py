"""The native block and stack calls at the sizes where their kernels change form: ragged token counts around the row pitches and
the GEMM tiles, several complexes and samples per call, in bfloat16 and float32, against the oracle."""
import pytest
import torch

from helpers import err_stats
from oracle import pairformer_oracle as O
from test_gpu_parity import PRECISE_MAX_TOL, PRECISE_RMS_TOL, _check, _oracle_on

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    return torch.device("cuda:0")


@pytest.fixture(autouse=True)
def _no_grad_and_status():
    from kfold_b200 import _lib as L
    with torch.no_grad():
        yield
    assert L.device_status() == 0


def _compare(out, ref, precise, what):
    if precise:
        mx, r = err_stats(out, ref)
        assert mx < PRECISE_MAX_TOL and r < PRECISE_RMS_TOL, f"{what}: {mx:.3e} {r:.3e}"
    else:
        _check(*err_stats(out, ref), what)


@pytest.mark.parametrize("n,batch,precise", [(8, 1, False), (24, 1, False), (25, 2, False), (63, 1, False), (129, 2, False), (257, 1, False),
                                             (40, 2, True)])
def test_pair_block_ragged(dev, n, batch, precise):
    from kfold_b200 import modules as M
    import synth
    dt = torch.float32 if precise else torch.bfloat16
    z, pm, m = synth.pair_inputs(n, n, 128, batch, valid=n - n // 10)
    s = synth.single_inputs(n, n, 384, batch)
    z, s = z.to(dt), s.to(dt)
    w = synth.pairformer_block_weights(n, 128, 384)
    blk = M.PairformerBlock(128, 384).to(dev)
    blk.load_state_dict(w, strict=True)
    zo, so = blk(z.to(dev), s.to(dev), pm.to(dev), m.to(dev))
    assert zo.dtype == dt and so.dtype == dt

    def run(z_, s_, pm_, m_, w_):
        zr, sr = O.pairformer_block(z_, s_, pm_, m_, w_, row_chunk=32)
        return torch.cat([zr.reshape(-1), sr.reshape(-1)])

    ref = _oracle_on(dev, run, z.float(), s.float(), pm, m, w)
    _compare(zo.float().cpu(), ref[: zo.numel()].view(zo.shape), precise, f"block N={n} z")
    _compare(so.float().cpu(), ref[zo.numel():].view(so.shape), precise, f"block N={n} s")


@pytest.mark.parametrize("l,groups,samples,own_s,precise", [(9, 1, 1, False, False), (37, 2, 3, False, False), (130, 1, 2, True, False),
                                                            (33, 2, 2, True, True), (45, 1, 3, False, True)])
def test_token_stack_ragged(dev, l, groups, samples, own_s, precise):
    """Two blocks (c = 256, 8 heads x 32): shared and per-sample conditioning, bias given as an unpadded and as a pitched tensor."""
    from kfold_b200 import modules as M
    import synth
    rng, blocks, c, heads = synth._Rng(l), 2, 256, 8
    w = {}
    for i in range(blocks):
        w.update(synth._prefixed(f"blocks.{i}.attention", synth.apb_weights(rng, c, 384)))
        w.update(synth._prefixed(f"blocks.{i}.transition", synth.conditioned_transition_weights(rng, c, 384)))
    a = rng.normal(groups, samples, l, c)
    s = rng.normal(groups, samples if own_s else 1, l, 384)
    bias = rng.normal(groups, 1, blocks, heads, l, l)
    mask = synth.token_mask(l, valid=l - l // 8).view(1, 1, l).expand(groups, 1, l).contiguous()
    stack = M.CachedGlobalTransformerStack(c, 384, heads, blocks).to(dev)
    stack.load_state_dict(w, strict=True)
    ref = _oracle_on(dev, O.global_transformer_stack, a, s, bias, mask, w, heads, blocks)
    pitched = torch.zeros(groups, 1, blocks, heads, l, (l + 15) // 16 * 16)
    pitched[..., :l] = bias
    for given in (bias.to(dev), pitched.to(dev)[..., :l]):
        with torch.autocast("cuda", dtype=torch.bfloat16, enabled=not precise):
            out = stack(a.to(dev), s.to(dev), given, mask.to(dev))
        _compare(out.float().cpu(), ref, precise, f"token stack L={l}")


@pytest.mark.parametrize("l,groups,samples,c,heads", [(65, 4, 3, 768, 16), (130, 2, 5, 768, 16), (257, 1, 4, 768, 16), (200, 3, 4, 512, 8),
                                                         (1100, 1, 2, 768, 16)])
def test_token_stack_shared_bias(dev, l, groups, samples, c, heads):
    """Head dims 48 and 64, enough samples per complex for the attention that adds one bias tile to several of them: odd sample
    counts, ragged tokens, scattered masks, heads whose bias lies far above and below zero."""
    from kfold_b200 import modules as M
    import synth
    rng = synth._Rng(l)
    w = synth._prefixed("blocks.0.attention", synth.apb_weights(rng, c, 384))
    w.update(synth._prefixed("blocks.0.transition", synth.conditioned_transition_weights(rng, c, 384)))
    a, s = rng.normal(groups, samples, l, c), rng.normal(groups, 1, l, 384)
    bias = rng.normal(groups, 1, 1, heads, l, l).bfloat16().float()
    bias[:, :, :, 1] = 256.0
    bias[:, :, :, 2] = -256.0
    mask = synth.token_mask(l, valid=l - l // 8).view(1, 1, l).expand(groups, 1, l).clone()
    mask[0, 0, :33] = False
    mask[-1, 0, 5::7] = False
    stack = M.CachedGlobalTransformerStack(c, 384, heads, 1).to(dev)
    stack.load_state_dict(w, strict=True)
    ref = _oracle_on(dev, O.global_transformer_stack, a, s, bias, mask, w, heads, 1)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        out = stack(a.to(dev), s.to(dev), bias.to(dev), mask.to(dev))
    _compare(out.float().cpu(), ref, False, f"token stack L={l}")


@pytest.mark.parametrize("starting", [True, False])
@pytest.mark.parametrize("n,batch,c,heads", [(25, 2, 128, 4), (33, 1, 128, 8), (65, 2, 96, 4), (130, 1, 128, 4), (257, 1, 128, 4)])
def test_triatt_rows_masks_and_stabiliser(dev, n, batch, c, heads, starting):
    """Pair rows around the tile and row-group sizes, with rows whose first 32 or 64 keys, scattered keys or all keys are masked, and
    heads whose logits all lie far above or below zero (a constant bias, which softmax ignores): every way the stabiliser moves."""
    from kfold_b200 import functional as F
    from kfold_b200 import packing
    import synth
    z, pm, _ = synth.pair_inputs(n, n, c, batch)
    g = torch.Generator().manual_seed(n)
    holes = torch.rand(pm.shape, generator=g) < 0.2
    rows = torch.arange(n) % 5
    keys = torch.arange(n)
    off = ((rows[:, None] == 1) & (keys < 32)) | ((rows[:, None] == 2) & (keys < 64)) | ((rows[:, None] == 3) & holes) | (rows[:, None] == 4)
    pm = pm & ~(off if starting else off.transpose(-1, -2))
    w = synth.triatt_weights(synth._Rng(n), c, heads)
    w["layer_norm.weight"][0], w["layer_norm.bias"][0] = 0.0, 1.0
    w["linear.weight"] *= (torch.arange(heads) % 2 == 0).float()[:, None]
    w["linear.weight"][1::2, 0] = torch.tensor([256.0, -256.0]).repeat(heads)[: heads // 2]
    zb = z.bfloat16()
    out = F.triangle_attention(zb.to(dev), pm.to(dev), packing.pack_triatt(w, heads, dev), starting).float().cpu()
    ref = _oracle_on(dev, O.triangle_attention, zb.float(), pm, w, heads, starting)
    _check(*err_stats(out, ref), f"triatt N={n} starting={starting}")


@pytest.mark.parametrize("n,batch,c,heads", [(8, 1, 128, 8), (40, 2, 96, 4), (72, 1, 128, 4), (72, 2, 128, 2)])
def test_triatt_fp32_key_split(dev, n, batch, c, heads):
    """float32 attention at key counts that leave some of a block's eight warps without keys, with one and two query rows per lane,
    masked keys and rows without any key."""
    from kfold_b200 import functional as F
    from kfold_b200 import packing
    import synth
    z, pm, _ = synth.pair_inputs(n, n, c, batch)
    pm = pm & ((torch.arange(n) % 3 != 1) | (torch.arange(n)[:, None] % 2 == 0)) & (torch.arange(n)[:, None] != 5)
    w = synth.triatt_weights(synth._Rng(n), c, heads)
    out = F.triangle_attention(z.to(dev), pm.to(dev), packing.pack_triatt(w, heads, dev, precise=True), True).cpu()
    ref = _oracle_on(dev, O.triangle_attention, z, pm, w, heads, True)
    mx, r = err_stats(out, ref)
    assert mx < PRECISE_MAX_TOL and r < PRECISE_RMS_TOL, f"{mx:.3e} {r:.3e}"


@pytest.mark.parametrize("rows", [1, 3, 33, 5000])
@pytest.mark.parametrize("c", [128, 256])
def test_layernorm_bf16_rows(dev, c, rows):
    """The 16-byte LayerNorm at row counts that leave part of a warp's rows empty and that make warps loop."""
    from kfold_b200 import functional as F
    g = torch.Generator().manual_seed(rows)
    x = (torch.randn(rows, c, generator=g) * 3 + 1).bfloat16()
    w, b = torch.rand(c, generator=g) + 0.5, torch.randn(c, generator=g)
    out = F.layer_norm(x.to(dev), w.to(dev), b.to(dev), 1e-5).float().cpu()
    ref = torch.nn.functional.layer_norm(x.float(), (c,), w, b, 1e-5)
    _check(*err_stats(out, ref), f"layernorm {rows} x {c}")
    if c == 256:    # same bits as the general kernel, which takes rows that are not contiguous
        wide = torch.zeros(rows, c + 8, dtype=torch.bfloat16)
        wide[:, :c] = x
        assert torch.equal(out, F.layer_norm(wide.to(dev)[:, :c], w.to(dev), b.to(dev), 1e-5).float().cpu())


@pytest.mark.parametrize("d", [6, 130, 132, 768])
def test_atoms_to_tokens_widths(dev, d):
    """The masked mean at widths that end inside a warp's channels and that are not whole vectors, with tokens of 0 to 40 atoms."""
    from kfold_b200 import _lib as L
    from kfold_b200 import functional as F
    g = torch.Generator().manual_seed(d)
    index = torch.cat([torch.zeros(40, dtype=torch.long), torch.randint(2, 30, (160,), generator=g)]).sort().values.view(1, 200)
    mask = torch.rand(1, 200, generator=g) < 0.8
    x = torch.randn(1, 3, 200, d, generator=g)
    launches = L.launch_count()
    out = F.aggregate_atoms_to_tokens(x.to(dev), index.to(dev), mask.to(dev), 31).cpu()
    assert L.launch_count() - launches == 3      # two for the tokens' ranges of atoms
    for t in range(31):
        rows = x[:, :, (index[0] == t) & mask[0]]
        ref = rows.mean(2) if rows.shape[2] else torch.zeros(1, 3, d)
        assert torch.allclose(out[:, :, t], ref, atol=1e-5), t


@pytest.mark.parametrize("d", [6, 130, 520, 1100])
@pytest.mark.parametrize("x_dtype,add_dtype", [(torch.bfloat16, None), (torch.float32, None), (torch.bfloat16, torch.float32), (torch.float32, torch.float32)])
def test_tokens_to_atoms_widths(dev, d, x_dtype, add_dtype):
    """Rows that are no, one and several groups of four pieces, copied and with something added: exact, the sum of two rounded numbers."""
    from kfold_b200 import functional as F
    g = torch.Generator().manual_seed(d)
    index = torch.randint(0, 9, (1, 65), generator=g)
    x = torch.randn(1, 2, 9, d, generator=g).to(x_dtype)
    add = None if add_dtype is None else torch.randn(1, 2, 65, d, generator=g).to(add_dtype)
    out = F.broadcast_tokens_to_atoms(x.to(dev), index.to(dev), None if add is None else add.to(dev)).cpu()
    ref = x[:, :, index[0]]
    assert torch.equal(out, ref if add is None else (ref.float() + add.float()).to(out.dtype))


@pytest.mark.parametrize("c", [6, 128, 130, 300])
def test_coord_embed_widths(dev, c):
    from kfold_b200 import functional as F
    g = torch.Generator().manual_seed(c)
    q, r, w = torch.randn(1, 37, c, generator=g), torch.randn(1, 3, 37, 6, generator=g), torch.randn(c, 6, generator=g)
    mask = torch.rand(1, 37, generator=g) < 0.8
    out = F.coord_embed(q.to(dev), r.to(dev), w.to(dev), mask.to(dev)).cpu()
    q, r, w = q.double().unsqueeze(1), r.double() * mask[:, None, :, None], w.double()
    # seven float32 roundings of partial sums that the magnitudes' sum bounds
    assert ((out - (q + r @ w.T)).abs() <= 7 * 2.0 ** -24 * (q.abs() + r.abs() @ w.abs().T)).all()


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("rows,k", [(1, 8), (37, 128), (300, 264), (65, 520), (40, 1032)])
def test_ln_linear_fp32_rows(dev, rows, k, bf16):
    """The split LayerNorm at the edges of its register forms (up to 128, 256, 512, 1024 channels, above) from both row types."""
    from kfold_b200 import functional as F
    from kfold_b200 import packing
    g = torch.Generator().manual_seed(k)
    x = torch.randn(rows, k, generator=g) * 2 + 0.5
    x = x.bfloat16() if bf16 else x
    lw, lb, w = torch.rand(k, generator=g) + 0.5, torch.randn(k, generator=g), torch.randn(64, k, generator=g) / k ** 0.5
    out = F.ln_linear_fp32(x.to(dev), lw.to(dev), lb.to(dev), packing.split3_weights(w).to(dev)).cpu()
    ref = (torch.nn.functional.layer_norm(x.double(), (k,), lw.double(), lb.double(), 1e-5) @ w.double().T).float()
    mx, r = err_stats(out, ref)
    assert mx < PRECISE_MAX_TOL and r < PRECISE_RMS_TOL, f"{mx:.3e} {r:.3e}"


def _hooked_cases(dev):
    """(module, its call, a submodule that the module calls)"""
    from kfold_b200 import modules as M
    from kfold_b200.confidence import ConfidencePairSingleBlock
    g = torch.Generator(device=dev).manual_seed(11)
    rnd = lambda *shape, dt=torch.bfloat16: torch.randn(shape, generator=g, device=dev, dtype=dt)
    n = 41
    z, s = rnd(1, n, n, 128), rnd(1, n, 384)
    m = torch.ones(1, n, dtype=torch.bool, device=dev)
    pm = torch.ones(1, n, n, dtype=torch.bool, device=dev)
    a, c, bias = rnd(1, 2, n, 256, dt=torch.float32), rnd(1, 1, n, 384, dt=torch.float32), rnd(1, 1, 2, 8, n, n)
    q, qc, p = rnd(1, 2, 64, 128, dt=torch.float32), rnd(1, 1, 64, 128, dt=torch.float32), rnd(1, 1, 2, 32, 128, 16, dt=torch.float32)
    am = torch.ones(1, 1, 64, dtype=torch.bool, device=dev)
    with torch.device(dev):
        tri, blk, conf = M.TriangularBlock(128), M.PairformerBlock(128, 384), ConfidencePairSingleBlock(384, 128, 16)
        tok, atm = M.CachedGlobalTransformerStack(256, 384, 8, 2), M.LocalTransformerStack(128, 128, 16, 4, 2)
    return {"triangular": (tri, lambda: tri(z, pm), tri.tri_mul_in), "pairformer": (blk, lambda: blk(z, s, pm, m), blk.attention),
            "confidence": (conf, lambda: conf(z, s, pm, m), conf.pair_block.transition_z),
            "token": (tok, lambda: tok(a, c, bias, m.unsqueeze(1)), tok.blocks[1].transition),
            "atom": (atm, lambda: atm(q, qc, p, am), atm.blocks[0].transition)}


@pytest.mark.parametrize("which", ["triangular", "pairformer", "confidence", "token", "atom"])
def test_hooks_of_submodules_fire(dev, which):
    """A forward hook on a submodule sees that submodule's output, and what it returns is used; the submodules called one by one
    give what the native call gives, to the rounding of the bf16 results that lie between them."""
    mod, call, sub = _hooked_cases(dev)[which]
    flat = lambda o: torch.cat([t.float().reshape(-1) for t in (o if isinstance(o, tuple) else (o,))])
    with torch.autocast("cuda", dtype=torch.bfloat16):
        one = flat(call())
        seen = []
        handle = sub.register_forward_hook(lambda m, args, out: seen.append(out.shape))
        hooked = flat(call())
        assert len(seen) == 1
        handle.remove()
        handle = sub.register_forward_hook(lambda m, args, out: out * 0)
        changed = flat(call())
        handle.remove()
        again = flat(call())
    _check(*err_stats(hooked, one), f"{which}: one by one against one call")
    assert torch.equal(again, one) and not torch.allclose(changed, one, rtol=0.1, atol=0.1)


def _token_weights(rng, blocks, c):
    import synth
    w = {}
    for i in range(blocks):
        w.update(synth._prefixed(f"blocks.{i}.attention", synth.apb_weights(rng, c, 384)))
        w.update(synth._prefixed(f"blocks.{i}.transition", synth.conditioned_transition_weights(rng, c, 384)))
    return w


@pytest.mark.parametrize("l", [33, 40])
@pytest.mark.parametrize("pattern", ["mask per sample", "conditioning of all complexes"])
def test_token_stack_other_sharing_patterns(dev, l, pattern):
    """What the one native call does not take runs block by block: against the oracle, with the bias given at a wider pitch than
    its own, and with no more launches a block than its own seven (the conditioning is projected once for all blocks)."""
    from kfold_b200 import _lib as L
    from kfold_b200 import modules as M
    import synth
    groups, samples, c, heads = 2, 2, 256, 8
    rng = synth._Rng(l)
    a, bias = rng.normal(groups, samples, l, c), rng.normal(groups, 1, 3, heads, l, l)
    s = rng.normal(groups, 1, l, 384) if pattern == "mask per sample" else rng.normal(1, 1, l, 384)
    mask = synth.token_mask(l, valid=l - 4).view(1, 1, l).repeat(groups, samples if pattern == "mask per sample" else 1, 1)
    if pattern == "mask per sample":
        mask[1, 1, : l // 2] = False
    pitched = torch.zeros(groups, 1, 3, heads, l, (l + 15) // 16 * 16 + 8)
    pitched[..., :l] = bias
    pitched = pitched.to(dev)[..., :l]
    launches = []
    for blocks in (2, 3):
        w = _token_weights(synth._Rng(7), blocks, c)
        stack = M.CachedGlobalTransformerStack(c, 384, heads, blocks).to(dev)
        stack.load_state_dict(w, strict=True)
        args = (a.to(dev), s.to(dev), pitched[:, :, :blocks], mask.to(dev))
        with torch.autocast("cuda", dtype=torch.bfloat16):
            stack(*args)
            before = L.launch_count()
            out = stack(*args)
            launches.append(L.launch_count() - before)
        ref = _oracle_on(dev, O.global_transformer_stack, a, s.expand(groups, 1, l, 384), bias[:, :, :blocks], mask, w, heads, blocks)
        _compare(out.float().cpu(), ref, False, f"token stack L={l}, {pattern}")
    assert launches[1] - launches[0] <= 7, launches


def test_a_block_with_a_mask_shared_by_its_complexes(dev):
    """(1, N) for two complexes: operator by operator, to the rounding of the bf16 results between them what the one call gives."""
    from kfold_b200 import modules as M
    g = torch.Generator(device=dev).manual_seed(3)
    n = 41
    z, s = (torch.randn(*shape, generator=g, device=dev).bfloat16() for shape in ((2, n, n, 128), (2, n, 384)))
    m = (torch.arange(n, device=dev) < n - 5).unsqueeze(0)
    pm = (m[:, :, None] & m[:, None, :]).expand(2, n, n)
    with torch.device(dev):
        blk = M.PairformerBlock(128, 384)
    for got, ref in zip(blk(z, s, pm, m), blk(z, s, pm, m.expand(2, n))):
        _check(*err_stats(got.float(), ref.float()), "shared mask")


@pytest.mark.parametrize("n,batch,c", [(24, 1, 64), (63, 2, 128), (65, 1, 256), (129, 1, 128), (200, 1, 256), (450, 1, 256)])
def test_trimul_statistics_of_the_contraction(dev, n, batch, c):
    """The output projection's LayerNorm statistics, taken by its kernel or (c = 256 beyond L2) by a pass: row counts around the tiles,
    two, four and eight stages per tile, several column tiles."""
    from kfold_b200 import functional as F
    from kfold_b200 import packing
    import synth
    z, pm, _ = synth.pair_inputs(n, n, c, batch, pad_frac=0.1)
    w = synth.trimul_weights(synth._Rng(n), c)
    zb = z.bfloat16()
    for direction in ("outgoing", "incoming"):
        out = F.triangle_multiplication(zb.to(dev), pm.to(dev), packing.pack_trimul(w, dev), direction).float().cpu()
        _check(*err_stats(out, _oracle_on(dev, O.triangle_multiplication, zb.float(), pm, w, direction)), f"trimul {direction} N={n} C={c}")


@pytest.mark.parametrize("n,batch", [(33, 2), (70, 1)])
def test_block_with_a_mask_that_is_not_symmetric(dev, n, batch):
    """Starting and ending node read the pair mask along its two directions; one launch scans both."""
    from kfold_b200 import modules as M
    import synth
    z, pm, m = synth.pair_inputs(n, n, 128, batch)
    s = synth.single_inputs(n, n, 384, batch)
    pm = pm & (torch.arange(n)[:, None] + 7 > torch.arange(n) // 2) & (torch.arange(n) != 3)
    w = synth.pairformer_block_weights(n)
    blk = M.PairformerBlock().to(dev)
    blk.load_state_dict(w, strict=True)
    zb, sb = z.bfloat16(), s.bfloat16()
    zo, so = blk(zb.to(dev), sb.to(dev), pm.to(dev), m.to(dev))
    zr, sr = O.pairformer_block(zb.float(), sb.float(), pm, m, w)
    _check(*err_stats(zo.float().cpu(), zr), "z")
    _check(*err_stats(so.float().cpu(), sr), "s")


@pytest.mark.parametrize("b,m,n,k", [(1, 19000, 512, 520), (1, 9601, 1024, 600), (3, 6500, 776, 712), (20, 1100, 520, 520), (40, 200, 512, 640)])
def test_gemm_of_cta_pairs(dev, b, m, n, k):
    """Tiles of two CTAs: even and odd counts of row blocks, rows, columns and K that end inside a tile, one and several waves."""
    from kfold_b200 import _lib as L
    g = torch.Generator(device=dev).manual_seed(m)
    a = torch.randn(b, m, k, generator=g, device=dev).bfloat16()
    w = torch.randn(b, n, k, generator=g, device=dev).bfloat16()
    d = torch.full((b, m, n), float("nan"), device=dev, dtype=torch.bfloat16)
    L.check(L.lib().kfb_gemm_bf16(L.ptr(a), L.ptr(w), L.ptr(d), None, b, m, n, k, k, k, n, m * k, n * k, m * n, 0, L.stream_ptr()))
    prev = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = False
    ref = torch.matmul(a.float(), w.float().transpose(1, 2))
    torch.backends.cuda.matmul.allow_tf32 = prev
    # identical bf16 operands and float32 sums on both sides; the result is off by half a unit in its last place, 2^-9 of itself
    assert ((d.float() - ref).abs() <= 1e-4 * k ** 0.5 + 2.0 ** -8 * ref.abs()).all()


@pytest.mark.parametrize("rows", [9473, 9601, 19200])
def test_transition_of_cta_pairs(dev, rows):
    """Gated tiles and tiles with a prefetched residual, at 75, 76 and 150 row blocks."""
    from kfold_b200 import functional as F
    from kfold_b200 import packing
    import synth
    w = synth.transition_weights(synth._Rng(rows), 256, 4)
    x = torch.randn(1, rows, 256, generator=torch.Generator().manual_seed(rows)).bfloat16()
    out = F.transition(x.to(dev), packing.pack_transition(w, dev), residual=True).float().cpu()
    _check(*err_stats(out, x.float() + _oracle_on(dev, O.transition, x.float(), w)), f"transition rows={rows}")


@pytest.mark.parametrize("m,n,k,ldd,shift,bias", [(9472, 512, 520, 512, 0, None), (9601, 776, 712, 776, 0, 0), (9601, 776, 712, 777, 0, None),
                                                  (9473, 520, 456, 528, 4, None), (9600, 512, 448, 512, 0, 1)],
                         ids=["one wave", "ragged columns with bias", "odd pitch", "destination off by 8 bytes", "bias off by 4 bytes"])
def test_gemm_of_cta_pairs_with_one_epilogue_group(dev, m, n, k, ldd, shift, bias):
    """Tiles of two CTAs that one group of warps takes: exactly one wave of them, or columns that the copy engine cannot store.  Nothing
    is written between the rows."""
    from kfold_b200 import _lib as L
    g = torch.Generator(device=dev).manual_seed(m + n)
    a = torch.randn(m, k, generator=g, device=dev).bfloat16()
    w = torch.randn(n, k, generator=g, device=dev).bfloat16()
    col_bias = None if bias is None else torch.randn(n + 4, generator=g, device=dev)[bias:bias + n]
    buf = torch.full((m * ldd + 16,), 7.0, device=dev, dtype=torch.bfloat16)
    d = buf[shift:shift + m * ldd].view(m, ldd)
    L.check(L.lib().kfb_gemm_bf16(L.ptr(a), L.ptr(w), L.ptr(d), L.ptr(col_bias), 1, m, n, k, k, k, ldd, 0, 0, 0, 0, L.stream_ptr()))
    prev = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = False
    ref = torch.matmul(a.float(), w.float().T) + (0.0 if col_bias is None else col_bias)
    torch.backends.cuda.matmul.allow_tf32 = prev
    # (the bound of the test above)
    assert ((d[:, :n].float() - ref).abs() <= 1e-4 * k ** 0.5 + 2.0 ** -8 * ref.abs()).all()
    assert (d[:, n:] == 7.0).all() and (buf[:shift] == 7.0).all() and (buf[shift + m * ldd:] == 7.0).all()


def test_gated_tiles_of_cta_pairs_in_one_wave(dev):
    """37 row blocks of pairs x 2 gated tiles: one for each pair that 148 multiprocessors hold."""
    from kfold_b200 import functional as F
    from kfold_b200 import packing
    import synth
    w = synth.transition_weights(synth._Rng(3), 256, 1)
    x = torch.randn(1, 9472, 256, generator=torch.Generator().manual_seed(3)).bfloat16()
    out = F.transition(x.to(dev), packing.pack_transition(w, dev)).float().cpu()
    _check(*err_stats(out, _oracle_on(dev, O.transition, x.float(), w)), "transition in one wave of pairs")


@pytest.mark.parametrize("m,n,k", [(1, 384, 1536), (64, 32, 520), (96, 768, 768), (130, 772, 1096), (300, 1024, 2048)])
def test_gemm_with_k_shared_by_a_cluster(dev, m, n, k):
    """Few rows, float32 results: rows, columns and K that end inside a tile, shares of K of unequal length, one to three row blocks."""
    from kfold_b200 import _lib as L
    g = torch.Generator(device=dev).manual_seed(m)
    a = torch.randn(m, k, generator=g, device=dev).bfloat16()
    w = torch.randn(n, k, generator=g, device=dev).bfloat16()
    bias = torch.randn(n, generator=g, device=dev)
    d = torch.full((m, n), float("nan"), device=dev)
    L.check(L.lib().kfb_gemm_bf16(L.ptr(a), L.ptr(w), L.ptr(d), L.ptr(bias), 1, m, n, k, k, k, n, 0, 0, 0, 1, L.stream_ptr()))
    ref = a.double() @ w.double().T + bias.double()
    # products of bf16 numbers are exact; each of the K / 16 steps cuts the running sum, at most 6 sqrt(K) here, to 24 bits
    assert (d - ref).abs().max() <= k / 16 * 2.0 ** -23 * 6 * k ** 0.5


@pytest.mark.parametrize("n,batch,c,heads", [(8, 1, 128, 16), (24, 2, 256, 16), (40, 1, 128, 6), (136, 2, 128, 16)])
@pytest.mark.parametrize("transposed", [0, 1])
def test_pair_bias_in_one_pass(dev, n, batch, c, heads, transposed):
    """Rows that end inside a warp's sixteen, fewer heads than a fragment holds, both orders of the two positions."""
    from kfold_b200 import _lib as L
    g = torch.Generator(device=dev).manual_seed(n)
    z = torch.randn(batch, n, n, c, generator=g, device=dev).bfloat16()
    w = (torch.randn(heads, c, generator=g, device=dev) * c ** -0.5).bfloat16()
    lw, lb = 1 + 0.1 * torch.randn(c, generator=g, device=dev), 0.1 * torch.randn(c, generator=g, device=dev)
    out = torch.full((batch, heads, n, n), float("nan"), device=dev, dtype=torch.bfloat16)
    ws = torch.empty(L.lib().kfb_pair_bias_workspace_bytes(batch, n, c), dtype=torch.uint8, device=dev)
    L.check(L.lib().kfb_pair_bias_fwd(L.ptr(z), L.ptr(lw), L.ptr(lb), L.ptr(w), L.ptr(out), L.ptr(ws), ws.numel(), batch, n, c, heads, transposed,
                                      1e-5, 0, L.stream_ptr()))
    ref = torch.einsum("bijc,hc->bhij", torch.nn.functional.layer_norm(z.double(), (c,), lw.double(), lb.double(), 1e-5), w.double())
    ref = ref.transpose(-1, -2) if transposed else ref
    # operands and result are rounded to bf16, 2^-9 of themselves each: the sum's error stays within six sigma of c independent roundings
    assert (out.double() - ref).abs().max() <= 2.0 ** -8 * ref.abs().max() + 6 * 2.0 ** -9


@pytest.mark.parametrize("l,samples,c", [(96, 1, 768), (301, 2, 1024), (700, 3, 768), (1000, 4, 128), (64, 3, 256), (130, 1, 384)])
def test_adaln_behind_its_projection_in_a_captured_graph(dev, l, samples, c):
    """A replay has the projection of the gate / shift rows and the AdaLN that reads them back to back; every replay gets another
    conditioning, so that rows read too early are the last replay's.  One and several rows per warp, up to 592 blocks and more, and
    the kernel for other widths."""
    from kfold_b200 import modules as M
    from kfold_b200.graphs import GraphedCall
    g = torch.Generator().manual_seed(l)
    mod = M.AdaLN(c, 384)
    w = {k: torch.randn(p.shape, generator=g) * (p.shape[-1] ** -0.5 if p.dim() == 2 else 0.1) + (1.0 if k == "layernorm_s.weight" else 0.0)
         for k, p in mod.state_dict().items()}
    mod.load_state_dict(w, strict=True)
    mod = mod.to(dev)

    def three(a_, s_):
        with torch.autocast("cuda", dtype=torch.bfloat16):
            return tuple(mod(a_, s_[i]) for i in range(3))

    a = torch.randn(1, samples, l, c, generator=g)
    graphed = GraphedCall(three, a.to(dev), torch.zeros(3, 1, 1, l, 384, device=dev))
    for _ in range(3):
        s = torch.randn(3, 1, 1, l, 384, generator=g)
        outs = graphed(a.to(dev), s.to(dev))
        for i in range(3):
            ref = _oracle_on(dev, O.adaln, a, s[i].expand(1, samples, l, 384).contiguous(), w)
            _check(*err_stats(outs[i].float().cpu(), ref), f"AdaLN L={l} x {samples}, C={c}")


@pytest.mark.parametrize("n,batch,c", [(24, 1, 64), (65, 2, 128), (40, 1, 256)])
def test_nothing_is_written_past_the_reported_workspace(dev, monkeypatch, n, batch, c):
    """A caller may pass an arena whose tail holds something else: the triangle multiplication by itself, and in a block, whose workspace
    has room for its folded weights, leave that tail as it was and give the same result."""
    from kfold_b200 import functional as F
    from kfold_b200 import modules as M
    from kfold_b200 import packing
    import synth
    arenas = []

    def arena(device, nbytes, most_kept=None):
        arenas.append((torch.full((nbytes + tail,), 0xAB, dtype=torch.uint8, device=device), nbytes))
        return arenas[-1][0]

    monkeypatch.setattr(F, "_workspace", arena)
    z, pm, _ = synth.pair_inputs(n, n, c, batch)
    z, pm = z.bfloat16().to(dev), pm.to(dev)
    pk = packing.pack_trimul(synth.trimul_weights(synth._Rng(n), c), dev)
    torch.manual_seed(n)
    block = M.TriangularBlock(c).to(dev)
    for call in (lambda: F.triangle_multiplication(z, pm, pk, "outgoing"), lambda: F.triangle_multiplication(z, pm, pk, "incoming"),
                 lambda: block(z, pm)):
        results = []
        for tail in (0, 1 << 20):
            results.append(call())
            ws, nbytes = arenas[-1]
            assert (ws[nbytes:] == 0xAB).all()
        assert torch.equal(*results)


@pytest.mark.parametrize("rows", [1, 23, 9472, 20001])
@pytest.mark.parametrize("bf16", [False, True])
def test_atom_rows_of_128_channels(dev, rows, bf16):
    """The coordinate embedding and the projection to updates at 128 channels: one row, rows that leave a pair's second empty, as many as
    warps, more than go round once; masked atoms; three samples that share features and mask."""
    from kfold_b200 import _lib as L
    lib, samples = L.lib(), 3
    g = torch.Generator(device=dev).manual_seed(rows)
    rnd = lambda *shape: torch.randn(shape, generator=g, device=dev)
    dt, code = (torch.bfloat16, L.KFB_BF16) if bf16 else (torch.float32, L.KFB_FP32)
    mask = torch.rand(rows, generator=g, device=dev) < 0.8
    q, r, w = rnd(rows, 128).to(dt), rnd(samples, rows, 3), rnd(128, 3)
    out = torch.full((samples * rows * 128 + 8,), 7.0, device=dev)
    L.check(lib.kfb_coord_embed(L.ptr(q), L.ptr(r), L.ptr(w), L.ptr(mask), L.ptr(out), samples * rows, 128, 3, samples, rows, code, L.stream_ptr()))
    rm = r.double() * mask[:, None]
    ref = q.double() + rm @ w.double().T
    assert ((out[:-8].view(samples, rows, 128) - ref).abs() <= 4 * 2.0 ** -24 * (q.double().abs() + rm.abs() @ w.double().abs().T)).all()
    assert (out[-8:] == 7.0).all()
    x, lw, lb, wo = (rnd(samples * rows, 128) * 2 + 0.5).to(dt), rnd(128), rnd(128), rnd(3, 128)
    upd = torch.full((samples * rows * 3 + 8,), 7.0, device=dev)
    L.check(lib.kfb_ln_project(L.ptr(x), L.ptr(lw), L.ptr(lb), L.ptr(wo), L.ptr(mask), L.ptr(upd), samples * rows, 128, 3, 1e-5, samples, rows, code,
                               L.stream_ptr()))
    xn = torch.nn.functional.layer_norm(x.double(), (128,), lw.double(), lb.double(), 1e-5)
    ref = (xn @ wo.double().T).view(samples, rows, 3) * mask[:, None]
    # 128 products and a normalisation in float32
    assert ((upd[:-8].view(samples, rows, 3) - ref).abs() <= 2e-6 * (xn.abs() @ wo.double().abs().T).view(samples, rows, 3)).all()
    assert (upd[-8:] == 7.0).all()
