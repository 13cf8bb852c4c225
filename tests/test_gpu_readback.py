"""Read-back, bit for bit: ranges that begin and end inside the kernel's tiles, for blocks shorter
than a tile, than a 16-token group and off their grids, against the C restatement; the restore into an
engine's pages against the dense read-back rounded by torch."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H = 2


def _context(torch, w, vb, dt, n, seed=3, mode="nf4_asym", frac=0.02, heavy=False):
    from turboquant_pro_b200 import KVContext
    from turboquant_pro_b200.synth import make_kv

    k, v = make_kv(seed, H, n, dtype=np.float32)
    if heavy:  # tokens with more outliers than fixed slots, and more than the overflow list takes
        k[3, 0, :40] = 90.0 + np.arange(40)
        k[5:12, 1, :] = 200.0
    kw = dict(n_layers=2, n_seqs=2, n_kv_heads=H, n_q_heads=H, value_bits=vb, hot_window=w,
              max_tokens_per_seq=n + 8, kv_dtype=dt, seed=seed, key_mode=mode, outlier_frac=frac)
    ctx = KVContext(**kw)
    kt, vt = (torch.from_numpy(x).to(getattr(torch, dt)) for x in (k, v))
    ctx.append(1, kt[None].cuda(), vt[None].cuda(), seq_begin=1)
    return ctx, kt.float().numpy(), vt.float().numpy(), kw


@pytest.mark.parametrize("w,n", [(512, 1130), (100, 333), (64, 200), (37, 150), (9, 61), (2, 9)])
@pytest.mark.parametrize("vb", [3, 4])
def test_ranges_equal_the_restatement(w, n, vb):
    import torch

    from oracle import c_oracle as co
    from oracle import tq_oracle as orc

    ctx, k, v, _ = _context(torch, w, vb, "float16", n)
    s = orc.block_tokens(w)
    cent, bnd = orc.value_tables(128, vb)
    keys, vals = [], []
    nb = orc.n_cold_blocks(n, w)
    for b in range(nb):
        kb = co.encode_keys(np.ascontiguousarray(np.moveaxis(k[b * s:(b + 1) * s], 0, 1)),
                            orc.outlier_count(s, 0.02))
        vc = co.encode_values(np.ascontiguousarray(np.moveaxis(v[b * s:(b + 1) * s], 0, 1)),
                              np.ascontiguousarray(ctx.pi.T), bnd)
        keys.append(co.dequant_keys(kb["codes"], kb["scale"], kb["mean"], kb["out_idx"],
                                    kb["out_val"]))
        vals.append(co.dequant_values(vc["codes"], vc["norms"], cent, ctx.pi))
    keys = np.concatenate(keys + [np.moveaxis(k[nb * s:], 0, 1)], axis=1)
    vals = np.concatenate(vals + [np.moveaxis(v[nb * s:], 0, 1)], axis=1)
    cold = nb * s
    cuts = {(0, n), (0, 1), (n - 1, n), (cold - 1, cold), (cold - 1, min(cold + 1, n)), (cold, n),
            (s // 2, min(cold, s + 1)), (3, min(3 + 33, n)), (1, cold)}
    for a, b in sorted(cuts):
        gk, gv = ctx.dequant(1, 1, a, b)
        ok = [np.array_equal(got.cpu().numpy().view(np.uint32), want[:, a:b].view(np.uint32))
              for got, want in ((gk, keys), (gv, vals))]
        assert all(ok), (a, b, ok)
    assert torch.equal(ctx.dequant(1, 1, 1, n, values=False)[0].cpu(), torch.from_numpy(keys[:, 1:]))
    assert torch.equal(ctx.dequant(1, 1, 1, n, keys=False)[1].cpu(), torch.from_numpy(vals[:, 1:]))


@pytest.mark.parametrize("dt", ["float16", "bfloat16", "float32"])
@pytest.mark.parametrize("layout", ["plain", "heads_first", "off_grid", "other_type"])
def test_restore_into_pages_equals_the_dense_read_back(dt, layout):
    import torch

    from turboquant_pro_b200.connector import DeviceBlockStore
    from turboquant_pro_b200.synth import make_kv

    n, bs, pages = 777, 7, 120
    kind = getattr(torch, dt)
    store = DeviceBlockStore(2, H, max_requests=1, max_tokens=n, value_bits=3, dtype=dt, seed=4)
    k, v = (torch.from_numpy(x).to(kind).cuda() for x in make_kv(8, H, n))
    assert store.save("r", 1, k, v)
    if layout == "heads_first":     # [2, pages, H, bs, D] seen as [2, pages, bs, H, D]
        kv = torch.zeros((2, pages, H, bs, 128), dtype=kind, device="cuda").transpose(2, 3)
    elif layout == "off_grid":      # rows of odd length, beginning at an odd element
        kv = torch.zeros((2, pages, bs, H, 131), dtype=kind, device="cuda")[..., 1:129]
    elif layout == "other_type":    # float64 pages take the general path
        kv = torch.zeros((2, pages, bs, H, 128), dtype=torch.float64, device="cuda")
    else:
        kv = torch.zeros((2, pages, bs, H, 128), dtype=kind, device="cuda")
    want = kv.clone()
    table = torch.randperm(pages, generator=torch.Generator().manual_seed(1))[:-(-n // bs) + 2]
    table[3] -= pages               # an index counted from the end
    kd, vd = store.load("r", 1)
    pos = torch.arange(n)
    blk, row = table[pos // bs].cuda(), (pos % bs).cuda()
    want[0][blk, row] = kd.permute(1, 0, 2).to(kv.dtype)
    want[1][blk, row] = vd.permute(1, 0, 2).to(kv.dtype)
    for ids in (table.int().cuda(), table.tolist()):
        kv.zero_()
        before = kv._version
        assert store.load_into_paged("r", 1, kv, ids) == n
        assert torch.equal(kv, want) and kv._version > before
    with pytest.raises(ValueError):
        store.load_into_paged("r", 1, kv, table[:-(-n // bs) - 1])
    assert store.load_into_paged("r", 0, kv, table) == 0


@pytest.mark.parametrize("mode", ["nf4_asym", "polar"])
def test_tokens_of_a_page_outside_the_tensor_are_left_out(mode):
    import torch

    from turboquant_pro_b200 import KVContext
    from turboquant_pro_b200.synth import make_kv

    n, bs, pages = 777, 7, 120
    polar = mode == "polar"
    ctx = KVContext(n_kv_heads=H, value_bits=3, key_bits=3 if polar else 4, key_mode=mode,
                    outlier_frac=0.0 if polar else 0.02, max_tokens_per_seq=n, kv_dtype="float16", seed=4)
    k, v = (torch.from_numpy(x)[None].cuda() for x in make_kv(8, H, n, dtype=np.float16))
    ctx.append(0, k, v)
    kv = torch.zeros((2, pages, bs, H, 128), dtype=torch.float16, device="cuda")
    ids = torch.randperm(pages, generator=torch.Generator().manual_seed(1))[:-(-n // bs)]
    ctx.dequant_into_pages(0, 0, n, kv[0], kv[1], ids.cuda())
    assert ctx.status() == 0
    want = kv.clone()
    bad = ids.clone()
    for at, i in ((2, pages), (5, -1), (40, -(1 << 40)), (len(ids) - 1, 1 << 40)):
        want[:, ids[at]] = 0.0  # (cold pages and one of the window)
        bad[at] = i
    kv.zero_()
    ctx.dequant_into_pages(0, 0, n, kv[0], kv[1], bad.cuda())
    assert torch.equal(kv, want)
    assert ctx.status() == 4 and ctx.status() == 0


def test_pages_that_are_more_than_their_storage():
    """What indexing the pages refuses, negates or differentiates, the restore does too."""
    import torch
    from torch.autograd import forward_ad

    from turboquant_pro_b200.connector import DeviceBlockStore
    from turboquant_pro_b200.synth import make_kv

    n, bs, pages = 600, 16, 60
    store = DeviceBlockStore(1, H, max_requests=1, max_tokens=n, value_bits=3, dtype="float16", seed=4)
    assert store.save("r", 0, *(torch.from_numpy(x).cuda() for x in make_kv(8, H, n, dtype=np.float16)))
    table = torch.randperm(pages, generator=torch.Generator().manual_seed(1))[:-(-n // bs)].cuda()

    def fresh():
        return torch.zeros((2, pages, bs, H, 128), dtype=torch.float16, device="cuda")

    want = fresh()
    store.load_into_paged("r", 0, want, table)
    assert want.any()
    kv = torch._neg_view(fresh())
    store.load_into_paged("r", 0, kv, table)
    assert torch.equal(kv.resolve_neg(), want)
    with torch.inference_mode():
        kv = fresh()
        store.load_into_paged("r", 0, kv, table)
        assert torch.equal(kv, want)
    with pytest.raises(RuntimeError, match="[Ii]nference"):
        store.load_into_paged("r", 0, kv, table)
    with forward_ad.dual_level():
        kv = forward_ad.make_dual(fresh(), fresh() + 1.0)
        store.load_into_paged("r", 0, kv, table)
        primal, tangent = forward_ad.unpack_dual(kv)
        assert torch.equal(primal, want) and not tangent[:, table[0]].any()
    stack = torch.stack([fresh(), fresh()])
    torch.func.vmap(lambda x: (store.load_into_paged("r", 0, x, table), x)[1])(stack)
    assert torch.equal(stack[0], want) and torch.equal(stack[1], want)
