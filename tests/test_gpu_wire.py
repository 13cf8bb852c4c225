"""The batched export and import of blocks, bit for bit against the one-block forms: page images, pool
entries, metadata and cursors; tokens with more outliers than the page's slots and overflow list take,
every key grid, blocks off the 16-token grid, a pool that runs out."""

from __future__ import annotations

import numpy as np
import pytest
from test_gpu_readback import H, _context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,frac,vb,dt,w,n", [
    ("nf4_asym", 0.02, 3, "float16", 512, 1500), ("nf4", 0.036, 4, "bfloat16", 512, 1100),
    ("uniform", 0.0, 3, "float32", 512, 800), ("nf4_asym", 0.1, 4, "float16", 100, 500),
    ("uniform", 0.05, 3, "float16", 37, 200), ("nf4_asym", 0.5, 3, "float32", 2, 40)])
def test_batched_export_and_import_equal_the_one_block_forms(mode, frac, vb, dt, w, n):
    import torch

    from turboquant_pro_b200 import KVContext

    src, _, _, kw = _context(torch, w, vb, dt, n, mode=mode, frac=frac, heavy=True)
    nb = src.cold_blocks(n)
    one = [src.export_block(1, 1, b) for b in range(nb)]
    for first, count in ((0, nb), (1, nb - 1)):
        for want, got in zip(one[first:], src._export_blocks(1, 1, first, count), strict=True):
            assert set(want) == set(got)
            for name, x in want.items():
                if isinstance(x, np.ndarray):
                    assert x.dtype == got[name].dtype and x.shape == got[name].shape, name
                    assert x.tobytes() == got[name].tobytes(), name
                else:
                    assert x == got[name], name
    a, b = KVContext(**kw), KVContext(**kw)
    for blk in range(nb):
        a.import_block(1, 1, blk, one[blk])
    b._import_blocks(1, 1, 0, one[:2])
    b._import_blocks(1, 1, 2, one[2:])
    for name in ("pages", "pool_dec", "pool_val", "page_meta", "state"):
        assert torch.equal(a._regions[name], b._regions[name]), name
    if one[0]["outlier_idx"] is not None:
        bad = dict(one[0], outlier_idx=one[0]["outlier_idx"][::-1].copy())
        with pytest.raises(ValueError):
            b._import_blocks(1, 1, 0, [bad])
        # importing the same blocks again and again runs the pool out, in both forms alike
        rounds = {}
        for c, put in ((a, lambda: [a.import_block(1, 1, i, x) for i, x in enumerate(one)]),
                       (b, lambda: b._import_blocks(1, 1, 0, one))):
            c.clear(1, 1)
            for i in range(200):
                try:
                    put()
                except RuntimeError:
                    rounds[c is a] = i
                    break
        assert rounds[True] == rounds[False]
    with pytest.raises(RuntimeError):
        b._import_blocks(1, 1, b.geom.max_blocks, one[:1])


def test_batched_export_of_polarquant_keys():
    import torch

    from turboquant_pro_b200 import KVContext
    from turboquant_pro_b200.synth import make_kv

    k, v = make_kv(2, H, 900, dtype=np.float16)
    src = KVContext(n_kv_heads=H, value_bits=3, key_bits=3, key_mode="polar", outlier_frac=0.0,
                    max_tokens_per_seq=900, kv_dtype="float16", seed=1)
    src.append(0, torch.from_numpy(k)[None].cuda(), torch.from_numpy(v)[None].cuda())
    for b, got in enumerate(src._export_blocks(0, 0, 0, src.cold_blocks(900))):
        want = src.export_block(0, 0, b)
        assert set(want) == set(got)
        for name, x in want.items():
            same = x.tobytes() == got[name].tobytes() if isinstance(x, np.ndarray) else x == got[name]
            assert same, name


def test_imports_of_two_geometries_from_two_threads():
    """The kernel's shared-memory limit is the device's, not the context's: imports of a small page
    beside imports of the largest one."""
    import threading

    import torch

    from turboquant_pro_b200 import KVContext

    jobs, errors = [], []
    for w, vb, n in ((512, 4, 1100), (37, 3, 200)):
        src, _, _, kw = _context(torch, w, vb, "float16", n, frac=0.0)
        blks = [src.export_block(1, 1, b) for b in range(src.cold_blocks(n))]
        jobs.append((KVContext(**kw), blks))

    def work(ctx, blks):
        try:
            for _ in range(1500):
                ctx._import_blocks(1, 1, 0, blks[:1])
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=job) for job in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
