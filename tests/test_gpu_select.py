"""Top-k selection where its dispatch and its tiles change: rows on a cluster of CTAs, on one CTA, windows of a few columns,
ragged ends, more than one stretch per row, distributions on which the sampled threshold fails; and the page table."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def _rows(kind, rows, cols, g):
    x = torch.randn(rows, cols, generator=g)
    if kind == "ties":
        x = (x * 2).round() / 2
    elif kind == "constant":
        x = torch.full((rows, cols), 0.25)
    elif kind == "negative":
        x = -x.abs() - 1.0
    elif kind == "clustered":                    # the best entries all in one place, which the sample may miss
        x[:, cols // 3:cols // 3 + 300] += 50.0
    return x


@pytest.mark.parametrize("rows", [1, 37, 38, 149])
@pytest.mark.parametrize("cols,k", [(5, 8), (8063, 2048), (8070, 512), (40001, 2048), (131075, 2048)])
@pytest.mark.parametrize("kind", ["normal", "ties", "constant", "negative", "clustered"])
def test_selected_sets(rows, cols, k, kind):
    from sparse_mla_sm120_b200 import indexer
    if rows > 37 and (cols > 50000 or kind in ("negative", "clustered")):
        pytest.skip("the many-row kernels are covered at the smaller sizes")
    g = torch.Generator().manual_seed(rows + cols)
    x = _rows(kind, min(rows, 4), cols, g).repeat(-(-rows // min(rows, 4)), 1)[:rows].contiguous()
    ks = torch.randint(0, max(cols // 10, 1), (rows,), generator=g, dtype=torch.int32)
    ke = torch.randint(cols - cols // 10, cols + 1, (rows,), generator=g, dtype=torch.int32)
    ke[0] = ks[0]                                # an empty window
    got = indexer.topk_indices(x.to(DEV), ks.to(DEV), ke.to(DEV), k).cpu()
    cols_i = torch.arange(cols)
    masked = torch.where((cols_i >= ks[:, None]) & (cols_i < ke[:, None]), x, float("-inf"))
    for r in range(rows):
        # the oracle's choice with ties broken towards the lower column: a stable sort of the values
        order = torch.sort(masked[r], descending=True, stable=True).indices[:k]
        b = order[masked[r][order] > float("-inf")]
        a = got[r]
        assert torch.equal(torch.sort(a[a >= 0]).values.long(), torch.sort(b).values), r
        n = int((a >= 0).sum())
        assert bool((a[n:] == -1).all())         # padding last


@pytest.mark.parametrize("rows,cols,page", [(3, 5000, 64), (16, 20000, 48), (160, 3000, 64)])
def test_rows_through_a_page_table(rows, cols, page):
    from sparse_mla_sm120_b200 import indexer, pipeline
    from sparse_mla_sm120_b200._lib import native
    g = torch.Generator().manual_seed(5)
    x = torch.randn(rows, cols, generator=g).to(DEV)
    pages = -(-cols // page)
    table = torch.stack([torch.randperm(pages, generator=g) for _ in range(rows)]).to(torch.int32).to(DEV)
    ke = torch.full((rows,), cols - 100, dtype=torch.int32, device=DEV)
    ke[1] = 7
    got = native().topk(x, None, ke, 512, table, page)
    want = pipeline.positions_to_rows(indexer.topk_indices(x, None, ke, 512), table, page)
    assert torch.equal(got, want)
    wide = torch.zeros(rows, pages + 3, dtype=torch.int32, device=DEV)
    wide[:, :pages] = table
    assert torch.equal(native().topk(x, None, ke, 512, wide[:, :pages], page), want)


def test_copies_of_a_step():
    from sparse_mla_sm120_b200._lib import native
    g = torch.Generator().manual_seed(6)
    shapes = [(3, 128, 576), (7,), (5, 3), (1,), (33, 17), (0,), (9,), (2, 2), (4,)]
    src = [torch.randint(0, 255, s, generator=g, dtype=torch.uint8).to(DEV) for s in shapes]
    src[2] = torch.randn(5, 3, device=DEV)
    src[3] = torch.randn(1, dtype=torch.float64)                       # another type, from the host
    src[4] = torch.randint(0, 255, (17, 33), dtype=torch.uint8, device=DEV).t()        # not contiguous
    dst = [torch.zeros(s, dtype=torch.float32 if i in (2, 3) else torch.uint8, device=DEV) for i, s in enumerate(shapes)]
    native().copy_into(dst, src)
    for a, b in zip(dst, src):
        assert torch.equal(a, b.to(DEV).to(a.dtype))
    with pytest.raises(TypeError):
        native().copy_into(dst, src[:-1])


def test_copies_that_touch_each_other_run_in_order():
    """A destination that is also a source, or another destination: as if copied one after the other; a copy onto part of itself is
    refused, as Tensor.copy_ refuses it; a tensor onto itself is left alone."""
    from sparse_mla_sm120_b200._lib import native
    n = 1 << 22                                                        # many blocks per copy
    a, b, c = (torch.arange(n, device=DEV, dtype=torch.int32) * k for k in (1, 3, 7))
    want = a.clone()
    native().copy_into((b, c, a), (a, b, c))                           # a chain: everything becomes a
    for t in (a, b, c):
        assert torch.equal(t, want)
    native().copy_into((c, c), (torch.zeros_like(c), a * 5))           # the later one stays
    assert torch.equal(c, a * 5)
    native().copy_into((a, b), (a, c))
    assert torch.equal(a, want) and torch.equal(b, c)
    with pytest.raises(RuntimeError):
        native().copy_into((a[1:],), (a[:-1],))
    with pytest.raises(RuntimeError):
        a[1:].copy_(a[:-1])
