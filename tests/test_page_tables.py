"""Page tables of the indexed step: every table that a gather through it serves, and none that it refuses."""
import pytest
import torch

DEV = "cuda:0"


def test_tables_that_the_selection_cannot_read_go_through_the_gather(monkeypatch):
    """A table without a page for every column (no position may be dropped silently), with fewer rows than tokens, of another type
    or with its columns apart."""
    from sparse_mla_sm120_b200 import indexer, pipeline
    took = []

    class Native:
        def topk(self, logits, ks, ke, k, table, page):
            took.append("selection")
            return torch.zeros(logits.shape[0], k, dtype=torch.int32)
    logits = torch.zeros(3, 130)
    monkeypatch.setattr(pipeline, "native", Native)
    monkeypatch.setattr(indexer, "fp8_mqa_logits", lambda *a: logits)
    monkeypatch.setattr(indexer, "topk_indices", lambda lg, ks, ke, k: torch.tensor([[0, 70, -1]] * 3, dtype=torch.int32))
    monkeypatch.setattr(pipeline, "sparse_mla_decode_fwd", lambda q, kv, rows, *a, **k: (rows, rows))
    monkeypatch.setattr(pipeline, "positions_to_rows", lambda *a, real=pipeline.positions_to_rows: (took.append("gather"), real(*a))[1])
    kv = torch.zeros(8, 64, 1, 656, dtype=torch.uint8)

    def run(table):
        took.clear()
        out = pipeline.sparse_mla_indexed_decode_fwd(None, kv, None, None, None, None, None, None, 1.0, topk=3, block_table=table)
        return took[0], out[2]
    table = torch.tensor([[4, 1, 2], [0, 5, 3], [7, 6, 2]], dtype=torch.int32)
    assert run(table)[0] == "selection"
    assert run(table[:1].expand(3, -1))[0] == "selection"
    assert run(torch.cat([table, table]))[0] == "selection"
    assert run(torch.cat([table, table], dim=1)[:, :3])[0] == "selection"
    want = torch.tensor([[256, 70, -1], [0, 326, -1], [448, 390, -1]], dtype=torch.int32)
    for t in (table[:, :2], table[:, :2].contiguous(), table.long(), table.t().contiguous().t()):
        how, rows = run(t)
        assert how == "gather" and torch.equal(rows, want)
    with pytest.raises((RuntimeError, IndexError)):
        run(table[:, :1])                        # position 70 has no page
    with pytest.raises((RuntimeError, IndexError)):
        run(table[:2])                           # token 2 has no table


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["shared", "taller", "view", "overlapping", "short", "int64"])
def test_tables_of_an_indexed_step(kind):
    """The step through each kind of table against the same step through a plain copy of it."""
    from sparse_mla_sm120_b200 import pipeline
    from helpers import make_case
    tokens, keys, page = 5, 1000, 64
    pages = -(-keys // page)
    g = torch.Generator().manual_seed(4)
    case = make_case(2, tokens, 64, 64, pages + 4)
    qi = torch.randn(tokens, 64, 128, generator=g).to(torch.float8_e4m3fn).to(DEV)
    ki = torch.randn(keys, 128, generator=g).to(torch.float8_e4m3fn).to(DEV)
    scale, w = torch.rand(keys, generator=g).to(DEV), torch.randn(tokens, 64, generator=g).to(DEV)
    ks, ke = torch.zeros(tokens, dtype=torch.int32, device=DEV), torch.full((tokens,), keys, dtype=torch.int32, device=DEV)
    perm = lambda n=pages: torch.randperm(pages + 4, generator=g)[:n].to(torch.int32)
    table = torch.stack([perm() for _ in range(tokens + 2)]).to(DEV)
    if kind == "shared":
        table = table[0].unsqueeze(0).expand(tokens, -1)
    elif kind == "view":
        table = torch.cat([table, table], dim=1)[1:1 + tokens, 3:3 + pages]
    elif kind == "overlapping":
        table = torch.as_strided(perm(pages + 4).to(DEV), (tokens, pages), (1, 1))
    elif kind == "short":                        # enough for every window, though not for every key
        ke.fill_(keys - 2 * page)
        table = table[:tokens, :pages - 1].contiguous()
    elif kind == "int64":
        table = table[:tokens].long()

    def step(t):
        out, lse, rows = pipeline.sparse_mla_indexed_decode_fwd(
            case["q"].to(DEV), case["packed"].to(DEV), qi, ki, scale, w, ks, ke, case["sm_scale"], topk=128, block_table=t)
        return out, lse, rows
    plain = torch.zeros(tokens, pages, dtype=torch.int32, device=DEV)
    plain[:, :table.shape[1]] = table[:tokens]
    for a, b in zip(step(table), step(plain)):
        assert torch.equal(a, b)
