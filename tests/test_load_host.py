"""What the decoder is given for a chunk (host side of loading a database)."""
import pytest
import torch

from sseqs_b200 import database


def _forms(chunk):
    n = chunk.numel()
    wide = torch.zeros((n, 3), dtype=torch.uint8)
    wide[:, 1] = chunk
    return {"plain": chunk, "strided": torch.stack([chunk, chunk + 1], 1).reshape(-1)[::2],
            "column": wide[:, 1], "rows": chunk.view(2, -1), "expanded": chunk[:1].expand(n)}


@pytest.mark.parametrize("form", ["plain", "strided", "column", "rows", "expanded"])
def test_decoder_is_given_contiguous_bytes(form, monkeypatch):
    """Every view of a chunk reaches the decoder as its own bytes, one after
    another, on the device that the launch runs on."""
    monkeypatch.setattr(database, "DECODE_ON", "cpu", raising=False)
    chunk = torch.arange(80, dtype=torch.int64).to(torch.uint8)
    view = _forms(chunk)[form]
    seen = []
    monkeypatch.setattr(database.Database, "_add_batch",
                        lambda self, ci, j, ch: seen.append((ci, j, ch)))
    database.Database([view], bs=40, device="cpu")
    assert [(ci, j) for ci, j, _ in seen] == [(0, 0), (0, 1)]
    for _, _, ch in seen:
        assert ch.is_contiguous() and ch.numel() == 80
        assert torch.equal(ch.reshape(-1), view.reshape(-1))


def test_host_held_chunks_are_moved_to_the_decoding_device(monkeypatch):
    """A database kept on one device decodes on the other (here "meta" stands
    for the GPU); the packed chunk stays where it was asked for."""
    monkeypatch.setattr(database, "DECODE_ON", "meta", raising=False)
    seen = []
    monkeypatch.setattr(database.Database, "_add_batch",
                        lambda self, ci, j, ch: seen.append(ch.device.type))
    db = database.Database([torch.zeros(40, dtype=torch.uint8)], bs=40, device="cpu",
                           keep_packed=True)
    assert seen == ["meta"] and db.packed[0].device.type == "cpu"
