"""Packed tokenisation of a batch is the padded one without its padding."""
import pytest

from nanoplm_b200.data.tokenizer import ProtTokenizer, StudentTokenizer


@pytest.mark.parametrize("texts", [["A"], [""], ["ACD", "", "Zé\U0001f600x", "M" * 300], ["acgt", "U Z"]])
def test_pack(texts):
    t = StudentTokenizer()
    assert t.packs() and not hasattr(ProtTokenizer(), "packs")
    ids, lens = t.pack(texts)
    enc = t(texts, padding=True, return_tensors="pt")
    keep = enc["attention_mask"].numpy().astype(bool)
    assert ids.tolist() == enc["input_ids"].numpy()[keep].tolist() and lens.tolist() == keep.sum(1).tolist()
    t.encode_np = lambda *a, **k: None
    assert not t.packs()
