"""How the keys of the atoms behind a point of the batch's table are counted (csrc/attention_decode.cu splits by them)."""
import torch

from shuffle_exchange_b200.inference.v2.ragged.ragged_wrapper import RaggedBatchWrapper


class _Seq:
    def __init__(self, seen):
        self.seen_tokens = seen

    def kv_blocks(self):
        return torch.zeros(1, dtype=torch.int32)


def test_keys_of_the_last_atoms():
    w = RaggedBatchWrapper(1024, 8, 4, device="cpu")
    assert w.last_atoms_keys(3) == (0, 0)
    for seen, n in ((0, 300), (77, 1), (2000, 2), (9, 1)):
        w.insert_sequence(_Seq(seen), torch.zeros(n, dtype=torch.int64))
    w.finalize()
    assert w.atoms_longer_than(2) == 3 and w.atoms().shape[0] == 6
    assert w.last_atoms_keys(0) == (0, 0)
    assert w.last_atoms_keys(2) == (78 + 10, 78)
    assert w.last_atoms_keys(3) == (78 + 10 + 2002, 2002)
    assert w.last_atoms_keys(3) == (78 + 10 + 2002, 2002)
    w.clear()
    w.insert_sequence(_Seq(5), torch.zeros(1, dtype=torch.int64))
    w.finalize()
    assert w.last_atoms_keys(1) == (6, 6)                 # of this batch, not of the one before
    w.clear()
    w.finalize()
    assert w.last_atoms_keys(1) == (0, 0)
