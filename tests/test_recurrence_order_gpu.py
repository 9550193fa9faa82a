"""linear_recurrence takes up to 32 sequences longest first (two columns per lane): every sequence has its own rows and state,
whatever their number, order and lengths, and wherever the table lies."""
import pytest
import torch

from shuffle_exchange_b200.inference.v2.kernels import mixer_ops as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [[0], [5], [3, 0, 3], [9, 1, 40, 9], list(range(32)), list(range(33)), [1] * 32, [2] * 70])
@pytest.mark.parametrize("shift", [0, 1])
def test_every_sequence_by_itself(rows, shift):
    g = torch.Generator(device="cuda").manual_seed(len(rows))
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    H, n, dv, T, N = 64, 64, 128, max(1, sum(rows)), len(rows)
    k, q, v = mk(T, H * n) / 8, mk(T, H * n), mk(T, H * dv)
    decay, beta = (torch.rand(T, H, generator=g, device="cuda") for _ in range(2))
    state = mk(N, H, dv, n)
    slots = torch.randperm(N, generator=torch.Generator().manual_seed(1)).tolist()
    info = [[sum(rows[:i]), r, i % 2, slots[i]] for i, r in enumerate(rows)]
    table = torch.zeros(4 * N + 4, dtype=torch.int32, device="cuda")[shift: shift + 4 * N].view(N, 4)
    table.copy_(torch.tensor(info, dtype=torch.int32))
    got_state = state.clone()
    got = M.linear_recurrence(k, q, v, decay, beta, None, got_state, table, H, H, n, dv, True)
    for i, (first, r, _, slot) in enumerate(info):         # one at a time: the order of the sums is the same
        one = state.clone()
        want = M.linear_recurrence(k, q, v, decay, beta, None, one, table[i: i + 1].clone(), H, H, n, dv, True)
        assert torch.equal(got[first: first + r], want[first: first + r])
        assert torch.equal(got_state[slot], one[slot])         # without rows, too: kept, or zero where nothing was seen
        if r == 0:
            assert torch.equal(one[slot], state[slot] if i % 2 else torch.zeros_like(state[slot])), i
