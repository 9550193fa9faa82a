"""Host-side assembly of one ragged batch and its upload (reference: ``inference/v2/ragged/ragged_wrapper.py:31-292``).

All metadata of a forward pass lives in ONE pinned int32 staging buffer laid out as
``[token ids | token->sequence | token position | rows whose logits are wanted | block tables | attention atoms |
per-sequence info]`` and
is uploaded with a single ``cudaMemcpyAsync`` in ``finalize`` (the reference uses three pinned "fast host buffers",
``ragged/csrc/fast_host_buffer.cu``).  The attention atoms (one per 128-query tile of a sequence, with the KV extent
it attends to) are cut by the native scheduler ``sxbh_build_atoms`` (``csrc/host/ragged_host.cpp``) at ``finalize``
and consumed by the tensor-core paged attention kernels (``sxb_attn_fwd_atoms_keys``).

The upload is asynchronous and forwards may be queued without a synchronisation between them, so the batches take turns over
``STAGING_BUFFERS`` pinned buffers; a buffer is written again only when the upload that read it has completed.

The tables are filled through numpy views of the staging buffers and the device views are made once per batch: a slice of a
tensor costs 1 to 2 us, and a decode step of 4 requests through 4 layers took some 400 of them (0.95 of 1.2 ms per step)."""
from __future__ import annotations

import numpy as np
import torch

ATOM_Q_BLOCK = 128          # query rows of one attention atom = the kernel's q tile
ATOM_KV_BLOCK = 64
STAGING_BUFFERS = 4


class RaggedBatchWrapper:
    def __init__(self, max_ragged_batch_size: int, max_ragged_sequence_count: int, max_blocks_per_seq: int,
                 device=None) -> None:
        self.max_tokens, self.max_seqs, self.max_blocks = max_ragged_batch_size, max_ragged_sequence_count, max_blocks_per_seq
        self.device = device if device is not None else ("cuda" if torch.cuda.is_available() else "cpu")
        self.max_atoms = self.max_tokens // ATOM_Q_BLOCK + self.max_seqs
        n = 4 * self.max_tokens + self.max_seqs * self.max_blocks + 6 * self.max_atoms + 4 * self.max_seqs
        self._seq_meta = np.zeros((3, self.max_seqs), dtype=np.int32)          # start / in-flight tokens / seen tokens
        pin = torch.cuda.is_available()
        self._staging = [torch.zeros(n, dtype=torch.int32, pin_memory=pin) for _ in range(STAGING_BUFFERS if pin else 1)]
        self._uploaded = [None] * len(self._staging)          # per buffer: event behind the last upload from it
        self._host_views = [self._views(b) for b in self._staging]
        self._tables = [tuple(v.numpy() for v in views) for views in self._host_views]
        self._turn = 0
        self._host = self._staging[0]
        self._dev = torch.zeros(n, dtype=torch.int32, device=self.device)
        self._dev_views = self._views(self._dev)
        self.clear()

    def clear(self) -> None:
        self._n_tokens = 0
        self._n_seqs = 0
        self._n_atoms = 0
        self._n_logit_rows = 0
        self._finalized = False
        self._live = {}                                        # device views of the rows that this batch fills
        if self._uploaded[self._turn] is not None:            # the current buffer is in use by an upload: take the next one
            self._turn = (self._turn + 1) % len(self._staging)
            if self._uploaded[self._turn] is not None:
                self._uploaded[self._turn].synchronize()
                self._uploaded[self._turn] = None
            self._host = self._staging[self._turn]

    def _views(self, buf):
        T, S, B = self.max_tokens, self.max_seqs, self.max_blocks
        e = 4 * T + S * B
        f = e + 6 * self.max_atoms
        return (buf[0:T], buf[T:2 * T], buf[2 * T:3 * T], buf[3 * T:4 * T], buf[4 * T:e].view(S, B),
                buf[e:f].view(self.max_atoms, 6), buf[f:].view(S, 4))

    def insert_sequence(self, seq_descriptor, tokens: torch.Tensor, do_checks: bool = True, logit_rows=None) -> None:
        """``logit_rows``: indices among ``tokens`` whose logits the forward returns (default: the last token)."""
        n = tokens.numel()
        if do_checks:
            if self._n_tokens + n > self.max_tokens:
                raise RuntimeError(f"Ragged batch is full due to tokens: {self._n_tokens} + {n} > {self.max_tokens}")
            if self._n_seqs + 1 > self.max_seqs:
                raise RuntimeError("Ragged batch is full due to sequences")
        ids, t2s, pos, last, tables, _, info = self._tables[self._turn]
        i, seen = self._n_seqs, seq_descriptor.seen_tokens
        a, b = self._n_tokens, self._n_tokens + n
        blocks = seq_descriptor.kv_blocks()
        if (tokens.dim() > 1 and tokens.shape[-1] != n) or b > self.max_tokens or blocks.numel() > self.max_blocks:
            raise RuntimeError(f"tokens {tuple(tokens.shape)} at row {a} with {blocks.numel()} blocks do not fit a batch of "
                               f"{self.max_tokens} rows of tokens and {self.max_blocks} blocks per sequence")
        self._seq_meta[:, i] = (a, n, seen)
        ids[a:b] = tokens.to(device="cpu", dtype=torch.int32).reshape(-1).numpy()
        t2s[a:b] = i
        pos[a:b] = np.arange(seen, seen + n, dtype=np.int32)
        rows = [n - 1] if logit_rows is None else [int(r) for r in logit_rows]
        if any(r < 0 or r >= n for r in rows):
            raise ValueError(f"logit rows {rows} outside the {n} tokens of the sequence")
        for r in rows:
            last[self._n_logit_rows] = a + r
            self._n_logit_rows += 1
        info[i] = (a, n, seen, getattr(seq_descriptor, "state_slot", -1))
        tables[i, : blocks.numel()] = blocks.cpu().numpy()
        self._n_tokens, self._n_seqs = b, i + 1
        self._live = {}

    def finalize(self, padding: bool = False) -> None:
        if self._n_seqs:
            from ..kernels.atom_builder import AtomBuilder
            start, rows, seen = (torch.from_numpy(m[: self._n_seqs]) for m in self._seq_meta)
            _, self._n_atoms = AtomBuilder()(self._host_views[self._turn][5], start, rows, seen, ATOM_Q_BLOCK, ATOM_KV_BLOCK)
            # longest first: the kernels take the short tail (decode tokens, chunk remainders) on its own and need those
            # atoms contiguous; among equal short ones the one with most keys first, so that light ones end the grid
            # (the kernel for the long ones walks them from the end: a sequence's later tiles have more keys)
            live = self._tables[self._turn][5][: self._n_atoms]
            live[:] = live[np.lexsort((np.where(live[:, 2] <= 16, -live[:, 5], 0), -live[:, 2]))]
            self._atom_q_lens, self._atom_keys = live[:, 2].copy(), live[:, 5].copy()
            self._last_keys = {}
        self._live = {}
        self._dev.copy_(self._host, non_blocking=True)
        if self._dev.is_cuda:
            ev = self._uploaded[self._turn] = torch.cuda.Event()
            ev.record()
        self._finalized = True

    # device views ------------------------------------------------------------------------------
    def _rows(self, table: int, n: int) -> torch.Tensor:
        v = self._live.get(table)
        if v is None:
            v = self._live[table] = self._dev_views[table][:n]
        return v

    def input_ids(self):
        return self._rows(0, self._n_tokens)

    def token_to_seq(self):
        return self._rows(1, self._n_tokens)

    def token_positions(self):
        return self._rows(2, self._n_tokens)

    def last_token_index(self):
        """Batch rows whose logits are returned: every sequence's last token unless ``insert_sequence`` named others."""
        return self._rows(3, self._n_logit_rows)

    def seq_info(self):
        """int32 ``[n_seqs, 4]`` on the device: (first row, rows, tokens seen before this forward, state slot or -1)."""
        return self._rows(6, self._n_seqs)

    def host_seq_info(self):
        return self._host_views[self._turn][6][: self._n_seqs]

    def block_tables(self):
        return self._dev_views[4]

    def atoms(self):
        """int32 ``[n_atoms, 6]`` on the device: ``(seq, q_start_idx, q_len, global_q_idx, kv_blocks, total_extent)``."""
        return self._rows(5, self._n_atoms)

    def atoms_longer_than(self, q_len: int) -> int:
        """How many (leading) atoms have more than ``q_len`` queries; host-side, no synchronisation."""
        return int(np.count_nonzero(self._atom_q_lens > q_len)) if self._n_atoms else 0

    def last_atoms_keys(self, n: int):
        """``(keys that the last n atoms see together, keys that the longest of them sees)``; host-side, looked up once per
        batch."""
        if not self._n_atoms or n <= 0:
            return 0, 0
        got = self._last_keys.get(n)
        if got is None:
            keys = self._atom_keys[-n:]
            got = self._last_keys[n] = int(keys.sum(dtype=np.int64)), int(keys.max())
        return got

    def single_rows(self) -> bool:
        """Whether every sequence of the batch brings exactly one token (a pure decode step); host-side."""
        return self._n_tokens == self._n_seqs

    @property
    def current_tokens(self) -> int:
        return self._n_tokens

    @property
    def current_sequences(self) -> int:
        return self._n_seqs
