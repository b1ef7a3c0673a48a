"""Host-side helpers for the KDA path: device guard and the varlen index tables."""
from __future__ import annotations

import numpy as np
import torch

from . import _native

CHUNK = 64


def assert_blackwell(device=None):
    """Same guard as the reference's ``assert_blackwell`` (cula/utils.py:61-69): the kernels are
    compiled for sm_100a only."""
    if not torch.cuda.is_available():
        raise RuntimeError("cula_b200 needs a CUDA device (B200, sm_100a); there is no CPU fallback.")
    major, _ = torch.cuda.get_device_capability(device)
    if major != 10:
        raise RuntimeError(f"cula_b200 kernels are built for sm_100a; found compute capability {major}.x")


def prepare_chunk_indices(seqlens_cpu, chunk_size=CHUNK):
    """[NT, 2] int32 rows (sequence, chunk inside the sequence), sequence after sequence -- the table
    of fla.ops.utils.index.prepare_chunk_indices (fla/ops/utils/index.py:138-149) used at
    cula/kda/chunk.py:62-64."""
    lens = seqlens_cpu[1:] - seqlens_cpu[:-1]
    n_chunks = (lens + chunk_size - 1) // chunk_size
    seq = torch.repeat_interleave(torch.arange(len(lens), dtype=torch.int64), n_chunks)
    starts = torch.cumsum(n_chunks, 0) - n_chunks
    local = torch.arange(int(n_chunks.sum()), dtype=torch.int64) - torch.repeat_interleave(starts, n_chunks)
    return torch.stack([seq, local], dim=1).to(torch.int32)


def prepare_chunk_offsets(seqlens_cpu, chunk_size=CHUNK):
    """[N+1] int32: first global chunk of every sequence (cula/ops/chunk_delta_h.py:42-47)."""
    lens = seqlens_cpu[1:] - seqlens_cpu[:-1]
    n_chunks = (lens + chunk_size - 1) // chunk_size
    return torch.cat([torch.zeros(1, dtype=torch.int64), torch.cumsum(n_chunks, 0)]).to(torch.int32)


def prepare_uniform_cu_seqlens(batch, seqlen, device=None):
    """cu_seqlens of a fixed-length batch (cula/utils.py:215-218)."""
    return torch.arange(0, (batch + 1) * seqlen, seqlen, dtype=torch.int32, device=device)


class VarlenTables:
    """Device copies of the index tables of one packed batch."""

    def __init__(self, cu_seqlens, cu_seqlens_cpu=None):
        cpu = (cu_seqlens_cpu if cu_seqlens_cpu is not None else cu_seqlens.cpu()).to(torch.int64)
        if cpu.ndim != 1 or cpu.numel() < 1 or int(cpu[0]) != 0 or bool((cpu[1:] < cpu[:-1]).any()):
            raise ValueError("cu_seqlens must be a non-decreasing 1-D tensor starting at 0")
        # all tables in one host buffer and one copy: a new packed batch pays for this before its first launch
        bounds = cpu.numpy()
        lens = bounds[1:] - bounds[:-1]
        n = len(lens)
        n_chunks = (lens + CHUNK - 1) // CHUNK
        offsets = np.concatenate([[0], np.cumsum(n_chunks)])
        NT = int(offsets[-1])
        host = np.empty(3 * n + 2 + 2 * NT, dtype=np.int32)
        indices = host[:2 * NT].reshape(NT, 2)                      # (sequence, chunk inside the sequence)
        indices[:, 0] = np.repeat(np.arange(n), n_chunks)
        indices[:, 1] = np.arange(NT) - np.repeat(offsets[:-1], n_chunks)
        host[2 * NT:2 * NT + n + 1] = offsets
        host[2 * NT + n + 1:2 * NT + 2 * n + 2] = bounds
        # longest sequences first: their CTAs start first and the short ones fill in behind them
        host[2 * NT + 2 * n + 2:] = np.argsort(-lens, kind="stable")
        device = torch.from_numpy(host).to(cu_seqlens.device)
        self.n_seqs, self.num_chunks, self.total_tokens = n, NT, int(bounds[-1])
        self.chunk_indices = device[:2 * NT].view(NT, 2)
        self.chunk_offsets, self.cu_seqlens, self.seq_order = device[2 * NT:].split([n + 1, n + 1, n])
        self.seqlens_cpu = cpu
        self._native = self._segments = None

    @property
    def native(self):
        """The same tables as the host extension takes them."""
        if self._native is None:
            self._native = _native.host().Tables(self.cu_seqlens, self.chunk_indices, self.chunk_offsets, self.seq_order,
                                                 self.n_seqs, self.num_chunks, self.total_tokens)
        return self._native

    @property
    def segments(self):
        """The sequences of these tables as the side-by-side segments of one long sequence."""
        if self._segments is None:
            self._segments = _native.host().Segments(self.n_seqs, self.native)
        return self._segments


_TABLE_CACHE: list = []      # (source tensor, its version, cu_seqlens_cpu or None, tables), most recent last


def get_varlen_tables(cu_seqlens, cu_seqlens_cpu=None) -> VarlenTables:
    """Tables cached by tensor IDENTITY, as the reference caches its chunk indices (fla's ``tensor_cache``): an entry
    holds a reference to the caller's ``cu_seqlens`` tensor itself, so its address cannot be handed to another tensor
    while the entry lives, and is matched with ``is`` plus the tensor's version counter (an in-place edit
    invalidates it). Avoids a device->host sync on every call."""
    version = cu_seqlens._version
    for i in range(len(_TABLE_CACHE) - 1, -1, -1):
        src, ver, cpu, tab = _TABLE_CACHE[i]
        if src is cu_seqlens and ver == version and (cu_seqlens_cpu is None or cpu is None or cpu is cu_seqlens_cpu
                                                     or torch.equal(cpu, cu_seqlens_cpu)):
            return tab
    tab = VarlenTables(cu_seqlens, cu_seqlens_cpu)
    _TABLE_CACHE.append((cu_seqlens, version, cu_seqlens_cpu, tab))
    if len(_TABLE_CACHE) > 16:
        del _TABLE_CACHE[0]
    return tab
