"""Attention kernels with TMA multicast are for programs of one rank: every way in which a program comes to have several closes
them, wherever its keys and values lie."""
import os
import socket
import subprocess
import sys

import pytest
import torch.distributed as dist
import torch.multiprocessing as mp

from shuffle_exchange_b200.comm import comm
from shuffle_exchange_b200.native import lib


def _open():
    return lib.load().sxb_attn_note_ranks(1)


def _rank(rank, world, port, way):
    for k in ("RANK", "WORLD_SIZE", "LOCAL_RANK"):
        os.environ.pop(k, None)
    group = dict(init_method=f"tcp://127.0.0.1:{port}", rank=rank, world_size=world)
    if way != "before the library":
        assert _open() == 1
    if way == "own group":
        dist.init_process_group("gloo", **group)
        lib.call = lambda *a: None                # the kernel itself wants a GPU
        lib.attn_call("sxb_attn_fwd")
    else:
        comm.init_distributed(dist_backend="gloo", verbose=False, **group)
    assert _open() == (1 if world == 1 else 0)
    dist.destroy_process_group()
    assert _open() == (1 if world == 1 else 0)    # peers' mappings may outlive the group


@pytest.mark.parametrize("way", ["framework", "own group", "before the library"])
@pytest.mark.parametrize("world", [1, 2])
def test_a_group_of_several_ranks_closes_them(way, world):
    with socket.socket() as s:
        s.bind(("127.0.0.1", 0))
        port = s.getsockname()[1]
    mp.spawn(_rank, (world, port, way), nprocs=world)


@pytest.mark.parametrize("world,want", [("1", 1), ("8", 0)])
def test_a_launcher_that_starts_several_ranks_closes_them(world, want):
    code = "from shuffle_exchange_b200.native import lib; print(lib.load().sxb_attn_note_ranks(1))"
    r = subprocess.run([sys.executable, "-c", code], env={**os.environ, "WORLD_SIZE": world}, capture_output=True, text=True)
    assert r.stdout.strip().endswith(str(want)), r.stderr
