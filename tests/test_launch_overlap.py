"""When kernels without a partner on another GPU may be scheduled while the kernel before them still runs: not in a process that has a
communicator of several ranks, whose collectives let their successors start before they wait for their peers."""
import pytest

from mp_util import run_ranks


def _rank(rank, nranks, uid):
    from nccl_b200 import Communicator, _lib, get_unique_id
    lib = _lib.load()
    got = [lib.b200PlainLaunchesOverlap()]
    alone = Communicator(1, 0, get_unique_id())
    got.append(lib.b200PlainLaunchesOverlap())
    comm = Communicator(nranks, rank, uid)
    got.append(lib.b200PlainLaunchesOverlap())
    child = comm.split(0, rank)
    comm.destroy()
    got.append(lib.b200PlainLaunchesOverlap())   # the child has the ranks too
    single = child.split(rank, 0)
    child.destroy()
    got.append(lib.b200PlainLaunchesOverlap())
    single.destroy()
    alone.destroy()
    try:
        Communicator(nranks, nranks, uid)   # no such rank
    except Exception:
        pass
    return got + [lib.b200PlainLaunchesOverlap()]


@pytest.mark.parametrize("setting,want", [("1", [1, 1, 0, 0, 1, 1]), ("0", [0] * 6), ("2", [1] * 6)])
def test_plain_launches_overlap_only_without_peers(setting, want):
    env = {"NCCL_B200_HOST_ONLY": "1", "NCCL_SOCKET_IFNAME": "lo", "NCCL_B200_PDL": setting}
    assert list(run_ranks(_rank, 2, env=env, timeout=120).values()) == [want, want]
