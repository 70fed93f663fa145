"""Pair list of the binary64 step (``pp_pairs`` in the C ABI).

Both directions of a bond have the same length, stretch and, up to the sign,
direction cosines, bit for bit.  With a pair list the step computes each bond
once (``pp_pair_step``): one kernel over the pairs, one that sums every
node's slots in the reference's order.  The results are those of
``pp_fused_step``.
"""
import ctypes

from . import _lib
from ._lib import check, lib

#: Rows of at most this many slots are one load a lane in the one-kernel step,
#: which a second kernel beats only from ``MIN_BONDS`` directed bonds (one step,
#: one kernel against pairs: 23,000 bonds 5.2 against 6.0 us, 81,000 bonds 7.1
#: against 7.3, 97,000 bonds 7.7 against 7.4, 111,000 bonds 12.3 against 7.8,
#: 6.1M bonds 352 against 182).  Wider rows are a serial loop over their slots
#: there, so pairs are faster at every size (rows of 64: 39,000 bonds 7.7
#: against 6.4 us, 94,000 bonds 9.6 against 7.6; rows of 128: 6,800 bonds 9.8
#: against 6.8, 167,000 bonds 14.5 against 9.3, 2.9M bonds 139 against 76,
#: 42.7M bonds 1,959 against 954; rows of 256: 121,000 bonds 18.5 against
#: 9.7, 3.6M bonds 153 against 93).
NARROW = 32
MIN_BONDS = 100_000

_MAX_SLOTS = 2 ** 31 - 1
_MAX_PAIRS = 2 ** 30 - 1
_SMALL_BYTES = 2 ** 25
#: Slots, length, vector and two records.
_PAIR_BYTES = 8 + 8 + 24 + 64


def worthwhile(nnodes, max_neigh, bonds, device, steps=None):
    """Is the pair form of the fused step used for a model of this size?
    ``bonds`` counts the directed bonds, ``steps`` the run's steps where they
    are known."""
    return ((max_neigh > NARROW or bonds >= MIN_BONDS)
            and _repays(bonds, steps)
            and fits(nnodes, max_neigh, bonds, device))


def _repays(bonds, steps):
    """Do the steps of a run repay the list, which takes 0.1 ms (more, with many
    bonds) to build?  Calls on one kernel and on pairs break even at 50 steps of
    37,000 bonds, 27 of 167,000, 7 of 418,000, 4 to 6 of a million, 5 of 3.6
    million and 2 of 10.6 million; calls of one step take 0.79 against 0.89 ms
    (37,000 bonds), 1.01 against 1.12 (418,000) and 4.72 against 4.94 (10.6
    million)."""
    return steps is None or steps >= 2 + 6_000_000 / (bonds + 80_000)


def cy_worthwhile(nnodes, width, bonds, device, steps=None):
    """The same for PeriPy's CPU integrator, whose calls break even at 7 steps
    of 37,000 bonds and between 2 and 3 of 167,000; with 891,000 one step is
    faster on pairs (1.50 against 1.61 ms)."""
    return ((steps is None or steps * bonds >= 300_000)
            and fits(nnodes, width, bonds, device))


def fits(nnodes, max_neigh, bonds, device):
    """Do the indices and the memory of a pair list fit?  Its arrays take four
    bytes a slot and up to 52 a bond listed from both ends."""
    slots = nnodes * max_neigh
    return (slots <= _MAX_SLOTS and bonds <= _MAX_PAIRS
            and _room(4 * slots + 52 * bonds, device))


def _room(size, device):
    """May the pair list's arrays take so many bytes?  Half of the device memory
    that is free, and no more; for a small list that is not asked, and what
    torch keeps for reuse is only where the rest does not do (the three
    questions take as long as building the list)."""
    return (size <= _SMALL_BYTES or 2 * size <= _free_bytes(device)
            or 2 * size <= _free_bytes(device) + _cached_bytes(device))


def _free_bytes(device):
    import torch
    return torch.cuda.mem_get_info(device)[0]


def _cached_bytes(device):
    import torch
    return (torch.cuda.memory_reserved(device)
            - torch.cuda.memory_allocated(device))


class DevicePairs:
    """Device arrays of one pair list (see :meth:`build`)."""

    @classmethod
    def build(cls, fargs, device, stream, bonds, two_sided=False):
        """The pair list of the neighbour list (and volumes and corrections) of
        ``fargs``, or None where its arrays do not fit: a bond listed from one
        end only, or more than once, is a pair of its own, with up to twice
        the memory that :func:`fits` expects of ``bonds``.  Queued on ``stream`` (a handle,
        torch's current stream); the call waits for the count of the pairs,
        and for the rest only where the two directions of a bond may share a
        force.  With ``two_sided`` each direction keeps a force of its own,
        whatever the volumes and corrections."""
        import torch
        n, width = int(fargs.nnodes), int(fargs.max_neigh)

        def empty(shape, dtype):
            return torch.empty(shape, dtype=dtype, device=device)

        self = cls()
        args = ctypes.byref(fargs)
        self.slot_pair = empty((n, width), torch.int32)
        start = empty((n + 1,), torch.int32)
        scratch = empty((max(n, 1),), torch.int32)
        check(lib().pp_pair_count(args, self.slot_pair.data_ptr(),
                                  start.data_ptr(), scratch.data_ptr(),
                                  stream), "pp_pair_count")
        npairs = int(start[n].item())
        if npairs > _MAX_PAIRS or (2 * npairs > bonds and not _room(
                _PAIR_BYTES * npairs, device)):
            return None
        self.slots = empty((max(npairs, 1), 2), torch.int32)
        self.length = empty((max(npairs, 1),), torch.float64)
        self.vector = empty((3, max(npairs, 1)), torch.float64)
        s = self.struct = _lib.Pairs()
        s.npairs = npairs
        s.slots = self.slots.data_ptr()
        s.slot_pair = self.slot_pair.data_ptr()
        s.length = self.length.data_ptr()
        s.vector = self.vector.data_ptr()
        check(lib().pp_pair_fill(args, ctypes.byref(s), start.data_ptr(),
                                 scratch.data_ptr(), stream), "pp_pair_fill")
        s.symmetric = int(not two_sided and not fargs.bond_types
                          and scratch[0].item() == 0)
        self.force = empty((max(npairs, 1) * (1 if s.symmetric else 2), 4),
                           torch.float64)
        s.force = self.force.data_ptr()
        return self


class CyPairs:
    """Pair list of PeriPy's CPU integrator (``pp_cy_pairs``), built from the
    compact, symmetric rows of ``step`` (a ``_lib.CyStep``); queued on
    ``stream``, which the call waits for."""

    def __init__(self, step, device, stream):
        import torch
        n, width = int(step.nnodes), int(step.width)

        def empty(shape, dtype):
            return torch.empty(shape, dtype=dtype, device=device)

        self.row_state = empty((max(n, 1),), torch.int32)
        start = empty((n + 1,), torch.int32)
        differ = empty((1,), torch.int32)
        check(lib().pp_cy_pair_count(step.nlist, step.n_neigh, n, width,
                                     self.row_state.data_ptr(),
                                     start.data_ptr(), stream),
              "pp_cy_pair_count")
        npairs = int(start[n].item())
        self.nodes = empty((max(npairs, 1), 2), torch.int32)
        self.slot_pair = empty((max(n * width, 1),), torch.int32)
        self.length = empty((max(npairs, 1),), torch.float64)
        self.position = empty((max(n, 1), 3), torch.float64)
        s = self.struct = _lib.CyPairs()
        s.npairs = npairs
        s.nodes = self.nodes.data_ptr()
        s.slot_pair = self.slot_pair.data_ptr()
        s.length = self.length.data_ptr()
        s.row_state = self.row_state.data_ptr()
        s.position = self.position.data_ptr()
        check(lib().pp_cy_pair_fill(
            step.coords, step.u, step.volume, step.nlist, step.n_neigh, n,
            width, start.data_ptr(), ctypes.byref(s), differ.data_ptr(),
            stream), "pp_cy_pair_fill")
        s.symmetric = int(differ.item() == 0)
        self.term = empty((max(npairs, 1) * (1 if s.symmetric else 2), 4),
                          torch.float64)
        s.term = self.term.data_ptr()
