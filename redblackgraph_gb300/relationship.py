"""Relationship lookups on closed red/black graphs, on the GPU.

``calculate_relationship(a, b)`` mirrors redblackgraph/reference/calc_relationship.py:54-71:
for two rows of a transitive closure the common ancestor is the first index minimising
``a[j] + b[j]`` among the indices where both rows are non-zero, and the relationship name
comes from the generational distances MSB(a[j]) and MSB(b[j]) (lookup_relationship,
:23-51).  The sums wrap in the rows' dtype, as the numpy scalars of the reference's rows do
(the unsigned red one, the dtype's maximum, plus y gives y - 1).  The search runs in
``rbg_relationship_lookup`` (one CTA per query); ``lookup_many`` answers a whole batch of
(matrix, u, v) queries on resident device matrices in one launch.
"""
from __future__ import annotations

from dataclasses import dataclass
from typing import Sequence

import numpy as np
import torch

from . import _lib
from .device import numpy_dtype, require_cuda, stream_handle, to_device


@dataclass
class Relationship:
    """(common ancestor, name): redblackgraph/types/relationship.py:4-7."""
    common_ancestor: int
    relationship: str


def msb(x: int) -> int:
    """Bit position of the leading bit; 0 for x <= 1 (redblackgraph/reference/rbg_math.py:1-11)."""
    x = int(x)
    return x.bit_length() - 1 if x > 1 else 0


def _cousinth(generational: int) -> str:
    return {2: "1st cousin", 3: "2nd cousin", 4: "3rd cousin"}.get(generational,
                                                                    f"{generational - 1}th cousin")


def _grandparentith(removal: int) -> str:
    return {4: "2nd", 5: "3rd"}.get(removal, f"{removal - 2}th")


def relationship_name(da: int, db: int) -> str:
    """Name from the generational distances of u and v to their common ancestor
    (calc_relationship.py:23-51, including its rough edges)."""
    removal = abs(da - db)
    if da == 0 or db == 0:
        return {1: "parent", 2: "grandparent", 3: "great grandparent"}.get(
            removal, f"{_grandparentith(removal)} great grandparent")
    generational = min(da, db)
    if generational == 1 and removal == 0:
        return "sibling"
    if generational == 1 and removal == 1:
        return "aunt/uncle"
    if removal == 0:
        return _cousinth(generational)
    return f"{_cousinth(generational)} {removal} removed"


def decode(out: np.ndarray, dtypes) -> list[Relationship]:
    """Relationships from the raw (count, 3) lookup results and each query's matrix dtype."""
    x, y = out[:, 1].tolist(), out[:, 2].tolist()
    dtypes = list(dtypes)
    if any(np.dtype(dt).kind == "u" for dt in set(dtypes)):   # the raw results hold the values' bits
        mask = [0xFFFFFFFFFFFFFFFF if np.dtype(dt).kind == "u" else -1 for dt in dtypes]
        x, y = [a & m for a, m in zip(x, mask)], [b & m for b, m in zip(y, mask)]
    # the two MSBs (msb() in line)
    keys = [((a.bit_length() - 1 if a > 1 else 0), (b.bit_length() - 1 if b > 1 else 0)) for a, b in zip(x, y)]
    names: dict = {}
    res = []
    for j, key in zip(out[:, 0].tolist(), keys):
        if j >= 0:
            name = names.get(key)
            if name is None:
                name = names[key] = relationship_name(*key)
            res.append(Relationship(j, name))
        elif j == -2:
            raise IndexError("relationship query out of range")
        else:
            res.append(Relationship(-1, "No Relationship"))
    return res


def lookup_table(table_dev: torch.Tensor, count: int, stream=None) -> np.ndarray:
    """Run the lookups described by a device array of ``count`` rbg_lookup_t; returns the raw
    (count, 3) int64 results on the host."""
    out = torch.empty((max(count, 1), 3), dtype=torch.int64, device=table_dev.device)
    L = _lib.load()
    _lib.check(L.rbg_relationship_lookup(count, table_dev.data_ptr(), out.data_ptr(), stream_handle(stream)),
               "relationship_lookup")
    return out[:count].cpu().numpy()


_LOOKUP_DTYPE = np.dtype(_lib.RbgLookup)     # rbg_lookup_t


def lookup_many(queries, stream=None) -> list[Relationship]:
    """Answer many queries ``(W, u, v)`` (W a 2-D device tensor with contiguous rows, u and v two
    of its row indices) with one kernel launch."""
    queries = list(queries)
    if not queries:
        return []
    dev = queries[0][0].device
    # the fields of each distinct matrix once (`queries` holds the tensors), the vertices as columns
    mats, dts, seen = [], [], {}
    which, us, vs = [], [], []
    for W, u, v in queries:
        k = seen.get(id(W))
        if k is None:
            if W.ndim != 2 or not W.is_cuda or (W.shape[1] > 1 and W.stride(1) != 1):
                raise ValueError("queries take 2-D CUDA matrices with contiguous rows")
            dt = numpy_dtype(W.dtype)
            k = seen[id(W)] = len(mats)
            mats.append((W.data_ptr(), W.stride(0), W.shape[0], W.shape[1], 0, 0, _lib.dtype_code(dt), 0))
            dts.append(dt)
        rows, u, v = mats[k][2], int(u), int(v)
        if not (0 <= u < rows and 0 <= v < rows):
            raise IndexError(f"vertices ({u}, {v}) outside a matrix of {rows} rows")
        which.append(k)
        us.append(u)
        vs.append(v)
    table = np.array(mats, dtype=_LOOKUP_DTYPE)
    if len(mats) < len(which):           # else every query has a matrix of its own, in order
        table, dts = table[which], [dts[k] for k in which]
    table["u"] = us
    table["v"] = vs
    return decode(lookup_table(to_device(table.view(np.uint8), dev), len(queries), stream), dts)


def calculate_relationship(a: Sequence[int], b: Sequence[int]) -> Relationship:
    """Relationship between u and v given their closure rows a and b (calc_relationship.py:54-71)."""
    a = np.asarray(a)
    b = np.asarray(b)
    if a.shape != b.shape or a.ndim != 1:
        raise ValueError("a and b must be rows of the same length")
    dt = np.result_type(a.dtype, b.dtype)
    if dt.kind not in "iu":
        dt = np.dtype(np.int64)
    if a.size == 0:
        return Relationship(-1, "No Relationship")
    W = to_device(np.ascontiguousarray(np.stack([a.astype(dt), b.astype(dt)])), require_cuda())
    return lookup_many([(W, 0, 1)])[0]
