"""Predicate trees and their flat submission format.

A predicate is a tree of ``Cmp`` / ``In`` / ``And`` / ``Or`` / ``Not`` nodes
over attribute column slots. ``serialize`` flattens one tree exactly like
the engine's ``fv_pred_serialize`` (engine.cpp:1168-1224): nodes in the
pre-order of ``copy_tree`` (engine.cpp:600-622, node 0 is the root),
children and IN values in side arrays addressed by ``child0`` / ``val0``.
``concat`` joins per-query slices and rebases them like ``GpuConcat::build``
(engine.cpp:1232-1282) into the arrays ``fv_gpu_brute_batch`` /
``fv_gpu_graph_batch`` take.

Evaluation semantics (engine.cpp:397-431): NULL values are stored as NaN and
every comparison with NaN is false; ``NE`` is ``v == v and v != c``.
"""
from __future__ import annotations

import struct
from dataclasses import dataclass, field
from typing import List, Optional, Sequence

import numpy as np

from ._lib import (FV_CMP_EQ, FV_CMP_GE, FV_CMP_GT, FV_CMP_LE, FV_CMP_LT, FV_CMP_NE,
                   FV_NODE_AND, FV_NODE_CMP, FV_NODE_IN, FV_NODE_NOT, FV_NODE_OR, NODE_DTYPE,
                   QD_DTYPE, SPAN_DTYPE)

OPS = {"<": FV_CMP_LT, "<=": FV_CMP_LE, "==": FV_CMP_EQ, ">=": FV_CMP_GE, ">": FV_CMP_GT,
       "!=": FV_CMP_NE}


class Pred:
    def __and__(self, other):
        return And(self, other)

    def __or__(self, other):
        return Or(self, other)

    def __invert__(self):
        return Not(self)


@dataclass(frozen=True)
class Cmp(Pred):
    col: int
    op: str
    value: float

    def __post_init__(self):
        if self.op not in OPS:
            raise ValueError(f"unknown comparison {self.op!r}")


@dataclass(frozen=True)
class In(Pred):
    col: int
    values: tuple

    def __init__(self, col, values):
        object.__setattr__(self, "col", col)
        object.__setattr__(self, "values", tuple(float(v) for v in values))


class And(Pred):
    def __init__(self, *children):
        self.children = list(children)

    def __repr__(self):
        return "And(" + ", ".join(map(repr, self.children)) + ")"


class Or(Pred):
    def __init__(self, *children):
        self.children = list(children)

    def __repr__(self):
        return "Or(" + ", ".join(map(repr, self.children)) + ")"


class Not(Pred):
    def __init__(self, child):
        self.children = [child]

    def __repr__(self):
        return f"Not({self.children[0]!r})"


def to_json(p: Optional[Pred]):
    """A JSON-able nested list form of a tree (None = no filter)."""
    if p is None:
        return None
    if isinstance(p, Cmp):
        return ["cmp", p.col, p.op, p.value]
    if isinstance(p, In):
        return ["in", p.col, list(p.values)]
    kind = {And: "and", Or: "or", Not: "not"}[type(p)]
    return [kind] + [to_json(c) for c in p.children]


def from_json(j) -> Optional[Pred]:
    """Inverse of to_json."""
    if j is None:
        return None
    k = j[0]
    if k == "cmp":
        return Cmp(int(j[1]), j[2], float(j[3]))
    if k == "in":
        return In(int(j[1]), j[2])
    kids = [from_json(c) for c in j[1:]]
    if k == "not":
        return Not(kids[0])
    return (And if k == "and" else Or)(*kids)


@dataclass
class Serialized:
    nodes: np.ndarray     # NODE_DTYPE
    children: np.ndarray  # int32
    invals: np.ndarray    # float64


_record = struct.Struct("<8id").pack  # one NODE_DTYPE record
_query = struct.Struct("<5iIQ").pack  # one QD_DTYPE record
assert struct.calcsize("<8id") == NODE_DTYPE.itemsize
assert struct.calcsize("<5iIQ") == QD_DTYPE.itemsize
_KIND = {And: FV_NODE_AND, Or: FV_NODE_OR, Not: FV_NODE_NOT}


def _i32(v) -> int:
    if type(v) is int:  # (packing refuses what is beyond 32 bits)
        return v
    cell = np.zeros(1, np.int32)
    cell[0] = v  # refuses and converts as an assignment to a record does
    return int(cell[0])


def _flat_all(trees, recs: list, children: list, invals: list) -> list:
    """_flat of each tree (None: -1), refusing what a record cannot hold."""
    try:
        return [-1 if p is None else _flat(p, recs, children, invals) for p in trees]
    except struct.error as e:
        raise OverflowError(str(e)) from None


def _flat(n: Pred, recs: list, children: list, invals: list, at=(0, 0, 0)) -> int:
    """Appends a tree's records, children and IN values (node 0 = root,
    pre-order; indexes count from `at`) and returns its root's place. Records
    are packed bytes: assigning numpy records field by field took 20 us a
    filter, most of a 512-filter batch's time."""
    i, c0, v0 = len(recs) - at[0], len(children) - at[1], len(invals) - at[2]
    if isinstance(n, Cmp):
        v = n.value if type(n.value) is float else float(np.float64(n.value))
        recs.append(_record(FV_NODE_CMP, _i32(n.col), OPS[n.op], 0, c0, 0, v0, 0, v))
    elif isinstance(n, In):
        recs.append(_record(FV_NODE_IN, _i32(n.col), 0, 0, c0, len(n.values), v0, 0, 0.0))
        invals.extend(n.values)
    else:
        kind, kids = _KIND[type(n)], n.children
        recs.append(_record(kind, 0, 0, len(kids), c0, 0, v0, 0, 0.0))
        j = len(children)
        children.extend(kids)  # their places, once they have them
        for k in kids:
            children[j] = _flat(k, recs, children, invals, at)
            j += 1
    return i


def serialize(p: Pred) -> Serialized:
    """One tree -> flat arrays, node 0 = root (pre-order)."""
    recs, children, invals = [], [], []
    _flat_all([p], recs, children, invals)
    return Serialized(np.frombuffer(b"".join(recs), NODE_DTYPE).copy(),
                      np.asarray(children, np.int32), np.asarray(invals, np.float64))


@dataclass
class BatchPred:
    """Concatenated, rebased predicate arrays of one batch (GpuConcat)."""
    qd: np.ndarray
    nodes: np.ndarray
    children: np.ndarray
    invals: np.ndarray
    spans: np.ndarray
    spanoff: np.ndarray
    dedup: np.ndarray
    roots: np.ndarray = field(default=None)  # int32 per query (qd.proot)


def concat(preds: Sequence[Optional[Pred]], count: int,
           entries: Optional[Sequence[int]] = None) -> BatchPred:
    nq = len(preds)
    if type(count) is int and 0 <= count < 2 ** 64:
        qd = np.frombuffer(bytearray(_query(-1, 1, 0, 0, 0, 0, count) * nq), QD_DTYPE)
    else:
        qd = np.zeros(nq, QD_DTYPE)
        qd["proot"] = -1
        qd["need_eval"] = 1
        qd["total"] = count
    if entries is not None:
        e = entries
        if isinstance(e, (list, tuple, range)):
            e = np.asarray(e, qd["entry"].dtype)
        if isinstance(e, np.ndarray) and e.ndim == 1:
            if len(e) < nq:
                raise IndexError(f"{len(e)} entry nodes for {nq} queries")
            qd["entry"] = e[:nq]
        else:  # whatever takes an index
            for q in range(nq):
                qd[q]["entry"] = entries[q]
    recs, children, invals = [], [], []
    if nq - sum(p is None for p in preds) <= 8:
        # a few filters: every query's slice in place (the gather below costs
        # 45 us whatever the batch)
        roots = _flat_all(preds, recs, children, invals)
        if recs:
            qd["proot"] = roots
        return BatchPred(qd, np.frombuffer(bytearray(b"".join(recs)), NODE_DTYPE),
                         np.array(children, np.int32), np.array(invals, np.float64),
                         np.zeros(0, SPAN_DTYPE), np.zeros(0, np.uint64), np.zeros(nq, np.uint8),
                         np.array(roots, np.int32))
    # each distinct tree once, then every query's slice gathered from it with
    # its indexes moved to the slice's place
    place, size = {}, [(0, 0, 0)]  # tree -> its number; running ends of the three arrays
    which = []
    try:
        for p in preds:
            if p is None:
                which.append(-1)
                continue
            i = place.get(id(p))
            if i is None:
                i = place[id(p)] = len(place)
                _flat(p, recs, children, invals, size[-1])
                size.append((len(recs), len(children), len(invals)))
            which.append(i)
    except struct.error as e:
        raise OverflowError(str(e)) from None
    which = np.asarray(which, np.int64)
    has = which >= 0
    w = which[has]
    nodes = np.frombuffer(b"".join(recs), NODE_DTYPE)
    children = np.asarray(children, np.int32)
    invals = np.asarray(invals, np.float64)
    end = np.asarray(size, np.int64)
    start, length = end[:-1][w], np.diff(end, axis=0)[w]
    base = np.cumsum(length, axis=0) - length  # where each query's slices begin
    qd["proot"][has] = base[:, 0]

    def gather(a, k):
        n = length[:, k]
        return a[np.repeat(start[:, k] - base[:, k], n) + np.arange(int(n.sum()))]

    nodes = gather(nodes, 0)
    nodes["child0"] += np.repeat(base[:, 1], length[:, 0]).astype(np.int32)
    nodes["val0"] += np.repeat(base[:, 2], length[:, 0]).astype(np.int32)
    children = gather(children, 1) + np.repeat(base[:, 0], length[:, 1]).astype(np.int32)
    return BatchPred(qd, nodes, children, gather(invals, 2), np.zeros(0, SPAN_DTYPE),
                     np.zeros(0, np.uint64), np.zeros(nq, np.uint8),
                     qd["proot"].astype(np.int32))


def eval_numpy(p: Optional[Pred], cols: np.ndarray) -> np.ndarray:
    """Boolean mask of rows satisfying p; cols is [ncols, N] float64. Used by
    host-side tooling (selectivity estimates, workload construction)."""
    n = cols.shape[1]
    if p is None:
        return np.ones(n, bool)
    with np.errstate(invalid="ignore"):
        if isinstance(p, Cmp):
            v = cols[p.col]
            c = p.value
            return {"<": v < c, "<=": v <= c, "==": v == c, ">=": v >= c, ">": v > c,
                    "!=": (v == v) & (v != c)}[p.op]
        if isinstance(p, In):
            v = cols[p.col]
            m = np.zeros(n, bool)
            for x in p.values:
                m |= v == x
            return m
        if isinstance(p, And):
            m = np.ones(n, bool)
            for c in p.children:
                m &= eval_numpy(c, cols)
            return m
        if isinstance(p, Or):
            m = np.zeros(n, bool)
            for c in p.children:
                m |= eval_numpy(c, cols)
            return m
        if isinstance(p, Not):
            return ~eval_numpy(p.children[0], cols)
    raise TypeError(p)
