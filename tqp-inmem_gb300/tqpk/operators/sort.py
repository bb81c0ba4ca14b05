"""Drop-in ``tqp_sort`` (operators/sort.py:6-58).

The reference runs one stable torch.sort per key, last key first, each time
gathering the key through ``perm`` (:26-35), then slices ``perm[:limit]``
(:41-42) and gathers every input column (:44-54).  Here that loop is one
tqpk_argsort_keys call; with a limit the stable top-k of the first key, and of
the rows tied at its end by the next keys, returns the same rows as the full sort
followed by the slice.  A [N, w] key (the
reference ranks its rows with unique(dim=0)) is sorted by its 8-byte words,
which gives the same lexicographic order and ties; keys of more words than one
call takes are sorted key by key (tqpk_argsort_stable), last word of the last
key first.  [N, w] columns are gathered row by row.
When every input column comes from one tqp_hash_aggregate call, whose groups are
in ascending key-tuple order, and the sort keys are a prefix of those group keys,
all ascending, the stable sort is the identity: only the limit is applied.
"""
from __future__ import annotations

import torch

from .._lib import CLUSTER_SORT_ROWS, MAX_SORT_WORDS, ONE_CTA_SORT_ROWS, TOPK_MAX
from ..ops import (argsort_keys, argsort_stable, check_deferred, gather, gather_rows, sort_words, string_words, topk_keys,
                   topk_stable)
from ..variable import make_like, wait_ready
from .filter import _require_gpu


def _is_text(col) -> bool:
    return col.dim() == 2 and col.shape[1] > 1


def tqp_sort(gpu_enable, tensor_group, args, with_limit, name="sort"):
    _require_gpu(gpu_enable)
    check_deferred()
    limit = args["limit"] if with_limit else None
    input_ids = args["input ids"]
    rows = tensor_group[input_ids[0]].tensor.shape[0]
    key_ids, key_descs = args["key ids"], args["key orders"]
    k0 = tensor_group[key_ids[0]].tensor
    if k0.numel() * k0.element_size() >= 8_000_000_000:   # sort.py:22-23, 38-39
        raise RuntimeError("sort input exceeds in-memory limit")
    device = k0.device
    order = getattr(tensor_group[input_ids[0]], "_row_order", None)
    if (order is not None and not any(key_descs) and tuple(key_ids) == order[1][:len(key_ids)]
            and all(getattr(tensor_group[c], "_row_order", None) is order
                    and order[2].get(c) == tensor_group[c].tensor.data_ptr() for c in {*input_ids, *key_ids})):
        # every input column holds one group-by's output, whose rows are already in ascending
        # order of these keys: the stable sort is the identity, only the limit is left
        if limit is not None:
            for c in input_ids:
                v = tensor_group[c]
                tensor_group[c] = make_like(v, v.tensor[:limit], v.tensor_type)
        return rows
    wait_ready(*[tensor_group[k] for k in key_ids])
    perm = None                                           # identity until the first pass
    steps = []
    cols = [tensor_group[k].tensor for k in key_ids]
    if len(cols) == len(key_descs) and all(
            c.is_cuda and (c.dim() == 1 or c.shape[1] == 1 or
                           (c.shape[1] > 1 and c.dtype in (torch.int8, torch.uint8))) for c in cols):
        many = list(zip(cols, key_descs))
        words = sort_words(cols)
        few = words <= MAX_SORT_WORDS
        if limit is not None and 0 < limit <= TOPK_MAX and few and words > 1 and cols[0].shape[0] > CLUSTER_SORT_ROWS:
            # the top-k key by key: 6 M rows by a price and a tie-breaking id took 560 us of sorting the
            # ids first.  A table that one cluster sorts in a launch (~30-60 us) is sorted.
            perm = topk_keys(cols, key_descs, limit)
            many, key_ids = [], []
        elif limit is not None:              # all keys but the first, which ends the sort in a top-k
            many = many[1:] if not _is_text(cols[0]) else []
        # one numeric key of few rows: the one-key call below has less to set up (~5 us of a small limit's 100)
        if many and few and (len(many) > 1 or _is_text(many[0][0]) or many[0][0].shape[0] > ONE_CTA_SORT_ROWS):
            perm = argsort_keys([c for c, _ in many], [d for _, d in many])
            key_ids, key_descs = key_ids[:len(key_ids) - len(many)], key_descs[:len(key_descs) - len(many)]
    for key_id, desc in zip(reversed(key_ids), reversed(key_descs)):
        col = tensor_group[key_id].tensor
        if col.dim() == 2 and col.shape[1] > 1:
            if col.dtype not in (torch.int8, torch.uint8):
                raise NotImplementedError(f"2-D sort key of dtype {col.dtype}")
            steps += [(string_words(col, wd), desc) for wd in reversed(range((col.shape[1] + 7) // 8))]
        else:
            steps.append((col.reshape(-1), desc))
    for i, (key, desc) in enumerate(steps):
        last = i == len(steps) - 1
        if last and limit is not None:
            perm = topk_stable(key, limit, desc, perm)
        else:
            perm = argsort_stable(key, desc, perm)
    if perm is None:                                      # no key columns
        perm = torch.arange(rows, device=device, dtype=torch.int64)
    if limit is not None:
        perm = perm[:limit]
    wait_ready(*[tensor_group[k] for k in input_ids])
    flat, shapes = [], []
    for key_id in input_ids:                              # sort.py:44-54
        t = tensor_group[key_id].tensor
        if not t.is_cuda:
            t = t.to(device)
        flat.append(t)
    # every 1-D (or [N, 1]) column in one multi-column gather launch; [N, w] rows by row gather
    one_d = [i for i, t in enumerate(flat) if t.dim() == 1 or (t.dim() == 2 and t.shape[1] == 1)]
    outs = [None] * len(flat)
    if one_d:
        for i, o in zip(one_d, gather([flat[i].reshape(-1) for i in one_d], perm)):
            outs[i] = o.reshape(-1, 1) if flat[i].dim() == 2 else o
    for i, t in enumerate(flat):
        if outs[i] is None:
            outs[i] = gather_rows(t, perm)
    for key_id, out in zip(input_ids, outs):
        tensor_group[key_id] = make_like(tensor_group[key_id], out, tensor_group[key_id].tensor_type)
    return rows
