"""The selection plan (nsa_selection_plan_build) entry by entry, on both sides of the line between its one-launch and
three-launch builders."""
import pytest
import torch

from oracle import nsa_oracle as O
from tests.util import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,Hkv,G,T,S", [(1, 2, 4, 63, 3), (1, 1, 16, 64, 16), (2, 2, 3, 513, 5), (1, 2, 2, 1100, 16),
                                         (1, 1, 4, 2047, 16), (1, 1, 4, 2048, 16), (1, 1, 4, 2049, 16), (13, 5, 2, 200, 4)])
def test_every_entry(B, Hkv, G, T, S):
    nsa = pkg()
    L, lib = nsa._lib, nsa.lib()
    units, n_kt, nq, chunk = B * Hkv, (T + 63) // 64, 128 // G, 128
    idx = O.make_block_idx(B, Hkv, T, 64, S, seed=3)
    idx[:, :, ::5, -1] = idx[:, :, ::5, 0]                       # named twice: one pair
    idx[:, :, ::7, 0] = n_kt + 1                                 # after the query: no pair
    dims = L.dims(B, Hkv * G, Hkv, T, 64, L.DTYPE_BF16)
    n = lib.nsa_selection_plan_bytes(dims, S, 64)
    buf = torch.full((n,), 0x7f, dtype=torch.uint8, device="cuda")
    L.check(lib.nsa_selection_plan_build(L.ptr(idx.int().cuda()), dims, S, 64, L.ptr(buf), n, L.stream()))
    raw = buf.cpu()
    max_items = n_kt + n_kt // chunk + T * S // (chunk * nq) + 2
    at = 0

    def take(count, dtype=torch.int32):
        nonlocal at
        size = count * torch.empty(0, dtype=dtype).element_size()
        v = raw[at:at + size].view(dtype)
        at += (size + 255) // 256 * 256
        return v
    hdr = take(32, torch.int64)
    n_items = take(units)
    items = take(units * max_items * 4).view(units, max_items, 4)
    offsets = take(units * (n_kt + 1)).view(units, n_kt + 1)
    pairs, pos = take(units * T * S), take(units * T * S).view(units, T, S)
    lists = idx.view(units, T, S)
    nq_union = 128 // (1 << (G - 1).bit_length())
    n_pairs = union = 0
    for u in range(units):
        queries = [[] for _ in range(n_kt)]
        seen = set()
        for t in range(T):
            for j in sorted({int(x) for x in lists[u, t] if 0 <= x and 64 * x <= t}):
                queries[j].append(t)
                seen.add((t // nq_union, j))
        start = u * T * S
        want = []
        for j in range(n_kt):
            assert offsets[u, j] == start
            got = pairs[start:start + len(queries[j])]
            assert (got & 0xffffff).tolist() == queries[j] and ((got >> 24) & 0xf == 0xf).all()
            chunks = max(1, -(-(-(-len(queries[j]) // nq)) // chunk))
            want += [[u, j, chunk * k, chunks] for k in range(chunks)]
            start += len(queries[j])
        assert offsets[u, n_kt] == start and n_items[u] == len(want) and items[u, :len(want)].tolist() == want
        n_pairs += start - u * T * S
        union += len(seen)
        place = {(int(p) & 0xffffff, j): o for j in range(n_kt) for o, p in
                 zip(range(offsets[u, j], offsets[u, j + 1]), pairs[offsets[u, j]:offsets[u, j + 1]].tolist())}
        for t in range(0, T, 1 if T < 2000 else 37):
            named = set()
            for s in range(S):
                j = int(lists[u, t, s])
                ok = j >= 0 and 64 * j <= t and j not in named
                named.add(j)
                assert pos[u, t, s] == (place[t, j] if ok else -1)
    assert hdr[0] == union and hdr[1] == n_pairs and hdr[2] == 0      # (repeats count on smaller blocks only)
