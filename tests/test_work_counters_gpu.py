"""streamed_entries and streamed_chunked (needs a GB300) against their definition: the shorter list of
every edge an owner counts, the head's list of every edge counted at its tail, and the same once per
chunk of the owner's table: 2048 keys, or with split lists 256 of those that are not hubs."""
import numpy as np
import pytest

from katric_gb300 import Config

pytestmark = pytest.mark.gpu


def csr(n, e):
    src, dst = np.concatenate([e[:, 0], e[:, 1]]), np.concatenate([e[:, 1], e[:, 0]])
    order = np.argsort(src * n + dst)
    fo = np.zeros(n + 1, dtype=np.uint64)
    fo[1:] = np.cumsum(np.bincount(src, minlength=n))
    return fo, src[order], dst[order]


def ring_and_clique(ring, half, clique):
    v = np.arange(ring)
    i, j = np.triu_indices(clique, 1)
    return csr(ring + clique, np.concatenate([np.stack([v, (v + d) % ring], 1) for d in range(1, half + 1)] +
                                             [np.stack([i + ring, j + ring], 1)]))


def hubs_of(degree):
    """The vertices of the highest degree bins (128 per power of two, from degree 128 on) that together
    hold fewer than 2^15."""
    d = np.maximum(degree, 1)
    lg = np.floor(np.log2(d)).astype(np.int64)
    bin_ = lg * 128 + ((d >> np.maximum(lg - 7, 0)) & 127)
    bin_[degree < 128] = -1
    count = np.bincount(bin_[bin_ >= 0], minlength=4096)
    above = np.cumsum(count[::-1])[::-1]
    return (bin_ >= 0) & (above[np.maximum(bin_, 0)] < 1 << 15)


def expected(fo, src, dst, small, keys, hub):
    n = len(fo) - 1
    degree = np.diff(fo.astype(np.int64))
    up = (degree[src] < degree[dst]) | ((degree[src] == degree[dst]) & (src < dst))
    out = np.bincount(src[up], minlength=n)
    rest = np.bincount(src[up & ~hub[dst]], minlength=n)
    tail = up & (out[src] >= 2) & (out[src] <= small) & (out[dst] <= small)
    owner = (out[src] > small) & (out[dst] > 0) & ((out[dst] < out[src]) | ((out[dst] == out[src]) & (dst < src)))
    chunks = np.maximum(1, -(-rest // keys))
    at_tails = out[dst[tail]].sum()
    return (int(at_tails + out[dst[owner]].sum()),
            int(at_tails + (out - rest)[dst[owner]].sum() + (rest[dst[owner]] * chunks[src[owner]]).sum()))


def clique(n):
    i, j = np.triu_indices(n, 1)
    return csr(n, np.stack([i, j], 1))


@pytest.mark.parametrize("name,wide", [("clique-700", False), ("clique-2100", True), ("ring-300", False),
                                       ("ring-100", False)])
def test_streamed_entries(counter, name, wide):
    kind, size = name.split("-")
    fo, src, dst = clique(int(size)) if kind == "clique" else ring_and_clique(33000, int(size), 700)
    split = len(dst) >= 1 << 21 and not wide
    hub = hubs_of(np.diff(fo.astype(np.int64))) if split else np.zeros(len(fo) - 1, bool)
    hd = dst.astype(np.uint32)
    counter.count(fo, hd, Config(collect_stats=True, force_wide_offsets=wide))
    st = counter.stats()
    streamed, chunked = expected(fo, src, dst, 48, 256 if split else 2048, hub)
    assert st.streamed_entries == streamed and st.streamed_chunked == chunked
    assert (chunked > streamed) == (name in ("clique-2100", "ring-300"))
    counter.count(fo, hd, Config(collect_stats=True, intersection_method="merge", force_wide_offsets=wide))
    st = counter.stats()
    assert st.streamed_entries == streamed and st.streamed_chunked == streamed
