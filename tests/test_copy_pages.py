"""Copies of KV pages: what they move, and how much memory they take meanwhile (on the CPU, with the generator's own layout)."""
from types import SimpleNamespace

import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

from rpeg_b200.engine.generation import Generator


class _Buffers(TorchDispatchMode):
    """The largest tensor that an operation makes."""

    largest = 0

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        out = func(*args, **(kwargs or {}))
        if func is torch.ops.aten.index.Tensor or func is torch.ops.aten.clone.default:
            self.largest = max(self.largest, out.numel() * out.element_size())
        return out


def _generator(geometry, pages, limit):
    gen = SimpleNamespace(geometry=geometry, cfg=SimpleNamespace(n_layers=len(geometry)), dev=torch.device("cpu"), COPY_BYTES=limit, kcache=[], vcache=[])
    gen._upload = lambda arrays: Generator._upload(gen, arrays)
    sizes = [(cache, h, w) for h, dk, dv in geometry for cache, w in ((gen.kcache, dk), (gen.vcache, dv))]
    gen.kv_storage = torch.randn(sum(pages * h * 64 * w for _, h, w in sizes)).bfloat16()
    off = 0
    for cache, h, w in sizes:
        n = pages * h * 64 * w
        cache.append(gen.kv_storage[off:off + n].view(pages, h, 64, w))
        off += n
    return gen


@pytest.mark.parametrize("geometry", [[(2, 8, 8)] * 3, [(2, 8, 8), (1, 8, 4)], [(1, 12, 0), (0, 0, 0), (1, 12, 0)]])
@pytest.mark.parametrize("count", [0, 1, 17, 40])
@pytest.mark.parametrize("pages_in_buffer", [0.5, 1, 3, 100])
def test_pages_are_copied_within_the_buffer(geometry, count, pages_in_buffer):
    pages = 90
    row = sum(h * 64 * (dk + dv) * 2 for h, dk, dv in geometry) if len(set(geometry)) == 1 else max(h * 64 * max(dk, dv) * 2 for h, dk, dv in geometry)
    limit = int(row * pages_in_buffer)
    gen = _generator(geometry, pages, limit)
    perm = torch.randperm(pages, generator=torch.Generator().manual_seed(count)).tolist()
    src, dst = [perm[i // 2] for i in range(count)], perm[50:50 + count]
    want = [c.clone() for c in (*gen.kcache, *gen.vcache)]
    for c in want:
        for s, d in zip(src, dst):
            c[d] = c[s]
    with _Buffers() as seen:
        Generator._copy_pages(gen, src, dst)
    assert all(torch.equal(a, b) for a, b in zip(want, (*gen.kcache, *gen.vcache)))
    assert seen.largest <= limit
