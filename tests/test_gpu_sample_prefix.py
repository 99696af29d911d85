"""GPU: the sampler on states with empty chunks (4096 amplitudes each): whatever the prefixes
round to, an outcome of probability zero is never drawn and larger uniforms never give smaller
outcomes. Uniforms lie on and next to every chunk border, where the prefixes of one thread, of
the next thread (4 chunks) and of the next CTA (4096 chunks) meet."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CHUNK = 4096


def _empty(kind, chunks, rng):
    e = np.zeros(chunks, dtype=bool)
    if kind == "first of four":
        e[::4] = True
    elif kind == "last of four":
        e[3::4] = True
    elif kind == "random and tail":
        e[rng.random(chunks) < 0.5] = True
        e[::4096] = True
        e[chunks // 2:] = True
    elif kind == "whole blocks":
        e[: min(4096, chunks // 4)] = True
        e[chunks // 2: chunks // 2 + min(4096, chunks // 4)] = True
    return e


@pytest.mark.parametrize("kind", ["none", "first of four", "last of four", "random and tail", "whole blocks"])
@pytest.mark.parametrize("n", [16, 22, 24, 26])
def test_no_impossible_outcome_at_the_chunk_borders(built_lib, n, kind):
    import torch
    from damavand_gb300 import Circuit
    rng = np.random.default_rng(n)
    chunks = (1 << n) // CHUNK
    empty = _empty(kind, chunks, rng)
    if empty.all():
        empty[1] = False
    c = Circuit(n, "gpu")
    amps = c.state().torch()
    g = torch.Generator(device="cuda").manual_seed(n)
    v = torch.randn(chunks, 2 * CHUNK, generator=g, device="cuda", dtype=torch.float64)
    v *= torch.from_numpy(rng.uniform(0.1, 1.0, chunks)).cuda()[:, None]  # masses of no common size
    v[torch.from_numpy(empty).cuda()] = 0
    v /= torch.linalg.vector_norm(v)
    amps.copy_(torch.view_as_complex(v.view(-1, 2)))
    torch.cuda.synchronize()
    p = amps.real.square() + amps.imag.square()
    cdf = np.cumsum(p.view(chunks, CHUNK).sum(1).cpu().numpy())
    at = np.concatenate([cdf / cdf[-1], [1.0]])
    if len(at) > 2049:  # the borders next to an empty chunk and of a CTA's 4096, and a part of the others
        pick = np.zeros(len(at), dtype=bool)
        pick[rng.integers(0, len(at), 1024)] = True
        pick[4095::4096] = True
        pick[np.flatnonzero(empty)[:512]] = True
        pick[-3:] = True
        at = at[pick]
    u = np.sort((at[:, None] + np.spacing(at)[:, None] * np.arange(-12, 13)).ravel())
    u = u[(u > 0) & (u < 1)]
    got = c.sample_array(len(u), uniforms=u).astype(np.int64)
    assert got.min() >= 0 and got.max() < 1 << n
    drawn = p[torch.from_numpy(got).cuda()].cpu().numpy()
    assert np.count_nonzero(drawn == 0) == 0
    assert np.all(np.diff(got) >= 0)
