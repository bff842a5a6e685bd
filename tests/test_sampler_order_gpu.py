"""The cluster sampler's draw against float64: the token of (seed, row, step) is the one at which the masses, added up in the order (block, thread, vector,
element) over 512 threads a block, reach the uniform number's share.  Sizes at which threads, vectors and blocks run out."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def philox(counter, key):
    """Philox 4x32-10 (Salmon et al., 2011), first word; counter: four words, key: two, as Python numbers."""
    c, k, m = list(counter), list(key), 0xffffffff
    for _ in range(10):
        a, b = 0xD2511F53 * c[0], 0xCD9E8D57 * c[2]
        c = [(b >> 32) ^ c[1] ^ k[0], b & m, (a >> 32) ^ c[3] ^ k[1], a & m]
        k = [(k[0] + 0x9E3779B9) & m, (k[1] + 0xBB67AE85) & m]
    return c[0]


def order(V):
    """Tokens in the order in which their masses are added up."""
    blocks = 1 if V * 2 <= 102400 else 2 if V <= 102400 else 4
    size = ((V + blocks - 1) // blocks + 7) // 8 * 8
    t = np.arange(V)
    block, vec = t // size, t % size // 8
    return np.lexsort((t % 8, vec // 512, vec % 512, block))


@pytest.mark.parametrize("V", [8, 120, 4088, 4096, 4104, 8200, 51200, 51208, 102408, 151936, 152064])
def test_draw_follows_the_order(V):
    from nanorlhf_b200.ops import native
    R, seed = 48, 11
    g = torch.Generator(device="cuda").manual_seed(V)
    z = (torch.randn(R, V, generator=g, device="cuda") * 3).bfloat16()
    z[R // 2:, ::2] = -float("inf")                          # threads without mass
    ids, steps = torch.arange(100, 100 + R, dtype=torch.int32, device="cuda"), torch.arange(R, dtype=torch.int32, device="cuda") * 7
    tok = native.sample(z, 0.9, 1.0, seed, 0, ids, steps, impl=2).tolist()
    p = torch.softmax(z.double() / 0.9, -1).cpu().numpy()
    perm = order(V)
    for r in range(R):
        off = steps[r].item() * 32 // 4                      # 32 numbers a step, four of a counter
        u = (philox((off, 0, ids[r].item(), 0), (seed, 0)) + 0.5) * 2.0 ** -32
        at = int(np.flatnonzero(perm == tok[r])[0])
        cum = np.cumsum(p[r][perm])
        # float32: a thread adds up to 27 vectors of 8, then 16 threads, 32 parts and 4 blocks: under 300 roundings of a sum of at most 1
        tol = 300 * 2.0 ** -24
        assert p[r][tok[r]] > 0 and (cum[at - 1] if at else 0.0) - tol <= u <= cum[at] + tol, (r, u, cum[at])
