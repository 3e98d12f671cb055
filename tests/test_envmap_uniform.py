"""Sampling a uniform environment map: the closed form against the descent of
the probability pyramid bit for bit (numpy FP32), and renders lit by a
constant world against the oracle, which always descends."""
import numpy as np
import pytest

F = np.float32


def descend(uv, res):
    """worldLightSample's descent over a pyramid whose probabilities are all 1/4."""
    p = F(0.25)
    out = []
    for x, y in uv:
        cur, sx, sy = 1, 0, 0
        while cur < res:
            sx, sy, cur = 2 * sx, 2 * sy, 2 * cur
            left = F(p + p)
            if x < left:
                inv = F(F(1) / left)
                x, top = F(x * inv), F(p * inv)
            else:
                inv = F(F(1) / F(F(1) - left))
                x, top, sx = F(F(x - left) * inv), F(p * inv), sx + 1
            if y < top:
                y = F(y / top)
            else:
                y, sy = F(F(y - top) / F(F(1) - top)), sy + 1
        out.append((F(F(sx) + x) / F(res), F(F(sy) + y) / F(res)))
    return np.array(out, F)


def closed(uv, res):
    r = F(res)
    s = uv * r
    c = np.floor(s)
    return ((c + (s - c)) / r).astype(F)


@pytest.mark.parametrize("exponent", [0, 1, 2, 8, 11, 12])
def test_closed_form_equals_descent(exponent):
    res = 1 << exponent
    rng = np.random.default_rng(exponent)
    u = (rng.integers(0, 1 << 23, (400, 2)) / F(1 << 23)).astype(F)  # the generator's values: k / 2^23
    edges = np.array([[0, 0], [0.5, 0.5], [1 - 2.0 ** -23] * 2, [2.0 ** -23, 0.25], [0.75, 1 / res if res > 1 else 0]], F)
    uv = np.concatenate([u, edges])
    assert np.array_equal(descend(uv, res).view(np.uint32), closed(uv, res).view(np.uint32))


@pytest.mark.gpu
@pytest.mark.parametrize("exponent", [0, 1, 5])
def test_constant_world_matches_oracle(gpu_ctx, exponent):
    """The parity criterion of the other renders: 1e-3 relative on 99.9 % of the pixels."""
    import oracle_ctypes as O
    from raymond_b200 import api, materials as M, scenes
    from raymond_b200._abi import SceneDesc

    sc = scenes.cornell(seed=2, envmap_exponent=exponent)
    sc["light_materials"] = [("world", M.world((0.7, 0.9, 1.0, 1.0), 1.5))]  # seen through the room's open front
    desc = SceneDesc(sc)
    r = api.Renderer(api.Scene(gpu_ctx, desc), 96, 80)
    r.render(spp=1, max_depth=6, first_sample=3)
    cpu, _ = O.OracleScene(desc).render(96, 80, 1, 6, first_sample=3)
    ok = np.abs(r.film().astype(np.float64) - cpu) <= 1e-3 * np.abs(cpu) + 1e-6
    assert ok.all(axis=-1).mean() >= 0.999
