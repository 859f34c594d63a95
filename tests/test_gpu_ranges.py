"""The per-pass and fused steps against the float oracle on fields from all
over the float range: water films and fluxes down to subnormals, zeros, values
whose quotients and roots leave the range of the kernels' Newton forms,
negative heights; bit for bit.  With infinities and NaN the two steps are
compared with each other (the oracle carries an empty dirt layer, whose terms
no longer vanish); a NaN matches any NaN."""
import numpy as np
import pytest

import hydrogen as H
import oracle as O

pytestmark = pytest.mark.gpu

STATE = H.STATE_FIELDS


def fields(kind, n, seed):
    rng = np.random.default_rng(seed)

    def wide(lo, hi, zeros=0.2, signed=False):
        x = np.exp2(rng.uniform(lo, hi, (n, n)))
        x = np.where(rng.random((n, n)) < zeros, 0.0, x)
        if signed:
            x = np.where(rng.random((n, n)) < 0.5, -x, x)
        return x.astype(np.float32)

    f = {"rock": (64 * rng.random((n, n))).astype(np.float32), "water": wide(-20, 3), "sediment": wide(-30, 0)}
    for k in ("flux_l", "flux_r", "flux_t", "flux_b"):
        f[k] = wide(-20, 4)
    if kind == "films":  # depths and fluxes through the subnormals
        f["water"] = wide(-149, -5)
        for k in ("flux_l", "flux_r", "flux_t", "flux_b"):
            f[k] = wide(-149, 2, zeros=0.4)
    elif kind == "dry":
        f["water"] = wide(-10, 0, zeros=0.9)
        for k in ("flux_l", "flux_r", "flux_t", "flux_b"):
            f[k] = wide(-10, 0, zeros=0.9)
    elif kind == "huge":
        f["rock"] = wide(-10, 45, signed=True)
        f["water"] = wide(-10, 50)
        for k in ("flux_l", "flux_r", "flux_t", "flux_b"):
            f[k] = wide(-10, 52)
    elif kind == "negative":  # heights below zero: exhausted cells, H capped by a negative height
        f["rock"] = (f["rock"] - 60).astype(np.float32)
        f["sediment"] = wide(-30, 0, signed=True)
    elif kind == "nonfinite":
        for k in f:
            bad = rng.random((n, n)) < 0.002
            f[k][bad] = rng.choice(np.array([np.inf, -np.inf, np.nan], np.float32), bad.sum())
    return f


@pytest.mark.parametrize("kind", ["ordinary", "films", "dry", "huge", "negative", "nonfinite"])
@pytest.mark.parametrize("n,thermal,ks1", [(64, True, 0.05), (192, True, 0.0), (128, False, 0.05)])
def test_steps_over_the_float_range(kind, n, thermal, ks1):
    f = fields(kind, n, seed=n + len(kind))
    s = H.settings_config2()
    s.Ks[1] = ks1
    if not thermal:
        s.Kspeed[0] = 0.0
    worlds = []
    for _ in range(2):
        w = H.World(n)
        H.configure(w, "config2")
        w.set_erosion(s)
        w.set_options(H.options(H.RAIN_BERNOULLI, p=0.02, seed=3))
        for k, v in f.items():
            w.upload(k, v)
        worlds.append(w)
    ref = O.OracleWorld(n, 32)
    for k, v in f.items():
        ref.set(k, v)
    so, oo = O.erosion_from(s), O.options(2, 1, 0.5, p=0.02, seed=3)
    for step in range(3):
        for w, mode in zip(worlds, (H.MODE_PLAIN, H.MODE_FUSED)):
            w.step(1, mode)
        if kind != "nonfinite":
            ref.step(so, oo, 1)
        for k in STATE:
            a, b = worlds[0].download(k), worlds[1].download(k)
            pairs = [("fused", b, a)] if kind == "nonfinite" else [("per-pass", a, ref.get(k)), ("fused", b, ref.get(k))]
            for name, x, y in pairs:
                assert np.array_equal(x, y, equal_nan=True), \
                    f"step {step + 1} {name} {k}: {np.count_nonzero(~((x == y) | (np.isnan(x) & np.isnan(y))))} differ"


@pytest.mark.parametrize("layers", [1, 2])
@pytest.mark.parametrize("mode", [H.MODE_PLAIN, H.MODE_FUSED])
def test_flux_scale_of_a_hugely_negative_depth(mode, layers):
    """A depth of -3e38 over an outflow of less than one: the quotient is minus
    infinity, and so is the scale min(1, quotient)."""
    n = 64
    f = fields("ordinary", n, seed=5)
    f["water"][::7, ::5] = -3e38
    s = H.settings_config1()
    s.G = 0.0  # outflows from the old flux, whatever the depth
    w = H.World(n, layers=layers)
    w.set_erosion(s)
    w.set_options(H.options(H.RAIN_OFF))
    ref = O.OracleWorld(n, 32)
    for k, v in f.items():
        w.upload(k, v)
        ref.set(k, v)
    w.step(1, mode)
    ref.step(O.erosion_from(s), O.options(0, 1, 0.0), 1)
    hit = 0
    for k in ("water", "flux_l", "flux_r", "flux_t", "flux_b", "vel_u", "vel_v"):
        a, b = w.download(k), ref.get(k)
        hit += np.count_nonzero(~np.isfinite(b))
        assert np.array_equal(a, b, equal_nan=True), f"{k}: {np.count_nonzero(~((a == b) | (np.isnan(a) & np.isnan(b))))} differ"
    assert hit > 0
