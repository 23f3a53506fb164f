"""Arguments that do not fit q: an exception on the host, whichever path the call would take, and no launch."""

import pytest
import torch

B, T, H, K, V = 2, 128, 3, 64, 128


def arguments(cell, device="cpu"):
    delta, diag = cell in ("delta", "kda"), cell in ("gla", "kda")
    z = lambda *s, dtype=torch.float32: torch.zeros(*s, dtype=dtype, device=device)  # noqa: E731
    a = {"q": z(B, T, H, K, dtype=torch.bfloat16), "k": z(B, T, H, K, dtype=torch.bfloat16), "v": z(B, T, H, V, dtype=torch.bfloat16),
         "g": z(B, T, H, K) if diag else z(B, T, H), "initial_state": z(B, H, K, V)}
    if delta:
        a["beta"] = z(B, T, H)
    if not diag:
        a["dqk"] = z(H, K) + 1
    names = {"q": (H,), "k": (H,), "kw": (H, K), "state": (H, V)} | ({"w": (H,), "el": (H, V), "ew": (H, V)} if delta else {"vl": (H, V), "vw": (H, V)})
    return a, {n: z(*s) + 1 for n, s in names.items()}


def misfits(cell):
    """(what, change of the arguments and scales, exception)"""
    def put(name, f):
        def change(a, sc):
            where = sc if name.startswith("scale ") else a
            key = name.removeprefix("scale ")
            where[key] = f(where[key])
        return change

    a, sc = arguments(cell)
    yield "k of another length", put("k", lambda t: t[:, :64]), AssertionError
    yield "k of other heads", put("k", lambda t: t[:, :, :2]), AssertionError
    yield "v of another length", put("v", lambda t: t[:, :64]), AssertionError
    yield "k of another dtype", put("k", lambda t: t.half()), NotImplementedError
    yield "v of another dtype", put("v", lambda t: t.float()), NotImplementedError
    yield "k of one byte", put("k", lambda t: t.to(torch.int8)), NotImplementedError
    for name in ("g", "beta", "dqk", "initial_state"):
        if name in a:
            yield f"short {name}", put(name, lambda t: t[:, :-1]), AssertionError
            yield f"{name} transposed", put(name, lambda t: t.transpose(0, 1)), AssertionError
    for name in sc:
        yield f"short scale {name}", put(f"scale {name}", lambda t: t[:-1]), AssertionError


CASES = [(cell, *m) for cell in ("simple_gla", "gla", "delta", "kda") for m in misfits(cell)]
IDS = [f"{c[0]}-{c[1]}" for c in CASES]


@pytest.mark.parametrize("cell,what,change,error", CASES, ids=IDS)
def test_descriptor_refuses(cell, what, change, error, monkeypatch):
    from linquant_b200 import _cabi
    from linquant_b200.kernels.zoo import _common

    a, sc = arguments(cell)
    monkeypatch.setattr(_cabi, "status_word", lambda dev: torch.zeros(1, dtype=torch.int32))
    kw = dict(decay=_cabi.DECAY_DIAGONAL if cell in ("gla", "kda") else _cabi.DECAY_SCALAR, eta=1.0, sigma=1.0, tau=1.0, scale=1.0,
              chunk_size=64, bits=8, out=a["v"], final_state=None, rot_signs=None, keep=[])
    args = lambda: dict(q=a["q"], k=a["k"], v=a["v"], g=a["g"], beta=a.get("beta"), scales=sc, dqk=a.get("dqk"),  # noqa: E731
                        initial_state=a["initial_state"])
    _common.make_problem(**args(), **kw)  # the arguments as they are pass
    change(a, sc)
    with pytest.raises(error):
        _common.make_problem(**args(), **kw)


@pytest.mark.gpu
@pytest.mark.parametrize("cell", ["simple_gla", "gla", "delta", "kda"])
def test_calls_refuse(cell):
    from linquant_b200 import _cabi
    from linquant_b200.kernels import zoo

    for what, change, error in [*misfits(cell), ("k on the host", lambda a, sc: a.update(k=a["k"].cpu()), _cabi.LinQuantError)]:
        a, sc = arguments(cell, "cuda")
        change(a, sc)
        beta = (a.pop("beta"),) if "beta" in a else ()
        args = (a.pop("q"), a.pop("k"), a.pop("v"), a.pop("g"), *beta)
        for debug in (None, {}):
            with pytest.raises(error):
                getattr(zoo, f"chunk_{cell}_int8")(*args, sc, _debug=debug, **a)
