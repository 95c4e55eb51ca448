"""The key under which a tuned launch shape is kept in the autotuner's file."""
import hashlib
import json
from dataclasses import replace
from types import SimpleNamespace

from gpe_b200 import GpeParams
from gpe_b200.autotune import signature

BASE = [GpeParams(nx=32, ny=24, nz=16, precision=8), GpeParams(nx=64, ny=64, nz=64, precision=8)]


def key(prms, device="B200"):
    return signature(SimpleNamespace(prms=prms), device)


def test_key_tells_the_kernels_apart():
    """Runs whose right-hand sides step with other kernels are timed anew."""
    variants = [dict(), dict(omx=0.1), dict(Urhs=0.2), dict(diss_amp=0.3), dict(eqn_to_solve=2),
                dict(kahan=True), dict(order=4), dict(bcs=2)]
    keys = [key([replace(p, **v) for p in BASE]) for v in variants]
    assert len(set(keys)) == len(variants)
    # one trapped member is enough: the batch steps with its form
    assert key([replace(BASE[0], omy=0.1), BASE[1]]) not in (keys[0],)
    assert key(BASE) == key(BASE[::-1]) and key(BASE) != key(BASE, "another device")


def test_shapes_tuned_on_earlier_launches_are_not_applied():
    """Files written when the batch stepped one stage per launch had this key."""
    old = json.dumps({"shapes": sorted((p.nx, p.ny, p.nz) for p in BASE), "order": 2, "bcs": 1,
                      "precision": 8, "kahan": False, "device": "B200"}, sort_keys=True)
    assert key(BASE) != hashlib.sha1(old.encode()).hexdigest()[:16]
