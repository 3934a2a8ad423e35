"""A tuning file stands only for the set of kernel shapes that it was chosen
from: one written before the library had more shapes is not applied."""
from types import SimpleNamespace

from changa_gb300 import _native as N
from changa_gb300 import autotune


def test_a_choice_among_other_shapes_is_not_applied(built, monkeypatch, tmp_path):
    import torch
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda: "gpu")
    monkeypatch.setattr(autotune, "CACHE", str(tmp_path / "tuning.json"))
    req = SimpleNamespace(n_buckets=4, n_entries=40)
    ds = SimpleNamespace(lists=SimpleNamespace(n=32, cells=req, plist=req, bucket_starts=range(4)))
    now = autotune.signature(ds, "mixed")
    before = "gpu|mixed|n=32|cells=10|parts=10|nb=8"  # a key without the shapes
    other = now.replace("shapes=%d" % N.cuda_lib().changa_gb300_list_variant_count(), "shapes=17")
    old = {k: {"variant": v, "ms": 1.0, "all_ms": [1.0]} for k, v in
           zip(autotune.KERNELS["mixed"], (14, 10))}
    autotune._save({before: old, other: old})
    assert other != now and now not in autotune._load()
    lib = N.cuda_lib()
    saved = [lib.changa_gb300_get_list_variant(N.KERNEL_IDS[k]) for k in old]
    try:
        autotune._save({now: old})
        assert autotune.tune(ds) == dict(old, cached=True)  # one of the same shapes is
        assert [lib.changa_gb300_get_list_variant(N.KERNEL_IDS[k]) for k in old] == [14, 10]
    finally:
        for k, v in zip(old, saved):
            lib.changa_gb300_set_list_variant(N.KERNEL_IDS[k], v)
