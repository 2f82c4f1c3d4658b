"""Tuned launch shapes belong to the kernels they were measured on."""
import json

from cbc_b200 import _lib, autotune


def test_tables_of_the_one_form_kernels_are_not_reused(tmp_path):
    """Version 100 had one kernel form for every bubble count."""
    old = {autotune.cache_key("NVIDIA B200", 100, 2, "richardson", K): {} for K in (1, 16, 32)}
    path = tmp_path / "t.json"
    path.write_text(json.dumps(old))
    table = autotune.load_cache(str(path))
    version = int(_lib.lib().cbc_version())
    for K in (1, 16, 32):
        assert autotune.cache_key("NVIDIA B200", version, 2, "richardson", K) not in table
