"""The autotuner's cache in mpm_engine.cu: its key holds everything that selects the kernels it timed."""
import os
import re

ENGINE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mpm_cuda_b200", "csrc",
                      "mpm_engine.cu")


def test_key_holds_what_selects_the_kernels():
    """fused_fn takes dimension, material, configuration, fixed_scene and paged; the timing depends on the sizes and on
    the re-binning interval.  Every member takes part in the order, and every use of the cache goes through key_of."""
    with open(ENGINE) as f:
        src = f.read()
    body = src[src.index("struct TuneKey {"):src.index("struct Tuned {")]
    fields = set()
    for decl in re.findall(r"^    (?:int|long long|bool) ([\w, ]+);", body, re.M):
        fields |= {n.strip() for n in decl.split(",")}
    assert {"device", "dim", "mats", "particles", "blocks", "paged", "fixed_scene", "rebin_interval"} <= fields
    order = re.search(r"std::tie\((.*?)\)", body, re.S).group(1)
    assert fields == set(re.findall(r"k\.(\w+)", order))
    assert src.count("tune_cache()[key_of(*this)]") == 1 and src.count("tune_cache().find(key_of(*this))") == 1
    assert len(re.findall(r"tune_cache\(\)(?:\[|\.find)", src)) == src.count("key_of(*this)")
