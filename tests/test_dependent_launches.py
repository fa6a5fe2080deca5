"""The rule of launch.cuh, read from the sources: a kernel that is launched
dependently waits for the kernel before it (grid_wait), and loads through the
read-only path (__ldg, ldg4), which the compiler may move above the wait, only
what no kernel writes: twiddles, primes and their inverses, MMA fragments."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cheddar-fhe_b200", "csrc")
CONSTANT = re.compile(r"tw \+ m \+ i|(\w+\.)?(primes|qinvs) \+ g|jb\.frag \+ i|reinterpret_cast<const uint4 \*>\(tab\) \+ c")


def bodies(text):
    """Kernel name -> the text of its definition's body."""
    out = {}
    for m in re.finditer(r"__global__[^;{]*?\b(k\w+)\(const[^{;]*\{|__global__[^;{]*?\b(k\w+)\([^{;]*\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        out[m.group(1) or m.group(2)] = text[m.end():i]
    return out


def test_dependent_kernels_wait_and_load_plainly():
    seen = set()
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        kernels = bodies(text)
        # straight calls, and launches through a local `go`
        names = set(re.findall(r"launch_dependent\(\s*(k\w+?)[<,]", text)) - {"kern"}
        if "launch_dependent(kern" in text:
            names |= set(re.findall(r"\bgo\((k\w+?)<", text))
        for name in names:
            body = kernels[name]
            assert "grid_wait();" in body, name
            assert "ldg4(" not in body, name
            for arg in re.findall(r"__ldg\(((?:[^()]|\([^()]*\))*)\)", body):
                assert CONSTANT.fullmatch(arg), (name, arg)
        seen |= names
    assert {"k_ks_rows", "k_modswitch_cols", "k_fwd_rows16", "k_elem", "k64_bconv", "k_special_stages"} <= seen
