"""Rules that the kernels' correctness rests on and that no run shows reliably, checked on the source text."""
import pathlib
import re

KERNELS = pathlib.Path(__file__).resolve().parents[1] / "csrc" / "kernels"


def _code(path):
    text = re.sub(r"/\*.*?\*/", "", path.read_text(), flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def _functions(code):
    """(signature, body) of every device function of a file."""
    for m in re.finditer(r"__(?:global|device)__[^;{}]*?\)\s*\{", code):
        depth, at = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(code[at], 0)
            at += 1
        yield m.group(0), code[m.end():at]


def test_kernels_that_start_early_promise_nothing_about_their_inputs():
    """A kernel that waits for its predecessor while it is already running (pdl_wait, launch.h) reads what is written during its
    lifetime: no ``__restrict__`` (a const pointer would be read-only for that long) and no __ldg / __ldcg."""
    found = 0
    for path in sorted(KERNELS.glob("*.cu*")):
        code = _code(path)
        for signature, body in _functions(code):
            if "pdl_wait()" not in body or "void pdl_wait" in signature:
                continue
            found += 1
            where = f"{path.name}: {' '.join(signature.split())}"
            assert "__restrict__" not in signature, where
            assert not re.search(r"__ld(g|cg)\b|ld\.global\.nc", body), where
        # what these kernels call lies in the same files
        if "pdl_wait()" in code:
            assert not re.search(r"__ld(g|cg)\b|ld\.global\.nc", code), path.name
            assert not any("__restrict__" in s for s, _ in _functions(code) if "__global__" not in s), path.name
    assert found >= 15, "the kernels were not found in the sources"


def test_kernels_that_give_up_wait_for_their_loads():
    """A TMA load writes shared memory whenever it lands: a kernel whose waits have run out stays, for a bounded time, until its loads have landed.
    One CTA waits for the slots that it armed; a CTA pair's loads are counted in the leader, whose MMA thread waits for those it has not used."""
    found = {"single": 0, "pair": 0}
    for path in sorted(KERNELS.glob("*.cu*")):
        for signature, body in _functions(_code(path)):
            where = f"{path.name}: {' '.join(signature.split())}"
            if "tma_load_2d_pair(" in body:
                found["pair"] += 1
                issuer = body[body.rindex("tma_load_2d_pair("):]
                gave_up = issuer[issuer.index("if (!ok) {"):]
                assert re.match(r"if \(!ok\) \{[^}]*drain_pair_loads\(bar->full, \w*STAGES, stage, phase\);\s*\}", gave_up), where
                assert issuer.index("drain_pair_loads(") < issuer.rindex("cluster_sync()"), where
            elif "tma_load_2d(" in body:
                found["single"] += 1
                assert re.search(r"if \(armed & \(1u << s\)\)", body), where
    assert found["pair"] >= 2 and found["single"] >= 4, found
