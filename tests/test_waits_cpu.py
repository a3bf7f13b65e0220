"""No-GPU check of the kernels' source: a wait that gives up must not leave others waiting.

Every wait of the kernels is bounded, and its result is each thread's own: when one expires, some threads of a block see what they waited
for and others do not.  What stands under a condition on such a result must therefore be nothing that other threads have to take part in:
no block, named or cluster barrier (the others would wait for good, or a half count would be left for the next use), no warp shuffle
or vote, no access to tensor memory (a whole warp's).  A result that a vote made the warp's own may guard the warp's collectives, still no barrier."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "helios_glm53flash_b200", "csrc")
FILES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))
WAIT = re.compile(r"\b(mbar_wait|pt_wait|wait_u|poll_flag\w*)\b")
BARRIER = re.compile(r"bar\.sync|bar\.arrive|bar\.red|barrier\.c|__syncthreads|cluster\.sync|\bprep_sync\b|\bprep_publish\b")
COLLECTIVE = re.compile(r"__shfl\w*|__(all|any|ballot)_sync|__reduce_\w+_sync|\bwarp_(sum|max)\b|tmem_(ld|st)\d+")


def _clean(text):
    """comments out, line numbers kept"""
    text = re.sub(r"/\*.*?\*/", lambda m: "\n" * m.group().count("\n"), text, flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def _close(text, i, pair):
    """index behind the bracket that closes text[i]"""
    depth = 0
    while i < len(text):
        if text[i] == '"':
            i = text.index('"', i + 1)
        elif text[i] == pair[0]:
            depth += 1
        elif text[i] == pair[1]:
            depth -= 1
            if depth == 0:
                return i + 1
        i += 1
    raise ValueError("unbalanced")


def _guarded(text, i):
    """the statement that starts at text[i], with its else"""
    start = i
    while True:
        while text[i].isspace():
            i += 1
        m = re.compile(r"(?:if(?:\s+constexpr)?|for|while)\s*(?=\()").match(text, i)
        if m:
            i = _close(text, m.end(), "()")
            continue
        if text[i] == "{":
            i = _close(text, i, "{}")
        else:
            while text[i] != ";":
                i = _close(text, i, text[i] + {"(": ")", "{": "}"}[text[i]]) if text[i] in "({" else i + 1
            i += 1
        m = re.compile(r"\s*else\b").match(text, i)
        if not m:
            return text[start:i]
        i = m.end()


def _collectives(text):
    """functions of the file that hold a warp collective, or call one that does"""
    bodies = {}
    for m in re.finditer(r"__device__ __forceinline__ [\w:<>]+ (\w+)\(", text):
        end = _close(text, m.end() - 1, "()")
        brace = re.compile(r"\s*(?=\{)").match(text, end)
        if brace:
            bodies[m.group(1)] = text[brace.end():_close(text, brace.end(), "{}")]
    held = {n for n, b in bodies.items() if COLLECTIVE.search(b)}
    while True:
        more = {n for n, b in bodies.items() if n not in held and any(re.search(r"\b%s\b" % h, b) for h in held)}
        if not more:
            return held - {"mbar_wait"}
        held |= more


def faults(text):
    """(line, what, condition) of what stands under a condition on a wait's result and must not"""
    text = _clean(text)
    results = [(m.start(), m.group(1), "__all_sync" in m.group(2))                # (where, name, the warp's own)
               for m in re.finditer(r"\b(\w+)\s*=(?!=)\s*([^;{}]*);", text) if WAIT.search(m.group(2))]
    calls = _collectives(text)
    found = []
    for m in re.finditer(r"\bif\s*(?=\()", text):
        end = _close(text, m.end(), "()")
        cond = text[m.end():end]
        kinds = {n: whole for at, n, whole in results if at < m.start() and re.search(r"\b%s\b" % n, cond)}   # the last before
        if WAIT.search(cond):
            kinds[""] = "__all_sync" in cond
        if not kinds:
            continue
        body = _guarded(text, end)
        bad = [b.group() for b in BARRIER.finditer(body)]
        if "__all_sync" not in cond and not all(kinds.values()):
            bad += [c.group() for c in COLLECTIVE.finditer(body)] + [c for c in calls if re.search(r"\b%s(<\w+>)?\(" % c, body)]
        found += [(text.count("\n", 0, m.start()) + 1, b, cond) for b in bad]
    return found


@pytest.mark.parametrize("path", FILES, ids=[os.path.basename(f) for f in FILES])
def test_nothing_that_others_wait_for_hangs_on_a_single_threads_wait(path):
    assert faults(open(path).read()) == []


def test_the_reader_sees_the_forms_of_the_fault():
    wait = "const bool ok = tc::mbar_wait(&b, 0, &f, 1);"
    assert faults(wait + 'if (ok) { x(); if (w < 4) asm volatile("bar.arrive %0, 160;" ::"r"(1)); }')
    assert faults(wait + "if (ok) go(); else __syncthreads();")
    assert faults(wait + "if (a && ok) v = __shfl_xor_sync(~0u, v, 1);")
    assert faults("__device__ __forceinline__ void fin(int a) { s = warp_sum(a); }" + wait + "if (ok) fin(3);")
    assert faults(wait + "if (ok) tc::tmem_ld32(t, r);")
    assert not faults("const bool ok = __all_sync(~0u, tc::mbar_wait(&b, 0, &f, 1)) != 0; if (ok) v = __shfl_xor_sync(~0u, v, 1);")
    assert faults("const bool ok = __all_sync(~0u, tc::mbar_wait(&b, 0, &f, 1)) != 0; if (ok) { __syncthreads(); }")
    assert not faults(wait + "if (ok) { x(); } __syncthreads();")


def _conditions(text, at, names):
    """the conditions around text[at] that are formed from `names` alone, as one expression"""
    found = []
    for m in re.finditer(r"\bif\s*(?=\()", text):
        end = _close(text, m.end(), "()")
        if end <= at < end + len(_guarded(text, end)):
            cond = text[m.end():end]
            if set(re.findall(r"[A-Za-z_]\w*", cond)) <= names:
                found.append(cond.replace("&&", " and "))
    return " and ".join(found) or "True"


@pytest.mark.parametrize("n_tiles", [1, 2, 3, 4, 5, 6, 7, 8, 13])
def test_every_commit_that_arrives_at_both_ctas_of_a_pair_is_waited_for(n_tiles):
    """An arrival that nobody waits for may reach a CTA's shared memory after its end.  By the conditions in the source: the tiles whose
    products are announced on a barrier are the tiles that are waited for on it."""
    text = _clean(open(os.path.join(CSRC, "mla_pair_tc.cuh")).read())
    ring = int(re.search(r"\bFT_NBUF = (\d+)", _clean(open(os.path.join(CSRC, "mla_flash_tc.cu")).read())).group(1))
    names = {"t", "n_tiles", "FT_NBUF"}

    def tiles(at, which="t"):
        cond, env = _conditions(text, at, names), {"n_tiles": n_tiles, "FT_NBUF": ring}
        loop = range(n_tiles) if "t" in re.findall(r"\w+", which + " " + cond) else [0]
        return {eval(which, {}, {**env, "t": t}) for t in loop if eval(cond, {}, {**env, "t": t})}

    announced, seen = {}, {}
    for m in re.finditer(r"pt_commit\(leader, &ms\.(\w+)\[", text):
        announced.setdefault(m.group(1), set()).update(tiles(m.start()))
    assert set(announced) == {"s_full", "k_free", "pv_done", "v_free"}
    for m in re.finditer(r"(?:mbar_wait<FT_POLL_NS>|pt_wait)\(&ms\.(s_full|k_free|v_free)\[", text):
        # a slot's release is waited for by the tile that takes it over
        seen.setdefault(m.group(1), set()).update(tiles(m.start(), "t" if m.group(1) == "s_full" else "t - FT_NBUF"))
    for m in re.finditer(r"\bwait_pv\(([^,()]+), \d+\)", text):
        if "__any_sync" not in text[text.rindex("\n", 0, text.rindex("if (", 0, m.start())):m.start()]:
            seen.setdefault("pv_done", set()).update(tiles(m.start(), m.group(1)))
    assert seen["k_free"] == announced["k_free"] and seen["v_free"] == announced["v_free"]
    assert seen["s_full"] == announced["s_full"] == set(range(n_tiles))
    assert seen["pv_done"] == announced["pv_done"] == set(range(n_tiles))
