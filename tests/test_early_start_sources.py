"""Kernels that take their places while the kernel before them in the stream still runs: what the device code has to
keep to, checked on the sources.  Such a kernel is alive while its predecessor writes, and a read-only load
(``__ldg``, ``const __restrict__`` parameters) is allowed only for data that nothing writes while the kernel lives; nor
does the compiler keep it behind the wait."""
import functools
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "hades_b200" / "csrc"
WAITS = ("begin_after_previous", "wait_for_previous")
SETTLED = "load_settled"
NOT_FUNCTIONS = {"if", "for", "while", "switch", "return", "sizeof", "catch", "alignof", "decltype", "__launch_bounds__"}


def _source(path, seen):
    """A source with this library's headers in the place of their first inclusion, without comments."""
    seen.add(path.name)
    text = re.sub(r"//[^\n]*|/\*.*?\*/", " ", path.read_text(), flags=re.S)
    text = re.sub(r"\\\n", " ", text)

    def header(m):
        at = path.parent / m.group(1)
        return _source(at, seen) if at.parent == CSRC and at.name not in seen else ""

    return re.sub(r'#include "([\w./]+)"', header, text)


def _closing(text, at, left, right):
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == left) - (text[i] == right)
        if depth == 0:
            return i
    return len(text) - 1


def _functions(text):
    """(name, parameters, body) of everything that looks like a function definition."""
    for m in re.finditer(r"\b([A-Za-z_]\w*)\s*\(", text):
        if m.group(1) in NOT_FUNCTIONS:
            continue
        end = _closing(text, m.end() - 1, "(", ")")
        body = re.match(r"\s*(?:const\b|noexcept\b|override\b|->\s*[\w:<>\s*&]+?|\s)*\{", text[end + 1:end + 200])
        if body:
            at = end + body.end()
            yield m.group(1), text[m.end():end], text[at:_closing(text, at, "{", "}") + 1]


@functools.lru_cache(maxsize=None)
def _reached(path):
    """Of one source: the kernels that start early, and what they call by name (or what is called alike)."""
    functions = list(_functions(_source(path, set())))
    names = {}
    for f in functions:
        names.setdefault(f[0], []).append(f)
    early = [f for f in functions if f[0] not in WAITS and any(w + "()" in f[2] for w in WAITS)]
    seen, todo = [], list(early)
    while todo:
        f = todo.pop()
        if f in seen:
            continue
        seen.append(f)
        for called in re.findall(r"\b([A-Za-z_]\w*)\s*(?:<[^;{}()]*>\s*)?\(", f[2]):
            todo.extend(names.get(called, []))
    return early, seen


def _all():
    early, reached = [], []
    for path in sorted(CSRC.glob("*.cu")):
        e, r = _reached(path)
        early += e
        reached += r
    return early, reached


def test_the_wait_is_the_first_statement():
    early, _ = _all()
    assert len({f[0] for f in early}) >= 17
    for name, _, body in early:
        assert re.match(r"\{\s*(" + "|".join(WAITS) + r")\(\);", body), name
        assert ("wait_for_previous()" in body) == ("start_next()" in body), name


def test_what_starts_early_waits():
    early = {f[0] for f in _all()[0]}
    text = "".join(_source(p, set()) for p in sorted(CSRC.glob("*.cu")))
    launched = set(re.findall(r"HB_LAUNCH_NEXT(?:_IF\(\w+,|\()\s*\(*\s*(\w+)", text)) - {"true", "early", "kernel"}
    assert launched and launched <= early, launched - early


def test_no_read_only_loads_in_what_starts_early():
    early, reached = _all()
    assert {"warp_lookup_setassoc", "touch_runs", "resolve_run", "walk_list"} <= {f[0] for f in reached}
    loads = {name for name, _, body in reached if "__ldg" in body or re.search(r"\bld\.[\w.]*\bnc\b", body)}
    assert loads == {SETTLED}, sorted(loads)
    # rows and ids that the launch before, of the same call, does not write; the classes where a sort of the whole GPU,
    # which starts behind everything, reads them ("run")
    users = {name for name, _, body in reached if SETTLED + "(" in body}
    assert users == {"load_row16", "warp_put_rows", "segsum_kernel", "walk_list", "run"}, sorted(users)
    unaliased = {name for name, params, _ in early if "__restrict__" in params}
    assert not unaliased, sorted(unaliased)
