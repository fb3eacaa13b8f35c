"""A block of a warp-specialised kernel as its warps see it: who waits for which barrier, who arrives on it and
who issues something asynchronous, read from the kernel's source and played on the CPU.

``Kernel`` takes the part of the source between the first bounded wait's count and the teardown, and walks it
once per warp: control flow, integers and lambdas are followed, everything else is passed over (a condition
that an event depends on and that cannot be evaluated is an error).  ``nominal`` plays the warps in turn,
``skipped_or_early`` says which waits a parity alone does not keep to their phase, ``given_up`` plays them with
one wait that runs out."""

import copy
import functools
import itertools
import os
import re
from types import SimpleNamespace

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flashqla_b200", "csrc")
EVENT = re.compile(r"\b(mbar_wait(?:_uniform)?|mbar_arrive(?:_expect_tx|_if)?|umma_\w+|tma_(?:load|store)_2d|"
                   r"clc_try_cancel|bar_all|store_rows)\b|bar\.(?:sync|arrive)|uint4\*>\(p\.dv")
BARRIER = re.compile(r"&bars\[(.*?)\]|^(\w+)$")


def _close(text, at):
    """index behind the bracket that opens at `at`"""
    depth = 0
    for i in range(at, len(text)):
        depth += {"(": 1, "{": 1, "[": 1, ")": -1, "}": -1, "]": -1}.get(text[i], 0)
        if depth == 0:
            return i + 1
    raise ValueError(text[at:at + 80])


def _split(text, sep=","):
    """at separators outside of brackets"""
    parts, depth, start = [], 0, 0
    for i, ch in enumerate(text):
        depth += {"(": 1, "{": 1, "[": 1, ")": -1, "}": -1, "]": -1}.get(ch, 0)
        if ch == sep and depth == 0:
            parts.append(text[start:i])
            start = i + 1
    return [s.strip() for s in parts + [text[start:]]]


def _statement(text, at):
    """(node, index behind it)"""
    rest = text[at:]
    if m := re.match(r"(if|for|switch|while)\s*(constexpr)?\s*(?=\()", rest):
        end = _close(text, at + m.end())
        head = text[at + m.end() + 1:end - 1]
        body, end = _next(text, end)
        if m[1] != "if":
            return (m[1], head, body), end
        more = re.match(r"\s*else\b", text[end:])
        other, end = _next(text, end + more.end()) if more else (None, end)
        return ("if", head, body, other), end
    if rest[0] == "{":
        end = _close(text, at)
        return ("block", _parse(text[at + 1:end - 1])), end
    if m := re.match(r"(case\s+\w+|default)\s*:", rest):
        return ("label", m[1].replace("case", "").strip()), at + m.end()
    end = at
    while text[end] != ";":
        end = _close(text, end) if text[end] in "({[" else end + 1
    return ("do", text[at:end].strip()), end + 1


def _next(text, at):
    return _statement(text, at + len(text[at:]) - len(text[at:].lstrip()))


def _parse(text):
    nodes, at = [], 0
    while text[at:].strip():
        node, at = _next(text, at)
        nodes.append(node)
    return nodes


@functools.lru_cache(None)
def _python(expr):
    """A C++ expression over integers as a Python one."""
    expr = re.sub(r"\((?:int|uint32_t|long long|bool)\)", "", expr.strip())
    expr = re.sub(r"\b(0x[0-9a-f]+|\d+)u\b", r"\1", expr)
    expr = re.sub(r"bar_all<(\d+), (\d+)>", r"bar_all", expr)
    for open_ in reversed([m.start() for m in re.finditer(r"\(", expr)]):  # ternaries inside brackets first
        end = _close(expr, open_)
        inner = expr[open_ + 1:end - 1]
        if "?" in inner:
            expr = expr[:open_] + "(" + ", ".join(map(_python, _split(inner))) + ")" + expr[end:]
    at = _split(expr, "?")
    if len(at) > 1:
        rest = "?".join(at[1:])
        yes = _split(rest, ":")[0]
        return f"(({_python(yes)}) if ({_python(at[0])}) else ({_python(rest[len(yes) + 1:].lstrip(': '))}))"
    expr = expr.replace("&&", " and ").replace("||", " or ").replace(" / ", " // ")
    return re.sub(r"!(?!=)", " not ", re.sub(r"\btrue\b", "True", re.sub(r"\bfalse\b", "False", expr))).strip()


@functools.lru_cache(None)
def _code(expr):
    return compile(_python(expr), "<source>", "eval")


def _eval(expr, env):
    return eval(_code(expr), {}, env)


class Kernel:
    """One block: `config` holds what the source's names stand for (template arguments, parameters)."""

    def __init__(self, file, threads, config, text=None):
        src = text if text is not None else open(os.path.join(CSRC, file)).read()
        src = re.sub(r"//[^\n]*|^[ \t]*#[^\n]*", "", src, flags=re.M)
        src = re.sub(r"\b(pass|is|in|not)\b", r"\1_", src)  # names that Python has taken
        src = re.sub(r"(if \([^()]*\) )?(\{ const int it = [^;]*; )?FQLA_TRACE\([^;]*;( \})?", "", src)
        self.names = {}
        for body in re.findall(r"\benum \{(.*?)\}", src, flags=re.S):
            value = -1
            for item in _split(body):
                name, _, same = (x.strip() for x in item.partition("="))
                value = (self.names[same] if same in self.names else int(same)) if same else value + 1
                self.names[name] = value
        self.config, self.warps = dict(config), threads // 32
        self.shared = dict
        self.counts, self.eventful, self.bodies = {}, {}, {}
        env = {**self.names, **self.config}
        for head, bar, count in re.findall(r"(for \([^)]*\) )?mbar_init\(&bars\[(\w+)\], ([^;]+)\);", src):
            if head:
                first, last = re.search(r"= (\w+); i <= (\w+);", head).groups()
                for b in range(self.names[first], self.names[last] + 1):
                    self.counts[b] = _eval(count, env)
            elif bar in self.names:
                self.counts[self.names[bar]] = _eval(count, env)
        at = src.index("int tries = WAIT_TRIES;")
        self.nodes = _parse(src[at:src.index("\n  tc_fence_before();\n  __syncthreads();", at)])
        # functions that are a named barrier
        self.functions = {name: ([], [("do", barrier)], True) for name, barrier in re.findall(
            r"void (\w+)\(\) \{\s*(asm volatile\(\"bar\.sync \d+, \d+;\"[^;]*);", src)}

    # ---- one warp ---------------------------------------------------------------------------------------
    def warp(self, index, shared):
        """Generator of the warp's events: sends back what a wait (False: it ran out) or a vote gives."""
        env = {**self.names, **self.config, **shared, "warp": index, "lane": 0, "tid": 32 * index, "tries": 1,
               "WAIT_TRIES": 1, "elect_one": lambda: True, "__all_sync": lambda mask, x: x, "min": min, "max": max,
               "abs": abs, "__shfl_sync": lambda mask, x, lane: x, "INT_MAX": 2**31 - 1}
        lambdas = dict(self.functions)
        yield from self._run(self.nodes, env, lambdas, False)

    def _has_event(self, node, lambdas, leaves=True):
        """whether an event, or (`leaves`) a way out of a loop or lambda, stands in the node"""
        if node is None or node[0] == "label":
            return False
        key = id(node), leaves and node[0] != "for"  # (what leaves a loop without events is nothing)
        if key not in self.eventful:  # (a lambda is known before the code that calls it)
            text = node[1]
            if node[0] == "block":
                found = any(self._has_event(n, lambdas, leaves) for n in text)
            else:
                found = bool(EVENT.search(text) and "= [&]" not in text
                             or key[1] and node[0] == "do" and re.match(r"(break|return|continue)\b", text)
                             or any(n in lambdas and lambdas[n][2] for n in re.findall(r"\b(\w+)\(", text))
                             or any(self._has_event(n, lambdas, key[1]) for n in node[2:]))
            self.eventful[key] = found
        return self.eventful[key]

    def _value(self, expr, env, lambdas):
        """(a generator: an expression may hold a vote or call a lambda)"""
        if any(lambdas[n][2] for n in re.findall(r"\b(\w+)\(", expr) if n in lambdas):  # what waits, waits in order
            expr = expr.strip()
            for sign, ends in (("||", True), ("&&", False)):
                parts = _split(expr.replace(sign, "\0"), "\0")
                for part in parts if len(parts) > 1 else ():
                    value = yield from self._value(part, env, lambdas)
                    if bool(value) == ends or part is parts[-1]:
                        return value
            if expr[0] == "!":
                return not (yield from self._value(expr[1:], env, lambdas))
            if expr[0] == "(" and _close(expr, 0) == len(expr):
                return (yield from self._value(expr[1:-1], env, lambdas))
        if m := re.search(r"bar_all<(\d+), (\d+)>\(", expr):
            end = _close(expr, m.end() - 1)
            mine = yield from self._value(expr[m.end():end - 1], env, lambdas)
            result = yield "bar", int(m[1]), int(m[2]), bool(mine)
            return _eval(expr[:m.start()] + str(result) + expr[end:], env)
        for name in re.findall(r"\b(\w+)\(", expr):
            if name in lambdas and name not in env:
                at = re.search(rf"\b{name}\(", expr)
                end = _close(expr, at.end() - 1)
                args = [a for a in _split(expr[at.end():end - 1]) if a]
                result = yield from self._call(name, args, env, lambdas, False)
                expr = expr[:at.start()] + repr(result) + expr[end:]
        return _eval(expr, env)

    def _call(self, name, args, env, lambdas, one):
        params, body, _ = lambdas[name]
        values = []
        for a in args:
            m = BARRIER.match(a)
            try:
                values.append(_eval(m[1] if m and m[1] else a, env))
            except NameError:  # an address
                values.append(None)
        old = {p: env.get(p) for p in params}
        env.update(zip(params, values))
        result = yield from self._run(body, env, lambdas, one)
        env.update(old)
        return result[1] if result and result[0] == "return" else None

    def _run(self, nodes, env, lambdas, one):
        """(`one`: inside a branch that a single lane takes.)  Returns why the walk ended early, or None."""
        for node in nodes:
            kind = node[0]
            if kind == "block":
                out = yield from self._run(node[1], env, lambdas, one)
                if out:
                    return out
            elif kind == "if":
                if not (self._has_event(node[2], lambdas) or self._has_event(node[3], lambdas)
                        or EVENT.search(node[1])):
                    # an assignment under a condition counts if both can be followed
                    try:
                        branch = node[2] if _eval(node[1], env) else node[3]
                    except Exception:
                        continue
                    if branch:
                        yield from self._run([branch], env, lambdas, one)
                    continue
                cond = yield from self._value(node[1], env, lambdas)
                single = one or bool(re.search(r"elect_one\(\)|lane == 0|issuing\(\)", node[1]))
                branch = node[2] if cond else node[3]
                if branch:
                    out = yield from self._run([branch], env, lambdas, single if cond else one)
                    if out:
                        return out
            elif kind == "for":
                if not self._has_event(node[2], lambdas):
                    continue
                init, cond, step = _split(node[1], ";")
                if init:
                    self._assign(re.sub(r"^(?:int|bool|uint32_t) ", "", init), env)
                while not cond or (yield from self._value(cond, env, lambdas)):
                    out = yield from self._run([node[2]], env, lambdas, one)
                    if out and out[0] == "break":
                        break
                    if out and out[0] != "continue":
                        return out
                    for part in _split(step):
                        self._assign(part, env)
            elif kind == "switch":
                want = str((yield from self._value(node[1], env, lambdas)))
                body = node[2][1]
                labels = [i for i, n in enumerate(body) if n[0] == "label"]
                at = next((i for i in labels if body[i][1] == want), None)
                if at is None:
                    at = next(i for i in labels if body[i][1] == "default")
                out = yield from self._run([n for n in body[at + 1:] if n[0] != "label"], env, lambdas, one)
                if out and out[0] == "return":
                    return out
            elif kind == "do":
                out = yield from self._do(node[1], env, lambdas, one)
                if out:
                    return out
        return None

    def _assign(self, text, env):
        m = re.match(r"(?:\+\+(\w+)|([\w.]+(?:\[.*?\])?) ([\^+|-]?)= (.*))$", text, flags=re.S)
        if not m:
            return
        if m[1]:
            env[m[1]] += 1
            return
        value = _python(m[4] if not m[3] else f"{m[2]} {m[3]} ({m[4]})")
        if re.fullmatch(r"\w+", m[2]):
            value = eval(value, {}, env)
            env[m[2]] = copy.copy(value) if isinstance(value, SimpleNamespace) else value
        else:
            exec(f"{m[2]} = {value}", {}, env)

    def _do(self, text, env, lambdas, one):
        if text in ("break", "continue"):
            return (text,)
        if m := re.match(r"return (mbar_wait\w*\(.*\))$", text):
            yield from self._do(m[1], env, lambdas, one)
            return "return", env["tries"] > 0
        if m := re.match(r"return\b(.*)", text, flags=re.S):
            return "return", (yield from self._value(m[1], env, lambdas)) if m[1].strip() else None
        if m := re.match(r"auto (\w+) = \[&\]\s*(?:\((.*?)\))?\s*(?=\{)", text, flags=re.S):
            params = [re.split(r"[\s&*]+", p)[-1] for p in _split(m[2] or "") if p]
            if text not in self.bodies:  # (parsed once: nodes are told apart by identity)
                self.bodies[text] = _parse(text[m.end() + 1:_close(text, m.end()) - 1])
            body = self.bodies[text]
            lambdas[m[1]] = (params, body, False)
            lambdas[m[1]] = (params, body, any(self._has_event(n, lambdas, False) for n in body))
            return None
        if m := re.match(r'asm volatile\("bar\.(sync|arrive) (\d+), (\d+);"', text):
            yield ("bar" if m[1] == "sync" else "bar_arrive"), int(m[2]), int(m[3]), True
            return None
        if m := re.match(r"(\w+)(?:<.*?>)?\((.*)\)$", text, flags=re.S):
            name, args = m[1], [a for a in _split(m[2]) if a]
            if name.startswith("mbar_wait"):
                bar = _eval(BARRIER.match(args[0])[1], env)
                ok = yield "wait", bar, _eval(args[1], env) & 1
                if not ok:
                    env[args[2]] = 0
                return None
            if name == "mbar_arrive_if":
                name = "mbar_arrive"
                if not env["tries"] > 0:
                    return None
            if name in ("mbar_arrive", "mbar_arrive_expect_tx", "umma_commit"):
                b = BARRIER.match(args[0])
                bar = _eval(b[1] or b[2], env)
                yield "arrive", bar, 1 if one or name != "mbar_arrive" else 32
                return None
            if EVENT.match(name):
                if name != "store_rows" or _eval(args[3], env) > 0:  # (rows to store)
                    yield "issue", name, None
                return None
            if name in lambdas and name not in env:
                if lambdas[name][2]:
                    yield from self._call(name, args, env, lambdas, one)
                return None
        if m := re.match(r"uint64_t\* (\w+) = &bars\[(.*)\]$", text, flags=re.S):
            env[m[1]] = _eval(m[2], env)
            return None
        if text.startswith("*reinterpret_cast<uint4*>(p.dv"):
            yield "issue", "dv", None
            return None
        m = re.match(r"(?:const |constexpr )?(?:int|bool|uint32_t|long long|Item) (.*)$", text, flags=re.S)
        for part in _split(m[1] if m else text):
            if any(n in lambdas and lambdas[n][2] for n in re.findall(r"\b(\w+)\(", part)):
                name, _, expr = part.partition(" = ")
                env[name.strip()] = yield from self._value(expr.strip(), env, lambdas)
                continue
            assert not EVENT.search(part), part
            try:
                self._assign(part, env)
            except Exception:  # not an integer that can be followed
                pass
        return None


# ---- several warps --------------------------------------------------------------------------------------
class _Block:
    """The barriers of a block while its warps are played."""

    def __init__(self, kernel):
        self.kernel, self.done, self.pending, self.arrived = kernel, {}, dict(kernel.counts), {}
        shared = kernel.shared()
        self.warps = [kernel.warp(w, shared) for w in range(kernel.warps)]
        self.at = [next(g, None) for g in self.warps]  # the event each warp stands at

    def phase(self, bar, parity):
        """the phase that a wait for `parity` sees completed, or None"""
        done = self.done.get(bar, 0)
        return done - 1 if (done - 1) & 1 == parity else None

    def arrive(self, bar, n):
        """the phase that it counts for"""
        phase = self.done.get(bar, 0)
        self.pending[bar] -= n
        assert self.pending[bar] >= 0, f"barrier {bar}: more arrivals than its count"
        if self.pending[bar] == 0:
            self.done[bar], self.pending[bar] = phase + 1, self.kernel.counts[bar]
        return phase

    def go_on(self, w, value=None):
        try:
            self.at[w] = self.warps[w].send(value)
        except StopIteration:
            self.at[w] = None


def nominal(kernel):
    """[(warp, event, phase)] in an order in which the warps take turns; raises if they stop."""
    block, log, named = _Block(kernel), [], {}
    while any(e is not None for e in block.at):
        moved = False
        for w, e in enumerate(block.at):
            if e is None or (e[0] == "bar" and (w in named.get(e[1], {}))):
                continue
            value, phase = None, None
            if e[0] == "wait":
                phase = block.phase(e[1], e[2])
                if phase is None:
                    continue
                value = True
            elif e[0] == "arrive":
                phase = block.arrive(e[1], e[2])
            elif e[0].startswith("bar"):
                here = named.setdefault(e[1], {})
                here[w] = e
                moved = True
                if 32 * len(here) < e[2]:
                    if e[0] == "bar_arrive":
                        log.append((w, e, len(log)))
                        block.go_on(w)
                    continue
                phase = len(log)
                for other, ev in here.items():
                    if ev[0] == "bar":
                        log.append((other, ev, phase))
                        block.go_on(other, all(x[3] for x in here.values()))
                named[e[1]] = {}
                continue
            log.append((w, e, phase))
            block.go_on(w, value)
            moved = True
        if not moved:
            raise AssertionError(f"the warps stop: {[(w, e) for w, e in enumerate(block.at) if e]}")
    return log


def order(log):
    """(follows, waits, arrivals): follows(a, b) says whether event b of the log comes after event a in every
    run, by program order and by arrivals that a wait has seen complete; named barriers order nothing here."""
    nodes = {}  # (warp, n-th event) in program order
    seen, waits, arrivals = {}, [], {}
    for i, (w, e, phase) in enumerate(log):
        nodes[i] = seen.get(w)
        seen[w] = i
        if e[0] == "wait":
            waits.append((i, e[1], phase))
        elif e[0] == "arrive":
            arrivals.setdefault((e[1], phase), []).append(i)
    before = [0] * len(log)  # bit set of everything that comes before
    by_wait = {i: (b, k) for i, b, k in waits}
    for i in range(len(log)):
        prev = nodes[i]
        bits = 0 if prev is None else before[prev] | 1 << prev
        if i in by_wait:
            for a in arrivals.get(by_wait[i], []):
                bits |= before[a] | 1 << a
        before[i] = bits
    return (lambda a, b: bool(before[b] >> a & 1)), nodes, waits, arrivals


def skipped_or_early(kernel):
    """Waits that a parity alone does not keep to their phase: the phase before may still be open when the wait
    begins (it would be over at once), or the phase behind may be over before the wait has been (its parity would
    not come round).  Barriers whose phases the loads complete count by the arrival that goes with the loads."""
    log = nominal(kernel)
    follows, previous, waits, arrivals = order(log)
    name = {v: k for k, v in reversed(list(kernel.names.items()))}
    wrong = set()
    for i, bar, phase in waits:
        prev = previous[i]
        if any(prev is None or not (a == prev or follows(a, prev)) for a in arrivals.get((bar, phase - 1), [])):
            wrong.add((log[i][0], name[bar], "early"))
        after = arrivals.get((bar, phase + 1), [])
        complete = sum(log[a][1][2] for a in after) >= kernel.counts[bar]
        if complete and not any(follows(i, a) for a in after):
            wrong.add((log[i][0], name[bar], "skipped"))
    return sorted(wrong)


def given_up(kernel, warp, nth, last_first):
    """Plays the block with the `nth` wait of `warp` running out; whenever nobody can go on, the waits that are
    open run out one at a time (from the highest or the lowest warp).  Returns (warps left at a named barrier,
    [(warp, event)] that was signalled or issued by a warp behind a wait of its own that had run out)."""
    block, named, late = _Block(kernel), {}, []
    out, count = set(), [0] * kernel.warps
    while True:
        moved = False
        for w in range(kernel.warps):
            while (e := block.at[w]) is not None:
                if e[0] == "wait":
                    ok = block.phase(e[1], e[2]) is not None
                    if w == warp and count[w] == nth:
                        out.add(w)
                        ok = False
                    if not ok and w not in out:
                        break
                    count[w] += 1
                    block.go_on(w, ok)
                elif e[0].startswith("bar"):
                    here = named.setdefault(e[1], {})
                    if w in here:
                        break
                    here[w] = e
                    if e[0] == "bar_arrive":
                        block.go_on(w)
                    if 32 * len(here) == e[2]:
                        named[e[1]] = {}
                        for other, ev in here.items():
                            if ev[0] == "bar":
                                block.go_on(other, all(x[3] for x in here.values()))
                    elif e[0] == "bar":
                        moved = True
                        break
                else:
                    if w in out:
                        late.append((w, e))
                    if e[0] == "arrive":
                        block.arrive(e[1], e[2])
                    block.go_on(w)
                moved = True
        if not moved:
            open_ = [w for w, e in enumerate(block.at) if e is not None and e[0] == "wait"]
            if not open_:
                break
            out.add(open_[-1] if last_first else open_[0])
    return [(w, e) for w, e in enumerate(block.at) if e is not None], late


def waits_of(kernel, warp):
    return sum(1 for w, e, _ in nominal(kernel) if w == warp and e[0] == "wait")


def forward(no_o=False, extra=False, lead=0, n_it=7, partial=False, tiled=1, text=None):
    """The forward recurrence over n_it chunks, the first `lead` of them lead-in."""
    n_chunks = n_it - lead
    p = SimpleNamespace(h=extra, vnew=extra, tiled=tiled, o=not no_o, scale=1.0, Hv=1, N=1, lay=SimpleNamespace(
        cu=SimpleNamespace(ptr=0)), ht=1, M=0, ht_row=0)
    config = dict(NO_O=no_o, EXTRA=extra, STATE=no_o and not extra, PREP=12 if no_o else 16, p=p, n_it=n_it, lead=lead,
                  n_chunks=n_chunks, sp=SimpleNamespace(len=64 * n_chunks - (10 if partial else 0), bos=0, chunk_base=0),
                  CHUNK=64, tile_h=extra and tiled, tile_vn=extra and tiled, m_pass=False, hv=0, hq=0, n=0, D=128)
    return Kernel("fwd_tc.cu", 512 if no_o else 640, config, text=text)


def reverse(lead=0, n_it=7, partial=False, tiled=1, text=None):
    """The reverse recurrence likewise."""
    n_chunks = n_it - lead
    p = SimpleNamespace(dh=1, du=1, tiled=tiled, scale=1.0, Hv=1, dh0=1, dh0_row=0)
    config = dict(p=p, n_it=n_it, lead=lead, len_ext=64 * n_it - (10 if partial else 0), CHUNK=64, hv=0, hq=0, n=0, D=128,
                  sp=SimpleNamespace(len=64 * n_chunks, bos=0, chunk_base=0))
    return Kernel("bwd_dh_tc.cu", 512, config, text=text)


def items(clc=False, tiled=True, partial=(), n_items=4, text=None):
    """The chunk-parallel backward: one block that takes n_items items."""
    config = dict(TILED=tiled, CLC=clc, N_EPI=512, D=128, CHUNK=64,
                  p=SimpleNamespace(Hv=1000, next_item=0, dg_cumsum=0), total=n_items, raw=None, answers=0, blockIdx=SimpleNamespace(x=0), gridDim=SimpleNamespace(x=1))

    def shared():
        claims = itertools.count()
        return dict(
            ring=[None] * 4, stop_flag=[0] * 4, atomicAdd=lambda word, n: next(claims),
            finish=lambda raw, w: SimpleNamespace(valid=40 if w in partial else 64, row0=0, hv=0, hq=0, chunk_id=0),
            clc_block=lambda slot: next((w for w in [1 + next(claims)] if w < n_items), -1))

    kernel = Kernel("bwd_main_tc.cu", 544, config, text=text)
    kernel.shared = shared
    return kernel


CASES = [*itertools.chain(
    (("forward", dict(lead=lead, extra=extra, partial=partial)) for lead, extra, partial in
     itertools.product((0, 1, 2, 3), (False, True), (False, True))),
    (("forward", dict(no_o=True, extra=extra, partial=partial)) for extra, partial in
     itertools.product((False, True), (False, True))),
    (("reverse", dict(lead=lead, partial=partial)) for lead, partial in itertools.product((0, 1, 2, 3), (False, True))),
    (("items", dict(clc=clc, partial=partial)) for clc, partial in
     itertools.product((False, True), ((), (0, 2), (1, 3)))))]
