"""CompLL back end, fused CUDA target: ONE launch per DSL function.

The stage-by-stage target (emit_cuda.py) turns every ``reduce`` group and every
``map`` into a kernel of its own, so ``TbqEncode`` (three maps) crossed HBM three
times.  This module plans the same function as a sequence of *phases* and emits
one persistent kernel that runs them back to back:

* consecutive ``map`` / ``reduce`` stages over the same index range join one phase
  when every value they take from a vector written earlier in the phase is the
  element at their own index; that element is then forwarded in a register, each
  input is loaded once (128-bit loads, four consecutive elements per thread) and
  only the last value written to a vector is stored;
* a stage that needs the *result* of a reduction of the current phase, reads a
  freshly written vector at another index, or covers another range starts a new
  phase behind a grid barrier (cooperative launch; the barrier is bounded);
* a ``reduce`` accumulates while its phase streams by: per-thread partial, warp
  shuffle, one partial per block; behind the barrier every block folds the
  partials (no second kernel, no host round trip);
* sub-byte results (``uint<b>``) are packed at warp level: a thread builds the
  4*b-bit fragment of its four elements and ``__shfl_down_sync`` assembles whole
  32-bit words, which the owning lanes store;
* ``random<float>`` costs one Philox call per four elements.

Functions with library-lowered stages (``topk``, ``scatter``) keep the staged
target for those stages; a run of maps between them still becomes one kernel
(``fused_segments``: DgcEncode's two state updates are one pass).  The rules this replaces: one ``thrust::transform`` per map with one
thread per output byte and a serial pack loop (src/CompLL/GCGen/tree.py:197-244,
unit.py:469-482 of mark14wu/hipress).
"""
from __future__ import annotations

from dataclasses import dataclass, field

from . import frontend as F
from .emit_cuda import C_TYPES, SIZEOF, CompileError, Emitter, Sym


def _walk(e):
    """Every expression node below (and including) e, statements included."""
    if isinstance(e, list):
        for x in e:
            yield from _walk(x)
        return
    if e is None or isinstance(e, (str, int, float, bool, F.Type, tuple)):
        return
    yield e
    for f in getattr(e, "__dataclass_fields__", {}):
        v = getattr(e, f)
        if isinstance(v, (F.Expr, list)) or hasattr(v, "__dataclass_fields__"):
            yield from _walk(v)


@dataclass
class Item:
    kind: str                 # "map" | "reduce"
    target: str = ""          # map: vector written
    m: object = None          # map: F.Map
    sym: Sym = None           # reduce: the reduced symbol
    index: int = -1           # map: index into em.maps


@dataclass
class Phase:
    count: str                # C expression of the element count
    items: list = field(default_factory=list)
    written: list = field(default_factory=list)      # vectors written, in order
    reduced: set = field(default_factory=set)        # reduced symbols produced here
    read_elsewhere: set = field(default_factory=set)  # vectors read at an index other than the own one


class FusedPlan:
    """Phase plan of one function; ``ok`` is False when the staged target must be used."""

    def __init__(self, em: Emitter, stages: list | None = None):
        self.em = em
        self.stages = list(em.stages if stages is None else stages)
        self.phases: list[Phase] = []
        self.ok = True
        self.why = ""
        try:
            self._plan()
        except _NoFusion as e:
            self.ok, self.why = False, str(e)

    # -------------------------------------------------------------- analysis
    def _lambda_of(self, name_expr):
        em = self.em
        if not isinstance(name_expr, F.Name) or em.syms.get(name_expr.id, Sym("", "", None)).kind != "lambda":
            raise _NoFusion("map / reduce function is not a named lambda")
        return em.syms[name_expr.id]

    def _scalar_deps(self, node, seen=None) -> set:
        """Names of reduced symbols an expression (or lambda body) depends on."""
        em, out = self.em, set()
        seen = seen if seen is not None else set()
        for n in _walk(node):
            if isinstance(n, F.Name) and n.id in em.syms and n.id not in seen:
                s = em.syms[n.id]
                seen.add(n.id)
                if s.kind == "reduced":
                    out.add(n.id)
                elif s.kind == "derived":
                    out |= self._scalar_deps(s.expr, seen)
                elif s.kind == "lambda":
                    out |= self._scalar_deps(s.expr.body, seen)
                elif s.kind == "vector" and s.bits is not None:
                    out |= self._scalar_deps(s.bits, seen)
        return out

    def _vector_reads(self, lam: F.Lambda, own_index: str | None):
        """(vectors read at the own index, vectors read at any other index)."""
        em = self.em
        own, other = set(), set()
        for n in _walk(lam.body):
            if isinstance(n, F.Index) and isinstance(n.base, F.Name) and \
                    em.syms.get(n.base.id, Sym("", "", None)).kind in ("param_vector", "vector"):
                if own_index is not None and isinstance(n.idx, F.Name) and n.idx.id == own_index:
                    own.add(n.base.id)
                else:
                    other.add(n.base.id)
            elif isinstance(n, F.Call) and n.fn in em.syms and em.syms[n.fn].kind == "lambda":
                raise _NoFusion("a lambda that calls another lambda")
        return own, other

    def _count_of_map(self, m: F.Map) -> str:
        em = self.em
        if m.vec is not None:
            if not isinstance(m.vec, F.Name):
                raise _NoFusion("map over an expression")
            return f"c.n_{m.vec.id}"
        if isinstance(m.count, F.SizeOf) and isinstance(m.count.base, F.Name):
            return f"c.n_{m.count.base.id}"
        return f"(uint64_t)({em.expr(m.count, set())})"

    def _plan(self):
        em = self.em
        cur: Phase | None = None

        def close():
            nonlocal cur
            if cur is not None and cur.items:
                self.phases.append(cur)
            cur = None

        for st in self.stages:
            if st[0] in ("topk", "scatter"):
                raise _NoFusion("library-lowered stage")
            if st[0] == "reduce":
                for s in st[1]:
                    r: F.Reduce = s.expr
                    if not isinstance(r.vec, F.Name):
                        raise _NoFusion("reduce over an expression")
                    count = f"c.n_{r.vec.id}"
                    if cur is not None and r.vec.id in cur.written:
                        count = cur.count      # just produced over the phase's range
                    needs = self._scalar_deps(r.init)
                    if not (isinstance(r.fn, F.Name) and r.fn.id in ("smaller", "greater", "sum")
                            and r.fn.id not in em.syms):
                        lam = self._lambda_of(r.fn)
                        needs |= self._scalar_deps(lam.expr.body)
                        if self._vector_reads(lam.expr, None)[1]:
                            raise _NoFusion("a reducer that reads vectors")
                    if cur is None or cur.count != count or (needs & cur.reduced) or \
                            r.vec.id in cur.read_elsewhere:
                        close()
                        cur = Phase(count)
                    cur.items.append(Item("reduce", sym=s))
                    cur.reduced.add(s.name)
                continue
            target, m = em.maps[st[1]]
            lam = self._lambda_of(m.fn).expr
            count = self._count_of_map(m)
            if cur is not None and m.vec is not None and m.vec.id in cur.written:
                count = cur.count
            own_idx = lam.params[0][1] if (m.vec is None and lam.params) else None
            own, other = self._vector_reads(lam, own_idx)
            if m.vec is not None:
                own.add(m.vec.id)
            needs = self._scalar_deps(lam.body) | self._scalar_deps(em.syms[target].bits)
            if m.count is not None:
                needs |= self._scalar_deps(m.count)
            fresh = cur is None or cur.count != count or (needs & cur.reduced) or \
                bool(other & set(cur.written)) or target in cur.read_elsewhere or \
                (target in other)
            if fresh:
                close()
                cur = Phase(count)
            cur.items.append(Item("map", target=target, m=m, index=st[1]))
            cur.written.append(target)
            cur.read_elsewhere |= other
        close()
        if not self.phases:
            raise _NoFusion("nothing to launch")


class _NoFusion(Exception):
    pass


def fused_segments(em: Emitter) -> list:
    """For a function that keeps the staged target because of a library-lowered stage:
    the runs of consecutive ``map`` stages between the library calls that can still be
    one kernel.  Returns [(index of the run's first stage, number of stages, FusedPlan)].
    Kept simple on purpose: the function has no reduction, the run has at least two
    maps, none of them draws random numbers (the call sites are numbered per target)
    and the run plans as a single phase, so the kernel needs no grid barrier."""
    if em.reduces:
        return []
    out, i, n = [], 0, len(em.stages)
    while i < n:
        j = i
        while j < n and em.stages[j][0] == "map":
            j += 1
        run = em.stages[i:j]
        if len(run) >= 2:
            rnd = False
            for st in run:
                lam = em.syms.get(getattr(em.maps[st[1]][1].fn, "id", ""), None)
                if lam is None or any(isinstance(x, F.Random) for x in _walk(lam.expr.body)):
                    rnd = True
            plan = None if rnd else FusedPlan(em, run)
            if plan is not None and plan.ok and len(plan.phases) == 1:
                out.append((i, len(run), plan))
        i = max(j, i + 1)
    return out


def _ordered(r: F.Reduce) -> bool:
    """Whether the result of a reduction depends on the order of its steps (a sum of floats
    does, a minimum does not): such a function keeps its split over threads and blocks, so
    that the same input gives the same bits from one version to the next."""
    return not (isinstance(r.fn, F.Name) and r.fn.id in ("smaller", "greater"))


def _is_num(e, value: float) -> bool:
    return isinstance(e, F.Num) and float(e.text) == value


class FusedGen:
    """Emits the fused kernel and its launch for a plan that is ``ok``."""

    def __init__(self, plan: FusedPlan, tag: str = "fused", write_header: bool = True):
        self.plan, self.em = plan, plan.em
        self.name = self.em.fn.name
        self.tag = tag                    # kernel name: <function>_<tag>_kernel
        self.write_header = write_header  # the launch that runs last writes the concat headers

    # ------------------------------------------------------------ helpers
    def _apply(self, r: F.Reduce, a: str, b: str) -> str:
        return self.em._apply(r.fn, a, b)

    def _prologue_lines(self):
        rows = self.em.prologue().replace("scalars[", "red[").splitlines()
        return [r for r in rows if r.strip() not in ("Ctx c;", "c.seed = seed;")]

    def _elem_type(self, vec: str) -> str:
        s = self.em.syms[vec]
        return "uint32_t" if s.bits is not None else C_TYPES[s.type.name]

    # ------------------------------------------------------------- phases
    def _phase(self, pi: int, ph: Phase, last: bool) -> str:
        em = self.em
        need_in: dict[str, None] = {}
        need_frag: dict[str, None] = {}
        sites: list[int] = []
        fwd: dict[str, str] = {}
        body = []
        last_writer = {it.target: k for k, it in enumerate(ph.items) if it.kind == "map"}

        def scalar(e) -> str:
            # for use outside the loop over elements too, which the hooked forms belong to
            hook, em._binary_hook = em._binary_hook, None
            try:
                return em.expr(e, set())
            finally:
                em._binary_hook = hook

        def index_hook(sym, idx, local):
            own = em._own
            if own is None or not (isinstance(idx, F.Name) and idx.id == own and idx.id in local):
                return None
            if sym.name in fwd:
                return fwd[sym.name]
            if sym.bits is None:
                need_in[sym.name] = None
                return f"in_{sym.name}[u][e]"
            return frag_value(sym)

        def frag_value(sym):
            # a packed input read at the own index: the group's fragment is loaded once
            need_frag[sym.name] = None
            b = f"(uint32_t)({scalar(sym.bits)})"
            return f"((fr_{sym.name}[u] >> (e * {b})) & ((1u << {b}) - 1u))"

        def random_hook(site):
            sites.append(site)
            return f"hipress::u01(rg{site}.v[e])"

        def stream_value(vec: str) -> str:
            if vec in fwd:
                return fwd[vec]
            s = em.syms[vec]
            if s.bits is None:
                need_in[vec] = None
                return f"in_{vec}[u][e]"
            return frag_value(s)

        reducing = any(it.kind == "reduce" for it in ph.items)
        divisors: dict[str, None] = {}
        flags: list[str] = []

        def float_scalar(e, local):
            return isinstance(e, F.Name) and e.id not in local and e.id in em.syms and \
                em.syms[e.id].kind in ("param_scalar", "reduced", "derived", "extracted") and \
                em.syms[e.id].type.name == "float"

        def unit_draw(e):
            return isinstance(e, F.Random) and e.type == "float" and _is_num(e.lo, 0) and _is_num(e.hi, 1)

        def binary_hook(e, local, expr):
            if e.op == "/" and float_scalar(e.b, local) and not reducing:
                # one divisor for the whole phase; the elements run a second time, with `/`,
                # where a quotient may have come out wrong, so nothing may be accumulated
                divisors[e.b.id] = None
                num = f"(float)({expr(e.a)})"
                return f"(exact ? {num} / c.v_{e.b.id} : compll_div({num}, dv_{e.b.id}, bad))"
            if e.op == "+" and (unit_draw(e.a) or unit_draw(e.b)):
                # the draw is a multiple of 2^-24: exact, so one rounding either way
                first = None if unit_draw(e.a) else expr(e.a)     # sites count in source order
                site, em.rand_sites = em.rand_sites, em.rand_sites + 1
                sites.append(site)
                other = expr(e.b) if first is None else first
                return f"fmaf((float)(rg{site}.v[e] >> 8), 1.0f / 16777216.0f, (float)({other}))"
            return None

        def cond_hook(cond, local):
            # a condition on scalars alone: the loop is compiled for both of its values
            names = [n for n in _walk(cond) if isinstance(n, (F.Name, F.Index, F.Random, F.Call, F.SizeOf))]
            if not names or any(not isinstance(n, F.Name) or n.id in local or
                                em.syms[n.id].kind not in ("param_scalar", "reduced", "derived", "extracted")
                                for n in names):
                return None
            text = scalar(cond)
            if text not in flags:
                if flags:
                    return None
                flags.append(text)
            return "flag"

        em._index_hook, em._random_hook = index_hook, random_hook
        em._binary_hook, em._cond_hook = binary_hook, cond_hook
        decls, stores, whole_stores = [], [], []
        try:
            for k, it in enumerate(ph.items):
                if it.kind == "reduce":
                    r: F.Reduce = it.sym.expr
                    ty = C_TYPES[it.sym.type.name]
                    body.append(f"        acc_{it.sym.name} = "
                                f"{self._apply(r, 'acc_' + it.sym.name, '(' + ty + ')' + stream_value(r.vec.id))};")
                    continue
                tgt = em.syms[it.target]
                lam_sym = em.syms[it.m.fn.id]
                lam: F.Lambda = lam_sym.expr
                sub = tgt.bits is not None
                rty = "uint32_t" if sub else C_TYPES[tgt.type.name]
                lret = "uint32_t" if lam.ret.is_subbyte() else C_TYPES[lam.ret.name]
                var = f"r{pi}_{k}"
                decls.append(f"      {rty} {var}[4] = {{0, 0, 0, 0}};")
                pty, pname = lam.params[0]
                local = {pname}
                if it.m.vec is not None:       # map over a vector: the parameter is the element
                    em._own = None
                    pinit = f"({C_TYPES[pty.name]})({stream_value(it.m.vec.id)})"
                else:
                    em._own = pname
                    pinit = f"({C_TYPES[pty.name]})i"
                em._counter = pname
                em._return_to = "res"
                code = em.stmts(lam.body, local, lam.ret.is_subbyte(), indent="            ")
                em._return_to = None
                mask = ""
                if sub:
                    mask = f" & ((1u << (uint32_t)({scalar(tgt.bits)})) - 1u)"
                body.append(f"""        {{  // {it.target} = map(..., {lam_sym.name})
          const {C_TYPES[pty.name]} l_{pname} = {pinit};
          {lret} res = 0;
          do {{
{code}
          }} while (0);
          {var}[e] = (({rty})res){mask};
        }}""")
                fwd[it.target] = f"{var}[e]"
                if last_writer[it.target] == k:
                    if sub:
                        bits = f"(uint32_t)({scalar(tgt.bits)})"
                        stores.append(f"""      {{
        const uint32_t bits = {bits};
        const uint32_t frag = {var}[0] | ({var}[1] << bits) | ({var}[2] << (2 * bits)) | ({var}[3] << (3 * bits));
        compll_pack_store(c.v_{it.target}, (count * bits + 7) / 8, q, frag, bits);
      }}""")
                        whole_stores.append(stores[-1].replace(
                            f"compll_pack_store(c.v_{it.target}, (count * bits + 7) / 8, q, frag, bits)",
                            f"compll_pack_full(c.v_{it.target}, q, frag, bits)"))
                    else:
                        stores.append(f"      compll_store4(c.v_{it.target}, i0, count, {var});")
                        whole_stores.append(stores[-1] if rty != "float" else
                                            f"      reinterpret_cast<float4*>(c.v_{it.target})[q] = "
                                            f"make_float4({var}[0], {var}[1], {var}[2], {var}[3]);")
        finally:
            em._index_hook = em._random_hook = em._binary_hook = em._cond_hook = None
            em._own = None
            em._return_to = None
        # U groups of four elements per thread and trip, every load of a trip issued before
        # the first result is computed (a map only reads its own elements of the vectors
        # it also writes, so hoisting the loads over the stores is safe).
        # Four groups where nothing but packed fragments comes in or nothing goes out.  A phase
        # that streams floats in and out has enough loads with one group, but behind a header
        # (whose fields every block has to read first) or a barrier two pay: not where 32
        # registers are the limit (a sum, see _ordered: OnebitEncode of 64 M elements 244 us
        # with two, 228 with one) nor beside single bits (OnebitDecodeAccumulate 100 with two,
        # 90 with one; TernGradDecodeAccumulate 90 and 92).
        headed = bool(em.extracts) or len(self.plan.phases) > 1
        bits = [em.syms[v].bits for v in need_frag]
        two = headed and not any(isinstance(b, F.Num) and b.text == "1" for b in bits)
        U = 4 if not need_in or not stores else (2 if two else 1)
        if any(_ordered(r.expr) for r in em.reduces):
            U = 1
        # groups of a block in a grid that is not limited: a block that reads a header is
        # worth more of them (TernGradDecodeAccumulate of 16.8 M elements 28.8 us with one
        # group per thread and block, 25.4 with four), and a decode, whose loads are few,
        # still more (64 M elements, OnebitDecode 57 us with four and 53 with sixteen, TbqDecode
        # 59 and 57; the decode-accumulates lose up to 28 % with sixteen)
        self.unroll = (4 if need_in else 16) if headed else U
        # one test for the four elements of nearly every group, where loads of floats are to
        # overlap; the decodes are faster without it (TbqDecode of 64 M elements 65 us, now 59)
        skip = "!full && i >= count" if need_in else "i >= count"
        larr = [f"      {C_TYPES[em.syms[v].type.name]} in_{v}[{U}][4];" for v in need_in] + \
               [f"      uint32_t fr_{v}[{U}];" for v in need_frag]
        loads = [f"        compll_load4(c.v_{v}, i0, count, in_{v}[u]);" for v in need_in]
        for v in need_frag:
            b = f"(uint32_t)({em.expr(em.syms[v].bits, set())})"
            loads.append(f"        fr_{v}[u] = compll_load_frag(c.v_{v}, (c.n_{v} * {b} + 7) / 8, q, {b});")
        rngs = [f"      const hipress::Philox4 rg{s} = compll_rand4(c.seed, q, {s}u);" for s in sorted(set(sites))]
        reds = [it.sym for it in ph.items if it.kind == "reduce"]
        acc_init = [f"    {C_TYPES[s.type.name]} acc_{s.name} = ({C_TYPES[s.type.name]})"
                    f"({em.expr(s.expr.init, set())});" for s in reds]
        nl = "\n"
        header = ""
        if last and self.write_header:
            rows = []
            for tname, fields, _ in em.concats:
                for fname, off in fields:
                    s = em.syms[fname]
                    rows.append(f"      compll_store<{C_TYPES[s.type.name]}>(reinterpret_cast<uint8_t*>"
                                f"(p_{tname}) + {off}, c.v_{fname});")
            if rows:
                header = "    if (blockIdx.x == 0 && threadIdx.x == 0) {\n" + nl.join(rows) + "\n    }\n"
        def elements(skip_test: str) -> str:
            loop = f"""#pragma unroll
      for (int e = 0; e < 4; ++e) {{
        const uint64_t i = i0 + e;
        (void)i;
{skip_test}{nl.join(body)}
      }}"""
            if not divisors:
                return loop
            ok = " && ".join(f"dv_{d}.ok" for d in divisors)
            return f"""      auto elements = [&](auto exact_) {{
        constexpr bool exact = decltype(exact_)();
        uint32_t bad = 0;
{loop}
        return bad >> 31;
      }};
      if (!({ok}) || elements(CompllFlag<false>())) elements(CompllFlag<true>());"""

        main = f"""    for (; qb0 < groups; qb0 += stride * {U}) {{
{nl.join(larr)}
#pragma unroll
      for (int u = 0; u < {U}; ++u) {{   // past the end the loads return zeros and touch nothing
        const uint64_t q = qb0 + u * stride + threadIdx.x;
        const uint64_t i0 = q * 4;
        (void)q; (void)i0;
{nl.join(loads)}
      }}
#pragma unroll
      for (int u = 0; u < {U}; ++u) {{
      const uint64_t qb = qb0 + u * stride;   // the same for the whole block
      if (qb >= groups) break;
      const uint64_t q = qb + threadIdx.x;
      const uint64_t i0 = q * 4;
      const bool full = i0 + 3 < count;
      (void)full;
{nl.join(rngs)}
{nl.join(decls)}
{elements(f"        if ({skip}) continue;{nl}")}
{nl.join(stores)}
      }}
    }}
"""
        start = "    uint64_t qb0 = (uint64_t)blockIdx.x * blockDim.x;\n"
        # Blocks whose groups are all complete run without bounds tests and with 32-bit
        # indices.  TernGradEncode of 16.8 M elements took 56 us, of 67 M 207, and takes 37
        # and 139 with these loops: 36 instructions per element of its second phase were the
        # bound, 27 are left, 10 of them the random draws.  A trip of loads ahead cost more
        # in registers than it gained (39 and 148 us).  Functions with sums gain 1 to 3 % and
        # lose 7 % at 100 K elements, those of a single phase nothing: they keep one loop.
        whole = bool(need_in) and len(self.plan.phases) > 1 and not any(_ordered(r.expr) for r in em.reduces)
        if whole:
            floats = [v for v in need_in if em.syms[v].type.name == "float"]
            touched = sorted(set(floats) | {it.target for it in ph.items if it.kind == "map" and
                                            em.syms[it.target].bits is None and em.syms[it.target].type.name == "float"})
            address = " | ".join(f"reinterpret_cast<uint64_t>(c.v_{v})" for v in touched) or "0"
            wloads = [f"""        {{
          const float4 t = reinterpret_cast<const float4*>(c.v_{v})[q];
          in_{v}[u][0] = t.x; in_{v}[u][1] = t.y; in_{v}[u][2] = t.z; in_{v}[u][3] = t.w;
        }}""" if v in floats else f"        compll_load4(c.v_{v}, (uint64_t)q * 4, count, in_{v}[u]);" for v in need_in]
            wloads += [ld.replace(", q, ", ", (uint64_t)q, ") for ld in loads[len(need_in):]]
            wrngs = [f"      const hipress::Philox4 rg{s} = rand(q, {s}u);" for s in sorted(set(sites))]
            start += f"""    const uint32_t whole = compll_whole(count, {address});
    if (whole) {{
      const uint32_t step = (uint32_t)stride;
      for (uint32_t qw = (uint32_t)qb0; qw < whole; qw += step * {U}) {{
{nl.join(larr)}
#pragma unroll
      for (int u = 0; u < {U}; ++u) {{
        const uint32_t q = qw + u * step + threadIdx.x;
        if (u > 0 && qw + u * step >= whole) break;
{nl.join(wloads)}
      }}
#pragma unroll
      for (int u = 0; u < {U}; ++u) {{
      if (u > 0 && qw + u * step >= whole) break;
      const uint32_t q = qw + u * step + threadIdx.x;
      const uint64_t i0 = (uint64_t)q * 4;
      (void)i0;
{nl.join(wrngs)}
{nl.join(decls)}
{elements("")}
{nl.join(whole_stores)}
      }}
      }}
      // the block whose turn it is takes the groups that are left
      qb0 = whole / 256u % gridDim.x == blockIdx.x ? whole : groups;
    }}
"""
        main = self._per_width(start + main, need_frag, ph, flags)
        once = [f"    const CompllDivisor dv_{d} = compll_divisor(c.v_{d});" for d in divisors]
        if whole and sites:
            once.append("    const CompllRand rand(c.seed);")
        out = f"""  {{  // ---- phase {pi}: {', '.join((it.target if it.kind == 'map' else 'reduce ' + it.sym.name) for it in ph.items)}
{header}    const uint64_t count = {ph.count};
    const uint64_t groups = (count + 3) / 4;
{nl.join(acc_init + once)}
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
{main}{self._block_reduce(reds)}  }}
"""
        return out

    def _per_width(self, main: str, need_frag, ph: Phase, flags: list) -> str:
        """A width that is a scalar of the function (a parameter, a header field) makes every
        shift and mask of the packing a run-time one: the loop is compiled for the widths
        1, 2, 4 and 8 as well, and the kernel takes the one that applies.  So it is for both
        values of a condition on scalars (`flags`): as a branch in the loop
        TernGradEncode's cost 7 instructions per element."""
        em = self.em
        names = set()
        for v in list(need_frag) + [it.target for it in ph.items if it.kind == "map"]:
            bits = em.syms[v].bits
            if isinstance(bits, F.Name) and em.syms[bits.id].kind in ("param_scalar", "extracted"):
                names.add(bits.id)
        name = f"c.v_{names.pop()}" if len(names) == 1 else None
        if name is None and not flags:
            return "    {\n" + main + "    }\n"
        body = main if name is None else main.replace(name, "width")
        params = (["auto width_"] if name else []) + (["auto flag_"] if flags else [])
        head = ("      const uint32_t width = width_;\n" if name else "") + \
            ("      constexpr bool flag = decltype(flag_)();\n" if flags else "")

        def call(width):
            one = lambda f: f"loop({', '.join(([width] if name else []) + ([f'CompllFlag<{f}>()'] if flags else []))});"  # noqa: E731
            return f"if ({flags[0]}) {one('true')} else {one('false')}" if flags else one("")

        cases = call("") if name is None else \
            f"switch ({name}) {{ " + " ".join(f"case {w}: {call(f'CompllWidth<{w}>()')} break;" for w in (1, 2, 4, 8)) + \
            f" default: {call(f'(uint32_t){name}')} }}"
        return f"""    auto loop = [&]({', '.join(params)}) {{
{head}{body}    }};
    {cases}
"""

    def _block_reduce(self, reds) -> str:
        if not reds:
            return ""
        rows = ["    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;",
                "    for (int off = 16; off > 0; off >>= 1) {"]
        for s in reds:
            ty = C_TYPES[s.type.name]
            rows.append(f"      {{ {ty} o = __shfl_xor_sync(0xffffffffu, acc_{s.name}, off); "
                        f"acc_{s.name} = {self._apply(s.expr, 'acc_' + s.name, 'o')}; }}")
        rows.append("    }")
        rows.append("    __syncthreads();")
        rows.append("    if (lane == 0) { " + " ".join(f"sh[{s.slot}][warp] = (float)acc_{s.name};" for s in reds) + " }")
        rows.append("    __syncthreads();")
        rows.append("    if (threadIdx.x == 0) {")
        for s in reds:
            ty = C_TYPES[s.type.name]
            rows.append(f"      {{ {ty} a = ({ty})sh[{s.slot}][0]; for (int w = 1; w < 8; ++w) "
                        f"a = {self._apply(s.expr, 'a', '(' + ty + ')sh[' + str(s.slot) + '][w]')}; "
                        f"partials[{s.slot} * gridDim.x + blockIdx.x] = (float)a; }}")
        rows.append("    }")
        return "\n".join(rows) + "\n"

    def _fold(self, reds) -> str:
        """Behind the barrier: every block folds the per-block partials itself."""
        rows = []
        free = [s for s in reds if not _ordered(s.expr)]
        if free:
            # all together: every thread ends with the results, behind one barrier
            types = [C_TYPES[s.type.name] for s in free]
            part = lambda s, ty: f"({ty})__ldcg(&partials[{s.slot} * gridDim.x + w])"  # noqa: E731
            rows.append("  {")
            rows += [f"    {ty} f_{s.name} = ({ty})({self.em.expr(s.expr.init, set())});" for s, ty in zip(free, types)]
            rows.append("    for (unsigned w = threadIdx.x; w < gridDim.x; w += blockDim.x) {")
            rows += [f"      f_{s.name} = {self._apply(s.expr, 'f_' + s.name, part(s, ty))};" for s, ty in zip(free, types)]
            rows.append("    }\n    for (int off = 16; off > 0; off >>= 1) {")
            rows += [f"      {{ {ty} o = __shfl_xor_sync(0xffffffffu, f_{s.name}, off); "
                     f"f_{s.name} = {self._apply(s.expr, 'f_' + s.name, 'o')}; }}" for s, ty in zip(free, types)]
            rows.append("    }\n    if ((threadIdx.x & 31) == 0) {")
            rows += [f"      sh[{s.slot}][threadIdx.x >> 5] = (float)f_{s.name};" for s in free]
            rows.append("    }\n    __syncthreads();")
            for s, ty in zip(free, types):
                rows.append(f"    f_{s.name} = ({ty})sh[{s.slot}][0];\n    for (int w = 1; w < 8; ++w) f_{s.name} = "
                            f"{self._apply(s.expr, 'f_' + s.name, '(' + ty + ')sh[' + str(s.slot) + '][w]')};\n"
                            f"    red[{s.slot}] = (float)f_{s.name};\n"
                            f"    if (blockIdx.x == 0 && threadIdx.x == 0) scalars[{s.slot}] = red[{s.slot}];")
            rows.append("  }")
        for s in reds:
            if not _ordered(s.expr):
                continue
            ty = C_TYPES[s.type.name]
            init = self.em.expr(s.expr.init, set())
            load = '(' + ty + ')__ldcg(&partials[' + str(s.slot) + ' * gridDim.x + w])'
            # one warp, every lane in a fixed order; eight loads in flight
            fold = f"""    if (threadIdx.x < 32) {{
#pragma unroll 8
      for (unsigned w = threadIdx.x; w < gridDim.x; w += 32)
        a = {self._apply(s.expr, 'a', load)};
      for (int off = 16; off > 0; off >>= 1) {{
        {ty} o = __shfl_xor_sync(0xffffffffu, a, off);
        a = {self._apply(s.expr, 'a', 'o')};
      }}
      if (threadIdx.x == 0) sh[{s.slot}][0] = (float)a;
    }}
    __syncthreads();"""
            rows.append(f"""  {{
    {ty} a = ({ty})({init});
{fold}
    red[{s.slot}] = sh[{s.slot}][0];
    __syncthreads();
    if (blockIdx.x == 0 && threadIdx.x == 0) scalars[{s.slot}] = red[{s.slot}];
  }}""")
        return "\n".join(rows)

    # -------------------------------------------------------------- kernel
    def kernel_source(self) -> str:
        em, name = self.em, self.name
        phases = self.plan.phases
        nred = max(len(em.reduces), 1)
        pro = "\n".join(self._prologue_lines())
        parts = []
        for pi, ph in enumerate(phases):
            parts.append(self._phase(pi, ph, pi == len(phases) - 1))
            if pi != len(phases) - 1:
                reds = [it.sym for it in ph.items if it.kind == "reduce"]
                parts.append(f"  compll_grid_sync(sync, gen, sync + 2);\n{self._fold(reds)}\n{pro}\n")
        tail = ""
        if len(phases) > 1:
            tail = """  // the last block to leave clears the barrier words for the next launch
  __syncthreads();
  if (threadIdx.x == 0 && atomicAdd(sync + 1, 1u) == gridDim.x - 1) {
    sync[0] = 0;
    sync[1] = 0;
    sync[32] = 0;
  }
"""
        bound = ", 8" if any(_ordered(s.expr) for s in em.reduces) else ""   # kMaxBlocks resident
        return f"""
constexpr uint64_t {name}_{self.tag}_groups = {self.unroll};  // of four elements, per thread of a block

// One launch for the whole function: {len(phases)} phase(s){', grid barriers in between' if len(phases) > 1 else ''}.
__global__ void __launch_bounds__(256{bound}) {name}_{self.tag}_kernel({em.kernel_params()}, float* partials,
                                                       unsigned int* sync) {{
  __shared__ float sh[{nred}][8];
  float red[{nred}];
  for (int k = 0; k < {nred}; ++k) red[k] = 0.0f;
  unsigned int gen = 0;
  (void)gen; (void)sh; (void)partials; (void)sync;
  Ctx c;
  c.seed = seed;
{pro}
{''.join(parts)}{tail}}}
"""

    def launch_rows(self) -> str:
        """Body of the launcher: grid sizing and the (cooperative) launch."""
        name = self.name
        coop = len(self.plan.phases) > 1
        if coop:
            # all blocks resident; no more per SM than keep it busy, because every one of them
            # arrives at the same barrier word, 10 ns each.  TernGradEncode, 2 bits, us with
            # what fits / four / two blocks per SM: 0.5 M elements 14.3 / 14.3 / 12.3, 1 M
            # 18.4 / 16.4 / 14.3, 4 M 28.1 / 26.6 / 26.6, 8 M 41.0 / 38.9 / 41.0, 16 M 65.5 /
            # 63.5 / 73.7, 32 M 117 / 117 / 147, 64 M 215 / 219 / 274: four lose little anywhere
            most = "kMaxBlocks" if any(_ordered(s.expr) for s in self.em.reduces) else "kMaxBlocks / 2"
            rows = ("    if (blocks > (uint64_t)cap[dev]) blocks = cap[dev];\n"
                    f"    if (blocks > {most}) blocks = {most};")
        else:
            # nothing waits: a few thousand blocks, which the hardware gives to whichever SM is
            # free (a fixed share for every resident block costs about a tenth of the bandwidth),
            # and of a small array as many as fit (TbqDecodeAccumulate of 64 K elements 8.2 us
            # with several groups per thread, 6.2 with one)
            unroll = f"compll_gen_{name}::{name}_{self.tag}_groups"
            rows = ("    const uint64_t fit = blocks < (uint64_t)cap[dev] ? blocks : cap[dev];\n"
                    f"    blocks = (blocks + {unroll} - 1) / {unroll};\n"
                    "    if (blocks < fit) blocks = fit;\n"
                    "    if (blocks > 0x7FFFFFFFull) blocks = 0x7FFFFFFFull;")
        most_rows = "\n".join(f"    if (n_{pname} > most) most = n_{pname};"
                              for ty, pname in self.em.fn.params if ty.vector)
        return f"""  {{
    static int cap[64] = {{0}};           // blocks the device holds at once
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (cap[dev] == 0) {{
      int sms = 0, per = 0;
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, compll_gen_{name}::{name}_{self.tag}_kernel, 256, 0);
      cap[dev] = per * sms > 0 ? per * sms : 1;
    }}
    uint64_t most = work;
{most_rows}
    uint64_t blocks = (most / 4 + 255) / 256;
{rows}
    const int fgrid = blocks < 1 ? 1 : (int)blocks;
    unsigned int* sync = ticket;
    void* args[] = {{{', '.join('(void*)&' + a for a in self._arg_names())}, (void*)&partials, (void*)&sync}};
    cudaError_t e = {'cudaLaunchCooperativeKernel' if coop else 'cudaLaunchKernel'}(
        (const void*)compll_gen_{name}::{name}_{self.tag}_kernel, dim3(fgrid), dim3(256), args, 0, st);
    if (e != cudaSuccess) return (int)e;
  }}"""

    def _arg_names(self):
        a = []
        for ty, pname in self.em.fn.params:
            a += [f"p_{pname}", f"n_{pname}"] if ty.vector else [f"p_{pname}"]
        return a + ["scalars", "seed"]
