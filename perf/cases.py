"""Workloads of the coupled-cluster engine for timing: what a program that solves CC equations calls.

Every case goes through ``ccq_b200.lib.Context``, the binding of the C ABI, as the driver and the batched
solver do.  A pass of a resident case is one DIIS cycle of a solve (the amplitudes set to their start, the
iterations with energy, residuum and extrapolation, the amplitudes read back); of a host case one iteration of
a program that keeps its amplitude vector on the host; of a batch one DIIS cycle of several independent solves
that overlap; of a left case the left CCSD iterations and the triples corrections.  The Hamiltonians are seeded
synthetic ones with decaying factors and a gap, the amplitudes start where a solve starts.
"""
import itertools
import math

import numpy as np
import torch

from ccq_b200 import lib

DEV = 'cuda' if torch.cuda.is_available() else 'cpu'
F64 = torch.float64
DIIS = 5
T12 = ('T1A', 'T1B', 'T2A', 'T2B', 'T2C')
T3 = ('T3A', 'T3B', 'T3C', 'T3D')
T4 = ('T4A', 'T4B', 'T4C', 'T4D', 'T4E')
CYCLE = DIIS + 1


def _case(kind, method, orbs, occ_a, occ_b, froz=0, its=CYCLE, rhf=False, precision='fp64', tuned=False,
          act_occ=0, act_unocc=0, count=1):
    return dict(kind=kind, method=method, orbs=orbs, occ_a=occ_a, occ_b=occ_b, froz=froz, its=its, rhf=rhf,
                precision=precision, tuned=tuned, act_occ=act_occ, act_unocc=act_unocc, count=count)


def listed():
    named = [
        # a molecule in a minimal basis: every launch is tiny, latency and launches are all there is
        ('ccsd_8', _case('resident', 'CCSD', 8, 4, 4)),
        # CCSD of the small benchmark molecule (20 orbitals, 10 electrons)
        ('ccsd_20', _case('resident', 'CCSD', 20, 5, 5)),
        # an open shell with a frozen core and odd extents everywhere
        ('ccsd_33_open', _case('resident', 'CCSD', 33, 8, 6, froz=1)),
        # the largest system of the batched study, closed shell with the spin copies
        ('ccsd_48_rhf', _case('resident', 'CCSD', 48, 9, 9, rhf=True)),
        # many independent Hamiltonians of uneven size at once (16 to 30 orbitals)
        ('ccsd_batch_8', _case('batch', 'CCSD', 30, 6, 6, count=8)),
        # a small open-shell CCSDT
        ('ccsdt_13_open', _case('resident', 'CCSDT', 13, 4, 3)),
        # the Hamiltonian family of the warm-start study
        ('ccsdt_24', _case('resident', 'CCSDT', 24, 5, 5)),
        # the headline: 40 orbitals, 16 electrons, kernels picked by the autotuner as its users do
        ('ccsdt_40', _case('resident', 'CCSDT', 40, 8, 8, tuned=True)),
        # the same system for a program that keeps t_vec on the host, bulk contractions in split precision
        ('ccsdt_40_host_split', _case('host', 'CCSDT', 40, 8, 8, its=1, precision='split')),
        # active-space triples
        ('ccsdt_act_32', _case('resident', 'CCSDt', 32, 7, 7, its=DIIS, act_occ=2, act_unocc=5)),
        # quadruples
        ('ccsdtq_14', _case('resident', 'CCSDTQ', 14, 4, 4, rhf=True)),
        # left CCSD and CR-CC(2,3) of the 32-orbital benchmark molecule
        ('left_32', _case('left', 'CR-CC(2,3)', 32, 7, 7)),
    ]
    return [dict(c, name=n) for n, c in named]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    pick = rng.choice(('ccsd', 'ccsd', 'batch', 'ccsdt', 'ccsdt', 'host', 'act', 'quad', 'left'))
    if pick == 'ccsd':
        orbs = _log_int(rng, 7, 48)
        occ = max(2, int(orbs / rng.uniform(2.2, 5.5)))
        opened = rng.choice((0, 0, 1, 2)) if occ > 3 else 0
        return _case('resident', 'CCSD', orbs, occ, occ - opened, froz=rng.choice((0, 1)) if occ > 3 else 0,
                     rhf=opened == 0 and rng.random() < 0.4, tuned=rng.random() < 0.2)
    if pick == 'batch':
        orbs = rng.randint(16, 36)
        return _case('batch', 'CCSD', orbs, orbs // 5, orbs // 5, count=rng.randint(4, 10))
    if pick == 'ccsdt':
        orbs = _log_int(rng, 8, 36)
        occ = min(8, max(3, orbs // rng.choice((3, 4, 5))))
        opened = rng.choice((0, 0, 1))
        return _case('resident', 'CCSDT', orbs, occ, occ - opened, froz=rng.choice((0, 0, 1)) if occ > 3 else 0,
                     rhf=opened == 0 and rng.random() < 0.3, tuned=rng.random() < 0.3)
    if pick == 'host':
        orbs = rng.randint(20, 38)
        return _case('host', 'CCSDT', orbs, orbs // 5, orbs // 5, its=1,
                     precision='split' if rng.random() < 0.5 else 'fp64')
    if pick == 'act':
        orbs = rng.randint(14, 36)
        occ = min(8, orbs // 4)
        return _case('resident', 'CCSDt', orbs, occ, occ, its=DIIS, act_occ=rng.randint(1, 2),
                     act_unocc=rng.randint(2, 6))
    if pick == 'quad':
        orbs = rng.randint(9, 14)
        occ = rng.choice((3, 4))
        opened = rng.choice((0, 1))
        return _case('resident', 'CCSDTQ', orbs, occ, occ - opened, rhf=opened == 0 and rng.random() < 0.5)
    orbs = rng.randint(12, 34)
    return _case('left', 'CR-CC(2,3)', orbs, max(3, orbs // 5), max(3, orbs // 5), its=rng.randint(4, 6))


# ---- inputs ----------------------------------------------------------------------------------------------


def _members(case):
    """The systems of a case: one, or the uneven ones of a batch."""
    if case['kind'] != 'batch':
        return [(case['orbs'], case['occ_a'], case['occ_b'])]
    lo = 16
    sizes = [lo + (case['orbs'] - lo) * k // max(1, case['count'] - 1) for k in range(case['count'])]
    return [(n, n // 5, n // 5) for n in sizes]


def _hamiltonian(seed, orbs, occ_a, occ_b, froz):
    """Fock matrices over all orbitals and spin blocks <pq||rs> over the active ones, from factorised integrals
    with a diagonal closed-shell Fock matrix (singly occupied orbitals lie between occupied and virtual)."""
    g = torch.Generator(device='cpu').manual_seed(seed * 1009 + orbs)
    nf = 2 * orbs
    B = torch.randn(nf, orbs, orbs, generator=g, dtype=F64).to(DEV) * 0.03
    B = torch.tril(B) + torch.tril(B, -1).transpose(1, 2)
    u = torch.rand(orbs, generator=g, dtype=F64).to(DEV)
    eps = torch.cat([(-1.5 + 0.8 * u[:occ_b]).sort().values, (-0.25 + 0.1 * u[occ_b:occ_a]).sort().values,
                     (0.2 + 1.8 * u[occ_a:]).sort().values])
    Bm = B.reshape(nf, -1)
    e2 = (Bm.T @ Bm).reshape(orbs, orbs, orbs, orbs).permute(0, 2, 1, 3).contiguous()   # <pq|rs>
    def jk(occ):
        J = torch.einsum('piqi->pq', e2[:, :occ, :, :occ])
        K = torch.einsum('piiq->pq', e2[:, :occ, :occ, :])
        return J, K
    Ja, Ka = jk(occ_a)
    Jb, Kb = jk(occ_b)
    h = torch.diag(eps) - (2 * Jb - Kb)
    fa, fb = h + Ja + Jb - Ka, h + Ja + Jb - Kb
    v = e2[froz:, froz:, froz:, froz:].contiguous()
    vaa = v - v.permute(0, 1, 3, 2)
    return fa, fb, vaa.contiguous(), v


def _shape(name, oa, ob, va, vb):
    n, nb = int(name[1]), 'ABCDE'.index(name[2])
    return (oa,) * (n - nb) + (ob,) * nb + (va,) * (n - nb) + (vb,) * nb


def _dims(case):
    f = case['froz']
    return case['occ_a'] - f, case['occ_b'] - f, case['orbs'] - case['occ_a'], case['orbs'] - case['occ_b']


def _sign(p):
    return -1 if sum(p[j] < p[i] for i in range(len(p)) for j in range(i + 1, len(p))) % 2 else 1


def _antisym(x, groups):
    """x with its axes antisymmetrised within each group."""
    for g in groups:
        if len(g) < 2:
            continue
        acc = torch.zeros_like(x)
        for p in itertools.permutations(range(len(g))):
            axes = list(range(x.ndim))
            for q, w in enumerate(p):
                axes[g[q]] = g[w]
            acc += _sign(p) * x.permute(axes)
        x = acc
    return x


def _groups(name):
    n, nb = int(name[1]), 'ABCDE'.index(name[2])
    na = n - nb
    return [list(range(0, na)), list(range(na, n)), list(range(n, n + na)), list(range(n + na, 2 * n))]


def _guess(case, seed):
    """Amplitude blocks in mid-solve: antisymmetric, with the magnitudes of a solve's T1, T2 and T3."""
    g = torch.Generator(device=DEV).manual_seed(seed * 7 + 3)
    out = {}
    for name in T12 + T3:
        shp = _shape(name, *_dims(case))
        scale = {1: 3e-3, 2: 3e-3, 3: 1e-4}[int(name[1])]
        out[name] = _antisym(torch.randn(shp, generator=g, dtype=F64, device=DEV) * scale, _groups(name))
    return out


def _active(case):
    """ccq's act_occ_b and act_unocc_a."""
    return (max(case['occ_b'] - case['act_occ'], case['froz']), min(case['occ_a'] + case['act_unocc'], case['orbs']))


# ---- prepare and run --------------------------------------------------------------------------------------


def _context(case, seed, orbs, occ_a, occ_b):
    fa, fb, vaa, vab = (x.cpu().numpy() for x in _hamiltonian(seed, orbs, occ_a, occ_b, case['froz']))
    act = _active(case) if case['method'] == 'CCSDt' else None
    return lib.Context(case['froz'], occ_a, occ_b, orbs, case['method'], fa, fb, vaa, vab, vaa, rhf=case['rhf'],
                       diis_space=DIIS, active=act)


def prepare(case, seed):
    case = dict(case)
    st = dict(case=case)
    st['ctx'] = [_context(case, seed + 31 * k, *m) for k, m in enumerate(_members(case))]
    for ctx in st['ctx']:
        ctx.set_precision(lib.PREC_SPLIT if case['precision'] == 'split' else lib.PREC_FP64, 4)
        ctx.use_graph(2 if case['kind'] == 'batch' else 1)
    ctx = st['ctx'][0]
    if case['tuned']:
        ctx.autotune()
    if case['kind'] == 'left':
        for it in range(1, 2 * CYCLE + 1):
            st['e'] = ctx.iterate(it)[0]
        return st
    if case['kind'] == 'host':
        blocks = _guess(case, seed)
        st['t_in'] = torch.empty(ctx.t_size, dtype=F64).pin_memory()
        torch.cat([blocks[b].reshape(-1) for b in T12 + T3], out=(dev := torch.empty(ctx.t_size, dtype=F64, device=DEV)))
        st['t_in'].copy_(dev)
        st['t_out'] = torch.zeros(ctx.t_size, dtype=F64).pin_memory()
        return st
    if case['method'] in ('CCSDT', 'CCSDt', 'CCSDTQ'):
        st['zero'] = torch.zeros(ctx.t_size, dtype=F64).pin_memory()
        st['t'] = torch.zeros(ctx.t_size, dtype=F64).pin_memory()
    if case['method'] == 'CCSD':
        st['shapes'] = [{b: _shape(b, oa, ob, n - oa - case['froz'], n - ob - case['froz']) for b in T12}
                        for n, oa, ob in ((m[0], m[1] - case['froz'], m[2] - case['froz']) for m in _members(case))]
        st['zeros'] = [{b: np.zeros(s) for b, s in shp.items()} for shp in st['shapes']]
    if case['method'] == 'CCSDTQ':
        st['shapes4'] = {b: _shape(b, *_dims(case)) for b in T4}
        st['zeros4'] = {b: np.zeros(s) for b, s in st['shapes4'].items()}
    return st


def run(st):
    case, ctxs = st['case'], st['ctx']
    ctx, kind, method = ctxs[0], case['kind'], case['method']
    if kind == 'host':
        e, r, _ = ctx.iterate_host(1, st['t_in'].data_ptr(), st['t_out'].data_ptr())
        return {'e': e, 'res': r, 't': st['t_out']}
    if kind == 'left':
        ctx.lambda_init(st['e'])
        hist = [ctx.lambda_iterate(it)[:2] for it in range(1, case['its'] + 1)]
        return {'hist': np.array(hist), 'l': ctx.get_l(), 'e23': ctx.crcc23()}
    if method == 'CCSD':
        for c, z in zip(ctxs, st['zeros']):
            for b in T12:
                c.set_block(b, z[b])
        hist = []
        for it in range(1, case['its'] + 1):
            if len(ctxs) == 1:
                hist.append([ctx.iterate(it)[:2]])
                continue
            for c in ctxs:
                c.iterate_async(it)
            hist.append([c.iterate_wait()[:2] for c in ctxs])
        return {'hist': np.array(hist), 't': [{b: c.get_block(b, s[b]) for b in T12} if len(ctxs) == 1 else
                                              np.concatenate([c.get_block(b, s[b]).reshape(-1) for b in T12])
                                              for c, s in zip(ctxs, st['shapes'])]}
    ctx.set_t_ptr(st['zero'].data_ptr(), ctx.t_size)
    if method == 'CCSDTQ':
        for b in T4:
            ctx.set_block(b, st['zeros4'][b])
    hist = np.array([ctx.iterate(it)[:2] for it in range(1, case['its'] + 1)])
    ctx.get_t_ptr(st['t'].data_ptr(), ctx.t_size)
    out = {'hist': hist, 't': st['t']}
    if method == 'CCSDTQ':
        out['t4'] = {b: ctx.get_block(b, st['shapes4'][b]) for b in T4}
    return out


# ---- what a pass cannot do without ------------------------------------------------------------------------


def _c(n, k):
    return math.comb(n, k) if n >= k else 0


def _iteration_work(method, oa, ob, va, vb, rhf):
    """(flops, bytes) of one iteration: its ladder, hole-hole and ring products over unique index tuples, the
    integrals and amplitudes read once and the amplitudes written once."""
    n = oa + va
    levels = {'CCSD': 2, 'CR-CC(2,3)': 2, 'CCSDT': 3, 'CCSDt': 3, 'CCSDTQ': 4}[method]
    flops, elems = 0.0, 0.0
    for lev in range(1, levels + 1):
        for nb in range(lev + 1):
            na = lev - nb
            if rhf and nb > lev // 2:
                continue
            occ, vir = _c(oa, na) * _c(ob, nb), _c(va, na) * _c(vb, nb)
            elems += occ * vir
            if lev < 2:
                continue
            for pa, pb in ((2, 0), (1, 1), (0, 2)):
                if pa > na or pb > nb:
                    continue
                pair = _c(va, pa) * _c(vb, pb)
                flops += 2.0 * occ * _c(va, na - pa) * _c(vb, nb - pb) * pair * pair
                hole = _c(oa, pa) * _c(ob, pb)
                flops += 2.0 * vir * _c(oa, na - pa) * _c(ob, nb - pb) * hole * hole
            for s, (o, v) in enumerate(((oa, va), (ob, vb))):
                if (na, nb)[s] == 0:
                    continue
                ra, rb = (na - 1, nb) if s == 0 else (na, nb - 1)
                rest = _c(oa, ra) * _c(ob, rb) * _c(va, ra) * _c(vb, rb)
                flops += 2.0 * rest * o * v * (oa * va + ob * vb)
    ints = n ** 4 * (1.0 if rhf else 1.5)
    return flops, 8.0 * (ints + 2.0 * elems)


def work(case):
    flops = byts = 0.0
    for orbs, occ_a, occ_b in _members(case):
        f = case['froz']
        fl, by = _iteration_work(case['method'], occ_a - f, occ_b - f, orbs - occ_a, orbs - occ_b, case['rhf'])
        if case['method'] == 'CCSDt':
            m1, m2 = _active(case)
            oa, va = occ_a - f, orbs - occ_a
            share = (1 - _c(m1 - f, 3) / max(1, _c(oa, 3))) * (1 - _c(orbs - m2, 3) / max(1, _c(va, 3)))
            fl *= share
            by *= share
        flops += fl * case['its']
        byts += by * case['its']
    return {'bytes': byts, 'flops': flops}


# ---- the same in plain spin-orbital tensors ----------------------------------------------------------------


class _SpinOrbital:
    """CCSD and CCSDT iterations on dense spin-orbital tensors: occupied alpha, occupied beta, virtual alpha,
    virtual beta; amplitudes t1[i,a], t2[i,j,a,b], t3[i,j,k,a,b,c]."""

    def __init__(self, fa, fb, vaa, vab, oa, ob, froz):
        n = vab.shape[0]
        self.oa, self.ob, self.va, self.vb = oa, ob, n - oa, n - ob
        self.O, self.V = oa + ob, 2 * n - oa - ob
        ia, ib = torch.arange(n, device=fa.device), torch.arange(n, device=fa.device)
        # position of spatial orbital p of each spin among the spin orbitals
        pa = torch.where(ia < oa, ia, ia - oa + self.O)
        pb = torch.where(ib < ob, ib + oa, ib - ob + self.O + self.va)
        N = 2 * n
        fa, fb = fa[froz:, froz:], fb[froz:, froz:]
        v = torch.zeros(N, N, N, N, dtype=F64, device=fa.device)
        def put(P, Q, R, S, x):
            v[P[:, None, None, None], Q[None, :, None, None], R[None, None, :, None], S[None, None, None, :]] = x
        put(pa, pa, pa, pa, vaa)
        put(pb, pb, pb, pb, vaa)
        put(pa, pb, pa, pb, vab)
        put(pb, pa, pb, pa, vab.permute(1, 0, 3, 2))
        put(pa, pb, pb, pa, -vab.permute(0, 1, 3, 2))
        put(pb, pa, pa, pb, -vab.permute(1, 0, 2, 3))
        f = torch.zeros(N, N, dtype=F64, device=fa.device)
        f[pa[:, None], pa[None, :]] = fa
        f[pb[:, None], pb[None, :]] = fb
        O = self.O
        self.f, self.v = f, v
        self.h = f - torch.einsum('piqi->pq', v[:, :O, :, :O])
        self.dia = torch.diagonal(f)
        self.t = {1: torch.zeros(O, self.V, dtype=F64, device=fa.device),
                  2: torch.zeros(O, O, self.V, self.V, dtype=F64, device=fa.device)}

    def slices(self, name):
        n, nb = int(name[1]), 'ABCDE'.index(name[2])
        spins = [0] * (n - nb) + [1] * nb
        occ = (slice(0, self.oa), slice(self.oa, self.O))
        vir = (slice(0, self.va), slice(self.va, self.V))
        return tuple(occ[s] for s in spins) + tuple(vir[s] for s in spins)

    def get(self, name):
        return self.t[int(name[1])][self.slices(name)]

    def put(self, name, x):
        """The block and its images in every order of the spins."""
        n = int(name[1])
        sl = self.slices(name)
        done = set()
        for po in itertools.permutations(range(n)):
            for pv in itertools.permutations(range(n)):
                where = tuple((sl[p].start, sl[p].stop) for p in po) + tuple((sl[n + p].start, sl[n + p].stop) for p in pv)
                if where in done:
                    continue
                done.add(where)
                at = tuple(sl[p] for p in po) + tuple(sl[n + p] for p in pv)
                self.t[n][at] = _sign(po) * _sign(pv) * x.permute(list(po) + [n + p for p in pv])

    def dress(self):
        """The Hamiltonian transformed with exp(T1)."""
        O, t1 = self.O, self.t[1]
        N = O + self.V
        X = torch.eye(N, dtype=F64, device=t1.device)
        Y = X.clone()
        X[O:, :O] = -t1.T
        Y[:O, O:] = t1
        v = torch.einsum('pqrs,sz->pqrz', self.v, Y.T)
        v = torch.einsum('pqrs,rz->pqzs', v, Y.T)
        v = torch.einsum('pqrs,zq->pzrs', v, X)
        self.V2 = torch.einsum('pqrs,zp->zqrs', v, X).contiguous()
        h = X @ self.h @ Y.T
        self.F = h + torch.einsum('piqi->pq', self.V2[:, :O, :, :O])

    def energy(self):
        O, t1, t2 = self.O, self.t[1], self.t[2]
        w = self.v[:O, :O, O:, O:]
        return float((self.f[:O, O:] * t1).sum() + 0.25 * (w * t2).sum()
                     + 0.5 * torch.einsum('ijab,ia,jb->', w, t1, t1))

    def parts(self):
        o, v = slice(0, self.O), slice(self.O, None)
        return self.F, self.V2, o, v, self.t[2], self.t.get(3)

    def r1(self):
        F, W, o, v, t2, t3 = self.parts()
        r = F[v, o].T + torch.einsum('kc,ikac->ia', F[o, v], t2)
        r = r + 0.5 * torch.einsum('akcd,ikcd->ia', W[v, o, v, v], t2)
        r = r - 0.5 * torch.einsum('klic,klac->ia', W[o, o, o, v], t2)
        if t3 is not None:
            r = r + 0.25 * torch.einsum('klcd,iklacd->ia', W[o, o, v, v], t3)
        return r

    def one_body(self):
        F, W, o, v, t2, _ = self.parts()
        fvv = F[v, v] - 0.5 * torch.einsum('klcd,klad->ac', W[o, o, v, v], t2)
        foo = F[o, o] + 0.5 * torch.einsum('klcd,ilcd->ki', W[o, o, v, v], t2)
        return fvv, foo

    def r2(self):
        F, W, o, v, t2, t3 = self.parts()
        fvv, foo = self.one_body()
        woo = W[o, o, o, o] + 0.5 * torch.einsum('klcd,ijcd->klij', W[o, o, v, v], t2)
        ring = W[o, v, v, o] + 0.5 * torch.einsum('klcd,ljdb->kbcj', W[o, o, v, v], t2)
        r = W[v, v, o, o].permute(2, 3, 0, 1).clone()
        r += 0.5 * torch.einsum('abcd,ijcd->ijab', W[v, v, v, v], t2)
        r += 0.5 * torch.einsum('klij,klab->ijab', woo, t2)
        x = torch.einsum('bc,ijac->ijab', fvv, t2)
        r += x - x.permute(0, 1, 3, 2)
        x = torch.einsum('kj,ikab->ijab', foo, t2)
        r -= x - x.permute(1, 0, 2, 3)
        r += _antisym(torch.einsum('kbcj,ikac->ijab', ring, t2), [[0, 1], [2, 3]])
        if t3 is not None:
            r += torch.einsum('kc,ijkabc->ijab', F[o, v], t3)
            x = 0.5 * torch.einsum('bkcd,ijkacd->ijab', W[v, o, v, v], t3)
            r += x - x.permute(0, 1, 3, 2)
            x = 0.5 * torch.einsum('klcj,iklabc->ijab', W[o, o, v, o], t3)
            r += x - x.permute(1, 0, 2, 3)
        return r

    def r3_seed(self):
        """G with the residual = the signed sum of G over the permutations of ijk and of abc."""
        F, W, o, v, t2, t3 = self.parts()
        fvv, foo = self.one_body()
        oovv = W[o, o, v, v]
        vvvo = W[v, v, v, o] - torch.einsum('ld,lkbc->bcdk', F[o, v], t2)
        vvvo += 0.5 * torch.einsum('lmdk,lmbc->bcdk', W[o, o, v, o], t2)
        x = torch.einsum('bled,lkec->bcdk', W[v, o, v, v], t2)
        vvvo -= x - x.permute(1, 0, 2, 3)
        vvvo -= 0.5 * torch.einsum('lmde,lmkbec->bcdk', oovv, t3)
        ovoo = W[o, v, o, o] + 0.5 * torch.einsum('lcde,jkde->lcjk', W[o, v, v, v], t2)
        x = torch.einsum('lmjd,mkdc->lcjk', W[o, o, o, v], t2)
        ovoo += x - x.permute(0, 1, 3, 2)
        ovoo += 0.5 * torch.einsum('lmde,jmkdec->lcjk', oovv, t3)
        vvvv = W[v, v, v, v] + 0.5 * torch.einsum('lmde,lmbc->bcde', oovv, t2)
        oooo = W[o, o, o, o] + 0.5 * torch.einsum('lmde,jkde->lmjk', oovv, t2)
        ring = W[o, v, v, o] + torch.einsum('lmde,mkec->lcdk', oovv, t2)
        G = 0.25 * torch.einsum('bcdk,ijad->ijkabc', vvvo, t2)
        G -= 0.25 * torch.einsum('lcjk,ilab->ijkabc', ovoo, t2)
        G += torch.einsum('cd,ijkabd->ijkabc', fvv / 12, t3)
        G -= torch.einsum('lk,ijlabc->ijkabc', foo / 12, t3)
        G += torch.einsum('bcde,ijkade->ijkabc', vvvv / 24, t3)
        G += torch.einsum('lmjk,ilmabc->ijkabc', oooo / 24, t3)
        G += torch.einsum('lcdk,ijlabd->ijkabc', ring / 4, t3)
        return G

    def residual(self, name):
        n, sl = int(name[1]), self.slices(name)
        if n == 1:
            return self.r1()[sl]
        if n == 2:
            return self.r2()[sl]
        G = self.r3_seed()
        r = 0
        for po in itertools.permutations(range(3)):
            for pv in itertools.permutations(range(3)):
                at = tuple(sl[p] for p in po) + tuple(sl[3 + p] for p in pv)
                inv = [po.index(q) for q in range(3)] + [3 + pv.index(q) for q in range(3)]
                r = r + _sign(po) * _sign(pv) * G[at].permute(inv)
        return r

    def step(self, name, mask=None):
        self.dress()
        r = self.residual(name)
        n, sl = int(name[1]), self.slices(name)
        D = torch.zeros_like(r)
        eo, ev = self.dia[:self.O], self.dia[self.O:]
        for d in range(2 * n):
            e = -eo[sl[d]] if d < n else ev[sl[d]]
            D += e.reshape([-1 if q == d else 1 for q in range(2 * n)])
        x = self.get(name) - r / D
        self.put(name, x if mask is None else x * mask)


ORDER = ('T2A', 'T2C', 'T2B', 'T1A', 'T1B', 'T3A', 'T3D', 'T3B', 'T3C')
COPY = {'T1B': ('T1A', (0, 1)), 'T2C': ('T2A', (0, 1, 2, 3)), 'T3D': ('T3A', (0, 1, 2, 3, 4, 5)),
        'T3C': ('T3B', (2, 0, 1, 5, 3, 4))}


def _mask(case, name):
    oa, ob, va, vb = _dims(case)
    m1, m2 = _active(case)
    nb = 'ABCD'.index(name[2])
    occ = vir = None
    shp = _shape(name, oa, ob, va, vb)
    for d in range(3):
        spin = int(d >= 3 - nb)
        x = (torch.arange(shp[d], device=DEV) >= m1 - case['froz']).reshape([-1 if q == d else 1 for q in range(6)])
        y = (torch.arange(shp[3 + d], device=DEV) < m2 - (case['occ_a'], case['occ_b'])[spin])
        y = y.reshape([-1 if q == 3 + d else 1 for q in range(6)])
        occ = x if occ is None else occ | x
        vir = y if vir is None else vir | y
    return (occ & vir).to(F64)


def _iterate(case, so, blocks, its):
    """History of (energy, residuum) and the amplitudes after the iterations (DIIS at every sixth)."""
    vec = lambda: torch.cat([so.get(b).reshape(-1) for b in blocks])  # noqa: E731
    masks = {b: _mask(case, b) for b in T3} if case['method'] == 'CCSDt' else {}
    ring, hist = [], []
    prev = torch.zeros_like(vec())
    for it in range(1, its + 1):
        for b in ORDER:
            if b not in blocks:
                continue
            if case['rhf'] and b in COPY:
                so.put(b, so.get(COPY[b][0]).permute(COPY[b][1]).clone())
            else:
                so.step(b, masks.get(b))
        x = vec()
        if not masks:   # the active-space residuum runs over the compressed vector
            hist.append((so.energy(), float((x - prev).norm()) ** 0.5))
        else:
            hist.append((so.energy(), None))
        ring.append(x)
        prev = x
        if it % CYCLE == 0:
            d = torch.stack([ring[i + 1] - ring[i] for i in range(DIIS)])
            M = -torch.ones(CYCLE, CYCLE, dtype=F64)
            M[:DIIS, :DIIS] = (d @ d.T).cpu()
            rhs = torch.zeros(CYCLE, dtype=F64)
            rhs[DIIS] = -1.0
            c = torch.linalg.solve(M, rhs)
            x = sum(float(c[i]) * ring[i] for i in range(DIIS))
            at = 0
            for b in blocks:
                n = so.get(b).numel()
                so.put(b, x[at:at + n].reshape(so.get(b).shape).clone())
                at += n
            ring = []
    return hist


def exact(case, seed):
    if case['kind'] == 'left' or case['method'] == 'CCSDTQ':
        return None   # the left vector and the quadruples have no short dense form
    if case['method'] != 'CCSD' and case['its'] > 1 and case['orbs'] > 32:
        return None   # dense spin-orbital triples of this size take minutes
    blocks = T12 if case['method'] == 'CCSD' else T12 + T3
    hists, ts = [], []
    for k, (orbs, occ_a, occ_b) in enumerate(_members(case)):
        f = case['froz']
        so = _SpinOrbital(*_hamiltonian(seed + 31 * k, orbs, occ_a, occ_b, f), occ_a - f, occ_b - f, f)
        if case['method'] != 'CCSD':
            so.t[3] = torch.zeros((so.O,) * 3 + (so.V,) * 3, dtype=F64, device=DEV)
        if case['kind'] == 'host':
            start = _guess(case, seed)
            for b in blocks:
                so.put(b, start[b])
        hist = _iterate(case, so, blocks, case['its'])
        hists.append(hist)
        ts.append({b: so.get(b) for b in blocks})
    flat = lambda t: torch.cat([t[b].reshape(-1) for b in blocks]).cpu()  # noqa: E731
    if case['kind'] == 'host':
        return {'e': hists[0][0][0], 'res': hists[0][0][1], 't': flat(ts[0])}
    if case['method'] == 'CCSD':
        hist = np.array(hists).transpose(1, 0, 2)
        return {'hist': hist, 't': [{b: x.cpu() for b, x in ts[0].items()}] if len(ts) == 1 else [flat(t) for t in ts]}
    hist = None if case['method'] == 'CCSDt' else np.array(hists[0])
    return {'hist': hist, 't': flat(ts[0])}
