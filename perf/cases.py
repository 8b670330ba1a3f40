"""Timed work of the detector path: what a user of this package has it do, through its public entry points.

Twelve listed cases, each with the values the path meets in earnest: i.i.d. Rayleigh channels lifted to real
[[Re, -Im], [Im, Re]], uniform Gray PAM levels, SNR uniform over the case's range, and the budgets that the package
itself runs (the picks of detector.ARPEGGIO_PICKS, Chord's default schedule, the operating points of bench.py).

kind      entry point                                  stands for
detect    Detector.run                                 one-stage detection: a frame, a ragged batch, a full batch
soft      Detector.run_soft                            detection with list LLRs for a channel decoder
traj      soft.detect_llr                              trajectory LLRs on the RI map
warm      WarmDetector.run                             detection from the learned warm start
train     WarmMLP.train_step                           one optimisation step of the warm start's network
mdi       mdi.detect                                   the multi-stage detector (MMSE and SIC guesses, host walk)
chordj    chordfx.Kernel.chord                         Chord on a full int16 coupling matrix, as the solver interface

Inputs come from torch generators of the given seed alone."""
import math

import numpy as np
import torch

from arpeggio_b200 import chordfx, mdi, soft, warm
from arpeggio_b200.detector import Detector

PAM = {4: ((-1, 1), 1 / math.sqrt(2)), 16: ((-3, -1, 1, 3), 1 / math.sqrt(10)),
       64: ((-7, -5, -3, -1, 1, 3, 5, 7), 1 / math.sqrt(42))}
NB = {4: 1, 16: 2, 64: 3}


def listed():
    return [
        # one received frame inside its latency budget: the smallest call, launches and host time count
        dict(name='frame_x32', kind='detect', B=1, nt=32, nr=32, M=16, R=32, sweeps=32, policy='arpeggio',
             precision='int', start='rand', K=1, lo=14.0, hi=14.0),
        # the benchmark's batch: 32 users x 32 antennas, 16-QAM, the 32-user pick
        dict(name='batch_x32', kind='detect', B=65536, nt=32, nr=32, M=16, R=32, sweeps=32, policy='arpeggio',
             precision='int', start='rand', K=1, lo=6.0, hi=22.0),
        # 64 users x 64 antennas at the 64-user pick: the largest coupling matrices
        dict(name='batch_x64', kind='detect', B=8192, nt=64, nr=64, M=16, R=64, sweeps=64, policy='arpeggio',
             precision='int', start='bal', K=1, lo=10.0, hi=24.0),
        # a small cell: 8 users x 16 antennas, QPSK, an odd number of uses
        dict(name='cell_x8', kind='detect', B=49999, nt=8, nr=16, M=4, R=32, sweeps=32, policy='arpeggio',
             precision='int', start='bal', K=1, lo=5.0, hi=25.0),
        # FP32 fields, 24 users x 36 antennas (coordinates and rows no multiple of a tile), 64-QAM
        dict(name='float_x24', kind='detect', B=10007, nt=24, nr=36, M=64, R=32, sweeps=32, policy='arpeggio',
             precision='f32', start='bal', K=1, lo=12.0, hi=28.0),
        # Chord's synchronous rule at its default schedule (256 steps) in the same detector
        dict(name='chord_x32', kind='detect', B=16384, nt=32, nr=32, M=16, R=32, sweeps=128, policy='chord',
             precision='int', start='rand', K=1, lo=6.0, hi=22.0),
        # list LLRs for a decoder behind the 32-user detector
        dict(name='soft_x32', kind='soft', B=8192, nt=32, nr=32, M=16, R=32, sweeps=32, lo=8.0, hi=20.0),
        # trajectory LLRs: 16 chains of 256 steps on the 64-spin RI map
        dict(name='traj_x16', kind='traj', B=4096, nt=16, nr=16, M=16, R=16, S=256, lo=8.0, hi=18.0),
        # the learned warm start at its 32-user operating point (sampled starts, per-problem anneal counts)
        dict(name='warm_x32', kind='warm', B=32768, nt=32, nr=32, M=16, R=32, sweeps=24, lo=18.0, hi=24.0),
        # one training step of the warm start's network at the benchmark's rows per step
        dict(name='train_64k', kind='train', rows=65536),
        # the reference's full chain at its 16-user point: guesses, radii, three stages' sizes of sub-problems
        dict(name='mdi_x16', kind='mdi', B=8192, nt=16, nr=16, M=16, Ns=32, sweeps=64, lo=20.0, hi=20.0),
        # Chord on full coupling matrices: 32 users, two copy pairs (256 spins, four phases)
        dict(name='chordj_256', kind='chordj', B=1024, nt=32, P=4, R=8, S=256, lo=10.0, hi=20.0),
    ]


# ------------------------------------------------------------------------------------------------ drawn cases
CAP = 65536 * 32 * 64 * 64  # anneal tests of batch_x32 (uses x anneals x passes x coordinates)


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _batch(rng, per_use, cap, hi):
    """Uses, spread over the logarithm of 1 .. what `cap` allows at this cost per use."""
    return max(1, _logint(rng, 1, max(1, min(hi, int(cap / per_use)))))


def draw(rng):
    """One more case of the listed ranges: 4-64 users, 1-2 antennas per user, every constellation, 1 to 65536 uses."""
    kind = rng.choice(['detect'] * 6 + ['soft', 'traj', 'warm', 'train', 'mdi', 'chordj'])
    if kind == 'train':
        return dict(kind=kind, rows=16 * _logint(rng, 64, 4096))
    if kind == 'chordj':
        nt, P = rng.choice([(16, 1), (16, 2), (16, 4), (16, 6), (32, 2), (32, 4), (48, 2), (64, 2)])
        S, R = P * rng.choice([32, 64, 128]), rng.randint(1, 16)
        return dict(kind=kind, B=_batch(rng, S * R, 1024 * 8 * 256, 4096), nt=nt, P=P, R=R, S=S, lo=10.0, hi=20.0)
    nt = rng.randint(4, 64)
    nr = int(round(nt * rng.uniform(1.0, 2.0)))
    lo = rng.uniform(5.0, 18.0)
    c = dict(kind=kind, nt=nt, nr=nr, M=rng.choice([4, 16, 64]), lo=lo, hi=lo + rng.uniform(0.0, 8.0))
    if kind == 'traj':
        nt = rng.choice([8, 10, 16, 24, 32])
        c.update(nt=nt, nr=int(round(nt * rng.uniform(1.0, 2.0))), M=rng.choice([4, 16]), R=rng.randint(1, 24),
                 S=rng.choice([64, 128, 256]))
        c['B'] = _batch(rng, c['R'] * c['S'] * nt, 4096 * 16 * 256 * 16, 16384)
        return c
    if kind == 'mdi':
        nt = rng.randint(8, 32)
        c.update(nt=nt, nr=int(round(nt * rng.uniform(1.0, 1.5))), M=16, Ns=rng.choice([16, 32]),
                 sweeps=rng.choice([32, 64]), lo=20.0, hi=20.0)
        c['B'] = _batch(rng, c['Ns'] * c['sweeps'] * nt * nt, 8192 * 32 * 64 * 16 * 16, 8192)
        return c
    c.update(R=rng.choice([8, 16, 32, 33, 64]), sweeps=rng.choice([16, 24, 32, 64]))
    if kind == 'detect':
        c.update(policy=rng.choice(['arpeggio', 'arpeggio', 'arpeggio', 'chord']), K=rng.choice([1, 1, 1, 2, 3]),
                 precision=rng.choice(['int', 'int', 'f32']), start=rng.choice(['rand', 'bal']))
    elif kind == 'soft':
        c['M'] = rng.choice([4, 16])
    passes = c['sweeps'] * 2 * c.get('K', 1)
    # Chord and several copies flip more per test, FP32 fields and large matrices cost more per flip
    per = c['R'] * passes * (2 * nt) * (3 if c.get('policy') == 'chord' else 1) * (1 + (c.get('precision') == 'f32'))
    c['B'] = _batch(rng, per * (1 + nt / 32), CAP, 65536)
    return c


# ------------------------------------------------------------------------------------------------ inputs
def _uses(case, seed):
    """H (B, 2 nr, 2 nt), y (B, 2 nr), SNR (B) in dB and N0 (B) on the GPU."""
    B, nt, nr = case['B'], case['nt'], case['nr']
    lv, a = PAM[case['M']]
    g = torch.Generator(device='cuda').manual_seed(seed)
    l = torch.tensor(lv, dtype=torch.float32, device='cuda')[
        torch.randint(0, len(lv), (B, 2 * nt), generator=g, device='cuda')]
    H = torch.empty(B, 2 * nr, 2 * nt, device='cuda')
    re = torch.randn(B, nr, nt, generator=g, device='cuda') * (a / math.sqrt(2))
    H[:, :nr, :nt], H[:, nr:, nt:] = re, re
    re = torch.randn(B, nr, nt, generator=g, device='cuda') * (a / math.sqrt(2))
    H[:, nr:, :nt] = re
    H[:, :nr, nt:] = re.neg_()
    del re
    snr = case['lo'] + (case['hi'] - case['lo']) * torch.rand(B, generator=g, device='cuda', dtype=torch.float64)
    N0 = nt / 10 ** (snr / 10)
    n = torch.randn(B, 2 * nr, generator=g, device='cuda') * torch.sqrt(N0 / 2).float()[:, None]
    y = (H @ l[:, :, None])[..., 0] + n
    return H, y, N0


def _network(seed):
    """Weights of a warm-start network in the flat order of WarmMLP.LAYOUT: the refined single-coordinate move u
    (feature 10) carried through both hidden layers to logits (-u - b, 0, u - b) of a sharpness that leaves weak
    coordinates undecided, over small random weights everywhere."""
    g = torch.Generator().manual_seed(seed)
    W1 = torch.randn(256, 16, generator=g) * 0.02
    b1 = torch.randn(256, generator=g) * 0.02
    W2 = torch.randn(256, 256, generator=g) * 0.01
    b2 = torch.randn(256, generator=g) * 0.02
    W3t = torch.randn(256, 16, generator=g) * 0.02
    b3 = torch.zeros(16)
    W1[0, 10], W1[1, 10] = 1.0, -1.0
    W2[0, 0], W2[1, 1] = 1.0, 1.0
    W3t[0, 2], W3t[1, 0] = 6.0, 6.0
    b3[0], b3[2] = -4.0, -4.0
    return torch.cat([t.reshape(-1) for t in (W1, b1, W2, b2, W3t, b3)]).numpy()


def _train_inputs(case, seed):
    rows = case['rows']
    g = torch.Generator(device='cuda').manual_seed(seed)
    X = torch.randn(rows, 16, generator=g, device='cuda')
    X[:, 8] = 1.0   # the constant feature
    X[:, 11:] = 0.0  # unused features
    u = X[:, 10] + 0.3 * torch.randn(rows, generator=g, device='cuda')
    labels = (1 + (u > 0.7).to(torch.int8) - (u < -0.7).to(torch.int8)).to(torch.int8)
    return X.to(torch.bfloat16), labels


def _chord_problem(case, seed):
    """The integer problem of a one-stage detection with P copies per coordinate: J = -offdiag(G x 1 1^T) int16,
    h = h0 int32, units of 1/4096, Chord's default schedule."""
    B, nt, P, S = case['B'], case['nt'], case['P'], case['S']
    D = 2 * nt
    H, y, N0 = _uses(dict(case, nr=nt, M=16), seed)
    Hd, yd = H.double(), y.double()
    Q = Hd.transpose(1, 2) @ Hd
    A = Q + ((N0 / 2) / 5.0)[:, None, None] * torch.eye(D, device='cuda', dtype=torch.float64)
    z = torch.linalg.solve(A, (Hd.transpose(1, 2) @ yd[..., None]))[..., 0]
    x = (2 * torch.round((z - 1) / 2) + 1).clamp(-3, 3)
    h = 2 * (Hd.transpose(1, 2) @ (yd - (Hd @ x[..., None])[..., 0])[..., None])[..., 0]
    sc = torch.maximum(h.abs().amax(1), Q.abs().amax((1, 2)))
    J = -torch.round(Q / sc[:, None, None] * 4096).repeat(1, P, P).to(torch.int16)
    J.diagonal(dim1=1, dim2=2).zero_()
    hq = torch.round(h / sc[:, None] * 4096).to(torch.int32).repeat(1, P).contiguous()
    T = torch.full((S,), int(round(0.3 * 4096)), dtype=torch.int32, device='cuda')
    return dict(J=J.contiguous(), h=hq, h0=hq.clone(), T=T, c=torch.zeros_like(T), q=int(round(0.4 * 4096)), S=S)


# ------------------------------------------------------------------------------------------------ the interface
def prepare(case, seed):
    k = case['kind']
    st = dict(case=case, seed=seed)
    if k == 'train':
        st['X'], st['labels'] = _train_inputs(case, seed)
        st['mlp'] = warm.WarmMLP(P=2, rows=case['rows'], seed=0)
        st['mlp'].load_state_dict({'w': _network(0), 'P': 2, 'steps': 0})
        st['mlp'].reserve(case['rows'], train=True)
        return st
    if k == 'chordj':
        st['F'] = _chord_problem(case, seed)
        st['kernel'] = chordfx.Kernel()
        return st
    st['H'], st['y'], st['N0'] = _uses(case, seed)
    B, nt, nr, M = case['B'], case['nt'], case['nr'], case['M']
    if k == 'detect':
        chord = case['policy'] == 'chord'
        st['det'] = Detector(B, nt, nr, M, case['policy'], case['R'], case['K'], sweeps=case['sweeps'],
                             T0=0.3 if chord else 0.1, T1=0.3 if chord else 0.1, q=0.4 if chord else 0.0,
                             start=case['start'], precision=case['precision'])
        st['det'].set_noise(N0=st['N0'])
    elif k == 'soft':
        st['det'] = Detector(B, nt, nr, M, 'arpeggio', case['R'], 1, sweeps=case['sweeps'], T0=0.1, T1=0.1, q=0.0,
                             start='rand')
        st['det'].set_noise(N0=st['N0'])
        st['N0f'] = st['N0'].float()
    elif k == 'warm':
        mlp = warm.WarmMLP(P=2, seed=0)
        mlp.load_state_dict({'w': _network(0), 'P': 2, 'steps': 0})
        st['det'] = warm.WarmDetector(B, nt, nr, M, anneals=case['R'], sweeps=case['sweeps'], mlp=mlp, T0=0.085,
                                      T1=0.085, tau=0.8, conf_min=-(5.0 / 64) * 2 * nt, r_easy=4)
        st['det'].set_noise(N0=st['N0'])
    elif k == 'mdi':
        st['n0'] = nt / 10 ** (case['lo'] / 10)
        st['pick'] = dict(S=case['sweeps'], T0=0.1, T1=0.1, q=0.0, start='rand', Ns=case['Ns'])
    return st


def run(state):
    case = state['case']
    k = case['kind']
    if k == 'detect':
        det = state['det']
        bits, levels, dist = det.run(state['H'], state['y'], state['seed'])
        return dict(bits=bits, levels=levels, dist=dist, energies=det.de)
    if k == 'soft':
        bits, levels, dist, llr = state['det'].run_soft(state['H'], state['y'], state['seed'], state['N0f'])
        return dict(bits=bits, levels=levels, dist=dist, llr=llr)
    if k == 'warm':
        det = state['det']
        bits, levels, dist = det.run(state['H'], state['y'], state['seed'])
        return dict(bits=bits, levels=levels, dist=dist, energies=det.energies(), logits=det.Z)
    if k == 'traj':
        o = soft.detect_llr(state['H'], state['y'], state['N0'], case['M'], R=case['R'], S=case['S'],
                            seed=state['seed'])
        return {n: o[n] for n in ('llr', 'l_hat', 'best_l', 'best_d', 'm0', 'm1', 'mmse_levels', 'J', 'h0', 'scale')}
    if k == 'mdi':
        levels, ann, cnt, bits = mdi.detect(state['H'], state['y'], state['n0'], case['M'], state['seed'],
                                            state['pick'])
        return dict(levels=levels, bits=bits, anneals=ann, counters=[int(v) for n in sorted(cnt) for v in cnt[n]])
    if k == 'train':
        mlp = state['mlp']
        mlp.loss.zero_()
        mlp.train_step(state['X'], state['labels'], case['rows'])
        return dict(grad=mlp.grad, weights=mlp.w, loss=mlp.loss)
    s, e = state['kernel'].chord(state['F'], case['R'], state['seed'], P=case['P'])
    return dict(spins=s, energies=e)


def work(case):
    """Bytes: every input read and every output written once.  Operations: the Gram matrix and the solve of a use,
    one random word (a quarter of a Philox block of 100 operations) and one test per coordinate and pass, and the
    residual of every candidate; for the network its products, forward and backward."""
    k = case['kind']
    if k == 'train':
        r, n = case['rows'], 256 * 16 + 256 + 256 * 256 + 256 + 256 * 16 + 16
        return dict(bytes=r * 33 + 2 * 4 * n + 4 * 4 * n, flops=6.0 * r * (16 * 256 + 256 * 256 + 256 * 16))
    if k == 'chordj':
        B, R, S, N = case['B'], case['R'], case['S'], 2 * case['nt'] * case['P']
        return dict(bytes=B * (2 * N * N + 8 * N + R * (N + 8)) + 8 * S, flops=B * R * S * (N / case['P']) * 30.0)
    B, D, N2 = case['B'], 2 * case['nt'], 2 * case['nr']
    ins = B * 4 * (N2 * D + N2 + 1)
    bits = B * D * NB[case['M']]
    gram = B * (1.0 * N2 * D * (D + 1) + 2.0 * D ** 3 / 3)
    if k == 'traj':
        N, R, S = D * NB[case['M']], case['R'], case['S']
        return dict(bytes=ins + 4 * B * N * N + 4 * B * N + 3 * 4 * bits + 10 * B * D,
                    flops=gram + 30.0 * B * R * S * N)
    if k == 'mdi':
        return dict(bytes=ins + bits + B * D + 8 * B, flops=gram + 30.0 * B * 4 * case['Ns'] * 2 * case['sweeps'] * D)
    R, L = case['R'], case['sweeps'] * 2 * case.get('K', 1)
    b = ins + bits + B * D + 4 * B + (4 * bits if k == 'soft' else (4 if case.get('precision') == 'f32' else 8) * B * R)
    f = gram + 30.0 * B * R * L * D + 2.0 * B * R * N2 * D
    if k == 'warm':
        b += 64 * B * D
        f += 2.0 * B * D * (16 * 256 + 256 * 256 + 256 * 16)
    return dict(bytes=b, flops=f)


def exact(case, seed):
    """64-bit values of the outputs that are plain numbers of the inputs.  The detectors' other outputs are decided
    by their random draws: whole numbers, and the distances and LLRs of what was drawn."""
    k = case['kind']
    if k == 'train':
        X, labels = _train_inputs(case, seed)
        w = torch.from_numpy(_network(0)).cuda()
        wb = w.to(torch.bfloat16).double()
        wd = w.double()
        X = X.double()
        cut, o = [], 0
        for shp in ((256, 16), (256,), (256, 256), (256,), (256, 16), (16,)):
            n = int(np.prod(shp))
            cut.append((o, n, shp))
            o += n
        (W1, _, W2, _, W3, _), (_, b1, _, b2, _, b3) = ([v[a:a + n].view(s) for a, n, s in cut] for v in (wb, wd))
        h1 = torch.relu(X @ W1.T + b1)
        h2 = torch.relu(h1 @ W2.T + b2)
        z = (h2 @ W3 + b3)[:, :3]
        lab = labels.long()
        lp = z - torch.logsumexp(z, 1, keepdim=True)
        loss = -lp.gather(1, lab[:, None]).sum().reshape(1)
        dz = torch.zeros(case['rows'], 16, dtype=torch.float64, device='cuda')
        dz[:, :3] = lp.exp()
        dz[torch.arange(case['rows'], device='cuda'), lab] -= 1.0
        d2 = (dz @ W3.T) * (h2 > 0)
        d1 = (d2 @ W2) * (h1 > 0)
        grad = torch.cat([t.reshape(-1) for t in (d1.T @ X, d1.sum(0), d2.T @ h1, d2.sum(0), h2.T @ dz, dz.sum(0))])
        g = grad / case['rows']
        m, v = 0.1 * g, 0.001 * g * g
        neww = wd - 1e-3 * (m / 0.1) / (torch.sqrt(v / 0.001) + 1e-8)
        return dict(grad=grad, weights=neww, loss=loss)
    if k == 'traj':
        H, y, N0 = _uses(case, seed)
        H, y = H.double(), y.double()
        Q = H.transpose(1, 2) @ H
        g = (H.transpose(1, 2) @ y[..., None])[..., 0]
        if case['M'] == 16:
            J = torch.cat([torch.cat([4 * Q, 2 * Q], 2), torch.cat([2 * Q, Q], 2)], 1)
            h = torch.cat([4 * g, 2 * g], 1)
        else:
            J, h = Q.clone(), 2 * g
        J.diagonal(dim1=1, dim2=2).zero_()
        sc = torch.maximum(h.abs().amax(1), J.abs().amax((1, 2)))
        out = {n: None for n in ('llr', 'l_hat', 'best_l', 'best_d', 'm0', 'm1', 'mmse_levels')}
        out.update(J=-J / sc[:, None, None], h0=h / sc[:, None], scale=sc)
        return out
    return None
