"""The work that a user of this package has it do, as measurable cases.

Kinds of case, each through the package's public entry points:
  train   sgd_train / sgd_train_ex: host ratings in, host model out (the `cumf_sgd` job), from
          random rows with the deterministic schedule or from a deployed model with batch-Hogwild
  epoch   sgd_update on device-resident ratings and factors: one late epoch of the warm schedule,
          plain or with the copies of the most-rated rows (sgd_update + HotRows.merge)
  batch   Batch.run: epochs of many independent factorizations in one call
  rmse    dev_rmse: test RMSE of a device-resident model
  rank    evaluate: row- and column-wise AUC / MPR of a host model on a host test set
  text    dev_parse_text: rating text to 12-byte records
  warm    user_features + MLP.forward: starting rows for new users
  mlp     MLP.train: one pass of Adam over (features, rows) pairs
Ratings are integers 1..5 of users and items with power-law popularity; factors of the epoch
and evaluation cases are those of a model that has been trained for a while (they predict the
ratings up to noise), so that an epoch moves them as a late epoch does.  Batch-Hogwild workers
overwrite each other's updates as they meet, so two runs agree only as far as the learning rate
lets them: those cases continue a trained model at the low rates of the warm schedule (a run from
random rows does the same work, but ends at another of many equally good models each time).
"""
import math

import numpy as np
import torch

import cumf_sgd_gb300 as cm

STD = 1.1  # the ratings' standard deviation, by which sgd_train scales them
MEAN = 3.6 / STD
SIDE = 0.5  # entry that multiplies the other side's bias in a factor row
DTYPE = {"fp16": torch.float16, "fp16sr": torch.float16, "bf16": torch.bfloat16, "bf16sr": torch.bfloat16,
         "fp32": torch.float32}
D_IN_EXTRA = 3  # features beyond the k columns
HIDDEN = 512


def listed():
    return [
        # a refresh of a toy model, in full precision: latency of the whole call
        dict(name="train_small", kind="train", m=300, n=120, nnz=20_000, k=128, precision="fp32", iters=5, user_s=0.5,
             item_s=0.5, deterministic=0),
        # a small service's nightly refresh (0.9M ratings, popularity ~ 1/rank), 20 iterations as in the stock script
        dict(name="train_10k", kind="train", m=10_000, n=2_000, nnz=900_000, k=128, precision="fp16", iters=20,
             user_s=1.0, item_s=1.0, deterministic=0),
        # the same service's training from scratch where runs have to repeat bit for bit
        dict(name="train_deterministic", kind="train", m=10_000, n=2_000, nnz=900_000, k=128, precision="fp16",
             iters=4, user_s=0.5, item_s=0.5, deterministic=1),
        # one epoch at the benchmark shape, the library's defaults
        dict(name="epoch_large", kind="epoch", m=480_189, n=17_770, nnz=99_072_112, k=128, precision="fp16",
             user_s=0.39, item_s=0.46, hot=0.0),
        # the same epoch with the copies of the most-rated rows, as the benchmark runs it
        dict(name="epoch_large_copies", kind="epoch", m=480_189, n=17_770, nnz=99_072_112, k=128, precision="fp16",
             user_s=0.39, item_s=0.46, hot=0.5),
        # ordinary size, stochastic rounding, many items
        dict(name="epoch_bf16sr", kind="epoch", m=120_047, n=62_501, nnz=12_384_017, k=64, precision="bf16sr",
             user_s=0.39, item_s=0.46, hot=0.0),
        # many small tenants factorized together
        dict(name="batch", kind="batch", count=32, m=20_000, n=2_000, nnz=500_000, epochs=2),
        # test RMSE after training at the benchmark shape
        dict(name="rmse", kind="rmse", m=480_189, n=17_770, nnz=1_408_395, k=128, user_s=0.39, item_s=0.46),
        # ranking quality of a small service's model
        dict(name="rank", kind="rank", m=10_000, n=2_000, nnz=100_000, k=128, criterion="row_auc"),
        # import of a rating dump
        dict(name="text", kind="text", m=480_189, n=17_770, nnz=9_907_211, half=0),
        # 50,000 new users with 5% of the benchmark's ratings get starting rows
        dict(name="warm_start", kind="warm", m=50_000, n=17_770, nnz=5_214_321, k=128),
        # one pass of encoder training (short last batch)
        dict(name="mlp_train", kind="mlp", rows=100_003, k=128, batch=4096),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "epoch", "epoch", "batch", "rmse", "rank", "text", "warm", "mlp"])
    if kind == "train":
        det = rng.choice([0, 0, 1])
        nnz = _log(rng, 20_000, 2_000_000)
        m = max(200, min(60_000, nnz // rng.randint(40, 120)))
        return dict(kind=kind, m=m, n=max(100, m // rng.randint(2, 6)), nnz=nnz, k=rng.choice([32, 64, 128]),
                    precision=rng.choice(["fp16", "fp16", "bf16", "fp32"]), iters=rng.randint(2, 4 if det else 20),
                    user_s=0.5, item_s=rng.choice([0.5, 0.8]), deterministic=det)
    if kind == "epoch":
        precision = rng.choice(["fp16", "fp16", "bf16", "bf16sr", "fp16sr", "fp32"])
        k = rng.choice([32, 64, 128, 128, 256])
        cost = k / 128 * (2 if precision == "fp32" else 1)
        nnz = _log(rng, 500_000, int(99_072_112 / max(1.0, cost)))
        m = max(2_000, min(480_189, nnz // rng.randint(60, 250)))
        return dict(kind=kind, m=m, n=max(500, min(200_000, m // rng.randint(2, 27))), nnz=nnz, k=k,
                    precision=precision, user_s=0.39, item_s=0.46, hot=rng.choice([0.0, 0.0, 0.5]))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(8, 64), m=_log(rng, 2_000, 50_000), n=_log(rng, 500, 10_000),
                    nnz=_log(rng, 50_000, 1_000_000), epochs=rng.randint(1, 3))
    if kind == "rmse":
        m = _log(rng, 1_000, 480_189)
        return dict(kind=kind, m=m, n=max(200, m // rng.randint(2, 27)), nnz=_log(rng, 10_000, 4_000_000),
                    k=rng.choice([32, 64, 128, 256]), user_s=0.39, item_s=0.46)
    if kind == "rank":
        m, n = _log(rng, 500, 20_000), _log(rng, 500, 5_000)
        return dict(kind=kind, m=m, n=n, nnz=m * rng.randint(4, 20), k=rng.choice([32, 64, 128]),
                    criterion=rng.choice(["row_auc", "row_mpr", "col_auc"]))
    if kind == "text":
        return dict(kind=kind, m=_log(rng, 1_000, 1_000_000), n=_log(rng, 500, 500_000),
                    nnz=_log(rng, 5_000, 20_000_000), half=rng.choice([0, 0, 1]))
    if kind == "warm":
        m = _log(rng, 500, 100_000)
        return dict(kind=kind, m=m, n=_log(rng, 1_000, 50_000), nnz=m * rng.randint(20, 110), k=rng.choice([64, 128]))
    return dict(kind=kind, rows=_log(rng, 5_000, 200_000), k=rng.choice([64, 128]),
                batch=rng.choice([1024, 2048, 4096]))


# ---- inputs ---------------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _ids(count, rows, s, g):
    """`count` ids below `rows`, the popularity of rank x as x^-s, ranks relabelled at random."""
    u = torch.rand(count, generator=g, device="cuda", dtype=torch.float64)
    if s == 1.0:
        x = torch.exp(u * math.log(rows + 1))
    else:
        x = ((u * ((rows + 1) ** (1 - s) - 1)) + 1) ** (1 / (1 - s))
    rank = (x.floor() - 1).clamp_(0, rows - 1).long()
    return torch.randperm(rows, generator=g, device="cuda")[rank].to(torch.int32)


def _biases(m, n, g):
    return (torch.randn(m, generator=g, device="cuda") * 0.3, torch.randn(n, generator=g, device="cuda") * 0.3)


def _ratings(u, v, bu, bi, g):
    r = STD * (MEAN + bu[u.long()] + bi[v.long()]) + torch.randn(len(u), generator=g, device="cuda") * 0.9
    return torch.round(r).clamp_(1, 5)


def _records(u, v, r):
    return torch.stack((u, v, r.float().view(torch.int32)), 1).contiguous()


def _factors(bu, bi, k, g):
    """Rows whose products are MEAN + both biases, with a little noise on every entry."""
    a = math.sqrt(MEAN / (k - 2))
    P = torch.randn(len(bu), k, generator=g, device="cuda") * 0.03 + a
    Q = torch.randn(len(bi), k, generator=g, device="cuda") * 0.03 + a
    P[:, 0], P[:, 1] = bu / SIDE, SIDE
    Q[:, 0], Q[:, 1] = SIDE, bi / SIDE
    return P, Q


def _weights(d_in, d_out, g):
    parts = []
    for fi, fo in ((d_in, HIDDEN), (HIDDEN, HIDDEN), (HIDDEN, d_out)):
        lim = math.sqrt(6 / (fi + fo))
        parts += [((torch.rand(fo, fi, generator=g, device="cuda") * 2 - 1) * lim).reshape(-1),
                  torch.randn(fo, generator=g, device="cuda") * 0.02]
    return parts


def _problem(u, v, r, m, n):
    return cm.MFProblem.from_arrays(u.cpu().numpy(), v.cpu().numpy(), r.cpu().numpy(), m=m, n=n, pinned=True)


def _prepare_train(c, g):
    m, n = c["m"], c["n"]
    bu, bi = _biases(m, n, g)
    u, v = _ids(c["nnz"], m, c["user_s"], g), _ids(c["nnz"], n, c["item_s"], g)
    par = cm.Parameter(k=c["k"], num_workers=0, num_iters=c["iters"], lambda_p=0.05, lambda_q=0.05,
                       alpha=0.08 if c["deterministic"] else 0.001, beta=0.3, seed=11, gpu=0,
                       precision=c["precision"], deterministic=c["deterministic"])
    s = dict(prob=_problem(u, v, _ratings(u, v, bu, bi, g), m, n), par=par, model=None)
    if not c["deterministic"]:
        s["model"] = cm.MFModel.from_arrays(*((x * math.sqrt(STD)).cpu().numpy() for x in _factors(bu, bi, c["k"], g)), 0.0)
    return s


def _prepare_epoch(c, g):
    m, n, nnz, k = c["m"], c["n"], c["nnz"], c["k"]
    bu, bi = _biases(m, n, g)
    u, v = _ids(nnz, m, c["user_s"], g), _ids(nnz, n, c["item_s"], g)
    R = _records(u, v, _ratings(u, v, bu, bi, g) / STD)
    del u, v
    P, Q = _factors(bu, bi, k, g)
    s = dict(workers=cm.auto_workers(nnz, cm.device_info(0)[0], k, c["precision"]), plan=None, m=m, n=n)
    if c["hot"] > 0:
        per = cm.HotRows.per_copy(nnz, s["workers"], k, c["precision"], 0, c["hot"])
        plan = cm.HotRows(R.data_ptr(), nnz, m, n, per)
        plan.assign(R.data_ptr(), nnz)
        s.update(plan=plan, m=plan.m_rows, n=plan.n_rows)
    dt = DTYPE[c["precision"]]
    s["R"], s["P"], s["Q"] = R, torch.zeros(s["m"], k, dtype=dt, device="cuda"), torch.zeros(s["n"], k, dtype=dt,
                                                                                              device="cuda")
    s["P"][:m], s["Q"][:n] = P, Q
    if s["plan"]:
        s["plan"].spread(s["P"].data_ptr(), s["Q"].data_ptr(), k, c["precision"])
    s["lr"] = torch.from_numpy(cm.lr_schedule(0.04, 0.3, 0.0, 40)).cuda()
    s["status"] = torch.zeros(1, dtype=torch.int32, device="cuda")
    return s


def _batch_shapes(c):
    """Problem sizes spread over a factor of 16 around the case's, odd ones among them."""
    out = []
    for i in range(c["count"]):
        f = 4 ** (((i * 7) % 11) / 5 - 1)
        out.append((max(50, int(c["m"] * f) | 1), max(30, int(c["n"] * math.sqrt(f)) + i), int(c["nnz"] * f) + 13 * i,
                    (32, 64, 128)[i % 3]))
    return out


def _prepare_batch(c, g):
    shapes = _batch_shapes(c)
    pe, qe = sum(m * k for m, _, _, k in shapes), sum(n * k for _, n, _, k in shapes)
    P, Q = (torch.empty(e, dtype=torch.float16, device="cuda") for e in (pe, qe))
    lr = torch.from_numpy(cm.lr_schedule(0.04, 0.3, 0.0, 40)).cuda()
    probs, keep, po, qo = [], [lr], 0, 0
    for i, (m, n, nnz, k) in enumerate(shapes):
        bu, bi = _biases(m, n, g)
        u, v = _ids(nnz, m, 0.5, g), _ids(nnz, n, 0.5, g)
        R = _records(u, v, _ratings(u, v, bu, bi, g) / STD)
        p, q = _factors(bu, bi, k, g)
        P[po:po + m * k], Q[qo:qo + n * k] = p.reshape(-1), q.reshape(-1)
        probs.append(dict(d_R=R.data_ptr(), nnz=nnz, d_P=P.data_ptr() + 2 * po, m=m, n=n, d_Q=Q.data_ptr() + 2 * qo, k=k,
                          lambda_p=0.05, lambda_q=0.05, seed=100 + i, d_lr=lr.data_ptr(), lr_len=40))
        keep.append(R)
        po, qo = po + m * k, qo + n * k
    return dict(batch=cm.Batch(probs), keep=keep, P=P, Q=Q)


def _prepare_rmse(c, g):
    bu, bi = _biases(c["m"], c["n"], g)
    u, v = _ids(c["nnz"], c["m"], c["user_s"], g), _ids(c["nnz"], c["n"], c["item_s"], g)
    P, Q = _factors(bu, bi, c["k"], g)
    r = _ratings(u, v, bu, bi, g)
    return dict(u=u, v=v, r=r, R=_records(u, v, r), P=P * math.sqrt(STD), Q=Q * math.sqrt(STD))


def _prepare_rank(c, g):
    m, n, k = c["m"], c["n"], c["k"]
    pairs = torch.unique(_ids(c["nnz"], m, 0.3, g).long() * n + _ids(c["nnz"], n, 0.5, g).long())
    pairs = pairs[torch.randperm(len(pairs), generator=g, device="cuda")]
    u, v = torch.div(pairs, n, rounding_mode="floor").int(), (pairs % n).int()
    P, Q = (torch.randn(x, k, generator=g, device="cuda") * 0.3 for x in (m, n))
    z = (P[u.long()] * Q[v.long()]).sum(1) + torch.randn(len(u), generator=g, device="cuda") * 0.5
    r = torch.where(z > -0.6, 1.0, -1.0)
    return dict(u=u, v=v, r=r, P=P, Q=Q)


HEADER = b"%%MatrixMarket matrix coordinate real general\n%\n"


def _prepare_text(c, g):
    """Lines "u v r" (ids from 1), built as fixed-width fields whose leading zeros are dropped."""
    nnz = c["nnz"]
    u, v = _ids(nnz, c["m"], 0.39, g) + 1, _ids(nnz, c["n"], 0.46, g) + 1
    r = torch.randint(1, 6, (nnz,), generator=g, device="cuda")
    cols, keep = [], []
    for x in (u, v):
        for d in range(6, -1, -1):
            cols.append((torch.div(x, 10 ** d, rounding_mode="floor") % 10 + 48).to(torch.uint8))
            keep.append(x >= 10 ** d)
        cols.append(torch.full_like(cols[-1], 32))
        keep.append(torch.ones_like(keep[-1]))
    cols.append((r + 48).to(torch.uint8))
    keep.append(torch.ones_like(keep[-1]))
    if c["half"]:
        some = (torch.rand(nnz, generator=g, device="cuda") < 0.5) & (r < 5)
        cols += [torch.full_like(cols[-1], 46), torch.full_like(cols[-1], 53)]
        keep += [some, some]
    cols.append(torch.full_like(cols[-1], 10))
    keep.append(torch.ones_like(keep[-1]))
    body = torch.stack(cols, 1)[torch.stack(keep, 1)]
    head = HEADER + b"%d %d %d\n" % (c["m"], c["n"], nnz)
    start = cm.text_data_start(head + bytes(body[:64].cpu().numpy()))
    text = torch.cat((torch.frombuffer(bytearray(head), dtype=torch.uint8).cuda(), body))
    length = len(text)
    text = torch.cat((text, torch.zeros(256, dtype=torch.uint8, device="cuda")))
    return dict(text=text, length=length, start=start, out=torch.zeros(nnz, 3, dtype=torch.int32, device="cuda"))


def _warm_inputs(c, g):
    m, n, k = c["m"], c["n"], c["k"]
    bu, bi = _biases(m, n, g)
    u = torch.randint(0, m, (c["nnz"],), generator=g, device="cuda").int()
    v = _ids(c["nnz"], n, 0.46, g)
    r = _ratings(u, v, bu, bi, g)
    _, Q = _factors(bu, bi, k, g)
    return u, v, r, Q, _weights(k + D_IN_EXTRA, k, g)


def _prepare_warm(c, g):
    u, v, r, Q, w = _warm_inputs(c, g)
    k = c["k"]
    mlp = cm.MLP(k + D_IN_EXTRA, HIDDEN, k, seed=1)
    mlp.set(torch.cat(w).cpu().numpy())
    return dict(R=_records(u, v, r), Q=Q, mlp=mlp, X=torch.empty(c["m"], k + D_IN_EXTRA, device="cuda"),
                Y=torch.empty(c["m"], k, device="cuda"))


def _prepare_mlp(c, g):
    k = c["k"]
    mlp = cm.MLP(k + D_IN_EXTRA, HIDDEN, k, seed=1)
    mlp.set(torch.cat(_weights(k + D_IN_EXTRA, k, g)).cpu().numpy())
    X = torch.randn(c["rows"], k + D_IN_EXTRA, generator=g, device="cuda") * 0.5
    A = torch.randn(k + D_IN_EXTRA, k, generator=g, device="cuda") / math.sqrt(k)
    return dict(mlp=mlp, X=X, T=torch.tanh(X @ A))


def prepare(case, seed):
    g = _gen(seed)
    s = globals()["_prepare_" + case["kind"]](case, g)
    if case["kind"] == "rank":
        s = dict(prob=_problem(s["u"], s["v"], s["r"], case["m"], case["n"]),
                 model=cm.MFModel.from_arrays(s["P"].cpu().numpy(), s["Q"].cpu().numpy(), 0.0))
    s["case"] = case
    return s


# ---- one pass -------------------------------------------------------------------------------

def _run_train(c, s):
    if s["model"]:
        model = cm.sgd_train_ex(s["prob"], None, s["par"], s["model"])[0]
    else:
        model = cm.sgd_train(s["prob"], None, s["par"])
    return {"P": model.P, "Q": model.Q, "b": model.b}


def _run_epoch(c, s):
    k, P, Q = c["k"], s["P"], s["Q"]
    cm.sgd_update(s["R"].data_ptr(), c["nnz"], P.data_ptr(), s["m"], Q.data_ptr(), s["n"], k, c["precision"],
                  s["workers"], 0, s["lr"].data_ptr(), 30, 1, 0.05 / STD, 0.05 / STD, 5, s["status"].data_ptr(),
                  rows_copied=1 if s["plan"] else 0)
    if s["plan"]:
        s["plan"].merge(P.data_ptr(), Q.data_ptr(), k, c["precision"])
    return {"P": P[:c["m"]], "Q": Q[:c["n"]], "status": s["status"]}


def _run_batch(c, s):
    s["batch"].run(30, c["epochs"])
    return {"P": s["P"], "Q": s["Q"]}


def _run_rmse(c, s):
    return cm.dev_rmse(s["R"].data_ptr(), c["nnz"], s["P"].data_ptr(), c["m"], s["Q"].data_ptr(), c["n"], c["k"], 3.6)


def _run_rank(c, s):
    return cm.evaluate(s["prob"], s["model"], c["criterion"])


def _run_text(c, s):
    n = cm.dev_parse_text(s["text"].data_ptr(), s["length"], s["start"], s["out"].data_ptr(), c["nnz"])
    return {"n": n, "records": s["out"]}


def _run_warm(c, s):
    k = c["k"]
    cm.user_features(s["R"].data_ptr(), c["nnz"], s["Q"].data_ptr(), c["n"], k, c["m"], s["X"].data_ptr())
    s["mlp"].forward(s["X"].data_ptr(), c["m"], s["Y"].data_ptr())
    return {"X": s["X"], "Y": s["Y"]}


def _run_mlp(c, s):
    loss = s["mlp"].train(s["X"].data_ptr(), s["T"].data_ptr(), c["rows"], 1, c["batch"], 1e-3, 3)
    return {"loss": loss, "params": s["mlp"].get(0)}


def run(state):
    case = state["case"]
    return globals()["_run_" + case["kind"]](case, state)


# ---- what a pass cannot do without ----------------------------------------------------------

def _mlp_flops(rows, k):
    return 2 * rows * ((k + D_IN_EXTRA) * HIDDEN + HIDDEN * HIDDEN + HIDDEN * k)


def work(case):
    c, kind = case, case["kind"]
    if kind == "train":
        rows = (c["m"] + c["n"]) * c["k"]
        return {"bytes": 12 * c["nnz"] + 4 * rows, "flops": 12 * c["k"] * c["nnz"] * c["iters"]}
    if kind == "epoch":
        rows = (c["m"] + c["n"]) * c["k"] * (4 if c["precision"] == "fp32" else 2)
        return {"bytes": 12 * c["nnz"] + 2 * rows, "flops": 12 * c["k"] * c["nnz"]}
    if kind == "batch":
        sh = _batch_shapes(c)
        return {"bytes": sum(12 * z + 4 * (m + n) * k for m, n, z, k in sh),
                "flops": sum(12 * k * z * c["epochs"] for _, _, z, k in sh)}
    if kind == "rmse":
        rows = min(c["nnz"], c["m"]) + min(c["nnz"], c["n"])
        return {"bytes": 12 * c["nnz"] + 4 * rows * c["k"], "flops": 2 * c["k"] * c["nnz"]}
    if kind == "rank":
        return {"bytes": 12 * c["nnz"] + 4 * (c["m"] + c["n"]) * c["k"], "flops": 2 * c["k"] * c["m"] * c["n"]}
    if kind == "text":
        return {"bytes": c["nnz"] * (12 + 5 + len(str(c["m"])) + len(str(c["n"])) - 1), "flops": 0}
    if kind == "warm":
        k, d = c["k"], c["k"] + D_IN_EXTRA
        return {"bytes": 12 * c["nnz"] + 4 * c["n"] * k + 4 * c["m"] * (d + k),
                "flops": 2 * c["nnz"] * k + _mlp_flops(c["m"], k)}
    steps = -(-c["rows"] // c["batch"])
    params = (c["k"] + D_IN_EXTRA) * HIDDEN + HIDDEN * HIDDEN + HIDDEN * c["k"] + 2 * HIDDEN + c["k"]
    return {"bytes": 4 * c["rows"] * (2 * c["k"] + D_IN_EXTRA) + 12 * params * steps, "flops": 3 * _mlp_flops(c["rows"], c["k"])}


# ---- the same results in 64 bits --------------------------------------------------------------

def _exact_rmse(c, g):
    s = _prepare_rmse(c, g)
    total, step = 0.0, 1 << 20
    for a in range(0, c["nnz"], step):
        u, v = s["u"][a:a + step].long(), s["v"][a:a + step].long()
        e = s["r"][a:a + step].double() - (s["P"][u].double() * s["Q"][v].double()).sum(1)
        total += float((e * e).sum())
    return math.sqrt(total / c["nnz"])


def _exact_rank(c, g):
    s = _prepare_rank(c, g)
    u, v, P, Q = s["u"].long(), s["v"].long(), s["P"].double(), s["Q"].double()
    if c["criterion"].startswith("col"):
        u, v, P, Q = v, u, Q, P
    pos = s["r"] > 0
    u, v = u[pos], v[pos]
    rows, cols = len(P), len(Q)
    auc = mpr = 0.0
    active = npos = 0
    for a in range(0, rows, 2048):
        z = P[a:a + 2048] @ Q.T
        here = (u >= a) & (u < a + 2048)
        mark = torch.zeros_like(z, dtype=torch.bool)
        mark[u[here] - a, v[here]] = True
        inf = torch.full_like(z, math.inf)
        negs = torch.where(mark, inf, z).sort(1).values
        below = torch.searchsorted(negs, torch.where(mark, z, -inf))  # non-positives below each positive
        wins = torch.where(mark, below, 0).sum(1).double()
        p = mark.sum(1).double()
        q = cols - p
        ok = (p > 0) & (q > 0)
        auc += float((wins[ok] / q[ok] / p[ok]).sum())
        mpr += float(((p[ok] * q[ok] - wins[ok]) / q[ok]).sum())
        active, npos = active + int(ok.sum()), npos + int(p[ok].sum())
    return mpr / npos if c["criterion"].endswith("mpr") else auc / active


def _exact_warm(c, g):
    u, v, r, Q, w = _warm_inputs(c, g)
    m, k = c["m"], c["k"]
    u, v, r, Q = u.long(), v.long(), r.double(), Q.double()
    deg = torch.bincount(u, minlength=m).double()
    has, d = deg > 0, deg.clamp(min=1)
    mean = torch.zeros(m, dtype=torch.float64, device="cuda").index_add_(0, u, r) / d
    var = torch.zeros(m, dtype=torch.float64, device="cuda").index_add_(0, u, (r - mean[u]) ** 2) / d
    X = torch.zeros(m, k + D_IN_EXTRA, dtype=torch.float64, device="cuda")
    for a in range(0, c["nnz"], 1 << 20):
        i, j = u[a:a + (1 << 20)], v[a:a + (1 << 20)]
        X[:, :k].index_add_(0, i, ((r[a:a + (1 << 20)] - mean[i]) / d[i])[:, None] * Q[j])
    X[:, k] = torch.log1p(deg) / 4
    X[:, k + 1] = torch.where(has, (mean - 3) / 2, torch.zeros_like(mean))
    X[:, k + 2] = var / 2
    h, gelu = X, lambda x: torch.nn.functional.gelu(x, approximate="tanh")  # noqa: E731
    dims = [(HIDDEN, k + D_IN_EXTRA), (HIDDEN, HIDDEN), (k, HIDDEN)]
    for i, shape in enumerate(dims):
        h = h @ w[2 * i].double().reshape(shape).T + w[2 * i + 1].double()
        h = gelu(h) if i < 2 else h
    return {"X": X, "Y": h}


def exact(case, seed):
    """Where a pass has one right answer.  Hogwild epochs and training depend on the order in
    which the workers meet, so the start's own results are what they are held to."""
    f = globals().get("_exact_" + case["kind"])
    return f(case, _gen(seed)) if f else None
