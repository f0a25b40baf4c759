

def test_module_walk_sees_every_module_once():
    """Modules that hold one another, or share a part, as ``Module.modules()`` walks them."""
    import torch
    from spiraltorch_b200.models import contrastive
    enc = contrastive.ContrastiveEncoder(64, 128, 64, device="cpu", seed=1)
    enc.shared = torch.nn.Sequential(torch.nn.Identity())
    enc.wrapper = torch.nn.ModuleList([enc, enc.shared])
    assert {id(m) for m in contrastive._modules(enc)} == {id(m) for m in enc.modules()}
    assert len(contrastive._modules(enc)) == len(list(enc.modules()))
