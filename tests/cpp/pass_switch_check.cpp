// A simulator keeps running, with the same results, through switches of its GR pass
// in mid-run, those included that fail for want of memory at any of their
// allocations: cudaMalloc below stands in for the runtime's and refuses on demand.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include <dlfcn.h>

#include "cbm_sim.hpp"

static int mallocsLeft = -1;  // allocations that still succeed (-1: all)

extern "C" cudaError_t cudaMalloc(void **p, size_t bytes)
{
	static const auto real = (cudaError_t(*)(void **, size_t))dlsym(RTLD_NEXT, "cudaMalloc");
	if (mallocsLeft == 0) return cudaErrorMemoryAllocation;
	if (mallocsLeft > 0) mallocsLeft--;
	return real(p, bytes);
}

static void check(const std::string &e, const char *what)
{
	if (e.empty()) return;
	fprintf(stderr, "%s: %s\n", what, e.c_str());
	exit(1);
}

static std::vector<uint8_t> state(cbm::Simulator &sim, size_t i)
{
	std::vector<uint8_t> all;
	check(sim.sync(), "sync");
	for (cbm::Field f : {cbm::F_VM_GR, cbm::F_GESUM_GR, cbm::F_GISUM_GR, cbm::F_APBUF_GR, cbm::F_HIST_GR, cbm::F_THRESH_GR,
			cbm::F_GKCA_GR, cbm::F_VM_GO, cbm::F_APBUF_GO, cbm::F_VM_PC, cbm::F_VM_NC, cbm::F_VM_SC, cbm::F_PFPC_WEIGHT}) {
		std::vector<uint8_t> x(sim.net(i).fieldBytes(f));
		check(sim.exportField(i, f, 0, x.data(), x.size()), "export");
		all.insert(all.end(), x.begin(), x.end());
	}
	return all;
}

int main(int argc, char **argv)
{
	if (argc < 3) return 2;
	const uint32_t ring = 64;
	std::vector<std::string> paths(argv + 1, argv + argc - 1);
	const bool batch = paths.size() > 1;
	// a kind, then W, RW, S, B, M
	const int seq[][6] = {{1, 8, 1, 3, 2, 0}, {1, 4, 2, 2, 4, 0}, {3, 0, 1, 0, 0, 0}, {1, 2, 1, 4, 1, 0}, {0, 0, 1, 0, 0, 0},
		{1, 8, 1, 3, 2, 0}, {3, 0, 1, 0, 0, 0}, {0, 0, 1, 0, 0, 0}, {1, 1, 1, 4, 1, 0}};
	std::vector<cbm::State> a(paths.size()), b(paths.size());
	std::vector<cbm::State *> pa, pb;
	std::vector<std::vector<int>> seeds;
	for (size_t i = 0; i < paths.size(); i++) {
		check(a[i].load(paths[i]), "load");
		check(b[i].load(paths[i]), "load");
		pa.push_back(&a[i]);
		pb.push_back(&b[i]);
		seeds.push_back({5 + (int)i});
	}
	cbm::Simulator plain, sim;
	setenv("CBM_PASS_TMA", "0", 1);
	check(plain.create(pa, seeds, 0, ring), "create");
	unsetenv("CBM_PASS_TMA");
	check(sim.create(pb, seeds, 0, ring), "create");
	for (size_t i = 0; i < paths.size(); i++) {
		// about 4 % of MF spikes a step
		const uint32_t words = sim.net(i).mfWords(), mf = pa[i]->cp.numMF;
		std::vector<uint32_t> bits((size_t)words * ring, 0);
		uint64_t x = 88172645463325252ull + i;
		for (uint32_t t = 0; t < ring; t++)
			for (uint32_t m = 0; m < mf; m++) {
				x ^= x << 13; x ^= x >> 7; x ^= x << 17;
				if (x % 1000 < 40) bits[(size_t)t * words + m / 32] |= 1u << (m % 32);
			}
		for (cbm::Simulator *s : {&plain, &sim}) {
			check(s->net(i).uploadMFBits(bits.data(), 0, ring, s->stream()), "input");
			s->net(i).setPlastSteps(0, -0.002f, 0.002f);
			check(s->sync(), "input");
		}
	}
	uint64_t done = 0;
	auto steps = [&](uint32_t n, const std::string &at) {
		check(plain.runGraph(n, 4), "steps");
		check(sim.runGraph(n, 4), "steps");
		done += n;
		for (size_t i = 0; i < paths.size(); i++)
			if (state(plain, i) != state(sim, i)) check("the network differs from the plain pass's", at.c_str());
	};
	steps(39, "before any switch");  // the last steps of a run are launched one at a time
	int refused = 0;
	for (const int *q : seq) {
		cbm::PassGeometry g;
		g.kind = q[0]; g.W = q[1]; g.RW = q[2]; g.S = q[3]; g.B = q[4]; g.M = q[5];
		char at[96];
		for (int k = 0;; k++) {
			mallocsLeft = k;
			const std::string e = sim.usePassGeometry(g);
			const bool all = mallocsLeft > 0 || e.empty();
			mallocsLeft = -1;
			if (e.empty()) break;
			snprintf(at, sizeof at, "kind %d W %d, allocation %d refused", g.kind, g.W, k);
			if (all) check(e, "switch");
			if (e.find("allocat") == std::string::npos) check(e, at);
			refused++;
			steps(5, at);
		}
		snprintf(at, sizeof at, "kind %d W %d", g.kind, g.W);
		steps(11, at);
	}
	// a network whose tables do not fit at creation runs another pass
	{
		std::vector<cbm::State> c(paths.size());
		std::vector<cbm::State *> pc;
		for (size_t i = 0; i < paths.size(); i++) { check(c[i].load(paths[i]), "load"); pc.push_back(&c[i]); }
		int total = 0;
		{
			cbm::Simulator s;
			mallocsLeft = 1 << 30;
			check(s.create(pc, seeds, 0, ring), "create");
			total = (1 << 30) - mallocsLeft;
			mallocsLeft = -1;
		}
		cbm::Simulator s;
		mallocsLeft = total - 1;  // the default pass's last allocation fails, and all after it
		check(s.create(pc, seeds, 0, ring), "create without the event tables");
		mallocsLeft = -1;
		if (s.passGeometryInUse().kind == 1) check("the per-tile pass runs without its tables", "create");
	}
	FILE *f = fopen(argv[argc - 1], "w");
	if (!f) return 3;
	fprintf(f, "%llu steps, %d refused switches, batch %d\n", (unsigned long long)done, refused, (int)batch);
	fclose(f);
	return 0;
}
