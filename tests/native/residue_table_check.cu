// Prints the residue form's table of moduli (f4j_crt.cuh) for a host program to
// verify, and the configuration chosen for each precision and sum length.
// Launches no kernel.
#include "../../flag4j_gb300/csrc/f4j_split.cu"
#include <cstdio>

// the table is a constant of the program, for the host and the device alike
static_assert(crt_host.n > 0 && crt_host.cfg[0].nmod > 0, "built by the compiler");

int main() {
    printf("{\"cfgs\": [");
    for (int i = 0; i < crt_host.n; i++) {
        const CrtCfg& c = crt_host.cfg[i];
        printf("%s{\"nmod\": %d, \"nsq\": %d, \"words\": %d, \"sh\": %d, \"bits\": %.9g, \"qinv\": %.9g, \"mods\": [", i ? "," : "",
               c.nmod, c.nsq, c.words, c.sh, c.bits, c.qinv);
        for (int l = 0; l < c.nmod; l++)
            printf("%s[%.0f, %.9g, %.0f, %d, %d]", l ? "," : "", c.p[l], c.invp[l], c.u[l], c.c[l], crt_group(l));
        printf("], \"groups\": [");
        for (int g = 0; g < CRT_NG; g++) {
            printf("%s[%d", g ? "," : "", c.z0[g]);
            for (int j = 0; j < c.words; j++) printf(", %u", c.W[g][j]);
            printf("]");
        }
        printf("], \"NM\": [");
        for (int j = 0; j < c.words; j++) printf("%s%u", j ? "," : "", c.NM[j]);
        printf("]}");
    }
    printf("], \"picks\": [");
    bool first = true;
    for (long long k : {256ll, 8192ll, 100000ll, 1ll << 22})
        for (int s = 2; s <= S_MAX; s++) {
            printf("%s[%lld, %d, %d]", first ? "" : ",", k, s, crt_config(s, k));
            first = false;
        }
    printf("]}\n");
    return 0;
}
